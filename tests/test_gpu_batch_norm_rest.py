"""Channels-last BatchNorm whose elements are no whole number of channel periods, or of 16-byte vectors."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
# (n, c, h, w): odd channel counts and row counts, so that 1 to 7 elements are left over; few vectors; more than one wave of chunks
SHAPES = [(1, 3, 1, 3), (1, 9, 1, 2), (2, 35, 5, 5), (3, 287, 7, 7), (1, 401, 14, 13), (5, 509, 3, 3), (9, 92, 5, 5), (600, 77, 15, 15),
          (3, 3, 15, 15), (1, 9, 25, 27), (27, 35, 5, 5), (13, 287, 7, 7), (5, 401, 11, 13), (67, 509, 3, 3), (25, 92, 5, 5)]


def _image(shape, dtype, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    t = torch.randn(shape, generator=g, device="cuda") * scale + 0.3
    return t.to(dtype).contiguous(memory_format=torch.channels_last)


def _close(got, want, dtype, what):
    # one rounding of the result, and in front of it some ten fp32 steps on values of up to ten
    tol = {torch.float32: (1e-5, 1e-5), torch.bfloat16: (2.0 ** -8 + 1e-6, 1e-5), torch.float16: (2.0 ** -11 + 1e-6, 1e-5)}[dtype]
    assert torch.allclose(got.double(), want, rtol=tol[0], atol=tol[1]), (what, (got.double() - want).abs().max().item())


@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("dtype", list(DTYPES))
def test_forward(dtype, shape):
    from better_benchmark_b200 import kernels as k
    dt, c = DTYPES[dtype], shape[1]
    x = _image(shape, dt, 1)
    w, b = torch.rand(c, device="cuda") + 0.5, torch.randn(c, device="cuda")
    for relu in (False, True):
        y, mean, invstd = k.batch_norm_fwd(x, w, b, None, None, eps=1e-5, momentum=0.1, relu=relu)
        if c > 3:
            assert b"copy rings" in k.load().b200_last_kernel()
        d = x.double()
        m, v = d.mean((0, 2, 3)), d.var((0, 2, 3), unbiased=False)
        s = torch.rsqrt(v + 1e-5)
        want = (d - m.view(1, c, 1, 1)) * s.view(1, c, 1, 1) * w.double().view(1, c, 1, 1) + b.double().view(1, c, 1, 1)
        _close(y, want.relu() if relu else want, dt, "y")
        _close(mean, m, torch.float32, "mean")
        assert torch.allclose(invstd.double(), s, rtol=1e-5), "invstd"


@pytest.mark.parametrize("shape", SHAPES, ids=str)
@pytest.mark.parametrize("dtype", list(DTYPES))
def test_backward(dtype, shape):
    from better_benchmark_b200 import kernels as k
    dt, c = DTYPES[dtype], shape[1]
    x, dy, act = (_image(shape, dt, s) for s in (1, 2, 3))
    w = torch.rand(c, device="cuda") + 0.5
    d = x.double()
    m = d.mean((0, 2, 3)).float()
    s = torch.rsqrt(d.var((0, 2, 3), unbiased=False) + 1e-5).float()
    column = lambda t: t.double().view(1, c, 1, 1)  # noqa: E731
    count = x.numel() // c
    for a in (None, act):
        g = dy.double() if a is None else torch.where(a > 0, dy.double(), (dy.float() * 0.25).to(dt).double())
        xhat = (d - column(m)) * column(s)
        db, dw = g.sum((0, 2, 3)), (g * xhat).sum((0, 2, 3))
        want = (g - column(db) / count - xhat * column(dw) / count) * column(s) * column(w)
        rows, v = shape[0] * shape[2] * shape[3], 16 // dt.itemsize
        for want_dx in (True, False):
            dx, dweight, dbias = k.batch_norm_bwd(dy, x, m, s, w, act=a, slope=0.25, want_dx=want_dx)
            if want_dx and rows * c >= v and rows * c % (c // math.gcd(c, v) * v) != 0:   # few rows: the strided kernels
                assert (b"strided" in k.load().b200_last_kernel()) == (rows < 300 * v // 8)
            # fp32 chains of at most 16 additions a thread below fp64: a few 2^-24 of the magnitudes that are added
            for got, ref, parts in ((dbias, db, g.abs()), (dweight, dw, (g * xhat).abs())):
                assert bool(((got.double() - ref).abs() <= 40 * 2.0 ** -24 * (parts.sum((0, 2, 3)) + column(s).flatten() * g.abs().sum((0, 2, 3)))).all())
            if want_dx:
                _close(dx, want, dt, "dx")
            else:
                assert dx is None


def test_backward_with_a_small_scratch():
    """Room for the few partial rows of the strided kernels only: still taken, with the same result."""
    from better_benchmark_b200 import kernels as k
    shape, c = (69, 401, 14, 14), 401
    x, dy = (_image(shape, torch.bfloat16, s) for s in (1, 2))
    mean, invstd = torch.zeros(c, device="cuda"), torch.ones(c, device="cuda")
    want = k.batch_norm_bwd(dy, x, mean, invstd, None)
    splits = 69 * 196 // 16384 or 1
    small = torch.zeros(256 + splits * 2 * c * 8 + 4 * c * 4, dtype=torch.uint8, device="cuda")
    got = k.batch_norm_bwd(dy, x, mean, invstd, None, scratch=small)
    assert b"strided" in k.load().b200_last_kernel()
    assert torch.allclose(got[0].double(), want[0].double(), rtol=2.0 ** -7, atol=1e-5), "both rounded: at most one step apart"
    for a, b in zip(got[1:], want[1:]):
        assert torch.allclose(a, b, rtol=1e-4, atol=1e-2)
    with pytest.raises(ValueError, match="scratch"):
        k.batch_norm_bwd(dy, x, mean, invstd, None, scratch=small[:-16])
