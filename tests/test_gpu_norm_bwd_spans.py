"""LayerNorm / RMSNorm backward of rows off the 16-byte grid by the vector: CTAs that take rows of one alignment."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,n", [(d, n) for d in (torch.bfloat16, torch.float16) for n in (513, 769, 1010, 1011, 1522, 1523, 2034, 2035, 2546, 2547, 4082, 4083, 4095)]
                         + [(torch.float32, n) for n in (1025, 2042, 2043, 2554, 2555, 3066, 3067, 4090, 4091, 4095)], ids=str)
def test_spans(dtype, n):
    """Both sides of every change of geometry, every alignment of the first row, rows of a wider tensor; NaN lies beside the rows."""
    from better_benchmark_b200 import native
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows = (32 if n <= 1010 else 16) * sms + 5
    lib, stream = native.load(), torch.cuda.current_stream().cuda_stream
    code = {torch.float32: 0, torch.bfloat16: 1, torch.float16: 2}[dtype]
    ulp = {torch.float32: 2.0 ** -23, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype]
    g = torch.Generator(device="cuda").manual_seed(n)
    advertised = lib.b200_norm_bwd_scratch_bytes(n)
    for start, pitch, rms, scratch_bytes in ((0, n, False, advertised), (3, n, True, advertised), (5, n + 3, False, advertised),
                                             (1, n, False, 256 + 2 * 4 * n * 17), (7, n, False, 256 + 2 * 4 * n * 7)):
        size = (rows - 1) * pitch + n
        flat = [torch.full((size + 64,), float("nan"), device="cuda", dtype=dtype) for _ in range(2)]
        x, dy = (f[start:start + size].as_strided((rows, n), (pitch, 1)) for f in flat)
        x.copy_(torch.randn(rows, n, generator=g, device="cuda") * 2)
        dy.copy_(torch.randn(rows, n, generator=g, device="cuda"))
        out = torch.full((size + 64,), 7.0, device="cuda", dtype=dtype)
        dx = out[start:start + size].as_strided((rows, n), (pitch, 1))
        w = torch.randn(n, generator=g, device="cuda").to(dtype)
        mean = torch.randn(rows, generator=g, device="cuda")
        rstd = torch.rand(rows, generator=g, device="cuda") + 0.5
        mean[3], rstd[4] = float("nan"), float("inf")
        grads = torch.full((2, n), float("nan"), device="cuda")
        scratch = torch.zeros(scratch_bytes, device="cuda", dtype=torch.uint8)
        for special in (True, False):
            if not special:
                mean[3], rstd[4] = 0.5, 1.0
            rc = lib.b200_norm_bwd(x.data_ptr(), dy.data_ptr(), w.data_ptr(), None if rms else mean.data_ptr(), rstd.data_ptr(), dx.data_ptr(),
                                   grads[0].data_ptr(), None if rms else grads[1].data_ptr(), rows, n, pitch, pitch, code, code, int(rms),
                                   1, n, pitch, 0, n, scratch.data_ptr(), scratch_bytes, 0, stream)
            assert rc == 0
            ok = torch.ones(rows, dtype=torch.bool, device="cuda")
            if special:
                ok[3:5] = False
            assert not bool(torch.isnan(dx[ok]).any()), "special values stay in their rows"
        beside = torch.ones_like(out, dtype=torch.bool)
        beside[start:start + size].as_strided((rows, n), (pitch, 1)).fill_(False)
        assert bool((out[beside] == 7).all()), "nothing beside the rows is written"
        xd, gd, m, r = x.double(), dy.double(), mean.double()[:, None], rstd.double()[:, None]
        wg = gd * w.double()
        if rms:
            s2 = (wg * xd).sum(-1, keepdim=True)
            want = wg * r - xd * s2 * r ** 3 / n
            size_of = wg.abs() * r + (xd * r ** 3).abs() * (wg * xd).abs().sum(-1, keepdim=True) / n
            xhat = xd * r
        else:
            xhat = (xd - m) * r
            s1, s2 = wg.sum(-1, keepdim=True), (wg * xhat).sum(-1, keepdim=True)
            want = r / n * (n * wg - s1 - xhat * s2)
            size_of = r * (wg.abs() + wg.abs().mean(-1, keepdim=True) + xhat.abs() * (wg * xhat).abs().mean(-1, keepdim=True))
        # one rounding of the result; a row's sums have chains of at most 16 terms and some twenty additions, and six steps follow
        assert bool(((dx.double() - want).abs() <= ulp * want.abs() + 2.0 ** -24 * 44 * size_of + 6.2e-8).all())
        # a thread's sum over its rows: at most rows / 4 terms with seventeen or seven partial rows for all of them, then fp64
        chain = rows if scratch_bytes < advertised else 64
        for got, terms in ((grads[0], gd * xhat), (grads[1], gd)):
            if rms and got is not grads[0] and terms is gd:
                continue
            bound = 2.0 ** -24 * (3 + chain ** 0.5 * 2) * terms.abs().sum(0) + 1e-6
            assert bool(((got.double() - terms.sum(0)).abs() <= bound).all())
