"""LayerNorm / RMSNorm forward of rows off the 16-byte grid: groups of lanes with the parameters in shared memory, and a CTA per row."""
import pytest
import torch

pytestmark = pytest.mark.gpu

HALF = [57, 58, 121, 122, 185, 186, 249, 250, 257, 377, 378, 505, 506, 761, 762, 1017, 1018, 1024, 2661, 4089, 4090, 8191, 16377]


def _storage(rows, n, dtype, start, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    flat = torch.full((rows * n + 64,), float("nan"), device="cuda", dtype=dtype)
    flat[start:start + rows * n] = (torch.randn(rows * n, generator=g, device="cuda") * 2 + 0.3).to(dtype)
    return flat[start:start + rows * n].view(rows, n)


@pytest.mark.parametrize("dtype,n", [(d, n) for d in (torch.bfloat16, torch.float16) for n in HALF] + [(torch.float32, n) for n in (2049, 2050, 4001, 8189)],
                         ids=str)
def test_spans(dtype, n):
    """Both sides of every change of geometry; what lies beside the rows is NaN and stays out; parameters of either type, off the grid, none."""
    from better_benchmark_b200 import native
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows = (64 if n <= 128 else 25 if n < 250 else 48 if n <= 256 else 14 if n <= 505 else 25 if n <= 512 else 8 if n <= 1017 else 5) * sms + 3
    lib, stream = native.load(), torch.cuda.current_stream().cuda_stream
    eps, code = 1e-5, {torch.float32: 0, torch.bfloat16: 1, torch.float16: 2}
    ulp = {torch.float32: 2.0 ** -23, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype]
    par = torch.randn(4, n + 8, device="cuda")
    for start, wdt, shift, has_w, has_b, rms in ((0, dtype, 0, True, True, False), (3, dtype, 0, True, False, False), (6, dtype, 1, True, True, False),
                                                 (5, torch.float32, 0, True, True, False), (0, dtype, 0, False, False, True), (1, dtype, 0, False, True, False)):
        x = _storage(rows, n, dtype, start, n)
        flat = torch.full((rows * n + 64,), 7.0, device="cuda", dtype=dtype)
        y = flat[start:start + rows * n].view(rows, n)
        w, b = (par[i].to(wdt)[shift:shift + n] for i in (0, 1))
        stats = torch.empty(3, rows, device="cuda")
        rc = lib.b200_norm_fwd(x.data_ptr(), w.data_ptr() if has_w else None, b.data_ptr() if has_b else None, y.data_ptr(),
                               *(t.data_ptr() for t in stats), rows, n, n, n, code[dtype], code[wdt], code[dtype], eps, 0.0, int(rms), stream)
        on_grid = start * x.element_size() % 16 == 0 and n * x.element_size() % 16 == 0
        assert rc == 0 and (b"off-grid rows as vectors" in lib.b200_last_kernel()) == (n > 57 and not on_grid)
        assert bool((flat[:start] == 7).all()) and bool((flat[start + rows * n:] == 7).all()), "nothing beside the rows is written"
        d = x.double()
        mean = d.mean(-1, keepdim=True) * (0 if rms else 1)
        var = (d - mean).square().mean(-1, keepdim=True)
        rstd = (var + eps).rsqrt()
        want = (d - mean) * rstd
        scale = want.abs() + 1
        if has_w:
            want, scale = want * w.double(), scale * w.double().abs()
        if has_b:
            want, scale = want + b.double(), scale + b.double().abs()
        # one rounding of the result; in front of it some fp32 steps, and the sums: a chain of at most 64 terms of a lane and ten additions
        bound = ulp * want.abs() + 2.0 ** -24 * 80 * scale + 6.2e-8
        assert bool(((y.double() - want).abs() <= bound).all()), (start, ((y.double() - want).abs() - bound).max().item())
        assert torch.allclose(stats[0].double(), mean[:, 0], rtol=1e-5, atol=1e-5) and torch.allclose(stats[1].double(), rstd[:, 0], rtol=1e-5)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=str)
@pytest.mark.parametrize("n", [257, 377, 378, 505, 506, 761, 762, 1317, 4089, 4090])
def test_residual_and_gelu(dtype, n):
    """The three forms of the sum, the sum itself, the GELU prologue, and rows with infinities and NaN, which stay theirs."""
    from better_benchmark_b200 import kernels as k
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows = (14 if n <= 505 and n != 378 else 25 if n <= 505 else 64 if n <= 512 else 8 if n <= 1017 else 4) * sms + 1
    x, r = _storage(rows, n, dtype, 0, n), _storage(rows, n, dtype, 0, n + 1)
    x[5, n - 1], x[6, 0], x[7, n // 2] = float("nan"), float("inf"), float("-inf")
    w, b = torch.randn(n, device="cuda").to(dtype), torch.randn(n, device="cuda").to(dtype)
    kw = dict(eps=1e-6, residual=r, want_sum=True, want_mean=True, want_rstd=True)
    full, mean, rstd, _, total = k.norm_fwd(x, w, b, **kw)
    rounded = k.norm_fwd(x, w, b, round_sum=True, **kw)[0]
    both, mean2, rstd2, _, total2 = k.norm_fwd(x, w, b, round_sum="both", **kw)
    assert b"residual add, off-grid rows as vectors" in k.load().b200_last_kernel()
    gelu = k.norm_fwd(x, w, b, eps=1e-6, prologue="gelu_erf")[0]
    assert b"[off-grid rows as vectors]" in k.load().b200_last_kernel()
    s = x.float() + r.float()
    bad = torch.zeros(rows, dtype=torch.bool, device="cuda")
    bad[5:8] = True
    for t in (full, rounded, both):
        assert torch.equal(torch.isnan(t).any(-1), bad), "special values stay in their rows"
    assert not bool(torch.isnan(gelu[~bad]).any())
    ok = ~bad
    assert torch.equal(total[ok], s.to(dtype)[ok]) and torch.equal(total2[ok], total[ok])
    assert torch.equal(mean[ok], mean2[ok]) and torch.equal(rstd[ok], rstd2[ok])
    assert torch.equal(both[ok], torch.where(full.float().abs() > 3, full, rounded)[ok])
    ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    act = torch.nn.functional.gelu(x.double()).to(dtype)
    for got, at in ((full, x.double() + r.double()), (rounded, s.to(dtype).double()), (gelu, act.double())):
        d = at[ok]
        z = (d - d.mean(-1, keepdim=True)) * (d.var(-1, unbiased=False, keepdim=True) + 1e-6).rsqrt()
        want = z * w.double() + b.double()
        scale = (z.abs() + 1) * w.double().abs() + b.double().abs()
        # as above; an activation may round to the other neighbour, 2 ulp / 3 of what is normalised, and moves the row's statistics by less
        bound = ulp * want.abs() + (2.0 ** -24 * 80 + (2 * ulp if got is gelu else 0)) * scale + 6.2e-8
        assert bool(((got[ok].double() - want).abs() <= bound).all())
