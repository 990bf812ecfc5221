"""LayerNorm / RMSNorm backward of rows of at most 32 vectors: several rows per warp, fp64 partial rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rms", [False, True], ids=["layer", "rms"])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32], ids=str)
@pytest.mark.parametrize("vectors", [1, 3, 8, 9, 16, 17, 31, 32])
def test_narrow_rows(vectors, dtype, rms):
    """Every change of geometry; fewer rows than a CTA takes, one more than it does, several turns; small scratch; a chained finalize."""
    from better_benchmark_b200 import kernels as k
    n = vectors * (4 if dtype == torch.float32 else 8)
    ulp = {torch.float32: 2.0 ** -23, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype]
    for rows in (1, 3, 33, 4001, 60007):
        g = torch.Generator(device="cuda").manual_seed(n + rows)
        x, dy = ((torch.randn(rows, n, generator=g, device="cuda") * 2).to(dtype) for _ in range(2))
        w = torch.randn(n, generator=g, device="cuda").to(dtype)
        mean = None if rms else torch.randn(rows, generator=g, device="cuda")
        rstd = torch.rand(rows, generator=g, device="cuda") + 0.5
        xd, gd, r = x.double(), dy.double(), rstd.double()[:, None]
        wg = gd * w.double()
        if rms:
            xhat = xd * r
            want = wg * r - xd * (wg * xd).sum(-1, keepdim=True) * r ** 3 / n
            size = wg.abs() * r + (xd * r ** 3).abs() * (wg * xd).abs().sum(-1, keepdim=True) / n
        else:
            xhat = (xd - mean.double()[:, None]) * r
            want = r / n * (n * wg - wg.sum(-1, keepdim=True) - xhat * (wg * xhat).sum(-1, keepdim=True))
            size = r * (wg.abs() + wg.abs().mean(-1, keepdim=True) + xhat.abs() * (wg * xhat).abs().mean(-1, keepdim=True))
        small = torch.zeros(256 + 8 * 2 * n * 4, dtype=torch.uint8, device="cuda")
        for kw in (dict(), dict(two_launch=True), dict(scratch=small)):
            dx, dw, db = k.norm_bwd(x, dy, w, rstd, mean=mean, rms=rms, want_dweight=True, want_dbias=not rms, **kw)
            # one rounding of the result; chains of four additions in a lane, five between lanes, and six steps
            assert bool(((dx.double() - want).abs() <= ulp * want.abs() + 2.0 ** -24 * 24 * size + 6.2e-8).all())
            # a lane's chain in fp32: its rows (with four workers of at least eight groups: rows / 32), then fp64
            chain = 2.0 ** -24 * (rows // 32 + 8)
            assert bool(((dw.double() - (gd * xhat).sum(0)).abs() <= chain * (gd * xhat).abs().sum(0) + 1e-30).all())
            if not rms:
                assert bool(((db.double() - gd.sum(0)).abs() <= chain * gd.abs().sum(0) + 1e-30).all())
            again = k.norm_bwd(x, dy, w, rstd, mean=mean, rms=rms, want_dweight=True, want_dbias=not rms, **kw)
            assert torch.equal(again[0], dx) and torch.equal(again[1], dw), "bit-reproducible"
        assert int(small[:256].count_nonzero()) == 0, "the words are zero between launches"
    k.check_scratch_status()
