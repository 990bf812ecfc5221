"""Row reductions: several rows a warp (up to 256 vectors), rows that start and end off the 16-byte grid, and totals that leave fp32."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}


@pytest.mark.parametrize("op", ["sum", "mean", "amax", "amin"])
@pytest.mark.parametrize("dtype", list(DTYPES))
def test_lengths_and_alignments(dtype, op):
    """Around every change of the geometry (16, 32, 64, 128, 256 vectors), each start and pitch that a vector can meet."""
    from better_benchmark_b200 import kernels as k
    dt = DTYPES[dtype]
    v = 16 // dt.itemsize
    g = torch.Generator(device="cuda").manual_seed(7)
    for n in (1, 2, v - 1, v, v + 1, 15 * v + 3, 16 * v, 16 * v + 1, 32 * v, 32 * v + v - 1, 64 * v, 64 * v + 1, 128 * v,
              128 * v + 5, 256 * v, 256 * v + 1, 520 * v + 3):
        for rows in (1, 33, 700):
            for start, pad in ((0, 0), (1, 0), (v - 1, 1), (0, v)):
                base = torch.randn(rows, n + start + pad, generator=g, device="cuda").to(dt)
                x = base[:, start:start + n]
                got = k.row_reduce(x, op, out_dtype=torch.float32)
                d = x.double()
                if op in ("amax", "amin"):
                    assert torch.equal(got, getattr(d, op)(-1).float()), (n, rows, start, pad)
                    continue
                want = getattr(d, op)(-1)
                # chains of at most 2 n / (32 v) + 14 fp32 additions (and the product of the mean), each off by half an ulp of
                # at most the row's sum of magnitudes
                bound = (d.abs().sum(-1) / (n if op == "mean" else 1)) * 2.0 ** -24 * (2 * n / (32 * v) + 16)
                assert bool(((got.double() - want).abs() <= bound).all()), (n, rows, start, pad)


@pytest.mark.parametrize("n", [6, 60, 120, 250, 500])
def test_totals_beyond_fp32_on_the_way(n):
    """Chains that overflow although the sum is a number, infinities of one and of both signs, NaN, in rows next to ordinary ones."""
    from better_benchmark_b200 import kernels as k
    x = torch.ones(9, n, device="cuda")
    x[1, :n // 2] = 3e38
    x[1, n // 2:] = -3e38
    x[2, 1] = float("inf")
    x[3, 0], x[3, n - 1] = float("inf"), float("-inf")
    x[4, n // 2] = float("nan")
    x[5] = 3e38
    x[6] = -0.0
    got, want = k.row_reduce(x, "sum").cpu(), x.double().sum(-1).float().cpu()
    assert torch.allclose(got, want, rtol=1e-6, atol=0, equal_nan=True), (got, want)
    got, want = k.row_reduce(x, "amax").cpu(), x.amax(-1).cpu()
    assert torch.allclose(got, want, rtol=0, atol=0, equal_nan=True), (got, want)


@pytest.mark.parametrize("op", ["sum", "amax"])
@pytest.mark.parametrize("dtype,n,per_sm,path", [
    ("f32", 512, 17, b"several rows a warp"), ("f32", 1023, 17, b"several rows a warp"), ("f32", 1028, 17, b"vector, warp per row"),
    ("f32", 1024, 3, b"any alignment, CTA per row"), ("f32", 1023, 3, b"any alignment, CTA per row"), ("bf16", 4104, 63, b"vector, warp per row"), ("bf16", 4096, 17, b"any alignment, warp per row"),
    ("bf16", 4096, 8, b"any alignment, CTA per row"), ("bf16", 4001, 17, b"any alignment, warp per row"),
    ("f16", 4001, 40, b"any alignment, warp per row"), ("f32", 2049, 60, b"any alignment, warp per row"),
    ("bf16", 5001, 8, b"any alignment, CTA per row")])
def test_routes_of_longer_rows(dtype, n, per_sm, path, op):
    """Each kernel for rows of 64 vectors and more, at a number of rows that it takes."""
    from better_benchmark_b200 import kernels as k
    dt = DTYPES[dtype]
    rows = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + 3
    x = torch.randn(rows, n, generator=torch.Generator(device="cuda").manual_seed(n), device="cuda").to(dt)
    got = k.row_reduce(x, op, out_dtype=torch.float32)
    assert path in k.load().b200_last_kernel(), k.load().b200_last_kernel()
    d = x.double()
    if op == "amax":
        assert torch.equal(got, d.amax(-1).float())
    else:
        bound = d.abs().sum(-1) * 2.0 ** -24 * (2 * n / (32 * 16 // dt.itemsize) + 16)   # as above
        assert bool(((got.double() - d.sum(-1)).abs() <= bound).all())
