"""Softmax of long rows with more rows than SMs: clusters or two sweeps; fp32 rows with 16-bit results that keep their exponentials."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("log", [False, True])
@pytest.mark.parametrize("n,dtype,out_dtype,path", [
    (32772, torch.float32, torch.float32, b"cluster"), (65536, torch.float32, torch.float32, b"cluster"),
    (65540, torch.float32, torch.float32, b"two sweeps"), (65537, torch.float32, torch.float32, b"cluster"),
    (131072, torch.float32, torch.float16, b"cluster"), (131075, torch.float32, torch.bfloat16, b"cluster"),
    (131076, torch.float32, torch.bfloat16, b"two sweeps"), (65544, torch.bfloat16, torch.bfloat16, b"cluster"),
    (131072, torch.float16, torch.float16, b"cluster"), (131080, torch.bfloat16, torch.bfloat16, b"two sweeps"),
    (2909, torch.float32, torch.bfloat16, b"registers of a CTA"), (16384 + 3, torch.float32, torch.float16, b"registers of a CTA"),
], ids=str)
def test_many_long_rows(n, dtype, out_dtype, path, log):
    from better_benchmark_b200 import kernels as k
    rows = torch.cuda.get_device_properties(0).multi_processor_count + 1
    x = (torch.randn(rows, n, device="cuda") * 3).to(dtype)
    x[3, : n // 2] = float("-inf")
    x[4, 5], x[5, n - 1], x[6] = float("nan"), float("inf"), float("-inf")
    if dtype != torch.float16:
        x[7], x[7, 9] = -3e38, 3e38    # differences beyond what fp32 holds
        x[8], x[8, 9], x[8, 11] = -3e38, -2e38, float("-inf")   # and rows far below what -inf might be replaced by
        x[9], x[9, n - 1] = float("-inf"), -3e38
    got = k.softmax(x, log=log, out_dtype=out_dtype)
    assert path in k.load().b200_last_kernel(), k.load().b200_last_kernel()
    want = torch.log_softmax(x.double(), -1) if log else torch.softmax(x.double(), -1)
    poisoned = torch.isnan(got).all(-1)
    assert bool(poisoned[4:7].all()) and int(poisoned.sum()) == 3
    ok = ~poisoned
    ulp = {torch.float32: 2.0 ** -23, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[out_dtype]
    got, want = got[ok].double(), want[ok]
    if log:
        # the difference, the logarithm of the sum and their difference, each rounded once, and 2e-6 for the sum's own error
        finite = torch.isfinite(got) & (want.abs() < 1e30)
        bound = ulp * want.abs() + 2.0 ** -23 * want.abs() + 4e-6
        assert bool(((got - want).abs() <= bound)[finite].all())
        assert bool((got[~finite] < -6e4).all())
    else:
        # the exponent's difference may be off by half an ulp of 30 and the exponential by two of its own
        assert bool(((got - want).abs() <= ulp * want + 4e-6 * want + 6.2e-8 * (out_dtype == torch.float16) + 1e-38).all())


@pytest.mark.parametrize("n,dtype,path", [(98304, torch.bfloat16, b"two sweeps"), (50000, torch.float32, b"cluster"), (65536, torch.float32, b"cluster"),
                                          (81920, torch.float16, b"cluster"), (81928, torch.float16, b"two sweeps"), (98307, torch.bfloat16, b"cluster")])
def test_full_last_rows(n, dtype, path):
    """Two rows an SM: the sweeps lose nothing to an SM without a row."""
    from better_benchmark_b200 import kernels as k
    rows = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    x = (torch.randn(rows, n, device="cuda") * 3).to(dtype)
    for log in (False, True):
        got = k.softmax(x, log=log)
        assert path in k.load().b200_last_kernel(), k.load().b200_last_kernel()
        for i in (0, rows - 1):
            want = torch.log_softmax(x[i].double(), -1) if log else torch.softmax(x[i].double(), -1)
            ulp = {torch.float32: 2.0 ** -23, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype]
            # one rounding of the result; in front of it the difference, the exponential and the sum, as above
            bound = (ulp + 2.0 ** -23) * want.abs() + 4e-6 * (1 if log else want) + 6.2e-8 * (dtype == torch.float16)
            assert bool(((got[i].double() - want).abs() <= bound + 1e-38).all())
