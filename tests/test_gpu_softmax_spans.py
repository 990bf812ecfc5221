"""Masked softmax of many 16-bit rows off the 16-byte grid: groups of lanes that keep the mask, and a CTA per row."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(rows, n, dtype, mask, scale, start, log, batches=4):
    """x, out and what lies around them in one storage each, so that an access outside is seen (NaN in, a changed guard out)."""
    from better_benchmark_b200 import kernels as k
    g = torch.Generator(device="cuda").manual_seed(n + rows)
    size = rows * n
    xs = torch.full((size + 64,), float("nan"), device="cuda", dtype=dtype)
    xs[start:start + size] = (torch.randn(size, generator=g, device="cuda") * 3).to(dtype)
    ys = torch.full((size + 64,), 7.0, device="cuda", dtype=dtype)
    x, y = (t[start:start + size].view(batches, rows // batches, n) for t in (xs, ys))
    k.softmax(x, mask=mask, scale=scale, log=log, out=y)
    shared = mask is None and n < 256 or mask is not None and mask.shape[1] == 1
    fills = 121 < n <= 128 or 249 < n <= 256   # the other kernel's slots, and one more of this one's
    by_vectors = (n > 1017 and mask is not None or shared) and not fills and not (start % 8 == 0 and n % 8 == 0)
    assert (b"off-grid rows as vectors" in k.load().b200_last_kernel()) == by_vectors
    assert bool((ys[:start] == 7).all()) and bool((ys[start + size:] == 7).all()), "nothing beside the rows is written"
    t = x.double() * (1.0 if scale is None else scale)
    if mask is not None:
        t = t + mask.double()
    return y, torch.log_softmax(t, -1) if log else torch.softmax(t, -1)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16], ids=str)
@pytest.mark.parametrize("n", [1, 7, 9, 50, 57, 58, 114, 121, 122, 185, 249, 250, 257, 377, 378, 505, 506, 761, 762, 1017, 1018, 1241, 2047, 4089, 4090, 8191])
def test_spans(dtype, n):
    """Both sides of every change of geometry; every alignment of the first row; masks per batch, per row and none."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    per_sm = next(r for most, r in ((57, 44), (99, 160), (185, 52), (234, 250), (249, 96), (390, 25), (505, 5), (512, 72), (1017, 11), (8191, 2)) if n <= most)
    rows = (per_sm * sms + 15) // 4 * 4
    ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    g = torch.Generator(device="cuda").manual_seed(n)
    key = torch.where(torch.rand(4, 1, n, generator=g, device="cuda") < 0.7, 0.0, -10000.0).to(dtype)
    per_row = torch.randn(4, rows // 4, n, generator=g, device="cuda").to(dtype)
    cases = [(key, 0.125, 0, False), (None, None, 3, False), (per_row, None, 0, True), (key, 0.5, 5, True)]
    for start in (1, 2, 4, 6, 7):
        cases.append((key, None, start, False))
    for mask, scale, start, log in cases:
        y, want = _run(rows, n, dtype, mask, scale, start, log)
        # one rounding of the result, and fp32 steps in front of it (of a log-probability also in its terms, which may be 1e4)
        bound = ulp * want.abs() + (4e-6 * want.abs().clamp(max=1e4) + 2e-5 if log else 2e-6 * want + 6.2e-8)
        assert bool(((y.double() - want).abs() <= bound).all()), (n, start, log, ((y.double() - want).abs() - bound).max().item())


@pytest.mark.parametrize("n", [41, 333, 1001, 1241])
def test_special_values(n):
    """Masks of -inf and of the type's lowest value, rows without a key, infinities and NaN in one row, which stay there."""
    from better_benchmark_b200 import kernels as k
    rows = 8000
    x = torch.randn(2, rows // 2, n, device="cuda").half()
    x[0, 5, 3], x[0, 6, 0], x[1, 7, n - 1], x[1, 9] = float("nan"), float("inf"), float("-inf"), float("-inf")
    for low in (float("-inf"), torch.finfo(torch.float16).min):
        mask = torch.zeros(2, 1, n, device="cuda", dtype=torch.float16)
        mask[0, :, n // 2:] = low
        mask[1, :, 1:] = low
        for log in (False, True):
            got = k.softmax(x, mask=mask, scale=0.5, log=log)
            t = x.double() * 0.5 + mask.double()
            want = torch.log_softmax(t, -1) if log else torch.softmax(t, -1)
            assert torch.equal(torch.isnan(got), torch.isnan(want))
            assert torch.allclose(got.double(), want.to(got.dtype).double(), rtol=2e-3, atol=1e-6 if not log else 2e-2, equal_nan=True)
    full = torch.full((2, 1, n), float("-inf"), device="cuda", dtype=torch.float16)
    assert bool(torch.isnan(k.softmax(x, mask=full)).all())


@pytest.mark.parametrize("n", [41, 100, 333, 716, 1241])
def test_probabilities_below_the_normal_range(n):
    """bf16 holds numbers down to 2^-133 and so does fp32 below its normal range: probabilities there are not lost."""
    from better_benchmark_b200 import kernels as k
    rows = 200 * torch.cuda.get_device_properties(0).multi_processor_count
    x = torch.full((rows, n), -80.0, device="cuda", dtype=torch.bfloat16)
    x[:, 7] = 0.0
    mask = torch.linspace(0.0, -12.0, n, device="cuda").to(torch.bfloat16)
    mask[7] = 0.0
    got, want = k.softmax(x, mask=mask).double(), torch.softmax(x[:1].double() + mask.double(), -1)
    assert 0 < want.min() < 2.0 ** -130 and int((want < 2.0 ** -126).sum()) > n // 4
    # bf16's rounding: half a step of eight significant bits, at most 2^-8 of the value, below the normal range half of 2^-133; in front of it
    # those of fp32's exponential and of its product with the sum's inverse, 2^-21 of the value and steps of 2^-149 there
    assert bool(((got - want).abs() <= (2.0 ** -8 + 2.0 ** -21) * want + 2.0 ** -134 + 2.0 ** -147).all())


@pytest.mark.parametrize("n,group", [(41, 8), (100, 8), (333, 16), (716, 32)])
def test_masks_that_few_rows_share(n, group):
    """A group of lanes keeps its part of the mask, so masks for fewer rows than two turns of a CTA go by the element; so do rows that just fill
    that kernel's slots. The results are the same."""
    from better_benchmark_b200 import kernels as k
    rows = 208 * torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator(device="cuda").manual_seed(n)
    least = 2 * 256 // group
    x = torch.randn(rows, n, generator=g, device="cuda").half()
    masks = torch.randn(rows, n, generator=g, device="cuda").half()
    for share in (1, least // 2, least, 4 * least):
        for outer in (1, 2):
            batched = x[:rows // (outer * share) * outer * share].view(outer, -1, share, n)
            mask = masks[:batched.shape[0] * batched.shape[1]].view(outer, -1, 1, n)
            got = k.softmax(batched, mask=mask, scale=0.5)
            assert (b"off-grid rows as vectors" in k.load().b200_last_kernel()) == (share >= least), share
            want = torch.softmax(batched.double() * 0.5 + mask.double(), -1)
            assert bool(((got.double() - want).abs() <= (2.0 ** -11 + 2e-6) * want + 6.2e-8).all())
    every = masks[:1].expand(rows, n)
    k.softmax(x, mask=every)
    assert b"off-grid rows as vectors" in k.load().b200_last_kernel(), "one mask for all rows"
    for full in (125, 251, 509):
        x = torch.randn(rows, full, generator=g, device="cuda").half()
        got = k.softmax(x, mask=x[0])
        assert (b"[elements in registers]" in k.load().b200_last_kernel()) == (full < 256)
        want = torch.softmax(x.double() + x[0].double(), -1)
        assert bool(((got.double() - want).abs() <= (2.0 ** -11 + 2e-6) * want + 6.2e-8).all())
