"""Norm backward whose column sums are added up by the CTAs of the same launch, by some that start after the workers, or by a kernel chained to it."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(rows, n, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x, dy = (torch.randn(rows, n, generator=g, device="cuda").to(dtype) for _ in range(2))
    return x, dy, torch.rand(n, generator=g, device="cuda") + 0.5, x.float().mean(1), torch.rsqrt(x.float().var(1, unbiased=False) + 1e-5)


def _sums(x, dy, mean, rstd):
    xhat = (x.double() - mean.double()[:, None]) * rstd.double()[:, None]
    return (dy.double() * xhat).sum(0), dy.double().sum(0), (dy.double() * xhat).abs().sum(0), dy.double().abs().sum(0)


@pytest.mark.parametrize("rows,n,dtype", [(1, 64, torch.float32), (7, 768, torch.bfloat16), (9, 1024, torch.float32), (2369, 264, torch.bfloat16),
                                          (300, 2048, torch.float16), (1024, 1040, torch.bfloat16), (1025, 4096, torch.bfloat16),
                                          (2000, 2056, torch.float32), (1500, 8192, torch.float32), (64, 16384, torch.bfloat16)])
def test_column_sums_and_scratch_words(rows, n, dtype):
    from better_benchmark_b200 import kernels as k
    x, dy, w, mean, rstd = _inputs(rows, n, dtype, rows)
    want_w, want_b, abs_w, abs_b = _sums(x, dy, mean, rstd)
    scratch = torch.zeros(256 + 64 * 2 * n * 4, dtype=torch.uint8, device="cuda")   # also: fewer workers than the GPU has room for
    for buffer in (None, scratch):
        for want_db in (True, False):
            first = None
            for _ in range(3):
                dx, dw, db = k.norm_bwd(x, dy, w, rstd, mean=mean, rms=False, want_dbias=want_db, scratch=buffer)
                if first is not None:
                    assert torch.equal(dw, first), "bit-reproducible"
                first = dw
            # a column's chain in fp32: at most rows / 64 rows a worker, and its warps; an ulp of the magnitudes for each
            depth = (rows // 8 + 16) * 2.0 ** -24
            assert bool(((dw.double() - want_w).abs() <= depth * abs_w + 1e-30).all())
            if want_db:
                assert bool(((db.double() - want_b).abs() <= depth * abs_b + 1e-30).all())
    assert int(scratch[:256].count_nonzero()) == 0, "the words are zero between launches"
    k.check_scratch_status()


def test_two_streams_at_once():
    """Launches that wait for their own workers only: two that overlap, each with a scratch of its own, end and agree with one alone."""
    from better_benchmark_b200 import kernels as k
    cases = [_inputs(3000, 768, torch.bfloat16, 1), _inputs(1100, 4096, torch.bfloat16, 2), _inputs(500, 1024, torch.float32, 3)]
    want = [k.norm_bwd(x, dy, w, rstd, mean=mean, rms=False, want_dbias=True) for x, dy, w, mean, rstd in cases]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(2)]
    scratch = [torch.zeros(64 << 20, dtype=torch.uint8, device="cuda") for _ in range(2)]
    got = [[], []]
    for i in range(40):
        for s in range(2):
            x, dy, w, mean, rstd = cases[(i + s) % 3]
            with torch.cuda.stream(streams[s]):
                got[s].append(((i + s) % 3, k.norm_bwd(x, dy, w, rstd, mean=mean, rms=False, want_dbias=True, scratch=scratch[s])))
    torch.cuda.synchronize()
    for outs in got:
        for which, out in outs:
            assert all(torch.equal(a, b) for a, b in zip(out, want[which]))


@pytest.mark.parametrize("rows,n,dtype", [(1100, 4096, torch.bfloat16), (1100, 2056, torch.float32), (1030, 16384, torch.bfloat16), (300, 768, torch.bfloat16),
                                          (300, 64, torch.bfloat16), (300, 2048, torch.float32)])
def test_two_launches_need_no_zeroed_words(rows, n, dtype):
    """The two-launch form neither reads nor writes the words in front of the scratch."""
    from better_benchmark_b200 import kernels as k
    x, dy, w, mean, rstd = _inputs(rows, n, dtype, rows)
    want = k.norm_bwd(x, dy, w, rstd, mean=mean, rms=False, want_dbias=True, two_launch=True)
    scratch = torch.full((256 + 600 * 2 * n * 4,), 0xa5, dtype=torch.uint8, device="cuda")
    got = k.norm_bwd(x, dy, w, rstd, mean=mean, rms=False, want_dbias=True, two_launch=True, scratch=scratch)
    for a, b in zip(got, want):
        assert not bool(torch.isnan(a).any()) and torch.allclose(a.float(), b.float(), rtol=1e-5, atol=1e-3)
    assert bool((scratch[:256] == 0xa5).all())


@pytest.mark.parametrize("rows,n,dtype", [(1100, 4096, torch.bfloat16), (1100, 2056, torch.float32), (1030, 16384, torch.bfloat16), (300, 768, torch.bfloat16),
                                          (5000, 264, torch.bfloat16), (300, 64, torch.bfloat16), (300, 2048, torch.float32)])
def test_a_noted_error_shows_in_the_sums(rows, n, dtype):
    """With an error still noted in the words no sums are formed: they are NaN, not what the memory held, and the status says why."""
    from better_benchmark_b200 import kernels as k
    from better_benchmark_b200 import native
    x, dy, w, mean, rstd = _inputs(rows, n, dtype, rows)
    scratch = torch.zeros(256 + 600 * 2 * n * 4, dtype=torch.uint8, device="cuda")
    scratch[:16].view(torch.int32)[1] = 1
    want = k.norm_bwd(x, dy, w, rstd, mean=mean, rms=False, want_dbias=True)
    got = k.norm_bwd(x, dy, w, rstd, mean=mean, rms=False, want_dbias=True, scratch=scratch)
    assert torch.equal(got[0], want[0]) and bool(torch.isnan(got[1]).all()) and bool(torch.isnan(got[2]).all())
    assert native.load().b200_check_status(scratch.data_ptr(), torch.cuda.current_stream().cuda_stream) != 0
    assert int(scratch[:256].count_nonzero()) == 1


@pytest.mark.parametrize("rows,n,dtype", [(3000, 768, torch.bfloat16), (700, 2048, torch.bfloat16), (64, 512, torch.float32), (4000, 128, torch.bfloat16)])
def test_while_another_stream_holds_the_gpu(rows, n, dtype):
    """CTAs that find the GPU full of another stream's start late, and those that are there do not wait for them: the last one adds up."""
    from better_benchmark_b200 import kernels as k
    x, dy, w, mean, rstd = _inputs(rows, n, dtype, rows)
    scratch = torch.zeros(16 << 20, dtype=torch.uint8, device="cuda")
    want = k.norm_bwd(x, dy, w, rstd, mean=mean, rms=False, want_dbias=True, scratch=scratch)
    a = torch.randn(4096, 4096, device="cuda")
    a @ a
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    got = []
    for _ in range(6):
        with torch.cuda.stream(side):
            for _ in range(3):
                a @ a   # a few ms of every SM
        for _ in range(12):
            got.append(k.norm_bwd(x, dy, w, rstd, mean=mean, rms=False, want_dbias=True, scratch=scratch))
    torch.cuda.synchronize()
    for outs in got:
        assert all(torch.equal(p, q) for p, q in zip(outs, want))
    assert int(scratch[:256].count_nonzero()) == 0
