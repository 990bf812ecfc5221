"""Every entry point that takes scratch memory keeps its launches together in the stream, so that host threads on one stream can share a scratch."""
import re
import threading
from pathlib import Path

import pytest
import torch

CSRC = Path(__file__).resolve().parent.parent / "better-benchmark_b200" / "csrc"


def _entry_points():
    for src in sorted(CSRC.glob("*.cu")):
        text = src.read_text()
        for m in re.finditer(r'extern "C" int (b200_\w+)\(([^)]*)\) \{\n(.*?)\n\}\n', text, re.S):
            yield m.group(1), m.group(2), m.group(3)


def test_launches_of_a_call_are_held_together():
    held = forwarding = 0
    for name, arguments, body in _entry_points():
        if not re.search(r"\bvoid\* scratch\b", arguments) or "const void* scratch" in arguments:
            continue
        if re.search(r"return b200_\w+\(", body):   # hands the call on to one that holds
            forwarding += 1
            continue
        lock = body.find("LaunchesTogether together(st);")
        first_launch = re.search(r"return (?:rms \? )?(?:launch|dispatch)_\w+<", body)
        assert first_launch is not None and 0 <= lock < first_launch.start(), name
        held += 1
    assert held == 4 and forwarding == 2, (held, forwarding)


@pytest.mark.gpu
def test_threads_on_one_stream_share_the_scratch():
    """Norm backwards (row tiles, streaming, ragged), BatchNorm and column sums, each in a thread of its own on the default stream and on
    another one: what every call returns is what it returns alone."""
    from better_benchmark_b200 import kernels as k
    g = torch.Generator(device="cuda").manual_seed(3)

    def norm(rows, n, dtype):
        x, dy = (torch.randn(rows, n, generator=g, device="cuda").to(dtype) for _ in range(2))
        w, mean = torch.rand(n, generator=g, device="cuda") + 0.5, x.float().mean(1)
        rstd = torch.rsqrt(x.float().var(1, unbiased=False) + 1e-5)
        return lambda: k.norm_bwd(x, dy, w, rstd, mean=mean, rms=False, want_dbias=True)

    def batch_norm(channels):
        x, dy = (torch.randn(8, channels, 14, 14, generator=g, device="cuda").bfloat16().to(memory_format=torch.channels_last) for _ in range(2))
        w = torch.rand(channels, generator=g, device="cuda")
        mean, invstd = x.float().mean((0, 2, 3)), torch.rsqrt(x.float().var((0, 2, 3)) + 1e-5)
        return [lambda: k.batch_norm_fwd(x, w, w, None, None, eps=1e-5, momentum=0.1), lambda: k.batch_norm_bwd(dy, x, mean, invstd, w)]

    columns = torch.randn(20000, 40, generator=g, device="cuda")
    calls = [norm(1100, 4096, torch.bfloat16), norm(1200, 2048, torch.bfloat16), norm(1024, 2056, torch.float32), norm(1300, 2305, torch.bfloat16),
             *batch_norm(64), *batch_norm(144), lambda: (k.col_reduce(columns, "sum"),)]
    want = [call() for call in calls]
    torch.cuda.synchronize()
    for stream in (torch.cuda.default_stream(), torch.cuda.Stream()):
        got, errors, start = {}, [], threading.Barrier(len(calls))

        def work(i):
            try:
                with torch.cuda.stream(stream):
                    start.wait()
                    got[i] = [calls[i]() for _ in range(60)]
            except BaseException as e:  # noqa: BLE001
                errors.append(e)

        threads = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        torch.cuda.synchronize()
        assert not errors, errors
        for i, outs in got.items():
            for out in outs:
                assert all(torch.equal(a, b) for a, b in zip(out, want[i])), i
