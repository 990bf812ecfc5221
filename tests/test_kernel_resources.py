"""Registers and spills of kernels whose launch geometry counts on them, from what ``ptxas -v`` printed when the
library was built here. An SM has 65 536 registers: a kernel of T threads a block keeps c blocks resident
up to 65 536 / (T c) registers a thread."""
import re

import pytest


def _resources(stem):
    """{mangled kernel name: (registers, bytes spilled)} of one source file."""
    from better_benchmark_b200 import build
    log = build.BUILD_DIR / f"{stem}.ptxas"
    if not log.exists():
        pytest.skip("the library was not built in this tree")
    out, name, spill = {}, None, 0
    for line in log.read_text().splitlines():
        if m := re.search(r"Compiling entry function '(\S+)'", line):
            name = m.group(1)
        elif m := re.search(r"(\d+) bytes spill stores", line):
            spill = int(m.group(1))
        elif (m := re.search(r"Used (\d+) registers", line)) and name:
            out[name], name = (int(m.group(1)), spill), None
    return out


# (source, pattern over the mangled name, registers, why)
LIMITS = [
    ("norm_fwd", r"norm_fwd_resident_kernel.*Li4ELi0ELb0ELb0E", 102, "CTA per row of 128 threads: five per SM"),
    ("norm_fwd", r"norm_fwd_resident_kernel.*Li4ELi(8|16|32)ELb0ELb0E", 85, "sub-warp rows, 256 threads: three CTAs per SM"),
    ("norm_bwd", r"norm_bwd_stream_kernelIfLi2ELb0E", 93, "fp32 RMSNorm, streaming, up to 352 threads: two CTAs per SM"),
    ("norm_bwd", r"norm_bwd_stream_kernelIfLi2ELb1E", 100, "fp32 LayerNorm, streaming, up to 320 threads: two CTAs per SM"),
]


@pytest.mark.parametrize("stem,pattern,limit,why", LIMITS)
def test_registers(stem, pattern, limit, why):
    kernels = {n: r for n, r in _resources(stem).items() if re.search(pattern, n)}
    assert kernels, f"no kernel matches {pattern}"
    for name, (registers, spilled) in kernels.items():
        assert registers <= limit and spilled == 0, f"{name}: {registers} registers, {spilled} bytes spilled ({why})"
