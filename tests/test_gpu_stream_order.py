"""Kernels start while their predecessor in the stream drains: what they read must be what it wrote.

Every call below reads a tensor that the operation before it in the stream has just changed (a torch kernel, a
copy, another call of the library), without synchronising. Each result must have the bits of the same call made
after a synchronisation.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _calls():
    """name -> (input shape, dtype, call); every call returns tensors that depend on its input."""
    import better_benchmark_b200.kernels as k
    w = torch.linspace(0.5, 1.5, 768, device="cuda")
    rstd, mean = torch.full((2000,), 0.7, device="cuda"), torch.full((2000,), 0.1, device="cuda")
    cl = lambda t: t.view(8, 28, 28, 64).permute(0, 3, 1, 2)  # noqa: E731
    ones = torch.ones(64, device="cuda")
    return {
        "cast": ((2000, 768), torch.float32, lambda x: k.cast_scale(x, torch.bfloat16)),
        "silu": ((2000, 768), torch.bfloat16, lambda x: k.cast_scale(x, torch.bfloat16, activation="silu")),
        "row sum": ((2000, 768), torch.float32, lambda x: k.row_reduce(x, "sum")),
        "column sum": ((2000, 768), torch.float32, lambda x: k.col_reduce(x, "sum")),
        "softmax": ((2000, 768), torch.float16, lambda x: k.softmax(x)),
        "softmax ragged": ((700, 1003), torch.float16, lambda x: k.softmax(x)),
        "layer norm": ((2000, 768), torch.bfloat16, lambda x: k.norm_fwd(x, w, w, eps=1e-5, want_rstd=True)[:3:2]),
        "residual": ((2000, 768), torch.bfloat16,
                     lambda x: k.norm_fwd(x, x[0], x[1], eps=1e-5, residual=x, want_sum=True, round_sum="both")[0::4]),
        "norm backward": ((2000, 768), torch.bfloat16, lambda x: k.norm_bwd(x, x, w, rstd, mean=mean, rms=False, want_dbias=True)),
        "norm backward, weight": ((2000, 768), torch.float32, lambda x: k.norm_bwd(x, x, x[0], rstd, rms=True)[:2]),
        "batch norm": ((8, 28, 28, 64), torch.bfloat16,
                       lambda x: k.batch_norm_fwd(cl(x), ones, ones, None, None, eps=1e-5, momentum=0.1)),
        "batch norm backward": ((8, 28, 28, 64), torch.bfloat16, lambda x: k.batch_norm_bwd(cl(x), cl(x), ones, ones, ones)),
        "batch norm nchw": ((8, 64, 28, 28), torch.float32,
                            lambda x: k.batch_norm_fwd(x, ones, ones, None, None, eps=1e-5, momentum=0.1)),
        "transpose": ((64, 49, 128), torch.bfloat16, lambda x: k.permute_copy(x, (0, 2, 1))),
    }


NAMES = ["cast", "silu", "row sum", "column sum", "softmax", "softmax ragged", "layer norm", "residual", "norm backward",
         "norm backward, weight", "batch norm", "batch norm backward", "batch norm nchw", "transpose"]


def _list(out):
    return [out] if isinstance(out, torch.Tensor) else [t for t in out if t is not None]


@pytest.mark.parametrize("name", NAMES)
def test_inputs_changed_just_before_the_call(name):
    shape, dtype, call = _calls()[name]
    g = torch.Generator(device="cuda").manual_seed(7)
    sources = [torch.randn(shape, generator=g, device="cuda").to(dtype) for _ in range(4)]
    want = []
    for s in sources:
        torch.cuda.synchronize()
        want.append(_list(call(s)))
    torch.cuda.synchronize()
    x = torch.empty_like(sources[0])
    got = []
    for i in range(40):   # a device copy, or a kernel, or both, and the call right behind it
        if i % 3 == 0:
            x.copy_(sources[i % 4])
        elif i % 3 == 1:
            torch.add(sources[i % 4], 0, out=x)
        else:
            x.zero_()
            torch.mul(sources[i % 4], 1, out=x)
        got.append(_list(call(x)))
    torch.cuda.synchronize()
    for i, out in enumerate(got):
        for a, b in zip(out, want[i % 4]):
            assert torch.equal(a, b), f"{name}, call {i}"


@pytest.mark.parametrize("name", ["cast", "layer norm", "norm backward", "batch norm", "batch norm backward", "softmax ragged"])
def test_capture_behind_a_copy_and_behind_a_join(name):
    """In a graph: behind a copy node, behind the join of two streams, and with the input replaced between replays."""
    shape, dtype, call = _calls()[name]
    g = torch.Generator(device="cuda").manual_seed(8)
    sources = [torch.randn(shape, generator=g, device="cuda").to(dtype) for _ in range(3)]
    want = [[t.clone() for t in _list(call(s))] for s in sources]
    torch.cuda.synchronize()
    source, x, z = sources[0].clone(), torch.empty_like(sources[0]), torch.empty_like(sources[0])
    side = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        x.copy_(source)
        first = _list(call(x))
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            torch.add(source, 0, out=z)
        x.copy_(source)
        torch.cuda.current_stream().wait_stream(side)
        second = _list(call(z))
        third = _list(call(z))
    for i in (1, 2, 0, 1):
        source.copy_(sources[i])
        graph.replay()
        for out in (first, second, third):
            for a, b in zip(out, want[i]):
                assert torch.equal(a, b), name
