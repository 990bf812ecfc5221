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
    seeds = torch.tensor([11, 12], device="cuda")
    res = torch.linspace(-1, 1, 2000 * 512, device="cuda").view(2000, 512)
    bias = torch.linspace(-2, 2, 64 * 256, device="cuda").view(1, 1, 64, 256).expand(2, 12, 64, 256)
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
        # kernels for ragged rows and columns: scalar loads, of vectors along the row as well as of the row itself
        "softmax ragged, masked": ((700, 1003), torch.float16, lambda x: k.softmax(x, mask=x)),
        "layer norm ragged": ((1000, 767), torch.bfloat16, lambda x: k.norm_fwd(x, x[0], x[1], eps=1e-5, want_rstd=True)[:3:2]),
        "norm backward ragged": ((2000, 767), torch.bfloat16,
                                 lambda x: k.norm_bwd(x, x, x[0], rstd, mean=mean, rms=False, want_dbias=True)),
        # the same rows by the vector, where there are more of them
        "softmax as vectors, masked": ((2000, 1003), torch.float16, lambda x: k.softmax(x, mask=x[0])),
        "layer norm as vectors": ((2000, 767), torch.bfloat16, lambda x: k.norm_fwd(x, x[0], x[1], eps=1e-5, want_rstd=True)[:3:2]),
        "norm backward as vectors": ((2000, 1601), torch.bfloat16,
                                     lambda x: k.norm_bwd(x, x, x[0], rstd, mean=mean, rms=False, want_dbias=True)),
        "transpose ragged": ((16, 501, 333), torch.float16, lambda x: k.permute_copy(x, (0, 2, 1))),
        "dropout norm": ((2000, 512), torch.bfloat16, lambda x: k.dropout_rms_norm(x, res, w[:512], seeds, 0, 1, p=0.1, eps=1e-6)),
        "batch norm backward, sums": ((8, 28, 28, 64), torch.bfloat16,
                                      lambda x: k.batch_norm_bwd(cl(x), cl(x), ones, ones, ones, want_dx=False)),
        "softmax dropout": ((24, 64, 256), torch.bfloat16, lambda x: k.softmax_dropout(x, bias, seeds, 1, p=0.1)),
    }


NAMES = ["cast", "silu", "row sum", "column sum", "softmax", "softmax ragged", "layer norm", "residual", "norm backward",
         "norm backward, weight", "batch norm", "batch norm backward", "batch norm nchw", "transpose",
         "softmax ragged, masked", "layer norm ragged", "norm backward ragged", "softmax as vectors, masked", "layer norm as vectors",
         "norm backward as vectors", "transpose ragged", "dropout norm", "softmax dropout",
         "batch norm backward, sums"]
KERNELS = {"softmax ragged, masked": b"b200_softmax [elements in registers]", "layer norm ragged": b"b200_norm_fwd [elements in registers]",
           "softmax as vectors, masked": b"b200_softmax [off-grid rows as vectors", "layer norm as vectors": b"b200_norm_fwd [off-grid rows as vectors]",
           "norm backward ragged": b"b200_norm_bwd finalize", "norm backward as vectors": b"b200_norm_bwd finalize", "transpose ragged": b"b200_transpose_copy [ragged 16-bit tiles]"}


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
    if name in KERNELS:
        from better_benchmark_b200 import native
        assert KERNELS[name] in native.load().b200_last_kernel(), native.load().b200_last_kernel()
    x = torch.empty_like(sources[0])
    side, main = torch.cuda.Stream(), torch.cuda.current_stream()
    got = []
    for i in range(48):   # a device copy, a kernel, both, or a kernel of another stream, and the call right behind it
        new = sources[i // 4 % 4]
        if i % 4 == 0:
            x.copy_(new)
        elif i % 4 == 1:
            torch.add(new, 0, out=x)
        elif i % 4 == 2:
            x.zero_()
            torch.mul(new, 1, out=x)
        else:   # an event wait lies between what wrote x and the call
            x.zero_()
            side.wait_stream(main)
            with torch.cuda.stream(side):
                torch.add(new, 0, out=x)
            main.wait_stream(side)
        got.append(_list(call(x)))
    torch.cuda.synchronize()
    for i, out in enumerate(got):
        for a, b in zip(out, want[i // 4 % 4]):
            assert torch.equal(a, b), f"{name}, call {i}"


@pytest.mark.parametrize("channels", [64, 768])
def test_results_of_one_call_read_by_the_next(channels):
    """The statistics of a backward without dx are written by its last kernel, and read by the call right behind it."""
    import better_benchmark_b200.kernels as k
    g = torch.Generator(device="cuda").manual_seed(9)
    images = [torch.randn((16, channels, 14, 14), generator=g, device="cuda").to(torch.bfloat16).contiguous(memory_format=torch.channels_last)
              for _ in range(5)]
    dy = images.pop()
    mean, invstd = torch.full((channels,), 0.1, device="cuda"), torch.full((channels,), 0.7, device="cuda")
    row = torch.randn((300, channels), generator=g, device="cuda")
    readers = {
        "cast": lambda dw, db: k.cast_scale(dw, torch.bfloat16),
        "row": lambda dw, db: k.row_reduce(db.view(1, -1), "sum"),
        "weight": lambda dw, db: k.norm_fwd(row, dw, db, eps=1e-5)[0],
        "batch norm": lambda dw, db: k.batch_norm_bwd(dy, images[0], mean, invstd, dw)[0],
    }
    for name, reader in readers.items():
        want = []
        for x in images:
            _, dw, db = k.batch_norm_bwd(dy, x, mean, invstd, None, want_dx=False)
            torch.cuda.synchronize()
            want.append(reader(dw, db))
            torch.cuda.synchronize()
        got = []
        for i in range(32):
            _, dw, db = k.batch_norm_bwd(dy, images[i % 4], mean, invstd, None, want_dx=False)
            got.append(reader(dw, db))
        torch.cuda.synchronize()
        for i, out in enumerate(got):
            assert torch.equal(out, want[i % 4]), f"{name}, call {i}"


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
