"""GPU parity at the edges of the kernels' ranges: row lengths and starts off the vector grid, ends of
tiles and groups, the smallest and largest sizes a variant takes.

Tolerances: a 16-bit result may differ from the fp64 value by half a step of its type (2^-8 of the value
for bf16, 2^-11 for fp16) plus what the fp32 arithmetic before it loses; fp32 results by a few fp32 ulps
(2^-23) times the length of the summation tree, far below the bounds used here.
"""
import pytest
import torch

pytestmark = pytest.mark.gpu

STEP = {torch.float32: 2.0 ** -21, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}


def _kernels():
    import better_benchmark_b200.kernels as k
    return k


def _randn(shape, dtype, seed, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(shape, generator=g) * scale).to(dtype).cuda()


def _near(got, want64, what, floor=1e-6):
    """|got - want| within half a step of got's type (a whole one for fp32 rounding before it) of the value."""
    err = (got.double() - want64).abs()
    bound = STEP[got.dtype] * want64.abs() + floor
    worst = (err - bound).max().item()
    assert worst <= 0, f"{what}: beyond the bound by {worst:.3e}"


@pytest.mark.parametrize("log", [False, True])
@pytest.mark.parametrize("dtype,out", [(torch.bfloat16, torch.float32), (torch.bfloat16, torch.bfloat16),
                                       (torch.float16, torch.float32), (torch.float32, torch.float32),
                                       (torch.float32, torch.float16)])
@pytest.mark.parametrize("rows,n,stride", [(3, 257, 257), (5, 1003, 1005), (2, 4097, 4099), (2, 32769, 32771),
                                           (300, 8195, 8195), (1, 131075, 131075)])
def test_softmax_rows_of_any_alignment(rows, n, stride, dtype, out, log):
    """The row held in registers, one CTA or a cluster per row: consecutive rows start on every residue
    of the 16-byte grid, and so do their outputs."""
    base = _randn((rows, stride), dtype, n, 3.0)
    x = base[:, stride - n:]
    got = _kernels().softmax(x, log=log, out_dtype=out)
    d = x.double()
    want = torch.log_softmax(d, -1) if log else torch.softmax(d, -1)
    _near(got, want, f"softmax {rows}x{n} {dtype}->{out} log={log}", floor=2e-6 if log else 1e-7)


@pytest.mark.parametrize("scale", [None, 0.125])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("keys", [1, 31, 33, 65, 255, 257, 511, 513, 1201, 8191])
def test_masked_softmax_of_ragged_rows(keys, dtype, scale):
    x, keep = _randn((2, 3, 5, keys), dtype, keys, 2.0), torch.rand(2, 1, 1, keys, device="cuda") < 0.8
    keep[..., 0] = True
    mask = torch.where(keep, 0.0, -10000.0).to(dtype)
    got = _kernels().softmax(x, mask=mask, scale=scale)
    _near(got, torch.softmax(x.double() * (scale or 1.0) + mask.double(), -1), f"masked softmax {keys} {dtype}", floor=1e-7)


def _layer_norm64(d, w, b, eps, rms):
    c = d if rms else d - d.mean(-1, keepdim=True)
    y = c * torch.rsqrt(c.square().mean(-1, keepdim=True) + eps) * w.double()
    return y if b is None else y + b.double()


@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,n", [(3, 2), (9, 33), (7, 65), (10, 129), (5, 257), (3, 511), (3, 513), (2, 8191),
                                    (2, 8193), (2, 16383), (2, 16385), (1300, 257), (1185, 511), (400, 513), (297, 2047), (3, 2049)])
def test_norm_fwd_of_ragged_rows(rows, n, dtype, rms):
    x, w, b = _randn((rows, n), dtype, n), _randn((n,), dtype, n + 1), None if rms else _randn((n,), dtype, n + 2)
    y = _kernels().norm_fwd(x, w, b, eps=1e-5, rms=rms)[0]
    _near(y, _layer_norm64(x.double(), w, b, 1e-5, rms), f"norm {rows}x{n} {dtype} rms={rms}", floor=2e-5)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("rows,n", [(1, 264), (9, 512), (1, 520), (13, 520), (4000, 768), (11, 776), (3, 1024), (5, 449), (3, 1023),
                                    (1184, 512), (1185, 512), (16384, 1024), (16385, 1024)])  # the last of one kernel, the first of the other
def test_residual_layer_norm_forms(rows, n, dtype):
    """A warp per row with its own copy ring (65..128 vectors), and ragged rows: the element-wise choice
    between the two forms is bit for bit a choice between the two single forms."""
    k = _kernels()
    x, r = _randn((rows, n), dtype, n, 2.0), _randn((rows, n), dtype, n + 1)
    w, b = _randn((n,), dtype, n + 2, 2.0), _randn((n,), dtype, n + 3)
    kw = dict(eps=1e-6, residual=r, want_sum=True, want_mean=True, want_rstd=True)
    full, mean, rstd, _, total = k.norm_fwd(x, w, b, **kw)
    rounded = k.norm_fwd(x, w, b, round_sum=True, **kw)[0]
    both, mean2, rstd2, _, total2 = k.norm_fwd(x, w, b, round_sum="both", **kw)
    s = x.float() + r.float()
    assert torch.equal(total, s.to(dtype)) and torch.equal(total2, total)
    assert torch.equal(mean, mean2) and torch.equal(rstd, rstd2)
    assert torch.equal(both, torch.where(full.float().abs() > 3, full, rounded))
    _near(full, _layer_norm64(x.double() + r.double(), w, b, 1e-6, False), f"fp32 form {rows}x{n} {dtype}", floor=4e-5)
    _near(rounded, _layer_norm64(s.to(dtype).double(), w, b, 1e-6, False), f"rounded form {rows}x{n} {dtype}", floor=4e-5)


@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("rows,n", [(1, 3), (7, 129), (600, 257), (9, 511), (700, 513), (5, 4095),   # ragged rows
                                    (600, 132), (40, 520), (5000, 264), (3, 4104),                   # last unit of columns half full
                                    (7, 4104), (150, 8196), (3, 8200), (2, 12040)])                  # units of 16 to 64 columns
def test_norm_bwd_edges(rows, n, dtype, rms):
    x, dy, w = _randn((rows, n), dtype, n), _randn((rows, n), dtype, n + 1), _randn((n,), torch.float32, n + 2)
    d, g = x.double(), dy.double() * w.double()
    mean = None if rms else x.float().mean(-1)
    c = d if rms else d - mean.double()[:, None]
    rstd = torch.rsqrt(c.square().mean(-1) + 1e-5).float()
    dx, dw, db = _kernels().norm_bwd(x, dy, w, rstd, mean=mean, rms=rms, want_dbias=not rms)
    xhat = c * rstd.double()[:, None]
    want = g - xhat * (g * xhat).mean(-1, keepdim=True)
    if not rms:
        want = want - g.mean(-1, keepdim=True)
    want = want * rstd.double()[:, None]
    scale = want.abs().max().item()
    _near(dx, want, f"dx {rows}x{n} {dtype}", floor=4e-6 * max(scale, 1.0))
    # fp32 chains per thread, fp64 above them: a few fp32 ulps of the largest partial sum
    floor = 2.0 ** -21 * max(1.0, rows ** 0.5) * 8
    _near(dw, (dy.double() * xhat).sum(0), f"dweight {rows}x{n}", floor=floor)
    if not rms:
        _near(db, dy.double().sum(0), f"dbias {rows}x{n}", floor=floor)
        alone = _kernels().norm_bwd(x, dy, w, rstd, mean=mean, rms=False, want_dweight=False, want_dbias=True)
        assert alone[1] is None and torch.equal(alone[2], db) and torch.equal(alone[0], dx)


@pytest.mark.parametrize("batch,rows,cols", [(1, 2, 2), (7, 49, 128), (5, 196, 64), (33, 3, 10), (2000, 5, 6), (9, 64, 66),
                                             (3, 129, 126), (2, 16, 1024), (2, 63, 65), (3, 65, 63), (2, 500, 333),
                                             (2, 501, 768), (1, 1, 300), (2, 300, 1), (1300, 33, 64),
                                             (3, 2, 1024), (4001, 2, 6), (700, 4, 64), (9, 8, 1000), (50, 16, 130), (5000, 6, 34),
                                             (2500, 12, 100), (4, 1024, 8), (1200, 32, 48)])   # even row counts: walks that start apart
def test_transpose_of_ragged_16_bit_matrices(batch, rows, cols):
    """Groups of small matrices (a last group that ends between two 16-byte boundaries among them) and
    64 x 64 tiles with ragged ends on either side; a view that starts off the 4-byte grid."""
    k = _kernels()
    x = _randn((batch, rows, cols), torch.float16, rows)
    assert torch.equal(k.permute_copy(x, (0, 2, 1)), x.transpose(1, 2).contiguous())
    flat = _randn((batch * rows * cols + 1,), torch.bfloat16, cols)
    y = flat[1:].view(batch, rows, cols)
    assert torch.equal(k.permute_copy(y, (0, 2, 1)), y.transpose(1, 2).contiguous())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_silu_over_the_whole_range(dtype):
    """Every 16-bit pattern against fp64: finite values down to the type's lowest (where the result is -0), infinities and NaN."""
    x = torch.arange(-32768, 32768, dtype=torch.int32).to(torch.int16).cuda().view(dtype)
    got = _kernels().cast_scale(x, dtype, activation="silu")
    want = (x.double() * torch.sigmoid(x.double()))
    finite = torch.isfinite(x)
    _near(got[finite], want[finite], f"silu {dtype}", floor=1.2e-7 if dtype == torch.float16 else 1e-34)
    assert torch.isnan(got[torch.isnan(x) | (x == float("-inf"))]).all()
    assert torch.equal(got[x == float("inf")], x[x == float("inf")])


@pytest.mark.parametrize("out", [torch.bfloat16, torch.float16])
def test_silu_where_the_exponential_overflows(out):
    """fp32 inputs around -88.72, where exp(-x) leaves fp32, and far below: -0 as x / inf gives it, never x times a residue."""
    x = torch.cat([torch.linspace(-90.0, -87.0, 4096), -torch.logspace(2, 38, 4096)]).cuda()
    got = _kernels().cast_scale(x, out, activation="silu")
    _near(got, x.double() * torch.sigmoid(x.double()), f"silu f32 -> {out}", floor=6e-8 if out == torch.float16 else 3e-37)
    assert (got[x < -89] == 0).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("n,c,hw", [(8, 64, 49), (8, 257, 64), (16, 511, 16), (8, 1022, 16), (33, 24, 7), (64, 100, 196),
                                    (1001, 92, 196), (64, 511, 512), (1, 24, 2),   # copy rings from one chunk to many
                                     (16, 2040, 49), (8, 2044, 49)])   # many channels in a small tensor: the flat kernels
def test_batch_norm_channels_last_of_any_channel_count(n, c, hw, dtype):
    """Channel patterns of up to 512 vectors, tensors of one chunk and of several per CTA, forward and
    backward against fp64."""
    k = _kernels()
    x = _randn((n, c, hw, 1), dtype, c, 2.0).contiguous(memory_format=torch.channels_last)
    dy = _randn((n, c, hw, 1), dtype, c + 1).contiguous(memory_format=torch.channels_last)
    act = _randn((n, c, hw, 1), dtype, c + 2).contiguous(memory_format=torch.channels_last)
    w, b = _randn((c,), torch.float32, c + 3), _randn((c,), torch.float32, c + 4)
    col = lambda t: t.double().view(1, c, 1, 1)  # noqa: E731
    d = x.double()
    mean64, var64 = d.mean((0, 2, 3)), d.var((0, 2, 3), unbiased=False)
    y, mean, invstd = k.batch_norm_fwd(x, w, b, None, None, eps=1e-5, momentum=0.1, relu=True)
    _near(mean, mean64, "mean", floor=2e-6)
    _near(invstd, torch.rsqrt(var64 + 1e-5), "invstd", floor=2e-6)
    _near(y, torch.relu((d - col(mean64)) * col(torch.rsqrt(var64 + 1e-5)) * col(w) + col(b)), f"y {n}x{c}x{hw}", floor=2e-5)
    for a in (None, act):
        dx, dw, db = k.batch_norm_bwd(dy, x, mean, invstd, w, act=a, slope=0.25)
        g = dy.double() if a is None else torch.where(a > 0, dy, dy * 0.25).double()
        xhat = (d - col(mean)) * col(invstd)
        s1, s2 = g.sum((0, 2, 3)), (g * xhat).sum((0, 2, 3))
        floor = 2.0 ** -21 * (n * hw) ** 0.5 * 8   # fp32 chains per thread, fp64 above them
        _near(db, s1, "dbias", floor=floor)
        _near(dw, s2, "dweight", floor=floor)
        want = (g - col(s1) / (n * hw) - xhat * col(s2) / (n * hw)) * col(w) * col(invstd)
        _near(dx, want, f"dx {n}x{c}x{hw}", floor=1e-5)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gelu_over_the_whole_range(dtype):
    """Every 16-bit pattern against x * erfc(-x / sqrt 2) / 2 in fp64; -inf and NaN give NaN, as
    (x / 2) * (erf(x / sqrt 2) + 1) does, +inf itself."""
    x = torch.arange(-32768, 32768, dtype=torch.int32).to(torch.int16).cuda().view(dtype)
    got = _kernels().cast_scale(x, dtype, activation="gelu_erf")
    d = x.double()
    want = 0.5 * d * torch.special.erfc(-d * 0.5 ** 0.5)
    finite = torch.isfinite(x)
    _near(got[finite], want[finite], f"gelu {dtype}", floor=6e-8 if dtype == torch.float16 else 1e-35)
    assert torch.isnan(got[torch.isnan(x) | (x == float("-inf"))]).all()
    assert torch.equal(got[x == float("inf")], x[x == float("inf")])


@pytest.mark.parametrize("activation", ["silu", "gelu_erf"])
@pytest.mark.parametrize("dtype,out", [(torch.bfloat16, torch.bfloat16), (torch.float16, torch.float16),
                                       (torch.float32, torch.bfloat16), (torch.float32, torch.float16)])
def test_activations_do_not_depend_on_position_or_alignment(dtype, out, activation):
    """Vectors, a tail behind the last whole vector, and a view off the 16-byte grid give the same bits."""
    bits = torch.arange(-32768, 32768, dtype=torch.int32).to(torch.int16).cuda()
    x = bits.view(dtype) if dtype != torch.float32 else bits.view(torch.bfloat16).float()
    run = lambda t: _kernels().cast_scale(t, out, activation=activation).view(torch.int16)  # noqa: E731
    want = run(x)
    shifted = torch.cat([x[:1], x])[1:]
    assert torch.equal(run(shifted), want)
    for start in (0, 32768 - 11, 65536 - 1024):   # every length modulo a vector
        for n in range(1, 20):
            assert torch.equal(run(x[start:].clone()[:n]), want[start:start + n]), (start, n)


@pytest.mark.parametrize("dtype,out", [(torch.bfloat16, torch.float32), (torch.float32, torch.float16), (torch.float16, torch.float16),
                                       (torch.float32, torch.float32)])
@pytest.mark.parametrize("activation", [None, "relu", "silu"])
def test_casts_on_both_sides_of_the_32_byte_path(dtype, out, activation):
    """Lengths around its smallest size (4096 units) with every kind of rest, starts on 32-, 16- and 2- or 4-byte boundaries."""
    unit = 32 // dtype.itemsize
    x = _randn((400000,), dtype, 3, 2.0)
    for n in (4096 * unit - 1, 4096 * unit, 4096 * unit + 1, 4099 * unit - 1, 399000):
        for start in (0, unit // 2, 1):
            t = x[start:start + n]
            got = _kernels().cast_scale(t, out, activation=activation)
            if activation == "silu":
                d = t.double()
                _near(got, d * torch.sigmoid(d), f"silu {n} {start}", floor=1.2e-7)
            else:
                assert torch.equal(got, (torch.relu(t) if activation else t).to(out)), (n, start)


@pytest.mark.parametrize("dtype,out", [(torch.bfloat16, torch.float32), (torch.float16, torch.float32), (torch.float32, torch.float32),
                                       (torch.float32, torch.bfloat16), (torch.float16, torch.float16)])
@pytest.mark.parametrize("mode", [0, 2, 8])
def test_casts_through_the_entry_point_to_results_of_every_alignment(dtype, out, mode):
    """A caller's result may start anywhere on its type's grid: 16 bytes off a 32-byte boundary 8 values widened to fp32
    leave as two stores. The bits are those of the aligned call, and nothing beside the result is written."""
    k = _kernels()
    unit = 32 // dtype.itemsize
    x = _randn((4099 * unit + 64,), dtype, 5, 2.0)
    y = torch.empty(x.numel() + 64, dtype=out, device="cuda")
    assert x.data_ptr() % 256 == 0 and y.data_ptr() % 256 == 0
    activation = {0: None, 2: "relu", 8: "silu"}[mode]
    for n in (0, 1, 8, 77, 1000, 4096 * unit - 1, 4096 * unit, 4099 * unit + 5):
        want = k.cast_scale(x[:n].clone(), out, activation=activation)
        for x_start in (0, unit // 2):
            x[x_start:x_start + n].copy_(x[:n].clone())
            for offset in (0, 4, 8, 16, 20, 32, 48):
                start = offset // y.element_size()
                y.fill_(7.0)
                k.check(k.load().b200_cast_scale(x.data_ptr() + x_start * x.element_size(), y.data_ptr() + offset, n, k._code(x),
                                                 k._DTYPE_CODE[out], 1.0, mode, k._stream()), "b200_cast_scale")
                assert torch.equal(y[start:start + n], want), (n, x_start, offset)
                assert (y[:start] == 7).all() and (y[start + n:] == 7).all(), (n, x_start, offset)


@pytest.mark.parametrize("dtype,n,c,hw", [(torch.bfloat16, 1001, 92, 196), (torch.bfloat16, 336, 92, 196),
                                          (torch.float32, 80, 485, 256), (torch.bfloat16, 64, 1022, 49)])
def test_batch_norm_takes_the_same_path_with_the_advertised_scratch(dtype, n, c, hw):
    """A scratch buffer of exactly the advertised size gives the bits that the larger default buffer gives."""
    from better_benchmark_b200 import native
    k = _kernels()
    x = _randn((n, c, hw, 1), dtype, c).contiguous(memory_format=torch.channels_last)
    w, b = _randn((c,), torch.float32, 1), _randn((c,), torch.float32, 2)
    scratch = torch.zeros(int(native.load().b200_batch_norm_scratch_bytes(c)), dtype=torch.uint8, device="cuda")
    want = k.batch_norm_fwd(x, w, b, None, None, eps=1e-5, momentum=0.1)
    path = native.load().b200_last_kernel()
    got = k.batch_norm_fwd(x, w, b, None, None, eps=1e-5, momentum=0.1, scratch=scratch)
    assert native.load().b200_last_kernel() == path
    for g, v in zip(got, want):
        assert torch.equal(g, v)


def test_threads_launch_one_kernel_with_different_shared_memory_sizes():
    """Host threads, each on its own stream, call one instantiation with rings of different sizes through the C ABI:
    a limit set for one launch must not reject another's."""
    import threading
    from better_benchmark_b200 import kernels, native
    lib = native.load()
    failures = []

    def work(x):
        y = torch.empty(x.shape[0], x.shape[2], x.shape[1], dtype=x.dtype, device="cuda")
        b, r, c = x.shape
        with torch.cuda.stream(torch.cuda.Stream()):
            args = (x.data_ptr(), y.data_ptr(), b, r, c, r * c, c, kernels._code(x), kernels._code(x), 1.0, 0,
                    torch.cuda.current_stream().cuda_stream)
            for _ in range(20000):
                if lib.b200_transpose_copy(*args) != 0:
                    failures.append(native.last_error())
                    return
            torch.cuda.current_stream().synchronize()
        if not torch.equal(y, x.transpose(1, 2)):
            failures.append("wrong values")

    # odd row counts: one instantiation, rings of 49 KB and 94 KB
    inputs = [_randn(shape, torch.bfloat16, shape[1]) for shape in [(8, 49, 128), (4, 201, 80)] * 2]
    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(x,)) for x in inputs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures


def test_threads_ask_for_occupancies_at_the_same_time():
    """First calls of many kernel / block-size pairs from several host threads (each with its own stream and
    scratch) give the bits that the same calls give afterwards, one by one."""
    import threading
    k = _kernels()
    sizes = [list(range(600 + 40 * t, 3400, 173)) for t in range(4)]
    data = {n: (_randn((7, n), torch.float16, n), _randn((7, n), torch.float16, n + 1), _randn((n,), torch.float32, n))
            for group in sizes for n in group}
    rstd = torch.ones(7, device="cuda")
    torch.cuda.synchronize()
    results, start = {}, threading.Barrier(len(sizes))

    def work(group):
        with torch.cuda.stream(torch.cuda.Stream()):
            scratch = torch.zeros(64 << 20, dtype=torch.uint8, device="cuda")
            start.wait()
            for n in group:
                x, dy, w = data[n]
                results[n] = k.norm_bwd(x, dy, w, rstd, rms=True, scratch=scratch)[:2]
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(group,)) for group in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for n, (x, dy, w) in data.items():
        for got, want in zip(results[n], k.norm_bwd(x, dy, w, rstd, rms=True)[:2]):
            assert torch.equal(got, want), n


def _graph_us(run, calls=10, replays=20):
    """Microseconds of one call: the fastest of many replays of a graph that holds several."""
    run()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(calls):
            run()
    best = float("inf")
    for _ in range(replays):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        graph.replay()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) * 1e3 / calls)
    return best


def _bn_bwd_us(n, c, hw):
    k = _kernels()
    x, dy = (_randn((n, c, hw, 1), torch.bfloat16, s).contiguous(memory_format=torch.channels_last) for s in (1, 2))
    mean, invstd, w = torch.zeros(c, device="cuda"), torch.ones(c, device="cuda"), torch.ones(c, device="cuda")
    return _graph_us(lambda: k.batch_norm_bwd(dy, x, mean, invstd, w))


def test_batch_norm_bwd_costs_the_same_for_an_odd_channel_count():
    """The same bytes with 92 and with 64 channels (12 MB a tensor): 17.6 and 17.1 us. Each thread's 4 x 8
    coefficients have to come from L1; fetched past it they cost 40.5 and 27.4 us."""
    odd, even = _bn_bwd_us(328, 92, 196), _bn_bwd_us(118, 64, 784)
    assert odd < 1.25 * even, (odd, even)


@pytest.mark.parametrize("n,c,hw,rings", [(1, 24, 2, True), (64, 120, 784, True), (8, 1024, 49, True), (8, 2040, 49, False),
                                          (80, 2040, 49, True)])
def test_batch_norm_channels_last_takes_the_faster_kernels(n, c, hw, rings):
    """Copy rings for every size, except for more than 1024 channels in less than 12 MB."""
    k = _kernels()
    x = _randn((n, c, hw, 1), torch.bfloat16, c).contiguous(memory_format=torch.channels_last)
    k.batch_norm_fwd(x, None, None, None, None, eps=1e-5, momentum=0.1)
    assert (b"copy rings" in k.load().b200_last_kernel()) == rings, k.load().b200_last_kernel()


@pytest.mark.parametrize("n,c,hw,dtype", [(2, 1, 2056, torch.float16), (3, 4, 1022, torch.float32), (9, 8, 57345, torch.bfloat16),
                                          (61, 16, 4099, torch.bfloat16), (41, 256, 441, torch.float32),
                                          (340, 64, 196, torch.float16)])
def test_batch_norm_channels_last_of_few_channels_and_power_of_two_counts(n, c, hw, dtype):
    """Many threads share a channel in the fold of the partial sums; power-of-two counts on both sides of 8 MB."""
    k = _kernels()
    x = _randn((n, c, hw, 1), dtype, c, 2.0).contiguous(memory_format=torch.channels_last)
    dy = _randn((n, c, hw, 1), dtype, c + 1).contiguous(memory_format=torch.channels_last)
    w, b = _randn((c,), torch.float32, c + 3), _randn((c,), torch.float32, c + 4)
    col = lambda t: t.double().view(1, c, 1, 1)  # noqa: E731
    d = x.double()
    mean64, var64 = d.mean((0, 2, 3)), d.var((0, 2, 3), unbiased=False)
    y, mean, invstd = k.batch_norm_fwd(x, w, b, None, None, eps=1e-5, momentum=0.1)
    assert c < 4 or b"copy rings" in k.load().b200_last_kernel(), k.load().b200_last_kernel()
    _near(mean, mean64, "mean", floor=2e-6)
    _near(invstd, torch.rsqrt(var64 + 1e-5), "invstd", floor=2e-6)
    _near(y, (d - col(mean64)) * col(torch.rsqrt(var64 + 1e-5)) * col(w) + col(b), f"y {n}x{c}x{hw}", floor=2e-5)
    dx, dw, db = k.batch_norm_bwd(dy, x, mean, invstd, w)
    xhat, floor = (d - col(mean)) * col(invstd), 2.0 ** -21 * (n * hw) ** 0.5 * 8   # as in the test above
    s1, s2 = dy.double().sum((0, 2, 3)), (dy.double() * xhat).sum((0, 2, 3))
    _near(db, s1, "dbias", floor=floor)
    _near(dw, s2, "dweight", floor=floor)
    _near(dx, (dy.double() - col(s1) / (n * hw) - xhat * col(s2) / (n * hw)) * col(w) * col(invstd), f"dx {n}x{c}x{hw}", floor=1e-5)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("c", [64, 92, 256])
@pytest.mark.parametrize("mb", [10, 24, 36])
def test_batch_norm_statistics_with_a_first_row_far_from_the_mean(mb, c, dtype):
    """The sums are shifted by the mean of sixteen rows, not by the first one: here that is five standard deviations off, which
    would multiply the error of invstd. Half an fp32 step (2^-24 of the value) for its rounding and as much for the sums."""
    n = int(mb * 1e6 / dtype.itemsize / c / 49) // 8 * 8
    x = _randn((n, c, 7, 7), torch.float32, mb + c, 2.0).add_(0.5)
    side = torch.arange(c, device="cuda") % 2 * 2.0 - 1.0
    x[0, :, 0, 0] = 0.5 + 2.0 * 5 * side
    x = x.to(dtype).contiguous(memory_format=torch.channels_last)
    ones = torch.ones(c, device="cuda")
    _, mean, invstd = _kernels().batch_norm_fwd(x, ones, ones, None, None, eps=1e-5, momentum=0.1)
    var64, mean64 = torch.var_mean(x.double(), (0, 2, 3), unbiased=False)
    worst = (invstd.double() * torch.sqrt(var64 + 1e-5) - 1).abs().max().item()
    assert worst <= 2.0 ** -23, f"invstd off by {worst:.2e}"
    assert ((mean.double() - mean64) / var64.sqrt()).abs().max().item() <= 2.0 ** -24


@pytest.mark.parametrize("c,mb,dtype", [(8, 300, torch.bfloat16), (64, 300, torch.float32), (1024, 300, torch.bfloat16)])
def test_batch_norm_statistics_of_long_sums(c, mb, dtype):
    """Hundreds of additions per thread, in three levels of fp32 sums below fp64 ones: through the wrapper, and through the entry point
    that brings room for 160 partial rows of 1024 channels. Half an fp32 step for the rounding of a result, as much for the sums."""
    k = _kernels()
    n = int(mb * 1e6 / dtype.itemsize / c / 49) // 8 * 8
    x = _randn((n, c, 7, 7), dtype, c, 2.0).contiguous(memory_format=torch.channels_last)
    ones = torch.ones(c, device="cuda")
    results = [k.batch_norm_fwd(x, ones, ones, None, None, eps=1e-5, momentum=0.1)[1:]]
    y, mean, invstd = torch.empty_like(x), torch.empty(c, device="cuda"), torch.empty(c, device="cuda")
    k.check(k.load().b200_batch_norm_fwd_static_scratch(
        x.data_ptr(), y.data_ptr(), ones.data_ptr(), ones.data_ptr(), None, None, mean.data_ptr(), invstd.data_ptr(), n, c, 49,
        x.stride(0), x.stride(1), x.stride(3), k._code(x), k.F32, 1e-5, 0.1, 0, k._stream()), "b200_batch_norm_fwd_static_scratch")
    results.append((mean, invstd))
    var64, mean64 = torch.var_mean(x.double(), (0, 2, 3), unbiased=False)
    for mean, invstd in results:
        worst = (invstd.double() * torch.sqrt(var64 + 1e-5) - 1).abs().max().item()
        assert worst <= 2.0 ** -23, f"invstd off by {worst:.2e}"
        assert ((mean.double() - mean64) / var64.sqrt()).abs().max().item() <= 2.0 ** -24


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("mb", [4, 10, 60])   # the three kinds of shift
def test_batch_norm_of_channels_whose_rows_add_up_to_more_than_fp32_holds(mb, dtype):
    """Sixteen rows of 3e37 have a finite mean but not a finite sum: mean 3e37 and variance 0 all the same, beside ordinary channels."""
    n = int(mb * 1e6 / dtype.itemsize / 64 / 49) // 8 * 8
    x = _randn((n, 64, 7, 7), dtype, mb, 2.0)
    x[:, 5] = 3e37
    x[:, 63] = -3e37
    x = x.contiguous(memory_format=torch.channels_last)
    ones = torch.ones(64, device="cuda")
    y, mean, invstd = _kernels().batch_norm_fwd(x, ones, ones, None, None, eps=1e-5, momentum=0.1)
    var64, mean64 = torch.var_mean(x.double(), (0, 2, 3), unbiased=False)
    _near(mean, mean64, "mean", floor=2e-6)
    _near(invstd, torch.rsqrt(var64 + 1e-5), "invstd", floor=2e-6)
    assert (y[:, [5, 63]] == 1).all()


@pytest.mark.parametrize("dtype,c", [(torch.bfloat16, 64), (torch.float32, 92), (torch.float16, 320), (torch.bfloat16, 1022)])
@pytest.mark.parametrize("partial_rows", [295, 148, 5, 1])
def test_batch_norm_with_room_for_few_partial_rows(partial_rows, dtype, c):
    """A caller's scratch of less than two partial rows per SM, down to one: the copy rings on fewer, wider CTAs, the statistics as
    close to fp64 as with all of them. Nothing behind the buffer is written."""
    k = _kernels()
    n = int(12e6 / dtype.itemsize / c / 49) // 8 * 8
    x = _randn((n, c, 7, 7), dtype, c, 2.0).contiguous(memory_format=torch.channels_last)
    w, b = _randn((c,), torch.float32, c + 3), _randn((c,), torch.float32, c + 4)
    size = 256 + (partial_rows + 1) * 2 * c * 4
    scratch = torch.full((size + 4096,), 77, dtype=torch.uint8, device="cuda")
    y, mean, invstd = k.batch_norm_fwd(x, w, b, None, None, eps=1e-5, momentum=0.1, scratch=scratch[:size])
    assert b"copy rings" in k.load().b200_last_kernel(), k.load().b200_last_kernel()
    assert (scratch[size:] == 77).all() and (scratch[:256] == 77).all()
    var64, mean64 = torch.var_mean(x.double(), (0, 2, 3), unbiased=False)
    # 2^-24 for the rounding of a result; the longest chains here are of 5000 vectors in one CTA, in three levels of sums
    assert (invstd.double() * torch.sqrt(var64 + 1e-5) - 1).abs().max().item() <= 2.0 ** -22
    assert ((mean.double() - mean64) / var64.sqrt()).abs().max().item() <= 2.0 ** -23
    col = lambda t: t.double().view(1, c, 1, 1)  # noqa: E731
    _near(y, (x.double() - col(mean64)) * col(torch.rsqrt(var64 + 1e-5)) * col(w) + col(b), f"y {partial_rows} rows", floor=2e-5)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_log_softmax_in_fp32_has_no_biased_sum(dtype):
    """Mean error of fp32 log-probabilities over 100 000 rows of 1003. An exponential whose errors have a mean shifts
    every row alike: 2.7e-8 with the pair exponential of 16-bit results, 1.3e-8 with expf (rounding of the logits'
    difference and of the logarithm alone). Rows scatter by 2.4e-7, their mean by 0.8e-9."""
    g = torch.Generator(device="cuda").manual_seed(5)
    total = 0.0
    for _ in range(10):
        x = (torch.randn((10000, 1003), generator=g, device="cuda") * 2).to(dtype)
        got = _kernels().softmax(x, log=True, out_dtype=torch.float32)
        total += (got.double() - torch.log_softmax(x.double(), -1)).mean().item() / 10
    assert abs(total) < 2.1e-8, total


def test_a_few_ragged_rows_cost_what_aligned_ones_do():
    """LayerNorm forward of 148 rows: 449 columns (elements) against 448 (vectors), 3.0 and 4.0 us. One warp per row whose
    16 weights and biases are fetched one after the other took 9.9."""
    k = _kernels()

    def us(n):
        x, w, b = _randn((148, n), torch.bfloat16, 1), _randn((n,), torch.bfloat16, 2), _randn((n,), torch.bfloat16, 3)
        return _graph_us(lambda: k.norm_fwd(x, w, b, eps=1e-5, want_rstd=True))

    ragged, aligned = us(449), us(448)
    assert ragged < 1.5 * aligned, (ragged, aligned)


def test_ragged_norm_bwd_costs_what_aligned_rows_do():
    """LayerNorm backward of 1200 rows: 513 columns (a CTA per row, 1200 partial rows) against 512, 10 us each.
    With the partial rows added up by 9 CTAs it took 32."""
    k = _kernels()

    def us(n):
        x, dy, w = _randn((1200, n), torch.bfloat16, 1), _randn((1200, n), torch.bfloat16, 2), torch.ones(n, device="cuda")
        mean, rstd = torch.zeros(1200, device="cuda"), torch.ones(1200, device="cuda")
        return _graph_us(lambda: k.norm_bwd(x, dy, w, rstd, mean=mean, rms=False, want_dbias=True))

    ragged, aligned = us(513), us(512)
    assert ragged < 1.5 * aligned, (ragged, aligned)


@pytest.mark.parametrize("rows,n,dtype,warp", [(16384, 1024, torch.bfloat16, True), (16385, 1024, torch.bfloat16, False),
                                               (40000, 896, torch.float16, True), (1184, 512, torch.float32, True),
                                               (1185, 512, torch.float32, False)])
def test_residual_layer_norm_takes_the_faster_kernel(rows, n, dtype, warp):
    k = _kernels()
    x, w = torch.zeros((rows, n), dtype=dtype, device="cuda"), torch.ones(n, dtype=dtype, device="cuda")
    k.norm_fwd(x, w, w, eps=1e-5, residual=x)
    assert (b"warp rings" in k.load().b200_last_kernel()) == warp, k.load().b200_last_kernel()


@pytest.mark.parametrize("heads", [1, 60])   # 10 rows: a CTA per row up to 2048 keys; 600: a warp per row up to 512
@pytest.mark.parametrize("keys", [66, 127, 129, 255, 257, 511, 513, 2047, 2049])
def test_masked_softmax_few_and_many_ragged_rows(keys, heads):
    x, keep = _randn((2, heads, 5, keys), torch.bfloat16, keys, 2.0), torch.rand(2, 1, 1, keys, device="cuda") < 0.8
    keep[..., 0] = True
    mask = torch.where(keep, 0.0, -10000.0).to(torch.bfloat16)
    for rounded in (False, True):
        got = _kernels().softmax(x, mask=mask, scale=0.3, round_intermediates=rounded)
        t = (x * torch.tensor(0.3, dtype=torch.float32)).to(x.dtype) + mask if rounded else x.double() * 0.30000001192092896 + mask.double()
        _near(got, torch.softmax(t.double(), -1), f"masked softmax {heads}x{keys} rounded={rounded}", floor=1e-7)


def test_a_few_ragged_softmax_rows_cost_what_aligned_ones_do():
    """Masked softmax of 8 rows of 511 and of 512 keys, 2.3 and 3.1 us. One warp per row that waited for each load before
    the next took 5.9."""
    k = _kernels()

    def us(n):
        x, m = _randn((1, 8, 1, n), torch.float16, 1), torch.zeros((1, 1, 1, n), dtype=torch.float16, device="cuda")
        return _graph_us(lambda: k.softmax(x, mask=m, scale=0.125))

    ragged, aligned = us(511), us(512)
    assert ragged < 1.25 * aligned, (ragged, aligned)


def test_transposes_of_two_rows_cost_what_the_bytes_cost():
    """The same 30 MB as [14648, 2, 1024] and [7324, 4, 1024] in 16 bits: 25 and 28 us. Two rows took 48 with a walk of
    one step and its index arithmetic per column pair."""
    k = _kernels()
    two, four = (_graph_us(lambda x=_randn(shape, torch.bfloat16, 1): k.permute_copy(x, (0, 2, 1)))
                 for shape in [(14648, 2, 1024), (7324, 4, 1024)])
    assert two < 1.2 * four, (two, four)


@pytest.mark.parametrize("rows,n", [(20000, 64), (9000, 256), (20000, 129), (9000, 513), (9000, 768), (4000, 2052), (2000, 4096)])
def test_norm_bwd_takes_its_largest_grid_with_the_advertised_scratch(rows, n):
    """Exactly the advertised bytes give the bits that the larger default buffer gives, and they are what two planes of
    partial rows take."""
    from better_benchmark_b200 import native
    lib = native.load()
    x, dy, w = _randn((rows, n), torch.float32, n), _randn((rows, n), torch.float32, n + 1), torch.ones(n, device="cuda")
    mean, rstd = torch.zeros(rows, device="cuda"), torch.ones(rows, device="cuda")
    size = int(lib.b200_norm_bwd_scratch_bytes(n))
    assert size <= 256 + 2 * (64 if n <= 256 else 8) * lib.b200_sm_count() * n * 4
    kw = dict(mean=mean, rms=False, want_dbias=True)
    want = _kernels().norm_bwd(x, dy, w, rstd, **kw)
    got = _kernels().norm_bwd(x, dy, w, rstd, scratch=torch.zeros(size, dtype=torch.uint8, device="cuda"), **kw)
    assert all(torch.equal(g, v) for g, v in zip(got, want))


@pytest.mark.parametrize("log", [False, True])
def test_masked_softmax_beyond_the_registers(log):
    """More than 8192 keys off the vector grid: the three sweeps."""
    k = _kernels()
    x, keep = _randn((2, 1, 3, 9001), torch.float16, 3, 2.0), torch.rand(2, 1, 1, 9001, device="cuda") < 0.8
    keep[..., 0] = True
    mask = torch.where(keep, 0.0, -10000.0).to(torch.float16)
    got = k.softmax(x, mask=mask, scale=0.5, log=log)
    assert b"three passes" in k.load().b200_last_kernel()
    t = x.double() * 0.5 + mask.double()
    _near(got, torch.log_softmax(t, -1) if log else torch.softmax(t, -1), "9001 keys", floor=2e-6 if log else 1e-7)


@pytest.mark.parametrize("dtype,n", [(torch.bfloat16, 40003), (torch.float32, 5001)])
def test_softmax_rows_over_strided_outer_dimensions(dtype, n):
    """Three outer dimensions that do not collapse, rows on every alignment: a CTA and a cluster per row."""
    base = _randn((2, 3, 5, 4, n + 1), dtype, 5, 2.0)
    for x in (base[:, ::2, 1:4, :, :n], base[:, :, ::2, 1:3, 1:]):
        for rows in (x, x[:, :, :, :, :3001]):
            got = _kernels().softmax(rows)
            _near(got, torch.softmax(rows.double(), -1), f"strided softmax {tuple(rows.shape)}", floor=1e-7)


@pytest.mark.parametrize("dtype,out", [(torch.bfloat16, torch.float32), (torch.float16, torch.float16), (torch.float32, torch.bfloat16)])
@pytest.mark.parametrize("n", [1003, 20483, 30001])   # one CTA a row, and on both sides of two (16-bit rows to fp32 logs)
def test_softmax_rows_with_infinite_logits(n, dtype, out):
    """-inf among finite logits has probability 0 and log-probability -inf; the other elements are as if it were not there."""
    x = _randn((6, n), dtype, n, 2.0)
    x[1, 3:200] = float("-inf")
    x[2, 1:] = float("-inf")
    x[3, :n // 2] = float("-inf")
    x[4, n - 1] = float("nan")
    x[5] = float("-inf")
    d = x.double()
    for scale in (None, 0.5):
        for log in (False, True):
            got = _kernels().softmax(x, log=log, out_dtype=out, scale=scale)
            t = d if scale is None else d * scale
            want = torch.log_softmax(t, -1) if log else torch.softmax(t, -1)
            assert torch.isnan(got[4:]).all()
            g, w = got[:4], want[:4]
            assert torch.equal(torch.isinf(g), torch.isinf(w)) and not torch.isnan(g).any()
            finite = torch.isfinite(w)
            _near(g[finite], w[finite], f"softmax with -inf, {n} log={log} scale={scale}", floor=2e-6 if log else 1.2e-7)


@pytest.mark.parametrize("dtype,out", [(torch.float32, torch.bfloat16), (torch.bfloat16, torch.bfloat16), (torch.float32, torch.float32),
                                       (torch.bfloat16, torch.float32), (torch.float32, torch.float16)])
@pytest.mark.parametrize("n", [1003, 20483, 30001, 70001])
def test_softmax_rows_with_logits_as_low_as_the_type_goes(n, dtype, out):
    """Finite differences whose product with log2(e) is not: probability 0, whatever the exponential makes of them on the way."""
    x = _randn((5, n), dtype, n, 2.0)
    x[0, 3:200] = -3e38
    x[1, 1:] = -3e38
    x[2, ::3] = -2.4e38
    x[2, 0] = 1e38          # the difference itself overflows
    x[3] = -3e38            # all alike: 1 / n
    x[4, :n // 2] = -1e30
    d = x.double()
    for scale in (None, 0.5):
        t = d if scale is None else d * scale
        _near(_kernels().softmax(x, out_dtype=out, scale=scale), torch.softmax(t, -1), f"low logits {n} {scale}", floor=1.2e-7)
        if out != torch.float16:
            got, want = _kernels().softmax(x, log=True, out_dtype=out, scale=scale), torch.log_softmax(t, -1)
            inside = want > -3.38e38
            _near(got[inside], want[inside], f"low logits, log {n} {scale}", floor=2e-6)
            assert (got[~inside] <= -3.38e38).all()


@pytest.mark.parametrize("mask_shape", [(1, 1, 1), (4, 1, 1), (1, 3, 1), (1, 1, 5), (4, 1, 5), (4, 3, 1), (1, 3, 5), (4, 3, 5)])
@pytest.mark.parametrize("n", [64, 100, 1000])
def test_softmax_of_every_broadcast_mask_and_outer_order(n, mask_shape):
    """Rows at one distance take a flat map beside operands that need several dimensions: x contiguous, with gaps in each
    outer dimension, and with its outer dimensions in another order; every row has the bits of the expanded call."""
    k = _kernels()
    m = _randn((*mask_shape, n), torch.float16, n)
    big = _randn((8, 6, 10, n), torch.float16, n + 1, 2.0)
    forms = (big[:4, :3, :5].contiguous(), big[::2, :3, :5], big[:4, ::2, :5], big[:4, :3, ::2],
             big[:5, :3, :4].permute(2, 1, 0, 3), big[:3, :4, :5].permute(1, 0, 2, 3))
    for x in forms:
        want = k.softmax(x.contiguous().view(60, n), mask=m.expand(4, 3, 5, n).contiguous().view(60, n), scale=0.5)
        assert torch.equal(k.softmax(x, mask=m, scale=0.5).reshape(60, n), want), (mask_shape, x.stride())
        assert torch.equal(k.row_reduce(x, "sum").reshape(60), k.row_reduce(x.contiguous().view(60, n), "sum"))


def test_transpose_of_small_matrices_with_gaps_between_them():
    """The batch stride is not rows * columns: one matrix per block."""
    k = _kernels()
    for dtype, rows, take, cols in ((torch.bfloat16, 60, 49, 128), (torch.float16, 10, 4, 96), (torch.bfloat16, 8, 2, 48)):
        x = _randn((37, rows, cols), dtype, rows)[:, :take]
        assert torch.equal(k.permute_copy(x, (0, 2, 1)), x.transpose(1, 2).contiguous())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_residual_layer_norm_of_strided_and_of_special_rows(dtype):
    """Padded rows through the warp kernel's copies; NaN and infinities stay in their rows."""
    k = _kernels()
    n = 768 if dtype == torch.bfloat16 else 384
    base, other = _randn((50, n + 32), dtype, 1, 2.0), _randn((50, n + 32), dtype, 2)
    base[7, 3], base[8, n - 1], other[9, 0] = float("nan"), float("inf"), float("-inf")
    x, r, w, b = base[:, :n], other[:, :n], _randn((n,), dtype, 3), _randn((n,), dtype, 4)
    for form in (False, True, "both"):
        y, total = [k.norm_fwd(x, w, b, eps=1e-6, residual=r, want_sum=True, round_sum=form)[i] for i in (0, 4)]
        assert b"warp rings" in k.load().b200_last_kernel()
        assert torch.equal(total.view(50, n)[:7], (x.float() + r.float()).to(dtype)[:7])
        assert torch.isnan(y[7:10]).all() and torch.isfinite(y[:7]).all() and torch.isfinite(y[10:]).all()
        if form is False:
            rest = torch.cat([torch.arange(7), torch.arange(10, 50)]).cuda()
            _near(y[rest], _layer_norm64((x.double() + r.double())[rest], w, b, 1e-6, False), "strided residual", floor=4e-5)
