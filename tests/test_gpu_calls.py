"""The native host side of the wrappers (csrc/calls.cpp) against the Python code that takes every other form: the same results, shapes, strides
and dtypes over layouts, dtypes and options, the same errors, and the same behaviour with threads, streams, modes and graphs."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu

F32, BF16, F16 = torch.float32, torch.bfloat16, torch.float16


class _Nothing:
    """Every call is left to the Python code."""

    def __getattr__(self, name):
        return lambda *args: None


class _Counting:
    def __init__(self, calls):
        self.calls, self.taken, self.left = calls, 0, 0

    def __getattr__(self, name):
        def call(*args):
            got = getattr(self.calls, name)(*args)
            if got is None:
                self.left += 1
            else:
                self.taken += 1
            return got
        return call


def _flat(result):
    if result is None or isinstance(result, torch.Tensor):
        return [result]
    return [t for r in result for t in _flat(r)]


def _outcome(call):
    try:
        return _flat(call())
    except Exception as e:  # noqa: BLE001  (the type and the text are compared)
        return type(e), str(e)


def _compare(monkeypatch, call, native=None):
    """`native`: whether the native code is to take the call (None: either)."""
    from better_benchmark_b200 import kernels as k
    calls = k._calls or k._load_calls()
    counting = _Counting(calls)
    monkeypatch.setattr(k, "_calls", counting)
    got = _outcome(call)
    monkeypatch.setattr(k, "_calls", _Nothing())
    want = _outcome(call)
    monkeypatch.setattr(k, "_calls", calls)
    if native is not None:
        assert (counting.taken > 0) == native
    if isinstance(want, tuple):
        assert got == want
        return
    assert isinstance(got, list) and len(got) == len(want), got
    for a, b in zip(got, want):
        if b is None:
            assert a is None
            continue
        assert (a.shape, a.stride(), a.dtype, a.device, a.requires_grad) == (b.shape, b.stride(), b.dtype, b.device, b.requires_grad)
        assert torch.allclose(a, b, rtol=0, atol=0, equal_nan=True)


def _t(*shape, dtype=F32, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    return torch.randn(*shape, generator=g, device="cuda").to(dtype)


@pytest.mark.parametrize("dtype", [F32, BF16, F16], ids=str)
def test_row_reduce_softmax_cast(monkeypatch, dtype):
    from better_benchmark_b200 import kernels as k
    forms = [_t(5, 33, dtype=dtype), _t(2, 3, 4, 40, dtype=dtype), _t(7, dtype=dtype), _t(6, 50, dtype=dtype)[:, :47],
             _t(2, 4, 3, 16, dtype=dtype).transpose(1, 2), _t(4, 6, dtype=dtype).t(), _t(2, 3, 4, 5, 6, 2, 2, 8, dtype=dtype),
             _t(2, 2, 2, 2, 2, 2, 2, 2, 4, dtype=dtype), _t(2, 3, 4, 8, dtype=dtype)[:, ::2, ::2], _t(0, 4, dtype=dtype), _t(4, 0, dtype=dtype),
             _t(3, 1, dtype=dtype), _t(1, 1, 9, dtype=dtype).expand(4, 2, 9), _t(3, 8, 4, 4, dtype=dtype).to(memory_format=torch.channels_last),
             torch.tensor(1.5, device="cuda", dtype=dtype), _t(3, 5, dtype=dtype).requires_grad_(), torch.nn.Parameter(_t(3, 5, dtype=dtype))]
    for x in forms:
        for op in ("sum", "mean", "amax", "none"):
            for options in ({}, dict(keepdim=True), dict(out_dtype=F32), dict(out_dtype=torch.int32), dict(keepdim=1)):
                _compare(monkeypatch, lambda: k.row_reduce(x, op, **options))
        for options in ({}, dict(log=True), dict(scale=0.125), dict(scale=2), dict(out_dtype=F32), dict(out_dtype=BF16),
                        dict(round_intermediates=True, scale=0.3), dict(scale="x")):
            _compare(monkeypatch, lambda: k.softmax(x, **options))
        for options in ({}, dict(scale=0.5), dict(relu=True), dict(activation="silu"), dict(activation="gelu_erf"), dict(activation="none")):
            for out in (F32, BF16, dtype, torch.float64, None):
                _compare(monkeypatch, lambda: k.cast_scale(x, out, **options))
    _compare(monkeypatch, lambda: k.row_reduce(_t(5, 33, dtype=dtype), "sum"), native=True)
    _compare(monkeypatch, lambda: k.cast_scale(_t(3, 8, 4, 4, dtype=dtype).to(memory_format=torch.channels_last), F32), native=True)
    _compare(monkeypatch, lambda: k.row_reduce(torch.zeros(3, 4), "sum"), native=False)
    _compare(monkeypatch, lambda: k.cast_scale(torch.zeros(3, device="cuda", dtype=torch.int32), F32), native=False)


@pytest.mark.parametrize("dtype", [F32, BF16], ids=str)
def test_masks(monkeypatch, dtype):
    from better_benchmark_b200 import kernels as k
    x = _t(2, 3, 5, 24, dtype=dtype)
    for shape in ((24,), (1, 24), (5, 24), (1, 1, 1, 24), (2, 1, 1, 24), (2, 1, 5, 24), (2, 3, 5, 24), (3, 1, 24), (1, 3, 1, 24), (2, 1, 5, 1),
                  (4, 24), (1, 2, 3, 5, 24)):
        for other in (dtype, F16):
            _compare(monkeypatch, lambda: k.softmax(x, mask=_t(*shape, dtype=other), scale=0.125))
    _compare(monkeypatch, lambda: k.softmax(x, mask=_t(2, 1, 1, 24, dtype=dtype)), native=True)
    _compare(monkeypatch, lambda: k.softmax(x, mask=_t(24, 5, dtype=dtype).t()))
    _compare(monkeypatch, lambda: k.softmax(x.transpose(1, 2), mask=_t(2, 5, 1, 24, dtype=dtype)))
    _compare(monkeypatch, lambda: k.softmax(x, out=torch.empty_like(x)), native=False)


@pytest.mark.parametrize("dtype", [F32, BF16, F16], ids=str)
def test_norms(monkeypatch, dtype):
    from better_benchmark_b200 import kernels as k
    from better_benchmark_b200.families import layer_norm
    for x in (_t(6, 40, dtype=dtype), _t(2, 3, 40, dtype=dtype), _t(6, 48, dtype=dtype)[:, :40], _t(4, 6, 40, dtype=dtype)[::2], _t(1, 40, dtype=dtype),
              _t(40, dtype=dtype), _t(0, 40, dtype=dtype), _t(40, 6, dtype=dtype).t()):
        for wt, bt in ((dtype, dtype), (F32, F32), (None, None), (F32, None), (F32, BF16), (torch.float64, None)):
            w = None if wt is None else _t(40, dtype=F32).to(wt)
            b = None if bt is None else _t(40, dtype=F32).to(bt)
            for options in (dict(want_mean=True, want_rstd=True), dict(rms=True, want_rstd=True), dict(want_var=True, correction=1.0, want_y=False),
                            dict(prologue="gelu_erf"), dict(out_dtype=F32), dict(keepdim=False, want_rstd=True), dict(prologue="none"),
                            dict(want_sum=True), dict(residual=_t(*x.shape, dtype=dtype, seed=2), want_sum=True, round_sum="both"),
                            dict(residual=_t(*x.shape, dtype=dtype, seed=2), round_sum=True),
                            dict(residual=_t(*x.shape, dtype=dtype, seed=2), out_dtype=F32), dict(residual=_t(3, 40, dtype=dtype))):
                _compare(monkeypatch, lambda: k.norm_fwd(x, w, b, eps=1e-5, **options))
    x, res, w, b = _t(6, 40, dtype=dtype), _t(2, 3, 40, dtype=dtype, seed=3), _t(40, dtype=dtype), _t(40, dtype=dtype)
    _compare(monkeypatch, lambda: k.norm_fwd(x, w, b, eps=1, want_rstd=True), native=True)
    for returns in (("y2",), ("y3",), ("sum3", "y2"), ("sum2", "y2"), ("sum2", "y3", "mean"), ("mean", "rstd", "y2"), ("y3", "y2"), ("sum3", "sum2", "y2")):
        for shapes in (([2, 3, 40], [6, 40]), ([2, -1, 40], [-1, 40]), ((1, 6, 40), (6, 40)), ([2, 4, 40], [6, 40]), ([2, 3, 40], [5, 40]), ([-1, -1, 40], [6, 40])):
            _compare(monkeypatch, lambda: layer_norm.residual_forward([x, res, w, b, *shapes], eps=1e-12, returns=returns))
    _compare(monkeypatch, lambda: layer_norm.residual_forward([x, res, w, b, [2, 3, 40], [6, 40]], eps=1e-12, returns=("sum3", "y2")), native=True)


@pytest.mark.parametrize("dtype", [F32, BF16], ids=str)
def test_norm_backward(monkeypatch, dtype):
    from better_benchmark_b200 import kernels as k
    for shape, heads in (((6, 40), None), ((2, 3, 40), None), ((2, 5, 4, 8), 4), ((2, 5, 4, 8), 3), ((2, 5, 4, 8), None), ((1, 1), None), ((6, 300), None)):
        x = _t(*shape, dtype=dtype)
        n = shape[-1] * (heads if heads == 4 else 1)
        rows = x.numel() // n
        rstd, mean = _t(rows).abs() + 0.5, _t(rows, seed=4)
        for dy in (_t(*shape, dtype=dtype, seed=5), _t(1, dtype=dtype).expand(shape), torch.tensor(0.5, device="cuda", dtype=dtype),
                   _t(*shape, dtype=F16), _t(2, 2, dtype=dtype)):
            for options in (dict(rms=True), dict(rms=False, mean=mean, want_dbias=True), dict(rms=False), dict(rms=True, want_dweight=False),
                            dict(rms=True, two_launch=True), dict(rms=False, mean=mean.double()),
                            dict(rms=True, scratch=torch.zeros(1 << 20, dtype=torch.uint8, device="cuda"))):
                for w in (_t(n), None, _t(n + 1)):
                    _compare(monkeypatch, lambda: k.norm_bwd(x, dy, w, rstd, heads=heads, **options))
    x = _t(6, 40, dtype=dtype)
    _compare(monkeypatch, lambda: k.norm_bwd(x, x, None, _t(6), rms=True), native=True)
    _compare(monkeypatch, lambda: k.norm_bwd(_t(6, 48, dtype=dtype)[:, :40], x, None, _t(6), rms=True), native=False)


@pytest.mark.parametrize("dtype", [F32, BF16], ids=str)
def test_batch_norm(monkeypatch, dtype):
    from better_benchmark_b200 import kernels as k
    from better_benchmark_b200.families import batch_norm_bwd
    for base in (_t(4, 8, 5, 5, dtype=dtype), _t(4, 8, 5, 5, dtype=dtype).to(memory_format=torch.channels_last), _t(4, 8, 1, 1, dtype=dtype), _t(4, 1, 3, 3, dtype=dtype),
                 _t(4, 8, 5, 5, dtype=dtype).permute(0, 2, 1, 3), _t(4, 8, 5, 6, dtype=dtype)[..., :5], _t(0, 8, 5, 5, dtype=dtype), _t(4, 8, 5, dtype=dtype)):
        c = base.shape[1]
        w, b = _t(c), _t(c, seed=1)
        for options in (dict(), dict(relu=True), dict(unbiased_factor=1.25), dict(scratch=torch.zeros(1 << 20, dtype=torch.uint8, device="cuda")),
                        dict(scratch=torch.zeros(16, dtype=torch.uint8, device="cuda"))):
            for p in ((w, b), (None, None), (w, None), (w, b.to(BF16)), (_t(c + 1), b)):
                def forward():
                    running = torch.zeros(c, device="cuda"), torch.ones(c, device="cuda")
                    return k.batch_norm_fwd(base, *p, *running, eps=1e-5, momentum=0.1, **options), running
                _compare(monkeypatch, forward)
        _compare(monkeypatch, lambda: k.batch_norm_fwd(base, w, b, None, None, eps=1e-5, momentum=0.1))
        _compare(monkeypatch, lambda: k.batch_norm_fwd(base, w, b, torch.zeros(c + 1, device="cuda"), None, eps=1e-5, momentum=0.1))
        dy, act = (torch.empty_strided(base.shape, base.stride(), dtype=dtype, device="cuda").normal_() if base.dim() == 4 else base for _ in range(2))
        mean, invstd = _t(c), _t(c).abs() + 0.1
        for options in (dict(), dict(act=act, slope=0.2), dict(want_dx=False), dict(inv_count=0.01), dict(act=act.float())):
            _compare(monkeypatch, lambda: k.batch_norm_bwd(dy, base, mean, invstd, w, **options))
            _compare(monkeypatch, lambda: k.batch_norm_bwd(dy, base, mean.view(1, c, 1, 1), invstd, None, **options))
        _compare(monkeypatch, lambda: k.batch_norm_bwd(dy.contiguous(), base, mean, invstd, w))
        _compare(monkeypatch, lambda: batch_norm_bwd.oracle_forward([dy, base, torch.stack([mean, mean], 1)[:, 0], invstd, w]))
    x = _t(4, 8, 5, 5, dtype=dtype)
    _compare(monkeypatch, lambda: k.batch_norm_fwd(x, None, None, None, None, eps=1e-5, momentum=0.1), native=True)
    _compare(monkeypatch, lambda: k.batch_norm_bwd(x, x, _t(8), _t(8), None), native=True)


def test_permutes(monkeypatch):
    from better_benchmark_b200 import kernels as k
    from better_benchmark_b200.families import permute
    for x in (_t(3, 5, 7), _t(3, 5, 7, dtype=BF16), _t(2, 3, 4, 8, dtype=F16), _t(2, 3, 4, 2, 2), _t(1, 1), _t(6), _t(4, 6)[:, ::2], _t(0, 3), _t(2, 2, 2, 2, 2, 2)):
        nd = x.dim()
        for dims in (tuple(range(nd)), tuple(reversed(range(nd))), tuple(range(nd - 2)) + (nd - 1, nd - 2) if nd > 1 else (0,), (-1,) * nd, (0,) * nd,
                     tuple(range(nd + 1)), list(range(1, nd)) + [0]):
            for options in ({}, dict(scale=0.5), dict(out_dtype=BF16), dict(out_dtype=torch.int32)):
                _compare(monkeypatch, lambda: k.permute_copy(x, dims, **options))
    x = _t(3, 5, 7)
    for shape in ((3, 7, 5), [21, 5], (-1, 5), (3, -1, 5), (3, 35), (2, 5), (-1, -1, 5), torch.Size([105])):
        _compare(monkeypatch, lambda: permute.transpose_forward([x, shape]))
    _compare(monkeypatch, lambda: permute.transpose_forward([x, (3, 7, 5)]), native=True)
    _compare(monkeypatch, lambda: permute.head_split_forward([_t(10, 32), None, (2, 5, 4, 8), (8, 5, 8)]), native=True)


def test_modes_subclasses_and_transforms(monkeypatch):
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode
    from better_benchmark_b200 import kernels as k

    class Functions(TorchFunctionMode):
        seen = 0

        def __torch_function__(self, func, types, args=(), kwargs=None):
            Functions.seen += 1
            return func(*args, **(kwargs or {}))

    class Dispatches(TorchDispatchMode):
        seen = []

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            self.seen.append(str(func))
            return func(*args, **(kwargs or {}))

    class Sub(torch.Tensor):
        pass

    x = _t(4, 40)
    with Functions():
        _compare(monkeypatch, lambda: k.softmax(x), native=False)
    assert Functions.seen > 0
    k.softmax(x)
    with Dispatches():
        k.softmax(x)
    assert any("empty" in s for s in Dispatches.seen), "a dispatch mode sees the allocation"
    _compare(monkeypatch, lambda: k.row_reduce(x.as_subclass(Sub), "sum").as_subclass(torch.Tensor), native=False)
    for call in (lambda t: k.softmax(t), lambda t: k.row_reduce(t, "sum")):
        with pytest.raises(Exception):
            torch.func.vmap(call)(x)
    torch.use_deterministic_algorithms(True)
    try:
        _compare(monkeypatch, lambda: k.softmax(x), native=True)
    finally:
        torch.use_deterministic_algorithms(False)


def test_streams_threads_and_graphs():
    from better_benchmark_b200 import kernels as k
    x, w = _t(64, 768, dtype=BF16), _t(768)
    want = k.norm_fwd(x, w, w, eps=1e-5, want_mean=True, want_rstd=True)
    torch.cuda.synchronize()
    results, errors = {}, []

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(50):
                    got = k.norm_fwd(x, w, w, eps=1e-5, want_mean=True, want_rstd=True)
                torch.cuda.current_stream().synchronize()
                results[i] = got
                with pytest.raises(k.UnsupportedLayout):
                    k.norm_fwd(x, w[:5], w, eps=1e-5)
        except BaseException as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for got in results.values():
        assert all(torch.equal(a, b) for a, b in zip(got[:3], want[:3]))
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        got = k.norm_fwd(x, w, w, eps=1e-5, want_mean=True, want_rstd=True)
    g.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(got[:3], want[:3]))


def test_residuals_with_strides_of_their_own(monkeypatch):
    """A residual counts as contiguous whatever the stride of a dimension of size one: the Python code refuses it, and so does the native code."""
    from better_benchmark_b200 import kernels as k
    x, w = _t(4, 1, 40, dtype=BF16), _t(40)
    residual = torch.empty_strided((4, 1, 40), (40, 8, 1), device="cuda", dtype=BF16).copy_(x)
    assert residual.is_contiguous() and residual.stride() != x.stride()
    _compare(monkeypatch, lambda: k.norm_fwd(x, w, w, eps=1e-5, residual=residual), native=False)
    with pytest.raises(k.UnsupportedLayout, match="strides"):
        k.norm_fwd(x, w, w, eps=1e-5, residual=residual)
