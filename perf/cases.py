"""Measured cases: single calls of the package's public entry points, as a training or inference program makes them.

``listed()`` holds the five configurations of ``workloads.py`` and seven more calls at sizes that the
package's own family cases and canonical directories use; ``draw`` spreads the same kinds of call over
their sizes, layouts, dtypes and options, odd sizes among them. Inputs are made on the GPU from the seed.
"""
import math

import torch

from better_benchmark_b200 import kernels
from better_benchmark_b200.families import (batch_norm_bwd, batch_norm_relu, layer_norm, masked_softmax,
                                            permute, rms_norm_bwd_heads, row_mean)

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
SIZE = {"f32": 4, "bf16": 2, "f16": 2}


def listed():
    return [
        # the cast of one fp32 master weight to the compute dtype: the smallest and most frequent call of a
        # training step, where launch and host work are the whole cost
        dict(name="weight_cast", kind="pointwise", op="cast", rows=768, cols=768, dtype="f32", out="bf16"),
        # per-row mean of an fp32 matrix (pooling, metrics)
        dict(name="row_mean", kind="row_reduce", op="mean", rows=8192, cols=4096, dtype="f32"),
        # LayerNorm forward of an encoder block, statistics kept for the backward
        dict(name="layer_norm", kind="norm", form="layer", rows=32768, cols=768, dtype="bf16", gelu=False),
        # residual add -> LayerNorm of an encoder block at a large batch
        dict(name="residual_layer_norm", kind="residual_norm", rows=65536, cols=768, dtype="bf16", keep_sum=True),
        # LayerNorm backward of an encoder block
        dict(name="layer_norm_backward", kind="norm_bwd", form="layer", rows=32768, cols=768, dtype="bf16"),
        # RMSNorm backward of a decoder block, dx stored head-major
        dict(name="rms_norm_backward_heads", kind="rms_bwd_heads", batch=4, seq=4096, heads=32, head_dim=128, dtype="bf16"),
        # attention probabilities: scaled scores with a key mask
        dict(name="masked_softmax", kind="masked_softmax", batch=16, heads=12, queries=512, keys=512, dtype="f16"),
        # log-probabilities over a vocabulary whose size is not a multiple of a vector, rows padded, fp32 out
        dict(name="vocabulary_log_softmax", kind="vocabulary", rows=4096, cols=20005, pad=3, dtype="bf16", out="f32", log=True),
        # BatchNorm2d training forward + ReLU, channels-last
        dict(name="batch_norm_relu", kind="batch_norm", n=256, c=64, h=56, w=56, layout="cl", dtype="bf16", relu=True),
        # BatchNorm2d training backward, channels-last
        dict(name="batch_norm_backward", kind="batch_norm_bwd", n=256, c=64, h=56, w=56, layout="cl", dtype="bf16", leaky=False),
        # SiLU of an activation tensor in storage order
        dict(name="silu", kind="pointwise", op="silu", rows=32768, cols=1536, dtype="bf16", out="bf16"),
        # patch matrices [49, channels] to channel-major, an odd inner extent
        dict(name="window_transpose", kind="transpose", batch=16384, rows=49, cols=128, dtype="bf16"),
    ]


MOST_BYTES = 400e6   # below the largest listed case


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _extent(rng, low, high):
    """A length: half of the time a multiple of 64, as models have it, otherwise whatever comes."""
    n = _log_int(rng, low, high)
    return max(64, n // 64 * 64) if rng.random() < 0.5 and high >= 64 else n


def draw(rng):
    kind = rng.choice(["pointwise", "row_reduce", "norm", "residual_norm", "norm_bwd", "rms_bwd_heads", "masked_softmax",
                       "vocabulary", "batch_norm", "batch_norm_bwd", "transpose"])
    half = rng.choice(["bf16", "f16"])
    while True:
        if kind == "pointwise":
            op = rng.choice(["cast", "relu", "gelu_erf", "silu"])
            pair = rng.choice([("f32", "bf16"), ("bf16", "f32"), ("f32", "f16")]) if op == "cast" else (half, half)
            case = dict(kind=kind, op=op, rows=_log_int(rng, 1, 65536), cols=_extent(rng, 16, 4096), dtype=pair[0], out=pair[1])
        elif kind == "row_reduce":
            case = dict(kind=kind, op=rng.choice(["mean", "sum", "amax"]), rows=_log_int(rng, 32, 65536),
                        cols=_extent(rng, 32, 8192), dtype=rng.choice(["f32", "bf16"]))
        elif kind == "norm":
            gelu = rng.random() < 0.25
            case = dict(kind=kind, form="layer" if gelu else rng.choice(["layer", "rms"]), rows=_log_int(rng, 64, 65536),
                        cols=_extent(rng, 64, 8192), dtype=half if gelu else rng.choice(["f32", "bf16", "f16"]), gelu=gelu)
        elif kind == "residual_norm":
            case = dict(kind=kind, rows=_log_int(rng, 64, 65536), cols=_extent(rng, 64, 4096), dtype=half,
                        keep_sum=rng.random() < 0.5)
        elif kind == "norm_bwd":
            case = dict(kind=kind, form=rng.choice(["layer", "rms"]), rows=_log_int(rng, 64, 65536),
                        cols=_extent(rng, 64, 4096), dtype=rng.choice(["f32", "bf16", "f16"]))
        elif kind == "rms_bwd_heads":
            case = dict(kind=kind, batch=rng.randint(1, 8), seq=_log_int(rng, 64, 4096), heads=rng.choice([4, 8, 12, 16, 32]),
                        head_dim=rng.choice([64, 128]), dtype=half)
        elif kind == "masked_softmax":
            case = dict(kind=kind, batch=_log_int(rng, 1, 64), heads=rng.choice([8, 12, 16]), queries=_log_int(rng, 16, 1024),
                        keys=_extent(rng, 32, 2048), dtype=half)
        elif kind == "vocabulary":
            cols = _log_int(rng, 1000, 131072)
            case = dict(kind=kind, rows=_log_int(rng, 16, 8192), cols=cols, pad=-cols % 8 if rng.random() < 0.5 else 0,
                        dtype=rng.choice(["f32", "bf16"]), out=rng.choice(["f32", "f32", "bf16"]), log=rng.random() < 0.5)
        elif kind in ("batch_norm", "batch_norm_bwd"):
            h = rng.choice([7, 8, 14, 16, 28, 32, 56])
            case = dict(kind=kind, n=_log_int(rng, 8, 256), c=_extent(rng, 16, 1024), h=h, w=h, layout=rng.choice(["cl", "nchw"]),
                        dtype=rng.choice(["bf16", "bf16", "f32"]))
            case.update(dict(relu=rng.random() < 0.7) if kind == "batch_norm" else dict(leaky=rng.random() < 0.4))
        else:
            case = dict(kind=kind, batch=_log_int(rng, 1, 8192), rows=_log_int(rng, 16, 1024), cols=_extent(rng, 32, 1024), dtype=half)
        if work(case)["bytes"] <= MOST_BYTES:
            return case


class _Source:
    """Seeded tensors on the GPU."""

    def __init__(self, seed):
        self.generator = torch.Generator(device="cuda").manual_seed(int(seed))

    def normal(self, shape, dtype, scale=1.0, shift=0.0):
        t = torch.randn(shape, generator=self.generator, device="cuda", dtype=torch.float32)
        return t.mul_(scale).add_(shift).to(DTYPES[dtype])

    def uniform(self, shape, dtype, low, high):
        t = torch.rand(shape, generator=self.generator, device="cuda", dtype=torch.float32)
        return t.mul_(high - low).add_(low).to(DTYPES[dtype])


def _image(source, case, scale=1.0, shift=0.0):
    t = source.normal((case["n"], case["c"], case["h"], case["w"]), case["dtype"], scale, shift)
    return t.contiguous(memory_format=torch.channels_last) if case["layout"] == "cl" else t


def prepare(case, seed):
    s, kind = _Source(seed), case["kind"]
    state = dict(case=case)
    if kind in ("pointwise", "row_reduce"):
        state["x"] = s.normal((case["rows"], case["cols"]), case["dtype"])
    elif kind in ("norm", "residual_norm"):
        cols, dt = case["cols"], case["dtype"]
        state["x"] = s.normal((case["rows"], cols), dt)
        state["weight"] = s.uniform((cols,), dt, 0.5, 1.5)
        state["bias"] = s.normal((cols,), dt, 0.02)
        if kind == "residual_norm":
            state["residual"] = s.normal((1, case["rows"], cols), dt)
    elif kind == "norm_bwd":
        cols = case["cols"]
        state["x"] = s.normal((case["rows"], cols), case["dtype"], 1.0, 0.1)
        state["dy"] = s.normal((case["rows"], cols), case["dtype"])
        state["weight"] = s.uniform((cols,), "f32", 0.5, 1.5)
        xf = state["x"].float()
        if case["form"] == "layer":
            state["mean"] = xf.mean(dim=1)
            state["rstd"] = torch.rsqrt(xf.var(dim=1, unbiased=False) + 1e-5)
        else:
            state["mean"] = None
            state["rstd"] = torch.rsqrt(xf.pow(2).mean(dim=1) + 1e-6)
    elif kind == "rms_bwd_heads":
        shape = (case["batch"], case["seq"], case["heads"], case["head_dim"])
        state["x"], state["dy"] = s.normal(shape, case["dtype"]), s.normal(shape, case["dtype"])
        state["weight"] = s.uniform((case["heads"] * case["head_dim"],), case["dtype"], 0.5, 1.5)
        state["rstd"] = torch.rsqrt(state["x"].float().view(case["batch"] * case["seq"], -1).pow(2).mean(-1) + 1e-6)
    elif kind == "masked_softmax":
        b, k = case["batch"], case["keys"]
        state["x"] = s.normal((b, case["heads"], case["queries"], k), case["dtype"], 4.0)
        lengths = torch.randint(max(1, k // 4), k + 1, (b,), generator=s.generator, device="cuda")
        keys = torch.arange(k, device="cuda")[None, :]
        mask = torch.where(keys < lengths[:, None], 0.0, -10000.0)
        state["mask"] = mask.to(DTYPES[case["dtype"]]).view(b, 1, 1, k)
    elif kind == "vocabulary":
        rows = s.normal((case["rows"], case["cols"] + case["pad"]), case["dtype"], 2.0)
        state["x"] = rows[:, :case["cols"]]
    elif kind in ("batch_norm", "batch_norm_bwd"):
        c = case["c"]
        state["x"] = _image(s, case, 2.0, 0.5)
        state["weight"] = s.uniform((c,), "f32", 0.5, 1.5)
        if kind == "batch_norm":
            state["bias"] = s.normal((c,), "f32", 0.1)
            state["running_mean"], state["running_var"] = torch.zeros(c, device="cuda"), torch.ones(c, device="cuda")
        else:
            state["dy"] = _image(s, case)
            if case["leaky"]:
                state["act"] = _image(s, case)
            xf = state["x"].float()
            state["mean"] = xf.mean(dim=(0, 2, 3))
            state["invstd"] = torch.rsqrt(xf.var(dim=(0, 2, 3), unbiased=False) + 1e-5)
    else:
        state["x"] = s.normal((case["batch"], case["rows"], case["cols"]), case["dtype"])
    return state


def run(state):
    case, x = state["case"], state["x"]
    kind = case["kind"]
    if kind == "pointwise":
        return kernels.cast_scale(x, DTYPES[case["out"]], activation=None if case["op"] == "cast" else case["op"])
    if kind == "row_reduce":
        return row_mean.oracle_forward([x]) if case["op"] == "mean" else kernels.row_reduce(x, case["op"])
    if kind == "norm":
        if case["form"] == "rms":
            y, _, rstd, _ = kernels.norm_fwd(x, state["weight"], None, eps=1e-6, rms=True, want_rstd=True)
            return y, rstd
        if case["gelu"]:
            y, mean, rstd, _ = kernels.norm_fwd(x, state["weight"], state["bias"], eps=1e-12, prologue="gelu_erf",
                                                want_mean=True, want_rstd=True)
            return y, mean, rstd
        return layer_norm.oracle_forward([x, state["weight"], state["bias"]], eps=1e-12)
    if kind == "residual_norm":
        returns = ("sum3", "y2") if case["keep_sum"] else ("y2",)
        return layer_norm.residual_forward([x, state["residual"], state["weight"], state["bias"],
                                            (1, case["rows"], case["cols"]), (case["rows"], case["cols"])],
                                           eps=1e-12, returns=returns)
    if kind == "norm_bwd":
        layer = case["form"] == "layer"
        dx, dw, db = kernels.norm_bwd(x, state["dy"], state["weight"], state["rstd"], mean=state["mean"], rms=not layer,
                                      want_dbias=layer)
        return (dx, dw, db) if layer else (dx, dw)
    if kind == "rms_bwd_heads":
        return rms_norm_bwd_heads.oracle_forward([x, state["dy"], state["weight"], state["rstd"]])
    if kind == "masked_softmax":
        return masked_softmax.oracle_forward([x, state["mask"]], scale=0.125)
    if kind == "vocabulary":
        return kernels.softmax(x, log=case["log"], out_dtype=DTYPES[case["out"]])
    if kind == "batch_norm":
        return batch_norm_relu.oracle_forward([x, state["running_mean"], state["running_var"], state["weight"], state["bias"]],
                                              relu=case["relu"])
    if kind == "batch_norm_bwd":
        if case["leaky"]:
            return batch_norm_bwd.leaky_relu_forward([state["dy"], state["act"], x, state["mean"], state["invstd"], state["weight"]])
        return batch_norm_bwd.oracle_forward([state["dy"], x, state["mean"], state["invstd"], state["weight"]])
    return permute.transpose_forward([x, (case["batch"], case["cols"], case["rows"])])


def work(case):
    """Every input once and every output once; the operations are a few per element and never the bound."""
    kind, size = case["kind"], SIZE[case["dtype"]]
    if kind == "pointwise":
        n = case["rows"] * case["cols"]
        return {"bytes": n * (size + SIZE[case["out"]]), "flops": {"cast": 1, "relu": 1, "silu": 6, "gelu_erf": 20}[case["op"]] * n}
    if kind == "row_reduce":
        return {"bytes": case["rows"] * (case["cols"] + 1) * size, "flops": case["rows"] * case["cols"]}
    if kind == "norm":
        n = case["rows"] * case["cols"]
        vectors = 2 if case["form"] == "layer" else 1
        return {"bytes": 2 * n * size + vectors * (case["cols"] * size + case["rows"] * 4), "flops": (28 if case["gelu"] else 8) * n}
    if kind == "residual_norm":
        n = case["rows"] * case["cols"]
        return {"bytes": (4 if case["keep_sum"] else 3) * n * size + 2 * case["cols"] * size, "flops": 16 * n}
    if kind in ("norm_bwd", "rms_bwd_heads"):
        heads = kind == "rms_bwd_heads"
        rows = case["batch"] * case["seq"] if heads else case["rows"]
        cols = case["heads"] * case["head_dim"] if heads else case["cols"]
        vectors = 2 if case.get("form") == "layer" else 1
        return {"bytes": 3 * rows * cols * size + vectors * 4 * (rows + cols) + cols * (size if heads else 4), "flops": 12 * rows * cols}
    if kind == "masked_softmax":
        n = case["batch"] * case["heads"] * case["queries"] * case["keys"]
        return {"bytes": 2 * n * size + case["batch"] * case["keys"] * size, "flops": 8 * n}
    if kind == "vocabulary":
        n = case["rows"] * case["cols"]
        return {"bytes": n * (size + SIZE[case["out"]]), "flops": 6 * n}
    if kind in ("batch_norm", "batch_norm_bwd"):
        n = case["n"] * case["c"] * case["h"] * case["w"]
        tensors = 2 if kind == "batch_norm" else 4 if case["leaky"] else 3
        return {"bytes": tensors * n * size + 8 * 4 * case["c"], "flops": 8 * n}
    n = case["batch"] * case["rows"] * case["cols"]
    return {"bytes": 2 * n * size, "flops": n}


def tolerance(case):
    """Copies, casts and maxima are exact. With 16-bit results a different evaluation order moves a small
    share of the values by one rounding step (2^-8 of the value for bf16, 2^-11 for fp16; rows that are
    normalised at both precisions of a sum by two); with fp32 results it is fp32 sums."""
    kind = case["kind"]
    if kind == "transpose" or (kind == "pointwise" and case["op"] in ("cast", "relu")) or \
            (kind == "row_reduce" and case["op"] == "amax"):
        return "exact"
    result = case["out"] if kind in ("pointwise", "vocabulary") else case["dtype"]
    if result == "f32":
        return {"rel": 1e-5, "max": 1e-4}
    if result == "f16":
        return {"rel": 5e-4, "max": 4e-3}
    return {"rel": 2e-3, "max": 2e-2}


def _both_forms(x, residual, weight, bias, eps):
    """LayerNorm of the sum at full precision where that result exceeds 3, of the rounded sum elsewhere."""
    def normalise(t):
        centred = t - t.mean(dim=-1, keepdim=True)
        rstd = torch.rsqrt(centred.square().mean(dim=-1, keepdim=True) + eps)
        return centred * rstd * weight.double() + bias.double()
    total = x.double() + residual.double()
    rounded = total.to(x.dtype)
    full = normalise(total)
    return rounded, torch.where(full.to(x.dtype).abs() > 3, full, normalise(rounded.double()))


def exact(case, seed):
    state = prepare(case, seed)
    x, kind = state["x"], case["kind"]
    d = x.double()
    if kind == "pointwise":
        op = case["op"]
        if op == "silu":
            return d * torch.sigmoid(d)
        if op == "gelu_erf":
            return 0.5 * d * (1 + torch.erf(d * math.sqrt(0.5)))
        return torch.relu(d) if op == "relu" else d
    if kind == "row_reduce":
        return d.amax(dim=-1) if case["op"] == "amax" else d.sum(dim=-1) if case["op"] == "sum" else d.mean(dim=-1)
    if kind == "norm":
        w = state["weight"].double()
        if case["form"] == "rms":
            rstd = torch.rsqrt(d.square().mean(dim=-1, keepdim=True) + 1e-6)
            return d * rstd * w, rstd
        if case["gelu"]:
            d = (0.5 * d * (1 + torch.erf(d * math.sqrt(0.5)))).to(x.dtype).double()
        mean = d.mean(dim=-1, keepdim=True)
        rstd = torch.rsqrt((d - mean).square().mean(dim=-1, keepdim=True) + 1e-12)
        y = (d - mean) * rstd * w + state["bias"].double()
        return (y, mean, rstd) if case["gelu"] else (y, mean.squeeze(-1), rstd.squeeze(-1))
    if kind == "residual_norm":
        total, y = _both_forms(x, state["residual"].view(x.shape), state["weight"], state["bias"], 1e-12)
        return (total.double().view(1, *x.shape), y) if case["keep_sum"] else y
    if kind in ("norm_bwd", "rms_bwd_heads"):
        shape = x.shape
        cols = state["weight"].numel()
        d, dy = d.reshape(-1, cols), state["dy"].double().reshape(-1, cols)
        rstd = state["rstd"].double().view(-1, 1)
        layer = case.get("form") == "layer"
        xhat = (d - state["mean"].double().view(-1, 1)) * rstd if layer else d * rstd
        g = dy * state["weight"].double()
        dx = g - xhat * (g * xhat).mean(dim=-1, keepdim=True)
        if layer:
            dx = dx - g.mean(dim=-1, keepdim=True)
        dx = dx * rstd
        dw = (dy * xhat).sum(dim=0)
        if kind == "rms_bwd_heads":
            return dx.view(shape).permute(0, 2, 1, 3).contiguous(), dw
        return (dx, dw, dy.sum(dim=0)) if layer else (dx, dw)
    if kind == "masked_softmax":
        return torch.softmax(d * 0.125 + state["mask"].double(), dim=-1)
    if kind == "vocabulary":
        return torch.log_softmax(d, dim=-1) if case["log"] else torch.softmax(d, dim=-1)
    if kind == "batch_norm":
        c, n = case["c"], x.numel() // case["c"]
        mean, var = d.mean(dim=(0, 2, 3)), d.var(dim=(0, 2, 3), unbiased=False)
        invstd = torch.rsqrt(var + 1e-5)
        column = lambda t: t.double().view(1, c, 1, 1)  # noqa: E731
        y = (d - column(mean)) * column(invstd) * column(state["weight"]) + column(state["bias"])
        return torch.relu(y) if case["relu"] else y, mean, invstd, 0.1 * mean, 0.9 + 0.1 * var * (n / (n - 1))
    if kind == "batch_norm_bwd":
        c, n = case["c"], x.numel() // case["c"]
        column = lambda t: t.double().view(1, c, 1, 1)  # noqa: E731
        dy = state["dy"].double()
        if case["leaky"]:
            slope = float(torch.tensor(0.2, dtype=torch.float32))
            dy = torch.where(state["act"] > 0, dy, (dy * slope).to(x.dtype).double())
        xhat = (d - column(state["mean"])) * column(state["invstd"])
        db, dw = dy.sum(dim=(0, 2, 3)), (dy * xhat).sum(dim=(0, 2, 3))
        dx = (dy - column(db) / n - xhat * column(dw) / n) * column(state["weight"]) * column(state["invstd"])
        return db, dw, dx
    return d.transpose(1, 2).contiguous()
