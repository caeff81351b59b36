"""The work that a user of this package has it do, as cases that can be timed.

Each case is one call sequence through the package's public entry points, in the form a training or inference
program makes it: forward and backward of a product, of a Linear layer, of an attention block, of a transformer
MLP, single-token decoding, and the optimizer step over a model's parameters.  Everything is f32; `precision`
"tf32" is the single-pass option of the matmul entry points, "3xtf32" their default.

`listed()` names the cases, `draw(rng)` gives another one of the same ranges, `prepare` builds what a program
holds before the call, `run` is one pass, `work` the bytes and operations no implementation can avoid and
`tolerance` how far two correct implementations may be apart.
"""
import math

import torch

import framework_b200 as F
from framework_b200 import DeviceTensor, _lib

# Upper ends of the drawn sizes: no drawn case costs more than the largest listed ones, odd sizes included.
MAX_FLOPS = {"3xtf32": 0.45e12, "tf32": 1.6e12}
MAX_ELEMENTS = 2.0e8           # of the largest tensor of a drawn case


def listed():
    return [
        # A layer of a small network on a small batch: every size below one tile, so only launches and host work count.
        {"name": "linear-small", "kind": "linear", "m": 32, "k": 64, "n": 32, "dropin": True},
        # The square product every tutorial starts with (forward and both gradients).
        {"name": "square-512", "kind": "matmul", "batch": 1, "shared": False, "m": 512, "k": 512, "n": 512,
         "bt": False, "precision": "3xtf32"},
        # Feature and class counts of real data sets are not multiples of anything.
        {"name": "ragged", "kind": "matmul", "batch": 1, "shared": False, "m": 1000, "k": 333, "n": 777,
         "bt": False, "precision": "3xtf32"},
        # Training step of a Linear layer with bias at transformer size.
        {"name": "linear-step", "kind": "linear", "m": 4096, "k": 1024, "n": 4096, "dropin": False},
        # A batch of sequences times one shared weight; the weight gradient sums over the batch.
        {"name": "shared-weight", "kind": "matmul", "batch": 64, "shared": True, "m": 1024, "k": 768, "n": 3072,
         "bt": False, "precision": "3xtf32"},
        # The largest square in the fast mode.
        {"name": "square-8192-tf32", "kind": "matmul", "batch": 1, "shared": False, "m": 8192, "k": 8192, "n": 8192,
         "bt": False, "precision": "tf32"},
        # Generating one token: one row against a weight that does not stay in L2, forward only.
        {"name": "decode-1", "kind": "decode", "m": 1, "k": 4096, "n": 4096, "backward": False},
        # A few rows, trained: forward and both gradients, bound by moving the weight.
        {"name": "rows-16", "kind": "decode", "m": 16, "k": 4096, "n": 4096, "backward": True},
        # Multi-head attention on head-split views, forward and backward.
        {"name": "attention", "kind": "attention", "b": 8, "t": 512, "h": 12, "d": 64},
        # The same with a sequence length as it comes: rows of scores are then not 16-byte aligned.
        {"name": "attention-ragged", "kind": "attention", "b": 4, "t": 333, "h": 12, "d": 64},
        # Transformer MLP: up-projection + bias + GELU, down-projection, all gradients.
        {"name": "mlp", "kind": "mlp", "m": 2048, "c": 768, "f": 3072},
        # Global-norm clip and AdamW over the parameters of a transformer: many tensors, large and tiny.
        {"name": "optimizer", "kind": "optimizer", "layers": 6, "c": 768, "f": 3072},
    ]


# --------------------------------------------------------------------------- drawn cases
def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """Spread over the logarithm of [lo, hi]; half of them round (multiples of 64, or of 8 below 128), half as they come."""
    v = _log_int(rng, lo, hi)
    if rng.random() < 0.5:
        unit = 64 if v >= 128 else 8
        v = max(unit, (v + unit // 2) // unit * unit)
    return max(lo, min(hi, v))


def _fit(sizes, cost, limit):
    """Halves the largest of `sizes` until cost(sizes) is within limit."""
    while cost(sizes) > limit:
        i = max(range(len(sizes)), key=lambda j: sizes[j])
        sizes[i] = max(1, (sizes[i] + 1) // 2)
    return sizes


def draw(rng):
    kind = rng.choice(["linear", "matmul", "matmul", "decode", "attention", "mlp", "optimizer"])
    if kind == "matmul":
        precision = "tf32" if rng.random() < 0.2 else "3xtf32"
        batch = 1 if rng.random() < 0.6 else _log_int(rng, 2, 64)
        shared = batch > 1 and rng.random() < 0.5
        s = [_size(rng, 64, 8192) for _ in range(3)]
        _fit(s, lambda v: 6.0 * batch * v[0] * v[1] * v[2], MAX_FLOPS[precision])
        _fit(s, lambda v: batch * max(v[0] * v[1], v[1] * v[2], v[0] * v[2]), MAX_ELEMENTS)
        return {"kind": kind, "batch": batch, "shared": shared, "m": s[0], "k": s[1], "n": s[2],
                "bt": rng.random() < 0.25, "precision": precision}
    if kind == "linear":
        s = [_size(rng, 16, 8192) for _ in range(3)]
        _fit(s, lambda v: 6.0 * v[0] * v[1] * v[2], MAX_FLOPS["3xtf32"])
        return {"kind": kind, "m": s[0], "k": s[1], "n": s[2], "dropin": rng.random() < 0.5}
    if kind == "decode":
        return {"kind": kind, "m": _log_int(rng, 1, 16), "k": _size(rng, 512, 8192), "n": _size(rng, 512, 8192),
                "backward": rng.random() < 0.4}
    if kind == "attention":
        d = rng.choice([32, 64, 64, 128])
        b, h, t = _log_int(rng, 1, 8), rng.choice([4, 8, 12, 16]), _size(rng, 64, 1024)
        while b * h * t * t > 3.0e7:
            t = (t + 1) // 2
        return {"kind": kind, "b": b, "t": t, "h": h, "d": d}
    if kind == "mlp":
        c = 64 * _log_int(rng, 2, 24)
        return {"kind": kind, "m": _size(rng, 64, 8192), "c": c, "f": 4 * c}
    c = 64 * _log_int(rng, 1, 16)
    return {"kind": kind, "layers": rng.randint(1, 12), "c": c, "f": 4 * c}


# --------------------------------------------------------------------------- inputs
def _flags(case):
    return _lib.PRECISION_TF32 if case.get("precision") == "tf32" else 0


def _parameter_shapes(case):
    """A transformer's parameters: per layer the attention and MLP weights, their biases and two norm gains and shifts."""
    c, f = case["c"], case["f"]
    layer = [(c, 3 * c), (3 * c,), (c, c), (c,), (c, f), (f,), (f, c), (c,), (c,), (c,), (c,), (c,)]
    return layer * case["layers"] + [(c,), (c,)]


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)

    def normal(*shape, scale=1.0):
        t = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32)
        return DeviceTensor.from_torch(t.mul_(scale) if scale != 1.0 else t)

    kind = case["kind"]
    state = {"kind": kind, "flags": _flags(case)}
    if kind in ("matmul", "linear", "decode"):
        m, k, n = case["m"], case["k"], case["n"]
        lead = (case["batch"],) if case.get("batch", 1) > 1 else ()
        wlead = () if case.get("shared", False) else lead
        state["x"] = normal(*lead, m, k)
        scale = 1.0 / math.sqrt(k)
        if case.get("bt", False):                      # a weight stored [out, in], read through a transposing view
            w = normal(*wlead, n, k, scale=scale)
            state["w"] = w.permute(tuple(range(len(wlead))) + (len(wlead) + 1, len(wlead)))
        else:
            state["w"] = normal(*wlead, k, n, scale=scale)
        state["dy"] = normal(*lead, m, n)
        if kind == "linear":
            state["layer"] = F.Linear(state["w"], normal(n, scale=0.02))
            state["dropin"] = case["dropin"]
        if kind == "decode":
            state["backward"] = case["backward"]
            state["bias"] = normal(n, scale=0.02)
            state["y"] = DeviceTensor.empty((m, n))    # decoding writes the same activation buffer for every token
    elif kind == "attention":
        b, t, h, d = case["b"], case["t"], case["h"], case["d"]
        q = normal(b, t, h, d, scale=1.0 / math.sqrt(d))        # the 1/sqrt(d) of the scores is folded into q
        k, v = normal(b, t, h, d), normal(b, t, h, d)
        state["q"] = q.permute((0, 2, 1, 3))
        state["kt"] = k.permute((0, 2, 3, 1))
        state["v"] = v.permute((0, 2, 1, 3))
        state["do"] = normal(b, t, h, d)
    elif kind == "mlp":
        m, c, f = case["m"], case["c"], case["f"]
        state.update(x=normal(m, c), w1=normal(c, f, scale=1.0 / math.sqrt(c)), b1=normal(f, scale=0.02),
                     w2=normal(f, c, scale=1.0 / math.sqrt(f)), b2=normal(c, scale=0.02), dy=normal(m, c))
    else:
        shapes = _parameter_shapes(case)
        offsets, total = [], 0
        for shape in shapes:                           # each tensor starts on a 256-byte boundary of a flat buffer
            offsets.append(total)
            total += (math.prod(shape) + 63) // 64 * 64
        flat = {}
        for name, scale in (("p", 0.02), ("m", 1e-3), ("v", 1e-3), ("g", 1e-2)):
            flat[name] = torch.randn(total, generator=gen, device="cuda").mul_(scale)
        flat["v"].square_()                            # second moments are positive
        state["flat"] = flat
        for name, buf in flat.items():
            state[name] = [DeviceTensor(buf[o:o + math.prod(s)], s) for o, s in zip(offsets, shapes)]
    return state


# --------------------------------------------------------------------------- one pass
def run(state):
    kind, flags = state["kind"], state["flags"]
    if kind == "matmul":
        x, w = state["x"], state["w"]
        y = F.matmul(x, w, flags=flags)
        dx, dw = F.matmul_backward(state["dy"], x, w, flags=flags)
        return [y.storage, dx.storage, dw.storage]
    if kind == "linear":
        x, dy, layer = state["x"], state["dy"], state["layer"]
        if state["dropin"]:                            # the two-call form: matmul, then the bias add, each with its backward
            y = layer.forward(x)
            dh, db = F.add_backward(dy, dy.shape, layer.bias.shape)
            dx, dw = F.matmul_backward(dh, x, layer.weight)
        else:
            y = layer.forward_fused(x)
            dx, dw, db = layer.backward(x, dy)
        return [y.storage, dx.storage, dw.storage, db.storage]
    if kind == "decode":
        x, w = state["x"], state["w"]
        y = F.matmul(x, w, state["bias"], out=state["y"])
        if not state["backward"]:
            return [y.storage]
        dx, dw = F.matmul_backward(state["dy"], x, w)
        return [y.storage, dx.storage, dw.storage]
    if kind == "attention":
        q, kt, v, do = state["q"], state["kt"], state["v"], state["do"]
        p = F.softmax(F.matmul(q, kt))
        o = F.matmul(p, v)
        merged = F.permute(o, (0, 2, 1, 3)).contiguous()                 # heads back beside each other: [b, t, h, d]
        do_heads = F.permute_backward(do, (0, 2, 1, 3), o.shape)
        dp, dv = F.matmul_backward(do_heads, p, v)
        ds = F.softmax_backward(dp, p)
        dq, dkt = F.matmul_backward(ds, q, kt)
        back = (do.shape[0], do.shape[1], do.shape[2], do.shape[3])
        dq = F.permute_backward(dq, (0, 2, 1, 3), back)
        dk = F.permute_backward(dkt, (0, 2, 3, 1), back)
        dv = F.permute_backward(dv, (0, 2, 1, 3), back)
        return [p.storage, merged.storage, dq.storage, dk.storage, dv.storage]
    if kind == "mlp":
        x, w1, b1, w2, b2, dy = (state[k] for k in ("x", "w1", "b1", "w2", "b2", "dy"))
        pre, act = F.matmul_bias_gelu(x, w1, b1)
        y = F.matmul(act, w2, b2)
        dact, dw2, db2 = F.matmul_backward(dy, act, w2, want_dbias=True)
        dpre, db1 = F.bias_gelu_backward(dact, pre, b1)
        dx, dw1 = F.matmul_backward(dpre, x, w1)
        return [t.storage for t in (pre, act, y, dw2, db2, db1, dx, dw1)]
    norm = F.clip_and_step(state["p"], state["m"], state["v"], state["g"], lr=1e-3, weight_decay=0.01, step=10,
                           max_grad_norm=1.0)
    return [norm, state["flat"]["p"], state["flat"]["m"], state["flat"]["v"], state["flat"]["g"]]


# --------------------------------------------------------------------------- floors and tolerances
def work(case):
    """Inputs read once, outputs written once; two operations per multiply-add of the products, as the mathematics
    counts them (the default precision spends three tensor-core passes on each)."""
    kind = case["kind"]
    if kind in ("matmul", "linear", "decode"):
        m, k, n = case["m"], case["k"], case["n"]
        batch = case.get("batch", 1)
        weights = 1 if case.get("shared", False) else batch
        x, w, y = batch * m * k, weights * k * n, batch * m * n
        flops = 2.0 * batch * m * k * n
        if kind == "decode" and not case["backward"]:
            return {"bytes": 4.0 * (x + w + y + n), "flops": flops}
        bias = 2 * n if kind == "linear" else (n if kind == "decode" else 0)
        return {"bytes": 4.0 * (2 * (x + w + y) + bias), "flops": 3.0 * flops}
    if kind == "attention":
        b, t, h, d = case["b"], case["t"], case["h"], case["d"]
        return {"bytes": 4.0 * (8 * b * t * h * d + b * h * t * t), "flops": 12.0 * b * h * t * t * d}
    if kind == "mlp":
        m, c, f = case["m"], case["c"], case["f"]
        return {"bytes": 4.0 * (4 * m * c + 2 * m * f + 4 * c * f + 2 * f + 2 * c), "flops": 12.0 * m * c * f}
    n = sum(math.prod(s) for s in _parameter_shapes(case))
    return {"bytes": 4.0 * 8 * n, "flops": 20.0 * n}


def tolerance(case):
    if case["kind"] == "optimizer":
        return {"rel": 1e-6}                           # elementwise f32 arithmetic
    if case.get("precision") == "tf32":
        return {"rel": 2e-3}                           # one pass over 11-bit operands
    # The tensor core's f32 accumulate loses about 7e-9 per element of an accumulation chain of up to 1024: 8e-6 for
    # one implementation, and two that cut or order the sums differently can be that far apart in either direction.
    return {"rel": 2e-5}
