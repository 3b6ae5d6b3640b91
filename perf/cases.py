"""Performance cases of the quantized projections: what an inference engine has this library do.

An engine loads a model's block-quantized matrices once (`Backend.upload`) and then, for every token
or batch of tokens, multiplies activations by all of them: one call per projection (`project`,
`project_multi`), a prepared list of projections (`plan` / `run`), or host buffers in and out
(`project_host`).  The number of activation rows M is 1 when a sequence decodes, 2..16 when a draft is
verified or a few sequences decode together, some tens in a busy server, and hundreds to thousands
while prompts are read.

`listed()` holds the cases, `draw()` makes more of the same ranges, `prepare()` builds what a program
has in hand before the call, `run()` is one pass through the public entry points, `exact()` what that
pass returns, in 64 bits.
"""
from __future__ import annotations

import numpy as np
import torch

import magnitude_b200 as mb

_TYPES = {"Q4_0": mb.TYPE_Q4_0, "Q8_0": mb.TYPE_Q8_0, "Q4_K": mb.TYPE_Q4_K, "Q5_K": mb.TYPE_Q5_K, "Q6_K": mb.TYPE_Q6_K,
          "MXFP4": mb.TYPE_MXFP4}
_BLOCK = {"Q4_0": (32, 18), "Q8_0": (32, 34), "Q4_K": (256, 144), "Q5_K": (256, 176), "Q6_K": (256, 210), "MXFP4": (32, 17)}
_DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}
_SIZE = {"bf16": 2, "f32": 4}
_STREAMING = 2       # the largest M that decodes with activations in 16-bit fixed point
_EXACT = 16          # the largest M whose weights stay exact integers; larger batches round them to 16 bits

_HIDDEN_8B = {"hidden": 4096, "q_rows": 4096, "kv_rows": 1024, "inter": 14336}      # 32 query / 8 kv heads of 128
_HIDDEN_32B = {"hidden": 5120, "q_rows": 8192, "kv_rows": 1024, "inter": 25600}     # 64 query / 8 kv heads of 128


def listed():
    return [
        # The smallest call: one K projection of an 8B-class layer for one token.  Launch and call overhead count.
        {"name": "call_q4k_m1", "kind": "call", "type": "Q4_K", "n": 1024, "k": 4096, "m": 1, "x": "bf16", "y": "f32", "copies": 1},
        # The reference's own boundary: a Q8_0 mat-vec whose fp32 activation and result live in host memory.
        {"name": "host_q8_0_m1", "kind": "host", "type": "Q8_0", "n": 4096, "k": 4096, "m": 1, "x": "f32", "y": "f32"},
        # All MLP projections of a 32-layer 8B-class model for one token, as one plan of independent jobs: every
        # byte of 3.2 GB of weights is read once.
        {"name": "mlp_plan_q4k_m1", "kind": "mlp_plan", "hidden": 4096, "inter": 14336, "type": "Q4_K", "m": 1, "x": "bf16", "y": "f32", "layers": 32},
        # Decoding one token through four layers of a 32B-class model (Q4_K_M mix) the way an engine does: per layer
        # the attention inputs in one plan, then O, gate/up and down in another, chained through the residual stream.
        {"name": "chain_q4km_m1", "kind": "chain", "type": "Q4_K", "type_down": "Q6_K", "m": 1, "layers": 4, **_HIDDEN_32B},
        # Verifying a draft of three tokens: the fused QKV projections of 16 layers as one plan.
        {"name": "plan_q4k_m4", "kind": "plan", "type": "Q4_K", "n": 6144, "k": 4096, "m": 4, "x": "bf16", "y": "f32", "copies": 16},
        # Verifying a longer draft: the down projections of six layers, one call each.
        {"name": "calls_q6k_m8", "kind": "call", "type": "Q6_K", "n": 4096, "k": 14336, "m": 8, "x": "bf16", "y": "f32", "copies": 6},
        # Sixteen sequences decoding together: all projections of two 8B-class layers (Q4_K_M mix).
        {"name": "layer_q4km_m16", "kind": "layer", "type": "Q4_K", "type_down": "Q6_K", "m": 16, "x": "bf16", "y": "f32", "layers": 2, **_HIDDEN_8B},
        # A busier server: forty-eight sequences through the same two layers.
        {"name": "layer_q4km_m48", "kind": "layer", "type": "Q4_K", "type_down": "Q6_K", "m": 48, "x": "bf16", "y": "f32", "layers": 2, **_HIDDEN_8B},
        # The last, partial piece of a prompt against a matrix of odd height, fp32 activations.
        {"name": "call_q5k_m333", "kind": "call", "type": "Q5_K", "n": 11003, "k": 3328, "m": 333, "x": "f32", "y": "bf16", "copies": 1},
        # Reading a prompt in pieces of 512 tokens, an engine's usual physical batch: one 8B-class layer.
        {"name": "layer_q4km_m512", "kind": "layer", "type": "Q4_K", "type_down": "Q6_K", "m": 512, "x": "bf16", "y": "bf16", "layers": 1, **_HIDDEN_8B},
        # Reading 2048 tokens: one gate projection.
        {"name": "call_q4k_m2048", "kind": "call", "type": "Q4_K", "n": 14336, "k": 4096, "m": 2048, "x": "bf16", "y": "bf16", "copies": 1},
        # The largest: 4096 tokens through all projections of one 32B-class layer.
        {"name": "layer_q4km_m4096", "kind": "layer", "type": "Q4_K", "type_down": "Q6_K", "m": 4096, "x": "bf16", "y": "bf16", "layers": 1, **_HIDDEN_32B},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 200)


def draw(rng):
    """A case of the same ranges: any kind, type and row count, sizes spread over their logarithm, odd ones among them."""
    limit = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(["call"] * 6 + ["plan"] * 3 + ["layer"] * 4 + ["chain"] * 2 + ["mlp_plan"] * 2 + ["host"])
        t = rng.choice(["Q4_K"] * 3 + ["Q6_K"] * 2 + ["Q8_0"] * 2 + ["Q5_K", "Q4_0", "MXFP4"])
        blk = _BLOCK[t][0]
        x, y = rng.choice(["bf16", "bf16", "f32"]), rng.choice(["bf16", "f32"])
        m = rng.choice([lambda: rng.randint(1, 2), lambda: rng.randint(3, 16), lambda: _log(rng, 17, 127), lambda: _log(rng, 128, 4096)])()
        if kind in ("call", "plan", "host"):
            n, k = _log(rng, 512, 32768), _log(rng, 1024, 16384) // blk * blk
            if rng.random() < 0.5:
                n = max(512, n // 256 * 256)
            if kind == "plan":
                m = rng.randint(1, 16)
                if m > 8:
                    x = "bf16"
            if kind == "host":
                m = min(m, 512)
            copies = 1
            if kind == "plan" or (m <= 127 and rng.random() < 0.7):
                copies = max(2, min(24, int(rng.uniform(1.5e8, 3.5e8) / (n * k * _BLOCK[t][1] / blk))))
            case = {"kind": kind, "type": t, "n": n, "k": k, "m": m, "x": x, "y": y}
            if kind != "host":
                case["copies"] = copies
        elif kind == "mlp_plan":
            case = {"kind": kind, "hidden": 256 * rng.randint(8, 24), "inter": 256 * rng.randint(22, 100), "type": t, "m": rng.randint(1, 16),
                    "x": "bf16", "y": "f32", "layers": rng.randint(2, 16)}
        else:
            head = 128
            heads, kv = rng.choice([(16, 2), (24, 8), (32, 8), (40, 8), (64, 8)])
            case = {"kind": kind, "type": rng.choice(["Q4_K", "Q4_K", "Q5_K", "Q8_0"]), "m": m}
            case["type_down"] = rng.choice(["Q6_K", case["type"]])
            if case["type"] == "Q8_0":
                case["type_down"] = "Q8_0"
            case.update(hidden=256 * rng.randint(8, 24), q_rows=heads * head, kv_rows=kv * head, inter=256 * rng.randint(22, 100))
            if kind == "chain":
                case.update(m=rng.randint(1, 2), layers=rng.randint(1, 4))
            else:
                case.update(x="bf16", y=y, layers=1 if m >= 128 else rng.randint(1, 3))
        if _cost(case) <= limit:
            return case


# ---- what a program has in hand -----------------------------------------------------------------

_BACKEND = None


def _backend():
    """One backend per process, as in an engine."""
    global _BACKEND
    if _BACKEND is None:
        _BACKEND = mb.Backend(0)
    return _BACKEND


def _rows(rng, t, n, k):
    """N(0, 0.02) rows through the library's reference quantizer.  A few hundred distinct rows are drawn and every
    row of the matrix is one of them, so that a large matrix is made quickly; the library treats all rows alike."""
    base = rng.standard_normal((min(n, 307), k), dtype=np.float32) * np.float32(0.02)
    packed = mb.quantize(_TYPES[t], base)
    return packed, rng.integers(0, len(base), n)


def _weight(be, rng, t, n, k):
    packed, index = _rows(rng, t, n, k)
    return be.upload(_TYPES[t], packed[index], n, k)


def _acts(gen, m, k, dtype):
    """N(0, 1) activations with one channel in a hundred twenty times larger, as hidden states have them."""
    x = torch.randn((m, k), generator=gen, device="cuda")
    big = torch.randperm(k, generator=gen, device="cuda")[: max(1, k // 100)]
    x[:, big] *= 20.0
    return x.to(_DTYPES[dtype])


def _layer_shapes(c):
    h, i, t, td = c["hidden"], c["inter"], c["type"], c["type_down"]
    return {"q": (t, c["q_rows"], h), "k": (t, c["kv_rows"], h), "v": (td, c["kv_rows"], h), "o": (t, h, c["q_rows"]),
            "gate": (t, i, h), "up": (t, i, h), "down": (td, h, i)}


def _layer_weights(be, rng, c):
    first = {name: _weight(be, rng, *s) for name, s in _layer_shapes(c).items()}
    # further layers hold the same values in memory of their own: every layer is read from HBM
    return [first] + [{name: w.clone() for name, w in first.items()} for _ in range(c["layers"] - 1)]


def prepare(case, seed):
    be = _backend()
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    c = dict(case)
    kind, m = c["kind"], c["m"]
    s = {"kind": kind, "be": be}
    if kind in ("call", "plan"):
        w = _weight(be, rng, c["type"], c["n"], c["k"])
        s["w"] = [w] + [w.clone() for _ in range(c["copies"] - 1)]
        s["x"] = [_acts(gen, m, c["k"], c["x"]) for _ in s["w"]]
        s["y"] = [torch.empty((m, c["n"]), dtype=_DTYPES[c["y"]], device="cuda") for _ in s["w"]]
        if kind == "plan":
            s["plan"] = be.plan([([w], x, [y]) for w, x, y in zip(s["w"], s["x"], s["y"])])
    elif kind == "host":
        s["w"] = _weight(be, rng, c["type"], c["n"], c["k"])
        x = _acts(gen, m, c["k"], c["x"]).cpu()
        s["x"] = x.view(torch.uint16).numpy() if c["x"] == "bf16" else x.numpy()
        s["xt"] = mb.TYPE_BF16 if c["x"] == "bf16" else mb.TYPE_F32
        s["yt"] = mb.TYPE_BF16 if c["y"] == "bf16" else mb.TYPE_F32
        s["y"] = np.zeros((m, c["n"]), dtype=np.uint16 if c["y"] == "bf16" else np.float32)
        s["bf16_out"] = c["y"] == "bf16"
    elif kind == "mlp_plan":
        h, i = c["hidden"], c["inter"]
        first = (_weight(be, rng, c["type"], i, h), _weight(be, rng, c["type"], i, h), _weight(be, rng, c["type"], h, i))
        layers = [first] + [tuple(w.clone() for w in first) for _ in range(c["layers"] - 1)]
        s["y"] = [torch.empty((c["layers"], m, n), dtype=_DTYPES[c["y"]], device="cuda") for n in (i, i, h)]
        jobs = []
        for (gate, up, down), g, u, d in zip(layers, *s["y"]):
            jobs += [([gate, up], _acts(gen, m, h, c["x"]), [g, u]), ([down], _acts(gen, m, i, c["x"]), [d])]
        s["plan"] = be.plan(jobs)
    elif kind == "chain":
        h, i = c["hidden"], c["inter"]
        s["embedding"] = torch.randn((m, h), generator=gen, device="cuda")
        s["stream"] = torch.empty((m, h), device="cuda")
        s["plans"], s["y"] = [], []
        for w in _layer_weights(be, rng, c):
            norm1, norm2 = (1.0 + 0.1 * torch.randn(h, generator=gen, device="cuda") for _ in range(2))
            q, k, v = (torch.empty((m, w[p].n), device="cuda") for p in ("q", "k", "v"))
            attn = _acts(gen, m, c["q_rows"], "f32") * 0.1          # what attention would have made of q, k and v
            act = torch.empty((m, i), device="cuda")
            same = c["type"] == c["type_down"]
            qkv = [([w["q"], w["k"], w["v"]], s["stream"], [q, k, v])] if same else \
                [([w["q"], w["k"]], s["stream"], [q, k]), ([w["v"]], s["stream"], [v])]
            a = be.plan(qkv, norms=[norm1] * len(qkv))
            b = be.plan([([w["o"]], attn, [s["stream"]]), ([w["gate"], w["up"]], s["stream"], [act]), ([w["down"]], act, [s["stream"]])],
                        waits=[False, True, True], swiglu=[False, True, False], accumulate=[True, False, True], norms=[None, norm2, None])
            s["plans"] += [a, b]
            s["y"] += [q, k, v, act]
    elif kind == "layer":
        s["w"] = _layer_weights(be, rng, c)
        s["x"] = {"hidden": _acts(gen, m, c["hidden"], c["x"]), "attn": _acts(gen, m, c["q_rows"], c["x"]), "act": _acts(gen, m, c["inter"], c["x"])}
        new = lambda w: torch.empty((m, w.n), dtype=_DTYPES[c["y"]], device="cuda")  # noqa: E731
        s["y"] = [{name: new(w) for name, w in layer.items()} for layer in s["w"]]
        s["same"] = c["type"] == c["type_down"]
    else:
        raise ValueError(f"unknown kind {kind!r}")
    return s


# ---- one pass -------------------------------------------------------------------------------------

def run(s):
    be, kind = s["be"], s["kind"]
    if kind == "call":
        for w, x, y in zip(s["w"], s["x"], s["y"]):
            be.project(w, x, out=y)
        return s["y"]
    if kind in ("plan", "mlp_plan"):
        s["plan"].run()
        return s["y"]
    if kind == "host":
        y = be.project_host(s["w"], s["x"], s["xt"], s["y"], s["yt"])
        return (y.astype(np.uint32) << 16).view(np.float32) if s["bf16_out"] else y
    if kind == "chain":
        s["stream"].copy_(s["embedding"])
        for plan in s["plans"]:
            plan.run()
        return {"stream": s["stream"], "parts": s["y"]}
    for w, y in zip(s["w"], s["y"]):
        x = s["x"]
        if s["same"]:
            be.project_multi([w["q"], w["k"], w["v"]], x["hidden"], [y["q"], y["k"], y["v"]])
        else:
            be.project_multi([w["q"], w["k"]], x["hidden"], [y["q"], y["k"]])
            be.project(w["v"], x["hidden"], out=y["v"])
        be.project(w["o"], x["attn"], out=y["o"])
        be.project_multi([w["gate"], w["up"]], x["hidden"], [y["gate"], y["up"]])
        be.project(w["down"], x["act"], out=y["down"])
    return s["y"]


# ---- the same results in 64 bits ---------------------------------------------------------------------

_E2M1 = [0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0, -0.0, -0.5, -1.0, -1.5, -2.0, -3.0, -4.0, -6.0]


def _values(t, packed, k):
    """The weights that rows of GGUF blocks stand for, [rows][k] in 64 bits."""
    elems, size = _BLOCK[t]
    b = torch.from_numpy(np.ascontiguousarray(packed).view(np.uint8).reshape(-1, size)).cuda()
    half = lambda at: b[:, at:at + 2].contiguous().view(torch.float16).double()  # noqa: E731
    nibbles = lambda q: torch.cat([q & 15, q >> 4], dim=-1)                       # noqa: E731
    if t == "Q8_0":
        v = half(0) * b[:, 2:].contiguous().view(torch.int8).double()
    elif t == "Q4_0":
        v = half(0) * (nibbles(b[:, 2:]).double() - 8)
    elif t == "MXFP4":
        v = torch.exp2(b[:, :1].double() - 127) * torch.tensor(_E2M1, device="cuda", dtype=torch.float64)[nibbles(b[:, 1:]).long()]
    elif t in ("Q4_K", "Q5_K"):
        s = b[:, 4:16]
        scale = torch.cat([s[:, :4] & 63, (s[:, 8:] & 15) | (s[:, :4] >> 6 << 4)], dim=1).double()
        least = torch.cat([s[:, 4:8] & 63, (s[:, 8:] >> 4) | (s[:, 4:8] >> 6 << 4)], dim=1).double()
        q = nibbles(b[:, size - 128:].reshape(-1, 4, 32)).reshape(-1, 8, 32)
        if t == "Q5_K":
            q = q | ((b[:, None, 16:48] >> torch.arange(8, device="cuda", dtype=torch.uint8)[None, :, None]) & 1) << 4
        v = (half(0) * scale)[:, :, None] * q.double() - (half(2) * least)[:, :, None]
    else:  # Q6_K: two halves of 128 weights, each four runs of 32
        low = nibbles(b[:, :128].reshape(-1, 2, 64)).reshape(-1, 2, 4, 32)
        high = (b[:, 128:192].reshape(-1, 2, 1, 32) >> torch.tensor([0, 2, 4, 6], device="cuda", dtype=torch.uint8)[None, None, :, None]) & 3
        scale = half(208) * b[:, 192:208].contiguous().view(torch.int8).double()
        v = scale[:, :, None] * ((low | high << 4).reshape(-1, 16, 16).double() - 32)
    return v.reshape(-1, k)


class _Weight64:
    def __init__(self, rng, t, n, k):
        packed, index = _rows(rng, t, n, k)
        self.v, self.index, self.n = _values(t, packed, k), torch.from_numpy(index).cuda(), n

    def __call__(self, x):
        return (x.double() @ self.v.T)[:, self.index]


def exact(case, seed):
    """What `run` returns on the state of `prepare(case, seed)`, from the same draws, in 64 bits."""
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    c = dict(case)
    kind, m = c["kind"], c["m"]
    if kind in ("call", "plan"):
        w = _Weight64(rng, c["type"], c["n"], c["k"])
        return [w(_acts(gen, m, c["k"], c["x"])) for _ in range(c["copies"])]
    if kind == "host":
        w = _Weight64(rng, c["type"], c["n"], c["k"])
        return w(_acts(gen, m, c["k"], c["x"])).cpu().numpy()
    if kind == "mlp_plan":
        h, i = c["hidden"], c["inter"]
        gate, up, down = _Weight64(rng, c["type"], i, h), _Weight64(rng, c["type"], i, h), _Weight64(rng, c["type"], h, i)
        y = ([], [], [])
        for _ in range(c["layers"]):
            x = _acts(gen, m, h, c["x"])
            y[0].append(gate(x))
            y[1].append(up(x))
            y[2].append(down(_acts(gen, m, i, c["x"])))
        return [torch.stack(v) for v in y]
    if kind == "chain":
        h = c["hidden"]
        stream = torch.randn((m, h), generator=gen, device="cuda").double()
        w = {name: _Weight64(rng, *s) for name, s in _layer_shapes(c).items()}
        normed = lambda x, g: x * torch.rsqrt((x * x).mean(dim=1, keepdim=True) + 1e-5) * g.double()  # noqa: E731
        parts = []
        for _ in range(c["layers"]):
            norm1, norm2 = (1.0 + 0.1 * torch.randn(h, generator=gen, device="cuda") for _ in range(2))
            attn = _acts(gen, m, c["q_rows"], "f32") * 0.1
            x = normed(stream, norm1)
            parts += [w["q"](x), w["k"](x), w["v"](x)]
            stream = stream + w["o"](attn)
            x = normed(stream, norm2)
            act = torch.nn.functional.silu(w["gate"](x)) * w["up"](x)
            parts.append(act)
            stream = stream + w["down"](act)
        return {"stream": stream, "parts": parts}
    w = {name: _Weight64(rng, *s) for name, s in _layer_shapes(c).items()}
    x = {"hidden": _acts(gen, m, c["hidden"], c["x"]), "attn": _acts(gen, m, c["q_rows"], c["x"]), "act": _acts(gen, m, c["inter"], c["x"])}
    source = {"o": "attn", "down": "act"}
    y = {name: p(x[source.get(name, "hidden")]) for name, p in w.items()}
    return [y] * c["layers"]


# ---- what a pass cannot do without ------------------------------------------------------------------

def _products(c):
    """(type, n, k, bytes of x counted here, bytes of y) of every product of a pass."""
    kind, m = c["kind"], c["m"]
    if kind in ("call", "plan", "host"):
        n, k = c["n"], c["k"]
        return [(c["type"], n, k, m * k * _SIZE[c["x"]], m * n * _SIZE[c["y"]])] * c.get("copies", 1)
    h, i = c["hidden"], c["inter"]
    if kind == "mlp_plan":
        t, xs, ys = c["type"], _SIZE[c["x"]], _SIZE[c["y"]]
        return [(t, i, h, m * h * xs, m * i * ys), (t, i, h, 0, m * i * ys), (t, h, i, m * i * xs, m * h * ys)] * c["layers"]
    xs, ys = _SIZE[c.get("x", "f32")], _SIZE[c.get("y", "f32")]
    t, td, q, kv = c["type"], c["type_down"], c["q_rows"], c["kv_rows"]
    # q, k, v, gate and up read the same hidden state
    one = [(t, q, h, m * h * xs, m * q * ys), (t, kv, h, 0, m * kv * ys), (td, kv, h, 0, m * kv * ys), (t, h, q, m * q * xs, m * h * ys),
           (t, i, h, 0, m * i * ys), (t, i, h, 0, m * i * ys), (td, h, i, m * i * xs, m * h * ys)]
    if kind == "chain":      # the activated product of gate and up is stored once, the residual stream read and written
        one[4] = (t, i, h, m * h * xs, m * i * ys)
        one[5] = (t, i, h, 0, 0)
    return one * c["layers"]


def work(case):
    nbytes = flops = 0.0
    for t, n, k, xb, yb in _products(case):
        elems, size = _BLOCK[t]
        nbytes += n * (k // elems) * size + xb + yb
        flops += 2.0 * case["m"] * n * k
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Four times the error seen against the product in 64 bits (rel: 2-norm, max: over max(|value|, rms))."""
    if case.get("y") == "bf16":
        return {"rel": 6.8e-3, "max": 2e-2}       # a bf16 result: seen 1.7e-3 and 5.1e-3
    if case["kind"] == "chain":
        return {"rel": 6e-4, "max": 6e-3}         # four layers of 16-bit fixed-point activations: seen 1.4e-4 and 1.5e-3
    if case["m"] <= _STREAMING:
        return {"rel": 2e-4, "max": 7e-4}         # activations in 16-bit fixed point: seen 4.9e-5 and 1.8e-4
    if case["m"] <= _EXACT:
        return {"rel": 1.2e-5, "max": 4e-5}       # exact integer weights, 32-bit sums: seen 3e-6 and 9.2e-6
    return {"rel": 1.2e-3, "max": 6e-3}           # both operands 16-bit floats: seen 3e-4 and 1.5e-3
