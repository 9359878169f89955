"""The work a program has this library do, as cases that can be timed: MoE expert layers of a decoder, through the public
classes of project_maya_b200.api.

A case is one pass of one kind of call:

  token   one decode token through `layers` resident layers (api.MoeLayer.forward, single token).  With `producer` each layer
          is the two-call decode layer - api.rms_router on the residual stream, then the layer on the x and logits it wrote -
          and with `residual` the layer also writes its output into the residual stack (hc).
  window  2..16 tokens of concurrent or speculative decode through `layers` layers (api.MoeLayer.forward).
  chunk   a prompt chunk, or a decode batch beyond 16 tokens, through one layer (api.MoePrefill.forward).

`graph` replays the pass as a CUDA graph captured once, as serving loops do; without it every pass is made of eager calls.
Weights are valid GGUF blocks: N(0, 0.02) values quantized by the library for Q8_0, Q4_K, IQ2_S and IQ3_S, random codes under
small super-scales for the other types.  Activations are N(0, 1); router logits are N(0, 1), with `zipf` > 0 plus the
log-probabilities of a Zipf law over a shuffled expert order (a few experts take most tokens, as trained routers show).
"""
from __future__ import annotations

import math

import numpy as np
import torch

from project_maya_b200 import api, synthetic

TYPES = {"Q8_0": api.Q8_0, "Q4_K": api.Q4_K, "IQ2_S": api.IQ2_S, "IQ3_S": api.IQ3_S, "Q5_K": api.Q5_K, "Q6_K": api.Q6_K,
         "IQ4_XS": api.IQ4_XS, "IQ3_XXS": api.IQ3_XXS, "IQ2_XXS": api.IQ2_XXS, "IQ1_S": api.IQ1_S}
CORE = ("Q8_0", "Q4_K", "IQ2_S", "IQ3_S")
# random codes need a super-scale that leaves weights of about 0.02: its place(s) in the block and its range
SCALES = {"Q5_K": ((0, 2), 5e-5, 2e-4), "Q6_K": ((208,), 1e-5, 3e-5), "IQ4_XS": ((0,), 1e-5, 3e-5), "IQ3_XXS": ((0,), 2e-4, 6e-4),
          "IQ2_XXS": ((0,), 2e-4, 6e-4), "IQ1_S": ((0,), 2e-3, 6e-3)}
# gate/up and down types that files mix: the down rows a step wider, as the usual quantization recipes store them
MIXES = (("Q4_K", "Q6_K"), ("Q5_K", "Q6_K"), ("IQ3_XXS", "IQ4_XS"), ("IQ2_XXS", "IQ3_XXS"), ("IQ1_S", "IQ2_XXS"), ("IQ2_S", "IQ3_S"))
MOST_BYTES = 7.6e9      # resident expert bytes of a case: what the largest listed layer holds
MOST_FLOPS = 2.4e12     # and its work


def _case(kind, T, H, FF, E, k, gu, d, **more):
    c = dict(kind=kind, T=T, H=H, FF=FF, E=E, k=k, gu=gu, d=d, half="", shared=0, act="bf16", router="softmax", zipf=0.0,
             layers=1, producer=False, residual=False, limit=0.0, graph=False)
    c.update(more)
    return c


def listed():
    return [
        # the smallest call: one token, one layer of a small model (28 MB of experts read), called eagerly - launches and host work
        dict(_case("token", 1, 2048, 1024, 64, 8, "Q4_K", "Q4_K", act="f32"), name="token_small"),
        # a mid-size model stored by the common 4-bit recipe (6-bit down rows), both calls of a decode layer, two layers
        dict(_case("token", 1, 4096, 1536, 128, 8, "Q4_K", "Q6_K", act="f32", layers=2, producer=True), name="token_mixed"),
        # the headline decode layer: 2-bit routed experts and an always-on 8-bit shared expert
        dict(_case("token", 1, 6144, 2048, 256, 8, "IQ2_S", "IQ2_S", shared=2048, zipf=1.1), name="token_shared"),
        # the serving form of decode: producer + layer of two 3-bit layers, replayed as a graph
        dict(_case("token", 1, 6144, 2048, 256, 8, "IQ3_S", "IQ3_S", layers=2, producer=True, graph=True), name="token_graph"),
        # sigmoid routing with a selection bias, clamped SwiGLU, odd k, and the residual-stack write: every option of the layer
        dict(_case("token", 1, 5120, 1536, 160, 6, "Q8_0", "Q8_0", shared=3072, router="sigmoid", limit=7.0, residual=True),
             name="token_sigmoid"),
        # the smallest window: a token and one draft token of the headline layer, shared expert included
        dict(_case("window", 2, 6144, 2048, 256, 8, "IQ2_S", "IQ2_S", shared=2048, zipf=1.1), name="window_2_shared"),
        # a speculative window of odd length over a mid-size model's 3/4-bit recipe
        dict(_case("window", 5, 4096, 1536, 128, 8, "IQ3_XXS", "IQ4_XS", act="f32"), name="window_5_mixed"),
        # eight concurrent streams, 4-bit experts, skewed routing, replayed as a graph
        dict(_case("window", 8, 7168, 2048, 256, 8, "Q4_K", "Q4_K", zipf=1.1, graph=True), name="window_8"),
        # the largest window: sixteen streams over 3-bit experts
        dict(_case("window", 16, 6144, 2048, 256, 8, "IQ3_S", "IQ3_S", zipf=1.1), name="window_16"),
        # a decode batch of 64 streams
        dict(_case("chunk", 64, 6144, 2048, 256, 8, "IQ3_S", "IQ3_S", zipf=1.1), name="chunk_64"),
        # a prompt of ragged length through the headline layer
        dict(_case("chunk", 777, 6144, 2048, 256, 8, "IQ2_S", "IQ2_S", shared=2048, zipf=1.1), name="chunk_777_shared"),
        # the largest: a full prompt chunk over a layer whose experts are half 8-bit, half 4-bit
        dict(_case("chunk", 4096, 6144, 2048, 256, 8, "Q8_0", "Q8_0", half="Q4_K"), name="chunk_4096"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _row(t, n):
    qk, nbytes = synthetic.BLOCK[TYPES[t]]
    return n // qk * nbytes


def _blob(c, gu, d):
    return 2 * c["FF"] * _row(gu, c["H"]) + c["H"] * _row(d, c["FF"])


def draw(rng):
    kind = rng.choice(("token", "window", "chunk"))
    half = ""
    if kind == "chunk":
        gu = d = rng.choice(CORE)
        if gu in ("Q8_0", "Q4_K"):
            H, FF = 256 * _log_int(rng, 4, 32), 256 * _log_int(rng, 2, 12)
            if rng.random() < 0.3:
                half = "Q4_K" if gu == "Q8_0" else "Q8_0"
        else:                                   # rows of 2-byte aligned blocks: whole multiples of 2048 values
            H, FF = 2048 * rng.randint(1, 4), 2048
        T = _log_int(rng, 17, 4096)
    else:
        gu, d = rng.choice(MIXES) if rng.random() < 0.4 else (rng.choice(CORE),) * 2
        step = 32 if gu == "Q8_0" else 256
        H, FF = step * _log_int(rng, 1024 // step, 8192 // step), step * _log_int(rng, 512 // step, 3072 // step)
        T = 1 if kind == "token" else _log_int(rng, 2, 16)
    k = 8 if rng.random() < 0.6 else rng.randint(1, 8)
    c = _case(kind, T, H, FF, 0, k, gu, d, half=half)
    big = max(_blob(c, t, t if kind == "chunk" else d) for t in (gu, half or gu))
    c["E"] = max(k, min(_log_int(rng, 8, 512), int(MOST_BYTES / big)))
    c["T"] = max(1, min(T, int(MOST_FLOPS / (6 * H * FF * k))))
    c["act"] = rng.choice(("f32", "bf16"))
    c["zipf"] = rng.choice((0.0, 1.1))
    c["limit"] = rng.choice((0.0, 0.0, 7.0))
    if rng.random() < 0.4:
        c["shared"] = 256 * rng.randint(2, 12)
    if kind != "chunk":
        c["router"] = rng.choice(("softmax", "softmax", "sigmoid"))
        c["graph"] = rng.random() < 0.4
    if kind == "token":
        c["producer"] = rng.random() < 0.4
        c["residual"] = rng.random() < 0.3
    return c


# ---------------------------------------------------------------------------------------------------------- inputs
def _fill(t, rows, seed, gen):
    """rows: uint8 [n, bytes] (rows contiguous, n of them spaced by their stride): every row filled with blocks of type t."""
    qk, nbytes = synthetic.BLOCK[TYPES[t]]
    n, row = rows.shape
    if t in CORE:                               # 256 values at a time: the generator's unit
        if rows.is_contiguous():
            api.synth_weights(TYPES[t], seed, 0.02, n * row // nbytes * qk // 256, 256, rows)
        else:
            for i in range(n):
                api.synth_weights(TYPES[t], seed + i, 0.02, row // nbytes * qk // 256, 256, rows[i])
        return
    places, lo, hi = SCALES[t]
    b = torch.randint(0, 256, (n * row // nbytes, nbytes), dtype=torch.uint8, device="cuda", generator=gen)
    for at in places:
        s = torch.rand(b.shape[0], device="cuda", generator=gen) * (hi - lo) + lo
        b[:, at:at + 2] = s.half().view(torch.uint8).view(-1, 2)
    rows.copy_(b.view(n, row))


def _experts(c, n, gu, d, seed, gen):
    e = torch.empty((n, _blob(c, gu, d)), dtype=torch.uint8, device="cuda")
    if gu == d:
        _fill(gu, e, seed, gen)
    else:
        at = 2 * c["FF"] * _row(gu, c["H"])
        _fill(gu, e[:, :at], seed, gen)
        _fill(d, e[:, at:], seed + 500000, gen)
    return e


def _logits(c, gen):
    l = torch.randn((c["T"], c["E"]), device="cuda", generator=gen)
    if c["zipf"]:
        pmf = torch.arange(1, c["E"] + 1, device="cuda", dtype=torch.float32) ** -c["zipf"]
        bias = torch.log(pmf) - torch.log(pmf).mean()
        l += bias[torch.randperm(c["E"], device="cuda", generator=gen)]
    return l


def _layer(c, seed, gen):
    """One resident layer and its inputs."""
    H, FF, E, T = c["H"], c["FF"], c["E"], c["T"]
    limit = c["limit"] or api.INF
    cfg = api.MoeLayerConfig(H, FF, E, c["k"], TYPES[c["gu"]], TYPES[c["d"]], n_ff_sh=c["shared"], limit=limit)
    randn = lambda *shape: torch.randn(shape, device="cuda", generator=gen)  # noqa: E731
    shared = None
    if c["shared"]:
        shared = torch.empty((1, cfg.shared_bytes), dtype=torch.uint8, device="cuda")
        _fill("Q8_0", shared, seed + 900000, gen)
        shared = shared[0]
    s = {"c": c, "logits": _logits(c, gen), "x": randn(T, H).to(torch.bfloat16 if c["act"] == "bf16" else torch.float32)}
    if c["kind"] == "chunk":
        if c["half"]:
            order = torch.randperm(E, device="cuda", generator=gen).tolist()
            pools = []
            for i, t in enumerate((c["gu"], c["half"])):
                members = sorted(order[i * E // 2:(i + 1) * E // 2])
                if members:
                    pools.append((TYPES[t], _experts(c, len(members), t, t, seed + 100000 * i, gen), members))
            s["layer"] = api.MoePrefill(cfg, None, shared, max_tokens=T, pools=pools)
        else:
            s["layer"] = api.MoePrefill(cfg, _experts(c, E, c["gu"], c["d"], seed, gen), shared, max_tokens=T)
        return s
    sigmoid = (randn(E) * 0.1, 2.5, True) if c["router"] == "sigmoid" else None
    s["layer"] = api.MoeLayer(cfg, _experts(c, E, c["gu"], c["d"], seed, gen), shared, max_tokens=T, sigmoid=sigmoid)
    if c["producer"]:
        s.update(h=randn(H), add=randn(H) * 0.1, norm=1.0 + 0.1 * randn(H), router=(randn(E, H) / math.sqrt(H)).to(torch.bfloat16),
                 h_out=torch.empty(H, device="cuda"))
    if c["residual"]:
        s["hc"] = (randn(T, 4, H), torch.sigmoid(randn(T, 4)), torch.softmax(randn(T, 4, 4), -1), torch.empty((T, 4, H), device="cuda"))
    return s


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    layers = [_layer(case, (seed * 16 + i) * 1000003, gen) for i in range(case["layers"])]
    if not case["graph"]:
        return {"layers": layers}
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        _pass(layers)
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        out = _pass(layers)
    return {"layers": layers, "graph": graph, "out": out}


# ------------------------------------------------------------------------------------------------------------ a pass
def _pass(layers):
    out = []
    for s in layers:
        logits, x = s["logits"], s["x"]
        if "router" in s:
            xv, lv = api.rms_router(s["h"], s["add"], s["norm"], 1e-6, s["router"], h_out=s["h_out"])
            out += [xv, lv, s["h_out"]]
            logits, x = lv.view(1, -1), xv.view(1, -1)
        if "hc" in s:
            out += [*s["layer"].forward(logits, x, hc=s["hc"]), s["hc"][3]]
        else:
            out += s["layer"].forward(logits, x)
    return out


def run(state):
    if "graph" in state:
        state["graph"].replay()
        return state["out"]
    return _pass(state["layers"])


# ------------------------------------------------------------------------------------------------- work and precision
def _distinct(c):
    """Experts that a pass reads, on average over routings drawn as the inputs are."""
    rng = np.random.default_rng(1)
    n = 0
    for _ in range(4):
        l = rng.standard_normal((c["T"], c["E"]))
        if c["zipf"] and not c["producer"]:
            l += np.log(np.arange(1, c["E"] + 1, dtype=np.float64) ** -c["zipf"])
        n += np.unique(np.argpartition(-l, c["k"] - 1, axis=1)[:, :c["k"]]).size
    return n / 4


def work(case):
    c, T, H, FF, E = case, case["T"], case["H"], case["FF"], case["E"]
    blob = _blob(c, c["gu"], c["d"])
    if c["half"]:
        blob = (blob + _blob(c, c["half"], c["half"])) / 2
    bytes_ = _distinct(c) * blob + T * (4 * E + H * (4 if c["act"] == "f32" else 2) + 8 * c["k"] + 4 * H)
    flops = 6 * T * c["k"] * H * FF
    if c["shared"]:
        bytes_ += 3 * c["shared"] * _row("Q8_0", H)
        flops += 6 * T * H * c["shared"]
    if c["producer"]:
        bytes_ += 2 * E * H + 16 * H
        flops += 2 * E * H
    if c["residual"]:
        bytes_ += T * 32 * H
        flops += T * 40 * H
    return {"bytes": c["layers"] * bytes_, "flops": c["layers"] * flops}


def tolerance(case):
    # Expert ids are exact.  Decode: activations and h are rounded to 8-bit blocks, the dots over them are exact integers
    # and the rest is 32-bit: two correct orders of the sums differ by a few 1e-6, and where that moves a value of h across
    # a rounding boundary (about one in 1e4) by one step of 1/127 of its block's largest - 2e-4 of the result in all.
    # Chunks multiply f16 operands (rounding 5e-4) after the same 8-bit rounding.
    return {"rel": 1e-3 if case["kind"] == "chunk" else 2e-4, "max": 2e-2 if case["kind"] == "chunk" else 4e-3, "differ": 0.0}
