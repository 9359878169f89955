"""The whole decode layer (route -> experts -> combine, shared expert alongside) through maya_moe_layer_decode, on
the benchmark configurations: C1 in full against the committed fixtures; C2 / C3 / C5 at their full shapes on
synthetic device-generated experts, checked against the oracle on the experts each token actually routed, and
through size-independent properties (window == token by token bit for bit; the expert-parallel partition's partial
outputs sum to the unpartitioned output)."""
import hashlib
import sys
from pathlib import Path

import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu
GOLDEN = Path(__file__).resolve().parent / "golden"
TOL, TIGHT = 1e-2, 2e-4


@pytest.fixture(scope="module")
def T(cuda):
    import torch
    return torch


@pytest.fixture(scope="module")
def api(cuda):
    from project_maya_b200 import api as a
    return a


def dev(T, a, dtype=None):
    t = T.from_numpy(np.ascontiguousarray(a))
    if dtype is not None:
        t = t.to(dtype)
    return t.cuda()


def layer_cfg(api, cfg, with_shared=True):
    return api.MoeLayerConfig(cfg["n_embd"], cfg["n_ff"], cfg["n_expert"], cfg["k"], cfg["gu_type"], cfg["d_type"],
                              cfg.get("n_ff_sh", 0) if with_shared else 0, cfg.get("sh_gu_type", H.Q8_0),
                              cfg.get("sh_d_type", H.Q8_0), cfg.get("limit", H.INF))


def synth_layer(T, api, cfg, n_expert, seed):
    """n_expert synthetic experts (N(0, 0.02) quantized on the device) + the shared expert when the config has one."""
    lc = layer_cfg(api, dict(cfg, n_expert=n_expert))
    experts = T.empty((n_expert, lc.blob_bytes), dtype=T.uint8, device="cuda")
    H_, FF = cfg["n_embd"], cfg["n_ff"]
    gu_bytes = 2 * FF * H.row_bytes(cfg["gu_type"], H_)
    for e in range(n_expert):
        api.synth_weights(cfg["gu_type"], seed * 100003 + 2 * e, 0.02, 2 * FF, H_, experts[e, :gu_bytes])
        api.synth_weights(cfg["d_type"], seed * 100003 + 2 * e + 1, 0.02, H_, FF, experts[e, gu_bytes:])
    shared = None
    if cfg.get("n_ff_sh"):
        shared = T.empty(lc.shared_bytes, dtype=T.uint8, device="cuda")
        sgu = 2 * cfg["n_ff_sh"] * H.row_bytes(cfg["sh_gu_type"], H_)
        api.synth_weights(cfg["sh_gu_type"], seed * 7 + 1, 0.02, 2 * cfg["n_ff_sh"], H_, shared[:sgu])
        api.synth_weights(cfg["sh_d_type"], seed * 7 + 2, 0.02, H_, cfg["n_ff_sh"], shared[sgu:])
    T.cuda.synchronize()
    return lc, experts, shared


def oracle_token(oracle, cfg, experts, shared, ids, w, x, limit=H.INF):
    """The oracle on one token, given the routing: only the routed experts' blobs are brought to the host."""
    H_, FF, k = cfg["n_embd"], cfg["n_ff"], cfg["k"]
    xq = oracle.quantize_q8_1(x)
    parts = np.stack([oracle.expert_q8_1(cfg["gu_type"], cfg["d_type"], experts[int(e)].cpu().numpy(), H_, FF, limit, xq)
                      for e in ids])
    sh = None
    if shared is not None:
        sh = oracle.expert_q8_1(cfg["sh_gu_type"], cfg["sh_d_type"], shared.cpu().numpy(), H_, cfg["n_ff_sh"], limit, xq)
    return oracle.combine_down(parts, w, sh)


def test_c1_full_against_fixtures(T, api, oracle):
    sys.path.insert(0, str(GOLDEN))
    import make_golden
    g = np.load(GOLDEN / "c1_reference_cpu.npz")
    cfg = H.CONFIGS["C1"]
    blobs = make_golden.c1_experts()
    assert hashlib.sha256(blobs.tobytes()).hexdigest() == str(g["experts_sha256"])
    layer = api.MoeLayer(layer_cfg(api, cfg), dev(T, blobs))
    logits = H.router_logits("C1", cfg["tokens"], cfg["n_expert"], None)
    x = H.activations("C1", cfg["tokens"], cfg["n_embd"], "f32")
    for t in range(cfg["tokens"]):                      # batch 1, 16 seeded tokens
        ids, w, out = layer.forward(dev(T, logits[t:t + 1]), dev(T, x[t:t + 1]))
        assert np.array_equal(ids.cpu().numpy()[0], g["ids"][t])                       # routing bit-exact
        assert (np.abs(w.cpu().numpy()[0] - g["weights"][t]) / g["weights"][t]).max() <= 1e-5
        o = out.cpu().numpy()[0]
        assert H.rel_err(o, g["out_oracle_q8_1"][t]) <= TOL
        assert H.rel_err(o, g["out_oracle_q8_1"][t]) <= TIGHT
        # against the reference's CPU rows (Q8_K activations): the gate the reference holds its own two paths to
        assert H.rel_err(o, g["out_cpu_rows"][t]) <= 3e-2
    # the same 16 tokens as one window: the same bits
    ids16, w16, out16 = layer.forward(dev(T, logits), dev(T, x))
    for t in range(cfg["tokens"]):
        _, _, one = layer.forward(dev(T, logits[t:t + 1]), dev(T, x[t:t + 1]))
        assert T.equal(out16[t], one[0])


@pytest.mark.parametrize("name,n_tok_check", [("C2", 3), ("C5", 2)])
def test_full_shape_single_token(T, api, oracle, name, n_tok_check):
    cfg = H.CONFIGS[name]
    lc, experts, shared = synth_layer(T, api, cfg, cfg["n_expert"], seed=11)
    layer = api.MoeLayer(lc, experts, shared)
    logits = H.router_logits(name, 8, cfg["n_expert"], cfg.get("zipf"))
    x = H.activations(name, 8, cfg["n_embd"], cfg["act"])
    ids_o, w_o = oracle.router_top10(logits, cfg["k"])
    for t in range(n_tok_check):
        xd = dev(T, x[t:t + 1], T.bfloat16)
        ids, w, out = layer.forward(dev(T, logits[t:t + 1]), xd)
        assert np.array_equal(ids.cpu().numpy()[0], ids_o[t])
        want = oracle_token(oracle, cfg, experts, shared, ids_o[t], w_o[t], x[t])
        got = out.cpu().numpy()[0]
        assert H.rel_err(got, want) <= TOL
        assert H.rel_err(got, want) <= TIGHT


def test_c3_window_of_eight(T, api, oracle):
    cfg = H.CONFIGS["C3"]
    n_expert = 64                                       # reduced expert count, full hidden / FFN widths
    lc, experts, _ = synth_layer(T, api, cfg, n_expert, seed=5)
    layer = api.MoeLayer(lc, experts)
    logits = H.router_logits("C3", 8, n_expert, cfg["zipf"])
    x = H.activations("C3", 8, cfg["n_embd"], "bf16")
    ids, w, out = layer.forward(dev(T, logits), dev(T, x, T.bfloat16))
    ids_o, w_o = oracle.router_top10(logits, cfg["k"])
    assert np.array_equal(ids.cpu().numpy(), ids_o)
    assert len(np.unique(ids_o)) < 8 * cfg["k"]         # the skew makes tokens share experts
    for t in range(8):
        _, _, one = layer.forward(dev(T, logits[t:t + 1]), dev(T, x[t:t + 1], T.bfloat16))
        assert T.equal(out[t], one[0])                  # window == token by token, bit for bit
    want = oracle_token(oracle, dict(cfg, n_expert=n_expert), experts, None, ids_o[0], w_o[0], x[0])
    assert H.rel_err(out[0].cpu().numpy(), want) <= TIGHT


def test_expert_parallel_partition_sums_to_whole(T, api, oracle):
    cfg = dict(H.CONFIGS["C5"], n_expert=32)
    lc, experts, _ = synth_layer(T, api, cfg, 32, seed=9)
    logits = H.router_logits("C5", 4, 32, 1.1)
    x = H.activations("C5", 4, cfg["n_embd"], "bf16")
    ld, xd = dev(T, logits), dev(T, x, T.bfloat16)
    _, _, whole = api.MoeLayer(lc, experts).forward(ld, xd)
    parts = []
    for n_ranks in (2, 8):
        per = 32 // n_ranks
        partial = [api.MoeLayer(lc, experts, expert_range=(r * per, (r + 1) * per)).forward(ld, xd)[2].cpu().numpy()
                   for r in range(n_ranks)]
        summed = np.stack([oracle.allreduce_in_order(np.stack([p[t] for p in partial])) for t in range(4)])
        parts.append(summed)
        assert H.rel_err(summed, whole.cpu().numpy()) <= 1e-5
    # a rank with none of a token's experts contributes exact zeros
    empty = api.MoeLayer(lc, experts, expert_range=(0, 0)).forward(ld, xd)[2]
    assert not bool(empty.any())


@pytest.mark.parametrize("n_ranks", [2, 8])
def test_width_sliced_shared_expert_sums_to_whole(T, api, oracle, n_ranks):
    """Expert-parallel ranks that each hold 1/n of the shared expert's FFN width (its gate/up rows and the same
    columns of the down rows): the rank-ordered sum of the partial outputs is the one-rank output up to the order of
    the shared expert's down sums; a slice that the staged kernels would have to run is refused."""
    cfg = dict(H.CONFIGS["C2"], n_expert=16)
    lc, experts, shared = synth_layer(T, api, cfg, 16, seed=21)
    logits = H.router_logits("C2", 3, 16, 1.1)
    x = H.activations("C2", 3, cfg["n_embd"], "bf16")
    ld, xd = dev(T, logits), dev(T, x, T.bfloat16)
    per, wid = 16 // n_ranks, cfg["n_ff_sh"] // n_ranks
    for t in range(3):
        whole = api.MoeLayer(lc, experts, shared).forward(ld[t:t + 1], xd[t:t + 1])[2].cpu().numpy()[0]
        partial = [api.MoeLayer(lc, experts, shared, expert_range=(r * per, (r + 1) * per),
                                shared_range=(r * wid, (r + 1) * wid)).forward(ld[t:t + 1], xd[t:t + 1])[2].cpu().numpy()[0]
                   for r in range(n_ranks)]
        summed = oracle.allreduce_in_order(np.stack(partial))
        assert H.rel_err(summed, whole) <= 1e-5
        assert np.abs(partial[-1]).max() > 0            # every rank carries a share
    sliced = api.MoeLayer(lc, experts, shared, shared_range=(0, wid))
    with pytest.raises(api.MayaError):
        sliced.forward(ld[:2], xd[:2])                   # two tokens: the staged kernels do not slice
    with pytest.raises(api.MayaError):
        api.MoeLayer(lc, experts, shared, shared_range=(16, wid)).forward(ld[:1], xd[:1])     # not a multiple of 32


@pytest.mark.parametrize("n_ranks", [2, 4, 8])
def test_width_sliced_experts_sum_to_whole(T, api, oracle, n_ranks):
    """Tensor-parallel ranks: every rank holds FFN rows [r * n_ff / N, (r + 1) * n_ff / N) of EVERY expert as blobs of
    their own (api.width_slice) and runs the same layer kernel on them; routing is replicated (same ids on every rank),
    the rank-ordered sum of the partial outputs is the one-rank output up to the order of the down sums.  At N = 8 a
    slice is one 256-value block wide."""
    cfg = dict(H.CONFIGS["C2"], n_expert=16)
    lc, experts, shared = synth_layer(T, api, cfg, 16, seed=23)
    logits = H.router_logits("C2", 3, 16, 1.1)
    x = H.activations("C2", 3, cfg["n_embd"], "bf16")
    ld, xd = dev(T, logits), dev(T, x, T.bfloat16)
    wid = cfg["n_ff"] // n_ranks
    ranks = []
    for r in range(n_ranks):
        c, ex, sh = api.width_slice(lc, experts, shared, r * wid, (r + 1) * wid)
        assert c.n_ff == wid and ex.shape == (16, c.blob_bytes) and sh.numel() == c.shared_bytes
        ranks.append(api.MoeLayer(c, ex, sh))
    whole_layer = api.MoeLayer(lc, experts, shared)
    for t in range(3):
        ids0, w0, whole = whole_layer.forward(ld[t:t + 1], xd[t:t + 1])
        parts = []
        for L in ranks:
            ids, w, out = L.forward(ld[t:t + 1], xd[t:t + 1])
            assert T.equal(ids, ids0) and T.equal(w, w0)
            parts.append(out.cpu().numpy()[0])
        assert H.rel_err(oracle.allreduce_in_order(np.stack(parts)), whole.cpu().numpy()[0]) <= 1e-5
        assert min(np.abs(p).max() for p in parts) > 0
    with pytest.raises(ValueError):
        api.width_slice(lc, experts, shared, 0, 100)       # not whole blocks


@pytest.mark.parametrize("t,shared", [(H.Q4_K, False), (H.Q8_0, False), (H.IQ2_S, True), (H.IQ3_S, True), (H.IQ3_S, False)])
@pytest.mark.parametrize("n_ff", [768, 256])
def test_fused_token_kernel_equals_staged_kernels_bitwise(T, api, oracle, t, shared, n_ff):
    """One token through the single fused kernel and through the separate launches: the same bits, and the oracle's
    values.  Odd sizes on purpose: the FFN and output rows do not divide evenly over the blocks.  FFN width 256 leaves
    fewer 32-row units than half the grid: the kernel then cuts every unit in two for two blocks."""
    n_embd, n_expert, k = 1024, 20, 6
    cfg = dict(n_embd=n_embd, n_ff=n_ff, n_expert=n_expert, k=k, gu_type=t, d_type=t, limit=7.0)
    if shared:
        cfg.update(n_ff_sh=512, sh_gu_type=H.Q8_0, sh_d_type=H.Q8_0)
    lc, experts, sh = synth_layer(T, api, cfg, n_expert, seed=21)
    lc.limit = 7.0
    fused = api.MoeLayer(lc, experts, sh, expert_range=(0, 17))
    staged = api.MoeLayer(lc, experts, sh, expert_range=(0, 17), staged=True)
    logits = H.router_logits("fused", 6, n_expert, 1.1)
    x = H.activations("fused", 6, n_embd, "bf16")
    ids_o, w_o = oracle.router_top10(logits, k)
    for i in range(6):
        ld, xd = dev(T, logits[i:i + 1]), dev(T, x[i:i + 1], T.bfloat16)
        ids_f, w_f, out_f = fused.forward_checked(ld, xd, api.LAYER_FUSED)
        ids_s, w_s, out_s = staged.forward(ld, xd)
        assert T.equal(ids_f, ids_s) and T.equal(w_f, w_s)
        assert np.array_equal(ids_f.cpu().numpy()[0], ids_o[i])
        assert T.equal(out_f, out_s), f"token {i}"
    assert fused.error() == 0
    # f32 activations and the oracle, experts 17..19 left to "another rank"
    xf = H.activations("fused32", 1, n_embd, "f32")
    _, _, out = fused.forward_checked(dev(T, logits[:1]), dev(T, xf), api.LAYER_FUSED)
    xq = oracle.quantize_q8_1(xf[0])
    parts = np.zeros((k, n_embd), np.float32)
    skip = np.zeros(k, np.uint8)
    for j, e in enumerate(ids_o[0]):
        if e < 17:
            parts[j] = oracle.expert_q8_1(t, t, experts[int(e)].cpu().numpy(), n_embd, n_ff, 7.0, xq)
        else:
            skip[j] = 1
    shv = oracle.expert_q8_1(H.Q8_0, H.Q8_0, sh.cpu().numpy(), n_embd, 512, 7.0, xq) if shared else None
    want = oracle.combine_down(parts, w_o[0], shv, skip)
    assert H.rel_err(out.cpu().numpy()[0], want) <= TIGHT


@pytest.mark.parametrize("t,n_embd,n_ff,n_ff_sh,k", [
    (H.Q4_K, 2048, 1024, 0, 8), (H.Q4_K, 7168, 512, 1024, 8), (H.Q8_0, 2080, 1056, 96, 6), (H.Q8_0, 6144, 256, 2048, 8),
    (H.IQ3_S, 6144, 2048, 0, 4), (H.IQ3_S, 4352, 1024, 288, 6), (H.IQ2_S, 6144, 1024, 2048, 8)])
def test_fused_kernel_at_the_widths_that_ranks_use(T, api, t, n_embd, n_ff, n_ff_sh, k):
    """What several ranks run a token with, whichever kernel is the faster one on a single GPU: the staged kernels' bits."""
    n_expert = 10
    cfg = dict(n_embd=n_embd, n_ff=n_ff, n_expert=n_expert, k=k, gu_type=t, d_type=t, limit=7.0)
    if n_ff_sh:
        cfg.update(n_ff_sh=n_ff_sh, sh_gu_type=H.Q8_0, sh_d_type=H.Q8_0)
    two = dev(T, np.stack([H.constructed_expert(t, t, n_embd, n_ff, H.rng_for("wide", t, e)) for e in range(2)]))
    experts = two[T.arange(n_expert, device="cuda") % 2].contiguous()
    sh = dev(T, H.constructed_expert(H.Q8_0, H.Q8_0, n_embd, n_ff_sh, H.rng_for("wide-shared", t))) if n_ff_sh else None
    layer = api.MoeLayer(layer_cfg(api, cfg), experts, sh, expert_range=(0, 8))
    logits, x = dev(T, H.router_logits("wide", 3, n_expert, 1.1)), dev(T, H.activations("wide", 3, n_embd, "bf16"), T.bfloat16)
    for i in (0, 1, 2, 0):
        got, want = (layer.forward_checked(logits[i:i + 1], x[i:i + 1], kernel) for kernel in (api.LAYER_FUSED, api.LAYER_STAGED))
        assert all(T.equal(a, b) for a, b in zip(got, want)), f"token {i}"
    assert layer.error() == 0 and want[2].abs().max() > 0


@pytest.mark.parametrize("gu,d,n_embd,n_ff,n_ff_sh,k,cut", [
    (H.Q8_0, H.Q8_0, 1344, 352, 0, 8, None),             # an odd number of blocks a row; 11 calls of a down row
    (H.Q8_0, H.Q8_0, 2080, 1056, 96, 6, None),           # three segments, the last of one block; two of a down row
    (H.Q4_K, H.Q4_K, 512, 512, 0, 8, None),              # down rows of 8 calls, four side by side
    (H.Q4_K, H.Q4_K, 512, 20480, 0, 1, None),            # experts wider than the fused kernel takes
    (H.Q4_K, H.Q6_K, 2304, 1536, 4128, 8, None),         # down in segments of 840 bytes
    (H.Q4_K, H.Q4_K, 2304, 1536, 4128, 6, 64),           # slices of the shared expert
    (H.Q5_K, H.Q8_0, 1536, 2304, 352, 5, None), (H.Q6_K, H.Q5_K, 1280, 768, 0, 7, None), (H.IQ4_XS, H.IQ3_XXS, 2560, 256, 0, 8, None),
    (H.IQ2_S, H.IQ3_S, 2304, 2304, 512, 3, None), (H.IQ2_S, H.IQ2_S, 2048, 1280, 0, 8, None), (H.IQ3_S, H.IQ3_S, 4352, 1024, 288, 6, None),
    (H.IQ3_XXS, H.IQ4_XS, 4096, 1536, 0, 8, None), (H.IQ2_XXS, H.IQ3_XXS, 1792, 512, 64, 8, None), (H.IQ1_S, H.IQ2_XXS, 2304, 768, 0, 8, None),
    (H.IQ3_S, H.IQ1_S, 2048, 2560, 1024, 8, None), (H.IQ1_S, H.IQ1_S, 1024, 512, 256, 1, None)])
def test_token_kernel_equals_staged_kernels_bitwise(T, api, gu, d, n_embd, n_ff, n_ff_sh, k, cut):
    """One token through the streamed single-token kernel and through the separate launches: the same bits, where segments,
    stages, units shared by two blocks and short down rows end unevenly; twice, so that the counters are seen again."""
    n_expert = 12
    cfg = dict(n_embd=n_embd, n_ff=n_ff, n_expert=n_expert, k=k, gu_type=gu, d_type=d)
    if n_ff_sh:
        cfg.update(n_ff_sh=n_ff_sh, sh_gu_type=H.Q8_0, sh_d_type=H.Q8_0)
    lc = layer_cfg(api, cfg)
    lc.limit = 7.0
    three = dev(T, np.stack([H.constructed_expert(gu, d, n_embd, n_ff, H.rng_for("tok", gu, d, e)) for e in range(3)]))
    experts = three[T.arange(n_expert, device="cuda") % 3].contiguous()
    sh = dev(T, H.constructed_expert(H.Q8_0, H.Q8_0, n_embd, n_ff_sh, H.rng_for("tok-shared", gu))) if n_ff_sh else None
    token = api.MoeLayer(lc, experts, sh, expert_range=(1, n_expert))
    staged = api.MoeLayer(lc, experts, sh, expert_range=(1, n_expert), staged=True)
    logits = dev(T, H.router_logits("tok", 4, n_expert, 1.1))
    x = dev(T, H.activations("tok", 4, n_embd, "f32"))
    for i in (0, 1, 2, 3, 0):
        got, want = token.forward_checked(logits[i:i + 1], x[i:i + 1], api.LAYER_TOKEN), staged.forward(logits[i:i + 1], x[i:i + 1])
        assert all(T.equal(a, b) for a, b in zip(got, want)), f"token {i}"
        assert T.isfinite(want[2]).all() and want[2].abs().max() > 0
    assert token.error() == 0
    if cut:                                                              # two slices of the shared expert add up to it
        out = [api.MoeLayer(lc, experts, sh, expert_range=(1, n_expert), **kw).forward_checked(logits[:1], x[:1], api.LAYER_TOKEN)[2].double()
               for kw in ({}, dict(shared_here=False), dict(shared_range=(0, cut)), dict(shared_range=(cut, n_ff_sh)))]
        assert ((out[2] + out[3] - out[1]) - out[0]).abs().max() <= 1e-5 * out[0].abs().max()


@pytest.mark.parametrize("gu,d,n_embd,n_ff,n_ff_sh,k", [
    (H.Q4_K, H.Q4_K, 2304, 1536, 0, 8), (H.IQ3_S, H.IQ1_S, 2048, 1280, 1024, 6), (H.Q8_0, H.Q8_0, 1344, 352, 2080, 1)])
def test_token_kernel_reports_a_wait_that_ran_out(T, api, gu, d, n_embd, n_ff, n_ff_sh, k):
    """The token kernel's waits for weight rows given no or one look: where one runs out the error word says so, no block writes an
    output or a residual row made of another block's missing h, and - with the word cleared - the next call is whole again: the
    counters of split units did not keep what the lost call left."""
    n_expert = 8
    cfg = dict(n_embd=n_embd, n_ff=n_ff, n_expert=n_expert, k=k, gu_type=gu, d_type=d)
    if n_ff_sh:
        cfg.update(n_ff_sh=n_ff_sh, sh_gu_type=H.Q8_0, sh_d_type=H.Q8_0)
    three = dev(T, np.stack([H.constructed_expert(gu, d, n_embd, n_ff, H.rng_for("lost", gu, d, e)) for e in range(3)]))
    experts = three[T.arange(n_expert, device="cuda") % 3].contiguous()
    sh = dev(T, H.constructed_expert(H.Q8_0, H.Q8_0, n_embd, n_ff_sh, H.rng_for("lost-shared", gu))) if n_ff_sh else None
    layer = api.MoeLayer(layer_cfg(api, cfg), experts, sh, max_tokens=1)
    rng = H.rng_for("lost", n_embd)
    logits, x = dev(T, H.router_logits("lost", 2, n_expert, None)), dev(T, H.activations("lost", 2, n_embd, "f32"))
    R_old, post, comb = (dev(T, rng.standard_normal(s).astype(np.float32)) for s in ((4, n_embd), 4, (4, 4)))
    lost = 0

    def call(i, kernel, polls=1 << 22):
        out, R_new = T.full((1, n_embd), -7.5, device="cuda"), T.full((4, n_embd), -7.5, device="cuda")
        layer.forward_checked(logits[i:i + 1], x[i:i + 1], kernel, polls, out=out, hc=(R_old, post, comb, R_new))
        return out, R_new

    want = [call(i, api.LAYER_STAGED) for i in range(2)]
    for polls in (0, 1, 0, 1, 1 << 22):
        out, R_new = call(1, api.LAYER_TOKEN, polls)
        err = layer.error()
        lost += err
        assert err == (1 if polls == 0 else 0 if polls > 1 else err)
        for got, full in ((out, want[1][0]), (R_new, want[1][1])):
            assert bool((got == -7.5).all()) if polls == 0 else bool(((got == full) | (got == -7.5)).all()) if err else T.equal(got, full)
        layer.scratch[8:12].zero_()                                      # the sticky word alone
        for i in (0, 1):
            out, R_new = call(i, api.LAYER_TOKEN)
            assert layer.error() == 0 and T.equal(out, want[i][0]) and T.equal(R_new, want[i][1])
    assert lost >= 2


def test_token_kernel_barrier_times_out_and_reports(T, api):
    """The token kernel's grid barrier, as the fused kernel's below: the call returns, the sticky word says so, nothing is written."""
    cfg = dict(n_embd=2304, n_ff=768, n_expert=8, k=4, gu_type=H.Q4_K, d_type=H.Q4_K)
    lc, experts, _ = synth_layer(T, api, cfg, 8, seed=3)
    layer = api.MoeLayer(lc, experts)
    logits, x = dev(T, H.router_logits("timeout", 1, 8, None)), dev(T, H.activations("timeout", 1, 2304, "f32"))
    layer.forward_checked(logits, x, api.LAYER_TOKEN)
    assert layer.error() == 0
    layer.scratch[:16].view(T.int32)[1] += 7
    out = T.full((1, 2304), -7.5, device="cuda")
    layer.forward_checked(logits, x, api.LAYER_TOKEN, out=out)
    assert layer.error() != 0 and bool((out == -7.5).all())


@pytest.mark.parametrize("t,n_embd,n_ff,n_ff_sh,n_expert,n_tok,sigmoid", [
    (H.IQ2_S, 1024, 256, 512, 12, 2, False), (H.Q4_K, 1280, 768, 1312, 12, 9, False),      # the shared expert's jobs: one; three of 4, 4, 1
    (H.Q8_0, 1056, 288, 4128, 300, 7, True), (H.IQ3_S, 4352, 512, 256, 600, 16, False),    # rows beyond 4096 values; 2 and 4 experts a thread
    (H.Q4_K, 512, 256, 8448, 8, 3, False)])                                                # too wide to ride: launches of its own
def test_window_with_shared_expert_equals_fused_tokens_bitwise(T, api, t, n_embd, n_ff, n_ff_sh, n_expert, n_tok, sigmoid):
    """A window whose shared expert rides in the routed experts' launches, behind the one launch that routes, quantizes and
    groups: every token has the fused single-token kernel's ids, weights and output, bit for bit."""
    cfg = dict(n_embd=n_embd, n_ff=n_ff, n_expert=n_expert, k=5, gu_type=t, d_type=t, n_ff_sh=n_ff_sh, sh_gu_type=H.Q8_0, sh_d_type=H.Q8_0)
    lc = layer_cfg(api, cfg)
    lc.limit = 7.0
    four = dev(T, np.stack([H.constructed_expert(t, t, n_embd, n_ff, H.rng_for("wsh", t, e)) for e in range(4)]))
    experts = four[T.arange(n_expert, device="cuda") % 4].contiguous()
    sh = dev(T, H.constructed_expert(H.Q8_0, H.Q8_0, n_embd, n_ff_sh, H.rng_for("wsh-shared", t)))
    route = (dev(T, (0.1 * H.rng_for("wsh", t).standard_normal(n_expert)).astype(np.float32)), 2.5, True) if sigmoid else None
    layer = api.MoeLayer(lc, experts, sh, expert_range=(1, n_expert), sigmoid=route)
    logits = dev(T, H.router_logits("wsh", n_tok, n_expert, 1.1))
    x = dev(T, H.activations("wsh", n_tok, n_embd, "bf16"), T.bfloat16)
    for _ in range(2):                                                   # twice: the launches leave their counters as they found them
        ids, w, out = layer.forward(logits, x)
        for i in range(n_tok):
            ids1, w1, out1 = layer.forward(logits[i:i + 1], x[i:i + 1])
            assert T.equal(ids[i], ids1[0]) and T.equal(w[i], w1[0]) and T.equal(out[i], out1[0]), f"token {i}"
    assert layer.error() == 0


def test_fused_kernel_many_calls_one_scratch(T, api):
    """The grid barrier's counter lives in the scratch: hundreds of calls, single tokens (fused) and windows interleaved."""
    cfg = dict(n_embd=512, n_ff=256, n_expert=8, k=4, gu_type=H.Q4_K, d_type=H.Q4_K)
    lc, experts, _ = synth_layer(T, api, cfg, 8, seed=3)
    layer = api.MoeLayer(lc, experts)
    logits = dev(T, H.router_logits("many", 16, 8, None))
    x = dev(T, H.activations("many", 16, 512, "f32"))
    first = layer.forward(logits[:1], x[:1])[2].clone()
    for i in range(300):
        if i % 50 == 7:
            layer.forward(logits, x)              # a 16-token window through the staged kernels, same scratch
        out = layer.forward(logits[:1], x[:1])[2]
    T.cuda.synchronize()
    assert T.equal(out, first)
    assert layer.error() == 0


@pytest.mark.parametrize("gu,d,n_ff_sh", [(H.Q4_K, H.Q6_K, 0), (H.IQ3_S, H.IQ3_S, 1056)])
def test_token_kernel_many_calls_one_scratch(T, api, gu, d, n_ff_sh):
    """The counters of units that two blocks share live in the scratch too: hundreds of tokens, whose experts change from call to call
    and some of which are another rank's, windows, fused tokens and replays of a captured token between them."""
    n_embd, n_ff, n_expert, k = 768, 1280, 12, 5
    cfg = dict(n_embd=n_embd, n_ff=n_ff, n_expert=n_expert, k=k, gu_type=gu, d_type=d)
    if n_ff_sh:
        cfg.update(n_ff_sh=n_ff_sh, sh_gu_type=H.Q8_0, sh_d_type=H.Q8_0)
    three = dev(T, np.stack([H.constructed_expert(gu, d, n_embd, n_ff, H.rng_for("manytok", gu, e)) for e in range(3)]))
    experts = three[T.arange(n_expert, device="cuda") % 3].contiguous()
    sh = dev(T, H.constructed_expert(H.Q8_0, H.Q8_0, n_embd, n_ff_sh, H.rng_for("manytok-shared", gu))) if n_ff_sh else None
    layer = api.MoeLayer(layer_cfg(api, cfg), experts, sh, expert_range=(2, n_expert))
    logits, x = dev(T, H.router_logits("manytok", 16, n_expert, None)), dev(T, H.activations("manytok", 16, n_embd, "f32"))
    want = [layer.forward_checked(logits[i:i + 1], x[i:i + 1], api.LAYER_STAGED) for i in range(16)]
    stream, graph = T.cuda.Stream(), T.cuda.CUDAGraph()
    T.cuda.synchronize()
    with T.cuda.graph(graph, stream=stream):
        replayed = layer.forward_checked(logits[3:4], x[3:4], api.LAYER_TOKEN)
    T.cuda.synchronize()
    for i in range(300):
        if i % 50 == 7:
            layer.forward(logits, x)
        if i % 50 == 23:
            graph.replay()
            assert all(T.equal(a, b) for a, b in zip(replayed, want[3]))
        if gu == d and i % 3 == 1:
            layer.forward_checked(logits[:1], x[:1], api.LAYER_FUSED)
        got = layer.forward_checked(logits[i % 16:i % 16 + 1], x[i % 16:i % 16 + 1], api.LAYER_TOKEN)
        assert all(T.equal(a, b) for a, b in zip(got, want[i % 16])), f"call {i}"
    assert layer.error() == 0


@pytest.mark.parametrize("t", [H.IQ2_S, H.Q4_K])
def test_layer_sigmoid_router_and_host_lane_hooks(T, api, oracle, t):
    """maya_moe_layer's options: sigmoid routing (selection bias, weight scale, normalisation: router_sigmoid's
    arithmetic) and the tier hooks cpu_part / cpu_flag (MoeDev's, glm_fast.hpp:299-300).  The fused single-token kernel,
    the staged kernels and the window path agree bit for bit; the ids are the oracle's sigmoid router's; the host lane's
    vector enters after the routed terms and before the shared expert (moe_down's order), only when its flag is set."""
    n_embd, n_ff, E, k = 1024, 512, 24, 4
    cfg = dict(n_embd=n_embd, n_ff=n_ff, n_expert=E, k=k, gu_type=t, d_type=t, n_ff_sh=256, sh_gu_type=H.Q8_0, sh_d_type=H.Q8_0)
    lc, experts, sh = synth_layer(T, api, cfg, E, seed=17)
    rng = H.rng_for("sigmoid-layer", t)
    bias = (0.3 * rng.standard_normal(E)).astype(np.float32)
    logits = H.router_logits("sigmoid-layer", 6, E, None)
    x = H.activations("sigmoid-layer", 6, n_embd, "bf16")
    cpu_part = rng.standard_normal((6, n_embd)).astype(np.float32)
    flags = np.array([1, 0, 1, 1, 0, 1], np.int32)
    ld, xd, bd = dev(T, logits), dev(T, x, T.bfloat16), dev(T, bias)
    cp, cf = dev(T, cpu_part), dev(T, flags)
    ids_o, w_o = oracle.router_sigmoid(logits, bias, k, 2.5, True)
    plain = api.MoeLayer(lc, experts, sh, sigmoid=(bd, 2.5, True))
    staged_plain = api.MoeLayer(lc, experts, sh, sigmoid=(bd, 2.5, True), staged=True)
    for i in range(6):
        hooked = api.MoeLayer(lc, experts, sh, sigmoid=(bd, 2.5, True), cpu_part=cp[i:i + 1], cpu_flag=cf[i:i + 1])
        hooked_staged = api.MoeLayer(lc, experts, sh, sigmoid=(bd, 2.5, True), cpu_part=cp[i:i + 1], cpu_flag=cf[i:i + 1], staged=True)
        ids_f, w_f, out_f = hooked.forward(ld[i:i + 1], xd[i:i + 1])
        ids_s, w_s, out_s = hooked_staged.forward(ld[i:i + 1], xd[i:i + 1])
        assert np.array_equal(ids_f.cpu().numpy()[0], ids_o[i]) and T.equal(ids_f, ids_s)
        assert np.abs(w_f.cpu().numpy()[0] - w_o[i]).max() <= 1e-6 and T.equal(w_f, w_s)
        assert T.equal(out_f, out_s), f"token {i}: fused and staged kernels differ"
        base = plain.forward(ld[i:i + 1], xd[i:i + 1])[2]
        assert T.equal(base, staged_plain.forward(ld[i:i + 1], xd[i:i + 1])[2])
        if flags[i]:
            assert not T.equal(out_f, base)
            assert H.rel_err((out_f - base).cpu().numpy()[0], cpu_part[i]) <= 1e-5
        else:
            assert T.equal(out_f, base)
    win = api.MoeLayer(lc, experts, sh, sigmoid=(bd, 2.5, True), cpu_part=cp, cpu_flag=cf)
    ids_w, _, out_w = win.forward(ld, xd)
    assert np.array_equal(ids_w.cpu().numpy(), ids_o)
    for i in range(6):
        one = api.MoeLayer(lc, experts, sh, sigmoid=(bd, 2.5, True), cpu_part=cp[i:i + 1], cpu_flag=cf[i:i + 1])
        assert T.equal(out_w[i], one.forward(ld[i:i + 1], xd[i:i + 1])[2][0]), f"window row {i}"
    with pytest.raises(api.MayaError):
        api.MoeLayer(lc, experts, sh, cpu_flag=cf[:1]).forward(ld[:1], xd[:1])        # a flag without the vector


def test_window_combine_carries_the_cross_rank_sum(T, api, oracle):
    """2..16 tokens on an expert-parallel rank: the rank-ordered sum of out[T][n_embd] runs inside the window's combine
    launch.  Three ranks on this GPU, one after another; what the ranks still to run would push is placed beforehand."""
    from project_maya_b200.peer import PeerGroup
    from test_gpu_allreduce import place_peer_pushes
    n_embd, n_ff, n_expert, k, nm, n_tok = 1024, 512, 12, 4, 3, 5
    cfg = dict(n_embd=n_embd, n_ff=n_ff, n_expert=n_expert, k=k, gu_type=H.Q4_K, d_type=H.Q4_K, n_ff_sh=256,
               sh_gu_type=H.Q8_0, sh_d_type=H.Q8_0)
    lc, experts, sh = synth_layer(T, api, cfg, n_expert, seed=9)
    logits = dev(T, H.router_logits("winar", n_tok, n_expert, 1.1))
    x = dev(T, H.activations("winar", n_tok, n_embd, "bf16"), T.bfloat16)
    per = n_expert // nm
    layers = [api.MoeLayer(lc, experts, sh, expert_range=(r * per, (r + 1) * per), shared_here=(r == 0)) for r in range(nm)]
    partial = [l.forward(logits, x)[2].clone() for l in layers]                     # each rank's own terms
    want = np.stack([oracle.allreduce_in_order(np.stack([p[t].cpu().numpy() for p in partial])) for t in range(n_tok)])
    ranks = PeerGroup.on_one_device(nm, stride=16 * n_embd, timeout_ms=200.0)
    for r in ranks:
        r.device_seq = False
    vecs = [p.reshape(-1) for p in partial]
    for mi in range(nm):
        place_peer_pushes(T, ranks, mi, 1, vecs, later_only=True)
    for r in range(nm):
        out = layers[r].forward(logits, x, peer=ranks[r])[2]
        T.cuda.synchronize()
        assert not ranks[r].poisoned()
        assert out.cpu().numpy().tobytes() == want.tobytes(), f"rank {r}"


@pytest.mark.parametrize("kernel", ["LAYER_FUSED", "LAYER_TOKEN"])
def test_single_tokens_on_several_streams_at_once(T, api, kernel):
    """Hundreds of launches on the legacy default stream and on others in flight together, a layer and a scratch a stream, and a captured
    one replayed between them - every output the same bits, no wait ran out."""
    cfg = dict(n_embd=2304, n_ff=768, n_expert=8, k=4, gu_type=H.Q4_K, d_type=H.Q4_K)
    lc, experts, _ = synth_layer(T, api, cfg, 8, seed=3)
    logits, x = dev(T, H.router_logits("streams", 1, 8, None)), dev(T, H.activations("streams", 1, 2304, "f32"))
    want = api.MoeLayer(lc, experts).forward_checked(logits, x, getattr(api, kernel))[2]
    side = [T.cuda.Stream(), T.cuda.Stream()]
    streams = [T.cuda.default_stream(), *side]
    layers = [api.MoeLayer(lc, experts) for _ in range(4)]
    T.cuda.synchronize()
    with T.cuda.stream(side[0]):
        layers[3].forward_checked(logits, x, getattr(api, kernel))
    side[0].synchronize()
    graph = T.cuda.CUDAGraph()
    with T.cuda.graph(graph, stream=side[0]):
        replayed = layers[3].forward_checked(logits, x, getattr(api, kernel))[2]
    outs = []
    for i in range(100):
        for s, layer in zip(streams, layers):
            with T.cuda.stream(s):
                outs.append(layer.forward_checked(logits, x, getattr(api, kernel))[2])
        if i % 10 == 0:
            with T.cuda.stream(side[1]):
                graph.replay()
    T.cuda.synchronize()
    assert all(layer.error() == 0 for layer in layers)
    assert all(T.equal(o, want) for o in [*outs, replayed])


@pytest.mark.parametrize("kernel", ["LAYER_FUSED", "LAYER_TOKEN"])
def test_single_token_starts_with_its_whole_grid_or_not_at_all(T, api, kernel):
    """A launch whose blocks wait for one another must not hold SMs while some of its blocks cannot start: another launch of that kind could
    have the SMs they need.  One block of a long product holds an SM (more shared memory than lies beside a block of the layer); on the
    default stream the layer's first block, once it runs, does not wait that long at the grid barrier."""
    cfg = dict(n_embd=2304, n_ff=768, n_expert=8, k=4, gu_type=H.Q4_K, d_type=H.Q4_K)
    lc, experts, _ = synth_layer(T, api, cfg, 8, seed=3)
    logits, x = dev(T, H.router_logits("whole", 1, 8, None)), dev(T, H.activations("whole", 1, 2304, "f32"))
    layer = api.MoeLayer(lc, experts)
    rows, cols = 256, 1 << 18
    w = T.zeros((1, rows * H.row_bytes(H.Q8_0, cols)), dtype=T.uint8, device="cuda")
    xq = api.mmq_quantize(T.ones((1, cols), device="cuda"), None, H.Q8_0)
    out = T.empty((1, rows), dtype=T.float32, device="cuda")
    product = api.mmq_product(w, H.Q8_0, rows, cols, w.shape[1], 1, xq, dev(T, np.array([0, 1], np.int32)), None, 1, out, rows)
    side = T.cuda.Stream()
    barrier, held = [], []
    for i in range(4):
        T.cuda.synchronize()
        begin, end = T.cuda.Event(enable_timing=True), T.cuda.Event(enable_timing=True)
        with T.cuda.stream(side):
            begin.record()
            api.mmq_run(product)
            end.record()
        layer.forward_checked(logits, x, getattr(api, kernel))
        T.cuda.synchronize()
        ns = layer.phase_ns()
        if i > 0:
            barrier.append(ns[3] - ns[2])
            held.append(begin.elapsed_time(end) * 1e6)
    assert layer.error() == 0
    assert min(held) > 4e5, "the product is over too soon for this test"
    assert max(barrier) < 1e5, f"{max(barrier)} ns at the barrier"


def test_fused_layer_barrier_times_out_and_reports(T, api):
    """The fused kernel's one wait on other blocks is bounded: with the scratch's epoch word set ahead of its arrival
    counter (a state no launch leaves behind) the grid barrier can never be satisfied; the call still returns after the
    time limit, every block having skipped the second phase, and the sticky error word says so."""
    cfg = dict(n_embd=512, n_ff=256, n_expert=8, k=4, gu_type=H.Q4_K, d_type=H.Q4_K)
    lc, experts, _ = synth_layer(T, api, cfg, 8, seed=3)
    layer = api.MoeLayer(lc, experts)
    logits = dev(T, H.router_logits("timeout", 1, 8, None))
    x = dev(T, H.activations("timeout", 1, 512, "f32"))
    layer.forward(logits, x)
    T.cuda.synchronize()
    assert layer.error() == 0
    words = layer.scratch[:16].view(T.int32)
    words[1] += 7                                  # the epoch word: the barrier now waits for arrivals that never come
    layer.forward(logits, x)
    T.cuda.synchronize()                           # returns: the wait gave up after its second
    assert layer.error() != 0


def test_layer_refusals(T, api):
    cfg = H.CONFIGS["C1"]
    lc = layer_cfg(api, cfg)
    experts = T.zeros((2, lc.blob_bytes), dtype=T.uint8, device="cuda")
    layer = api.MoeLayer(api.MoeLayerConfig(cfg["n_embd"], cfg["n_ff"], 2, 2, H.Q4_K, H.Q4_K), experts)
    with pytest.raises(api.MayaError) as e:
        layer.forward(T.zeros((17, 2), device="cuda"), T.zeros((17, cfg["n_embd"]), device="cuda"))
    assert e.value.status == -4
    with pytest.raises(api.MayaError):
        api.MoeLayer(api.MoeLayerConfig(cfg["n_embd"], cfg["n_ff"], 2, 9, H.Q4_K, H.Q4_K), experts)


@pytest.mark.parametrize("router_dtype", ["f32", "bf16"])
def test_rms_router_and_two_launch_layer(T, api, oracle, router_dtype):
    """maya_rms_router (residual add + RMS norm + router logits, one launch) against the oracle, and a decode layer
    as two launches: that kernel, then the fused layer kernel on its x and logits - the routing and the output are the
    oracle's on the same numbers."""
    cfg = dict(H.CONFIGS["C2"], n_expert=32)
    lc, experts, shared = synth_layer(T, api, cfg, 32, seed=33)
    Hd, E = cfg["n_embd"], 32
    rng = H.rng_for("rms-router-gpu", router_dtype)
    h = rng.standard_normal(Hd).astype(np.float32)
    add = (0.2 * rng.standard_normal(Hd)).astype(np.float32)
    nw = (1.0 + 0.1 * rng.standard_normal(Hd)).astype(np.float32)
    rw = (0.08 * rng.standard_normal((E, Hd))).astype(np.float32)
    if router_dtype == "bf16":
        rw = H.to_bf16_f32(rw)
    rw_d = dev(T, rw, T.bfloat16 if router_dtype == "bf16" else None)
    h_out = T.empty(Hd, dtype=T.float32, device="cuda")
    x, logits = api.rms_router(dev(T, h), dev(T, add), dev(T, nw), 1e-5, rw_d, h_out=h_out)
    T.cuda.synchronize()
    ho, xo, lo = oracle.rms_router(h, add, nw, 1e-5, rw)
    assert np.array_equal(h_out.cpu().numpy(), ho)
    assert H.rel_err(x.cpu().numpy(), xo) <= 2e-6
    assert np.abs(logits.cpu().numpy() - lo).max() <= 2e-5
    with pytest.raises(api.MayaError):                       # in place with an add: other blocks would read the sum
        hd = dev(T, h)
        api.rms_router(hd, dev(T, add), dev(T, nw), 1e-5, rw_d, h_out=hd)
    # launch 2: the layer on the first launch's outputs
    ids, w, out = api.MoeLayer(lc, experts, shared).forward(logits.reshape(1, E), x.reshape(1, Hd))
    T.cuda.synchronize()
    lg, xg = logits.cpu().numpy().reshape(1, E), x.cpu().numpy()
    ids_o, w_o = oracle.router_top10(lg, cfg["k"])
    assert np.array_equal(ids.cpu().numpy(), ids_o)
    want = oracle_token(oracle, cfg, experts, shared, ids_o[0], w_o[0], xg)
    assert H.rel_err(out.cpu().numpy()[0], want) <= TIGHT


@pytest.mark.parametrize("n", [8184, 8193, 12272, 12273, 12280, 12288, 12289])
@pytest.mark.parametrize("router_dtype", ["f32", "bf16"])
def test_rms_router_row_widths_around_the_shared_memory_limit(T, api, n, router_dtype):
    """Rows whose f32 image fills the 48 KB a kernel has without a raised limit - up to the last bytes, and beyond: x against
    float64, the logits against the float64 product with that x (f32 sums of n terms, added in up to 256 partial sums)."""
    rng = H.rng_for("rms-width", n, router_dtype)
    h, nw = (dev(T, rng.standard_normal(n).astype(np.float32)) for _ in range(2))
    rw = dev(T, (rng.standard_normal((5, n)) / np.sqrt(n)).astype(np.float32), T.bfloat16 if router_dtype == "bf16" else None)
    x, logits = api.rms_router(h, None, nw, 1e-6, rw)
    want = h.double() * T.rsqrt(h.double().pow(2).mean() + 1e-6) * nw.double()
    assert float((x.double() - want).abs().max()) <= 4e-6 * float(want.abs().max())
    assert float((logits.double() - rw.double() @ x.double()).abs().max()) <= 1e-5


def test_two_threads_with_calls_of_different_sizes(T, api):
    """The kernels' shared-memory limits are process-wide state: two host threads whose calls need different amounts are both
    served - on one stream, so that the GPU sees one call after another - and get the bits they get alone."""
    import threading
    rng = H.rng_for("two-threads")

    def mmvq(n_in):
        w = dev(T, H.constructed_blocks(H.Q8_0, 64, n_in, rng))
        xq = api.native_quantize_q8_1(dev(T, rng.standard_normal((8, n_in)).astype(np.float32)))
        return lambda: (api.native_mmvq(H.Q8_0, w, xq, n_in, 64, ncols=8),)

    def rms(n):
        h, nw, rw = (T.randn(s, device="cuda") for s in (n, n, (5, n)))
        return lambda: api.rms_router(h, None, nw, 1e-6, rw)

    def layer(n_embd, n_ff):
        lc, experts, _ = synth_layer(T, api, dict(n_embd=n_embd, n_ff=n_ff, n_expert=4, k=2, gu_type=H.Q4_K, d_type=H.Q4_K), 4, seed=9)
        m = api.MoeLayer(lc, experts)
        logits, x = T.randn(1, 4, device="cuda"), T.randn(1, n_embd, device="cuda")
        return lambda: m.forward(logits, x)

    for make, small, large in ((rms, (13000,), (50000,)), (mmvq, (5120,), (16384,)), (layer, (512, 256), (1024, 4096))):
        calls, failed = [make(*small), make(*large)], []
        gate, outs = threading.Barrier(2), [None, None]

        def work(i):
            try:
                gate.wait()
                for _ in range(500):
                    outs[i] = calls[i]()
            except Exception as e:
                failed.append(e)

        threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        T.cuda.synchronize()
        assert not failed, f"{make.__name__}: {failed[0]}"
        for call, out in zip(calls, outs):
            assert all(T.equal(a, b) for a, b in zip(call(), out))


def _word_area(T, r):
    """The {seq, value} words of rank r's receive buffer: they follow its 2 x nm x stride floats of rows."""
    return r.keep[0][r.mi][2 * r.nm * r.stride * 4:].view(T.int64).view(2, r.nm, r.stride)


def _words(seq, v):
    return ((np.uint64(seq) << np.uint64(32)) | v.view(np.uint32).astype(np.uint64)).view(np.int64)


def test_fused_layer_exchanges_flagged_words(T, api, oracle):
    """The cross-rank sum in the fused kernel's epilogue, on one GPU: rank 1 of 3 runs alone with the other ranks'
    {seq, value} words placed in its receive area beforehand.  Its output is rank 0's + its own + rank 2's vector, added
    in that order (bit for bit), and its own words land in both peers' areas with the call's sequence number."""
    from project_maya_b200.peer import PeerGroup
    cfg = dict(n_embd=1024, n_ff=512, n_expert=8, k=2, gu_type=H.Q8_0, d_type=H.Q8_0)
    lc, experts, _ = synth_layer(T, api, cfg, 8, seed=31)
    layer = api.MoeLayer(lc, experts, None)
    n = cfg["n_embd"]
    ranks = PeerGroup.on_one_device(3, stride=n, timeout_ms=50.0)
    logits = H.router_logits("words", 3, 8, 1.1)
    x = H.activations("words", 3, n, "bf16")
    ld, xd = dev(T, logits), dev(T, x, T.bfloat16)
    rng = np.random.default_rng(5)
    for t, seq in enumerate((1, 2, 3)):
        local = layer.forward(ld[t:t + 1], xd[t:t + 1])[2].cpu().numpy()[0]
        others = {m: rng.standard_normal(n).astype(np.float32) for m in (0, 2)}
        others[0][:4] = [0.0, -0.0, np.float32(1e-38), np.float32(3e38)]
        area = _word_area(T, ranks[1])
        for m, v in others.items():
            area[seq & 1, m, :n] = T.from_numpy(_words(seq, v)).cuda()
        got = layer.forward(ld[t:t + 1], xd[t:t + 1], peer=ranks[1])[2].cpu().numpy()[0]
        want = oracle.allreduce_in_order(np.stack([others[0], local, others[2]]))
        assert got.tobytes() == want.tobytes()
        for m in (0, 2):
            pushed = _word_area(T, ranks[m])[seq & 1, 1, :n].cpu().numpy()
            assert np.array_equal(pushed, _words(seq, local))
    assert not ranks[1].poisoned()


def test_fused_layer_word_exchange_sequence_wraps(T, api, oracle):
    """The device-side sequence count across 2^32 (the reference's own transport test starts at 0xffffffe0,
    tests/ds4_peer_allreduce_test.cu:143): preset to 0xfffffff8, 24 single-token calls on rank 1 of 2 with rank 0's words
    placed beforehand under the number each call will use.  The count never takes the value 0 (a zeroed word would
    match it): 0xffffffff is followed by 2, which also keeps the two receive slots alternating."""
    from project_maya_b200.peer import PeerGroup
    cfg = dict(n_embd=1024, n_ff=512, n_expert=8, k=2, gu_type=H.Q8_0, d_type=H.Q8_0)
    lc, experts, _ = synth_layer(T, api, cfg, 8, seed=31)
    layer = api.MoeLayer(lc, experts, None)
    n = cfg["n_embd"]
    ranks = PeerGroup.on_one_device(2, stride=n, timeout_ms=50.0)
    r = ranks[1]
    r.seq = 0xFFFFFFF8
    r.set_device_seq(True)
    ld, xd = dev(T, H.router_logits("wrap", 1, 8, 1.1)), dev(T, H.activations("wrap", 1, n, "bf16"), T.bfloat16)
    local = layer.forward(ld, xd)[2].cpu().numpy()[0]
    rng = np.random.default_rng(9)
    seq, seen = 0xFFFFFFF8, []
    for _ in range(24):
        seq = 2 if seq == 0xFFFFFFFF else seq + 1
        seen.append(seq)
        other = rng.standard_normal(n).astype(np.float32)
        _word_area(T, r)[seq & 1, 0, :n] = T.from_numpy(_words(seq, other)).cuda()
        got = layer.forward(ld, xd, peer=r)[2].cpu().numpy()[0]
        assert got.tobytes() == oracle.allreduce_in_order(np.stack([other, local])).tobytes(), hex(seq)
        pushed = _word_area(T, ranks[0])[seq & 1, 1, :n].cpu().numpy()
        assert np.array_equal(pushed, _words(seq, local))
    assert 0 not in seen and 0xFFFFFFFF in seen and 2 in seen
    assert all((a & 1) != (b & 1) for a, b in zip(seen, seen[1:]))         # the slots alternate across the wrap too
    r.set_device_seq(False)
    assert r.seq == seen[-1] and not r.poisoned()


def test_fused_layer_exchange_times_out_and_poisons(T, api):
    """A peer that never sends: the wait in the fused kernel's epilogue gives up after the time-out, records who it
    waited for and poisons the transport; later calls return at once and the device still answers."""
    import time
    from project_maya_b200.peer import PeerGroup
    cfg = dict(n_embd=1024, n_ff=512, n_expert=8, k=2, gu_type=H.Q8_0, d_type=H.Q8_0)
    lc, experts, _ = synth_layer(T, api, cfg, 8, seed=31)
    layer = api.MoeLayer(lc, experts, None)
    r = PeerGroup.on_one_device(2, stride=cfg["n_embd"], timeout_ms=20.0)[0]
    ld, xd = dev(T, H.router_logits("words", 1, 8, 1.1)), dev(T, H.activations("words", 1, cfg["n_embd"], "bf16"), T.bfloat16)
    t0 = time.time()
    layer.forward(ld, xd, peer=r)
    T.cuda.synchronize()
    assert time.time() - t0 < 2.0
    assert r.poisoned()
    f = r.failure_record()
    assert f.captured == 1 and f.sequence == 1 and f.rank == 0 and f.waited_for == 1 and f.elapsed_ns >= f.timeout_ns
    t0 = time.time()
    for _ in range(32):
        layer.forward(ld, xd, peer=r)
    T.cuda.synchronize()
    assert time.time() - t0 < 1.0
    assert layer.error() == 0                                   # the layer's own barrier is not affected
    assert bool((T.ones(4, device="cuda") * 2 == 2).all())


@pytest.mark.parametrize("t", list(H.MORE_TYPES))
def test_layer_with_further_block_types(T, api, oracle, t):
    """maya_moe_layer_decode on routed experts stored as Q5_K, Q6_K, IQ4_XS, IQ3_XXS or IQ2_XXS (the rest of
    glmf::moe_supported's table) with a Q8_0 shared expert beside them: single tokens (the token kernel) against the oracle, and
    a 5-token window equal to its tokens bit for bit."""
    n_embd, n_ff, E, k, n_sh = 1024, 512, 12, 4, 256
    cfg = dict(n_embd=n_embd, n_ff=n_ff, n_expert=E, k=k, gu_type=t, d_type=t, n_ff_sh=n_sh, sh_gu_type=H.Q8_0, sh_d_type=H.Q8_0)
    rng = H.rng_for("layer-more", t)
    experts_np = np.stack([H.constructed_expert(t, t, n_embd, n_ff, rng) for _ in range(E)])
    shared_np = H.constructed_expert(H.Q8_0, H.Q8_0, n_embd, n_sh, rng)
    experts, shared = dev(T, experts_np), dev(T, shared_np)
    lc = api.MoeLayerConfig(n_embd, n_ff, E, k, t, t, n_sh, H.Q8_0, H.Q8_0, 7.0)
    layer = api.MoeLayer(lc, experts, shared)
    logits = rng.standard_normal((5, E)).astype(np.float32)
    x = rng.standard_normal((5, n_embd)).astype(np.float32)
    ids_o, w_o = oracle.router_top10(logits, k)
    singles = []
    for i in range(5):
        ids, w, out = layer.forward(dev(T, logits[i:i + 1]), dev(T, x[i:i + 1]))
        assert np.array_equal(ids.cpu().numpy()[0], ids_o[i])
        want = oracle_token(oracle, cfg, experts, shared, ids_o[i], w_o[i], x[i], 7.0)
        assert H.rel_err(out.cpu().numpy()[0], want) <= 2e-4
        singles.append(out[0].clone())
    _, _, win = layer.forward(dev(T, logits), dev(T, x))
    for i in range(5):
        assert T.equal(win[i], singles[i])
    assert layer.error() == 0
