"""Which kernel a single token takes (maya_moe_layer_kernel): a rule on the layer's sizes, types and addresses, decided on the host."""
import ctypes as C
import itertools

import pytest

import helpers as H

CHOICE, FUSED, TOKEN, STAGED = range(4)
SMS = 148
TYPES = (H.Q8_0, H.Q4_K, H.Q5_K, H.Q6_K, H.IQ4_XS, H.IQ2_S, H.IQ3_S, H.IQ3_XXS, H.IQ2_XXS, H.IQ1_S)


def desc(gu, d, n_embd, n_ff, k, n_expert=256, n_ff_sh=0, at=1 << 20, gap=0, **more):
    from project_maya_b200._lib import MoeLayerDesc
    L = MoeLayerDesc(n_embd=n_embd, n_ff=n_ff, n_expert=n_expert, k=k, gu_type=gu, d_type=d, experts=at,
                     expert_stride=H.blob_bytes(gu, d, n_embd, n_ff) + gap, n_ff_sh=n_ff_sh, sh_gu_type=H.Q8_0, sh_d_type=H.Q8_0,
                     shared=1 << 30 if n_ff_sh else None, limit=H.INF, expert_lo=0, expert_hi=n_expert, shared_here=1)
    for name, v in more.items():
        setattr(L, name, v)
    return L


def kernel(lib, L, n_ranks=1, sms=SMS):
    return lib.maya_moe_layer_kernel(C.byref(L), n_ranks, sms)


@pytest.mark.parametrize("t,n_embd,n_ff,k,n_ff_sh,want", [
    # both sides of every line, each a layer on which the named kernel was timed as the faster one (or as fast)
    (H.Q8_0, 1312, 1120, 5, 0, FUSED), (H.Q8_0, 2528, 1056, 8, 0, FUSED), (H.Q8_0, 2720, 832, 8, 2816, FUSED), (H.Q8_0, 1824, 2016, 8, 0, FUSED),
    (H.Q8_0, 3200, 768, 6, 0, TOKEN), (H.Q8_0, 5504, 1568, 8, 0, TOKEN), (H.Q8_0, 5120, 1536, 6, 3072, TOKEN), (H.Q8_0, 2688, 704, 8, 512, TOKEN),
    (H.Q8_0, 1440, 2464, 8, 0, TOKEN), (H.IQ3_S, 2816, 768, 8, 512, TOKEN), (H.IQ3_S, 2560, 768, 8, 2560, FUSED), (H.IQ2_S, 3584, 1024, 5, 0, TOKEN),
    (H.Q4_K, 1280, 768, 8, 0, FUSED), (H.Q4_K, 1536, 1280, 7, 0, FUSED), (H.Q4_K, 1536, 1024, 8, 2816, FUSED), (H.Q4_K, 1536, 1536, 2, 3072, FUSED),
    (H.Q4_K, 2048, 1024, 8, 0, TOKEN), (H.Q4_K, 2560, 512, 8, 0, TOKEN), (H.Q4_K, 1280, 1280, 1, 1536, TOKEN), (H.Q4_K, 6656, 2048, 8, 2560, TOKEN),
    (H.IQ3_S, 1536, 768, 8, 0, FUSED), (H.IQ3_S, 6656, 512, 4, 0, FUSED), (H.IQ3_S, 2304, 1024, 4, 1792, FUSED), (H.IQ3_S, 2304, 2816, 3, 0, FUSED),
    (H.IQ3_S, 6144, 2048, 8, 0, TOKEN), (H.IQ3_S, 4352, 1280, 2, 0, TOKEN), (H.IQ3_S, 1280, 2560, 8, 0, TOKEN), (H.IQ3_S, 5120, 1024, 8, 2048, TOKEN),
    (H.IQ2_S, 6144, 2048, 8, 2048, FUSED), (H.IQ2_S, 7168, 512, 8, 0, FUSED), (H.IQ2_S, 2560, 1536, 8, 0, FUSED), (H.IQ2_S, 2560, 1280, 6, 0, FUSED),
    (H.IQ2_S, 6144, 2048, 8, 0, TOKEN), (H.IQ2_S, 5888, 1280, 5, 0, TOKEN)])
def test_core_types_take_the_faster_kernel(lib, t, n_embd, n_ff, k, n_ff_sh, want):
    assert kernel(lib, desc(t, t, n_embd, n_ff, k, n_ff_sh=n_ff_sh)) == want


def test_pairs_of_types_that_fit_shared_memory(lib):
    """Ring of the wider type and codebook of the larger one: on 6144 x 2048, top 8 of 256, 68 of the 100 pairs fit."""
    takes = {(g, d) for g, d in itertools.product(TYPES, TYPES) if g == d or kernel(lib, desc(g, d, 6144, 2048, 8)) == TOKEN}
    assert len(takes) == 68
    assert not takes & {(H.IQ2_S, H.IQ3_S), (H.IQ2_S, H.Q4_K), (H.IQ3_S, H.Q4_K), (H.IQ3_S, H.Q5_K), (H.Q8_0, H.IQ2_S)}
    assert {(H.Q4_K, H.Q6_K), (H.Q5_K, H.Q6_K), (H.IQ3_XXS, H.IQ4_XS), (H.IQ2_XXS, H.IQ3_XXS), (H.IQ1_S, H.IQ2_XXS)} <= takes
    # IQ2_S with IQ3_S: narrower experts, or fewer of them, leave the room
    assert kernel(lib, desc(H.IQ2_S, H.IQ3_S, 6144, 768, 8)) == TOKEN and kernel(lib, desc(H.IQ2_S, H.IQ3_S, 6144, 1024, 8)) == STAGED
    assert kernel(lib, desc(H.IQ2_S, H.IQ3_S, 2304, 2304, 3, n_ff_sh=512, n_expert=12)) == TOKEN


@pytest.mark.parametrize("t,n_embd,n_ff", [(H.Q8_0, 1024, 20480), (H.Q4_K, 512, 20480), (H.IQ3_S, 2048, 16384), (H.IQ2_S, 2048, 16384)])
def test_experts_too_wide_for_the_fused_kernel_take_the_other(lib, t, n_embd, n_ff):
    """The fused kernel holds nine columns of h whatever k is, the token kernel k of them."""
    assert kernel(lib, desc(t, t, n_embd, n_ff, 1, n_expert=8)) == TOKEN


def test_what_the_token_kernel_leaves_to_others(lib):
    core, mixed = (H.IQ3_S, H.IQ3_S, 6144, 2048, 8), (H.Q4_K, H.Q6_K, 4096, 1536, 8)
    for a, other in ((core, FUSED), (mixed, STAGED)):
        assert kernel(lib, desc(*a)) == TOKEN
        assert kernel(lib, desc(*a), n_ranks=2) == other                             # the cross-rank sum
        assert kernel(lib, desc(*a, at=(1 << 20) + 8)) == other                      # blobs off 16-byte boundaries
        assert kernel(lib, desc(*a, gap=8)) == other
        assert kernel(lib, desc(*a, staged=1)) == STAGED
        assert kernel(lib, desc(*a), sms=0) == other
        assert kernel(lib, desc(a[0], a[1], 16384, *a[3:])) == other        # more output rows a block than it holds
        assert kernel(lib, desc(*a, n_expert=2049)) == STAGED
    assert kernel(lib, desc(*mixed, n_ff_sh=1024, sh_gu_type=H.Q4_K, sh_d_type=H.Q4_K)) == STAGED
    assert kernel(lib, desc(*mixed, n_ff_sh=1024, sh_lo=0, sh_hi=512)) == STAGED      # a slice beside two types: refused there
    assert kernel(lib, desc(H.Q4_K, H.Q4_K, 4096, 1536, 8, n_ff_sh=1024, sh_lo=0, sh_hi=512)) == TOKEN
    assert kernel(lib, desc(H.Q4_K, H.Q4_K, 4096, 1536, 9)) == -4


def test_a_layers_outputs_lie_where_its_logits_do(monkeypatch):
    """MoeLayer.forward with its library replaced: ids, weights and out are allocated on the logits' device, contiguous and anew at each
    call, and a refused number of tokens leaves nothing behind."""
    import torch

    from project_maya_b200 import _lib, api

    class Fake:
        maya_row_bytes = staticmethod(lambda t, n: 144 * (n // 256))
        maya_moe_layer_scratch_bytes = staticmethod(lambda *a: 64)
        maya_moe_layer_decode = staticmethod(lambda L, logits, x, bf16, T, *a: 0 if T <= 4 else -4)

    monkeypatch.setattr(_lib, "load", lambda: Fake)
    monkeypatch.setattr(api, "_ptr", lambda t: None)             # (asks for CUDA tensors)
    cfg = api.MoeLayerConfig(256, 256, 8, 3, H.Q4_K, H.Q4_K)
    layer = api.MoeLayer(cfg, torch.empty((8, cfg.blob_bytes), dtype=torch.uint8, device="meta"), max_tokens=4)
    kept = None
    for T in (1, 4, 1):
        for device in ("cpu", "meta"):
            outs = layer.forward(torch.zeros((T, 8), device=device), torch.zeros((T, 256), device=device), stream=0)
            assert [(tuple(o.shape), o.dtype, o.device.type, o.is_contiguous()) for o in outs] == [
                ((T, 3), torch.int32, device, True), ((T, 3), torch.float32, device, True), ((T, 256), torch.float32, device, True)]
            if device == "cpu":
                assert kept is None or kept.data_ptr() != outs[2].data_ptr()
                kept = outs[2]
    held = len(layer._shapes)
    for T in (5, 6, 7):
        with pytest.raises(api.MayaError):
            layer.forward(torch.zeros((T, 8)), torch.zeros((T, 256)), stream=0)
    assert len(layer._shapes) == held


def test_a_layers_first_call_allocates_its_outputs_only(monkeypatch):
    """What a MoeLayer keeps from call to call is allocated when it is made, on its experts' device: a first call under graph capture would
    take it from the graph's own pool, which could then not be given back while the layer lives."""
    import torch

    from project_maya_b200 import _lib, api

    class Fake:
        maya_row_bytes = staticmethod(lambda t, n: 144 * (n // 256))
        maya_moe_layer_scratch_bytes = staticmethod(lambda *a: 64)
        maya_moe_layer_decode = staticmethod(lambda L, *a: 0)

    monkeypatch.setattr(_lib, "load", lambda: Fake)
    monkeypatch.setattr(api, "_ptr", lambda t: None)
    cfg = api.MoeLayerConfig(256, 256, 8, 3, H.Q4_K, H.Q4_K)
    layer = api.MoeLayer(cfg, torch.empty((8, cfg.blob_bytes), dtype=torch.uint8), max_tokens=4)
    calls = [(torch.zeros((T, 8)), torch.zeros((T, 256))) for T in (1, 4)]
    made = []

    class Watch(torch.utils._python_dispatch.TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            out = func(*args, **(kwargs or {}))
            if isinstance(out, torch.Tensor) and func.overloadpacket is not torch.ops.aten.expand:
                made.append(out.shape)
            return out

    for logits, x in calls:
        made.clear()
        with Watch():
            outs = layer.forward(logits, x, stream=0)
        assert made == [o.shape for o in outs]
