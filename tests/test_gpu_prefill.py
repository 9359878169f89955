"""The prompt path's grouped GEMM on the tensor cores (maya_mmq_quantize / maya_mmq_run / maya_mmq_run_glu) and the
whole prompt-path layer (api.MoePrefill).

Two bars.  Against the q8_1 oracle (the reference's GPU arithmetic: integer dots of q8_1 activations) the tolerance is
1e-2 in max-norm and in L2: the tensor-core path multiplies the same q8_1-rounded activations and the same dequantized
weights, each rounded to f16.  Against a float64 product of exactly those f16 operands (built here with numpy: the
oracle's q8_1 blocks as d * q, Q8_0 weights as q * d, Q4_K weights through the kernel's packed-half steps) the tolerance is 2e-5: that one pins the kernel itself - tile layout, descriptors,
the K loop, ragged groups - with only f32 accumulation order left over."""
import numpy as np
import pytest

import helpers as H

pytestmark = pytest.mark.gpu
TOL, PIN = 1e-2, 2e-5
MODEL = 1e-3   # rel-L2 from the reference's host model of its MMQ arithmetic (f16 scales and weights cost ~3e-4)
# Whole layers against the model: max-norm within the stated 1e-2.  Their rel-L2 gets 2e-2: the q8_1 rounding of h alone
# puts a down product ~1e-2 from the exact one, and two evaluations whose h differ by 1e-3 (f16 operands here, floats in the
# model) land up to ~1e-2 apart through flipped roundings; each product by itself is pinned to MODEL.
LAYER_L2 = 2e-2


@pytest.fixture(scope="module")
def T(cuda):
    import torch
    return torch


@pytest.fixture(scope="module")
def api(cuda):
    from project_maya_b200 import api as a
    return a


def dev(T, a):
    return T.from_numpy(np.ascontiguousarray(a)).cuda()


def synth_matrices(T, api, t, n, rows, cols, seed):
    w = T.empty((n, rows * H.row_bytes(t, cols)), dtype=T.uint8, device="cuda")
    for e in range(n):
        api.synth_weights(t, seed + e, 0.02, rows, cols, w[e])
    T.cuda.synchronize()
    return w


def q4k_f16_weights(raw, rows, cols):
    """Q4_K weights as the kernel's packed-half arithmetic makes them: dl = f16(d * sc), ml = f16(dmin * m),
    w = f16(q * dl - ml) with the product and difference exact before the one rounding (a fused multiply-add)."""
    blk = np.ascontiguousarray(raw).reshape(rows, cols // 256, 144)
    d = blk[:, :, 0:2].copy().view(np.float16).astype(np.float32)            # [rows, nb, 1]
    dmin = blk[:, :, 2:4].copy().view(np.float16).astype(np.float32)
    sc8 = blk[:, :, 4:16].astype(np.int32)
    qs = blk[:, :, 16:144]
    out = np.empty((rows, cols // 256, 8, 32), np.float64)
    for sb in range(8):
        if sb < 4:
            sc, mn = sc8[:, :, sb] & 63, sc8[:, :, sb + 4] & 63
        else:
            sc = (sc8[:, :, sb + 4] & 0x0F) | ((sc8[:, :, sb - 4] >> 6) << 4)
            mn = (sc8[:, :, sb + 4] >> 4) | ((sc8[:, :, sb] >> 6) << 4)
        dl = (d[:, :, 0] * sc).astype(np.float16).astype(np.float64)
        ml = (dmin[:, :, 0] * mn).astype(np.float16).astype(np.float64)
        q = qs[:, :, 32 * (sb // 2):32 * (sb // 2) + 32]
        q = ((q >> 4) if sb & 1 else (q & 0x0F)).astype(np.float64)
        out[:, :, sb, :] = (q * dl[:, :, None] - ml[:, :, None]).astype(np.float16).astype(np.float64)
    return out.reshape(rows, cols)


def xq_ld(cols):
    """Values in a row of the activation image: the cols f16 values d * q, then one sum correction per 32 values, padded
    with zeros to a multiple of 64."""
    return cols + ((cols // 32 + 63) // 64) * 64


def sum_corrections(x_rows, image):
    """xa of every 32-value group: f16(S) - sum(d * q), S the f32 sum of the unquantized values in the order of llama.cpp's
    quantize_mmq_q8_1 (4 consecutive values left to right, then a tree at distances 4, 2, 1); stored as f16."""
    rows, cols = x_rows.shape
    pt = x_rows.astype(np.float32).reshape(rows, cols // 32, 8, 4)
    part = ((pt[..., 0] + pt[..., 1]).astype(np.float32) + pt[..., 2]).astype(np.float32)
    part = (part + pt[..., 3]).astype(np.float32)
    for off in (4, 2, 1):
        part = (part[..., :off] + part[..., off:2 * off]).astype(np.float32)
    S = part[..., 0].astype(np.float16).astype(np.float32)
    sxr = image.astype(np.float32).reshape(rows, cols // 32, 32).astype(np.float64).sum(axis=2).astype(np.float32)   # exact
    return (S - sxr).astype(np.float32).astype(np.float16)


def q4k_constant_terms(raw, rows, cols):
    """-f16(dmin * m) of every 32-value group of Q4_K rows: the A operand of the sum-correction steps."""
    blk = np.ascontiguousarray(raw).reshape(rows, cols // 256, 144)
    dmin = blk[:, :, 2:4].copy().view(np.float16).astype(np.float32)[:, :, 0]
    sc8 = blk[:, :, 4:16].astype(np.int32)
    mn = np.stack([(sc8[:, :, sb + 4] & 63) if sb < 4 else ((sc8[:, :, sb + 4] >> 4) | ((sc8[:, :, sb] >> 6) << 4))
                   for sb in range(8)], axis=-1)
    return -(dmin[:, :, None] * mn.astype(np.float32)).astype(np.float16).astype(np.float64).reshape(rows, cols // 32)


def q8_1_image(oracle, x_rows):
    """What maya_mmq_quantize stores: f16 rows d * q with the rounding of llama.cpp's quantize_mmq_q8_1 as the reference's
    host model states it (tests/glm_dsa/glmd_mmq_ids_test.cu:300-312) - per 32 values d_inv = 127 / amax,
    q = round(x * d_inv) (half away from zero), d = 1 / d_inv - with d kept as f16 (clamped to 65504)."""
    rows, cols = x_rows.shape
    xb = x_rows.astype(np.float32).reshape(rows, cols // 32, 32)
    am = np.abs(xb).max(axis=2, keepdims=True).astype(np.float32)
    with np.errstate(divide="ignore", invalid="ignore"):
        d_inv = (np.float32(127.0) / am).astype(np.float32)
        v = (xb * d_inv).astype(np.float32)
        d = np.minimum((np.float32(1.0) / d_inv).astype(np.float32), np.float32(65504.0))
    q = np.where(am > 0, np.clip(np.sign(v) * np.floor(np.abs(v).astype(np.float64) + 0.5), -127, 127), 0.0).astype(np.float32)
    dh = np.where(am > 0, d.astype(np.float16).astype(np.float32), np.float32(0.0))
    return (dh * q).astype(np.float16).reshape(rows, cols)


def iq_f16_weights(oracle, t, raw, rows, cols):
    """IQ2_S / IQ3_S weights as the kernel makes them: the sub-block scale rounded to f16 (IQ2_S d (2 ls + 1) / 8, IQ3_S
    d (1 + 2 s)), times the codebook magnitude, rounded to f16 once more, with the sign.  The magnitudes and signs are
    recovered from the oracle's exact dequantization (magnitude = |y| / exact scale, a small integer)."""
    bb = 82 if t == H.IQ2_S else 110
    blk = np.ascontiguousarray(raw).reshape(rows, cols // 256, bb)
    d = blk[:, :, 0:2].copy().view(np.float16).astype(np.float32)[:, :, 0]                    # [rows, nb]
    y = oracle.dequantize(t, raw, rows * cols).reshape(rows, cols // 256, 8, 32).astype(np.float64)
    if t == H.IQ2_S:
        sc = blk[:, :, 74:82].astype(np.int32)                                                # [rows, nb, 8]
        ls = np.stack([sc & 15, sc >> 4], axis=-1)                                            # per half sub-block of 16
        mult = (2 * ls + 1).astype(np.float32) * np.float32(0.125)                            # [rows, nb, 8, 2]
        exact = (d[:, :, None, None] * mult).astype(np.float64)
        sc16 = (d[:, :, None, None] * mult).astype(np.float16).astype(np.float64)
        exact = np.repeat(exact, 16, axis=-1)
        sc16 = np.repeat(sc16, 16, axis=-1)                                                   # [rows, nb, 8, 32]
    else:
        sb = blk[:, :, 106:110].astype(np.int32)                                              # [rows, nb, 4]
        nib = np.stack([sb & 15, sb >> 4], axis=-1).reshape(rows, cols // 256, 8)
        mult = (1 + 2 * nib).astype(np.float32)
        exact = np.repeat((d[:, :, None] * mult).astype(np.float64)[..., None], 32, axis=-1)
        sc16 = np.repeat((d[:, :, None] * mult).astype(np.float16).astype(np.float64)[..., None], 32, axis=-1)
    with np.errstate(divide="ignore", invalid="ignore"):
        mag = np.where(exact != 0, np.rint(np.abs(y) / exact), 0.0)
    w = (sc16 * mag).astype(np.float16).astype(np.float64) * np.where(y < 0, -1.0, 1.0)
    return w.reshape(rows, cols)


def f16_weights(oracle, t, w_host, rows, cols):
    if t == H.Q4_K:
        return q4k_f16_weights(w_host, rows, cols)
    if t in (H.IQ2_S, H.IQ3_S):
        return iq_f16_weights(oracle, t, w_host, rows, cols)
    return oracle.dequantize(t, w_host, rows * cols).reshape(rows, cols).astype(np.float16).astype(np.float64)


COUNTS = [0, 3, 130, 128, 1, 0, 257]


@pytest.mark.parametrize("t", [H.Q4_K, H.Q8_0, H.IQ2_S, H.IQ3_S])
def test_grouped_product_ragged_groups(T, api, oracle, t):
    n, rows, n_tok = len(COUNTS), 256, 40
    cols = 2048 if t in (H.IQ2_S, H.IQ3_S) else 512        # the i-quants need rows that start on 16 bytes
    w = synth_matrices(T, api, t, n, rows, cols, 11)
    rng = H.rng_for("mmq", t)
    x = (rng.standard_normal((n_tok, cols)) * 1.5).astype(np.float32)
    bounds = np.concatenate([[0], np.cumsum(COUNTS)]).astype(np.int32)
    total = int(bounds[-1])
    row_tok = rng.integers(0, n_tok, total).astype(np.int32)
    dst_row = rng.permutation(total + 5)[:total].astype(np.int32)            # scattered, with holes
    xq = api.mmq_quantize(dev(T, x), dev(T, row_tok), t)
    xq_full = xq.cpu().numpy().view(np.float16).reshape(total, xq_ld(cols))
    xq_host, xa_host = xq_full[:, :cols], xq_full[:, cols:cols + cols // 32]
    assert np.array_equal(xq_host, q8_1_image(oracle, x[row_tok])), "mmq_quantize differs from the model's d * q"
    assert np.array_equal(xa_host, sum_corrections(x[row_tok], xq_host)), "the groups' sum corrections"
    assert not xq_full[:, cols + cols // 32:].any(), "the padding behind the corrections"
    xq_blocks = [oracle.quantize_q8_1(x[r]) for r in row_tok]

    ld = rows + 64
    dst = T.full((total + 5, ld), 7.0, dtype=T.float32, device="cuda")
    err = T.zeros(1, dtype=T.int32, device="cuda")
    p = api.mmq_product(w, t, rows, cols, w.shape[1], n, xq, dev(T, bounds), dev(T, dst_row), total, dst, ld, error=err)
    api.mmq_run(p)
    T.cuda.synchronize()
    assert int(err.item()) == 0
    got = dst.cpu().numpy()
    w_host = w.cpu().numpy()
    hit = np.zeros(total + 5, bool)
    for e in range(n):
        a, b = int(bounds[e]), int(bounds[e + 1])
        if a == b:
            continue
        wf, xf = f16_weights(oracle, t, w_host[e], rows, cols), xq_host[a:b].astype(np.float64)
        pin = xf @ wf.T
        if t == H.Q4_K:       # the constant term of a group times the group's unquantized sum, as the reference's MMQ forms it
            pin = pin + xa_host[a:b].astype(np.float64) @ q4k_constant_terms(w_host[e], rows, cols).T
        g = got[dst_row[a:b], :rows]
        assert H.rel_err(g, pin) <= PIN, f"expert {e}: not the product of its f16 operands"
        # the decode kernels' q8_1 dot on the group's edge rows.  Q4_K: the reference's two paths differ from each other
        # there (the decode dot takes the sum of the ROUNDED activations for the constant term, its MMQ - and this path -
        # the stored sum of the unquantized ones: ~1.1e-2 in rel-L2 on these weights), hence the wider bound
        for r in (a, b - 1):
            want = oracle.mmvq(t, w_host[e], xq_blocks[r], cols, rows)[0]
            tol = 3e-2 if t == H.Q4_K else TOL
            assert H.rel_err(got[dst_row[r], :rows], want) <= tol and H.rel_l2(got[dst_row[r], :rows], want) <= tol
        # the reference's own host model of its prompt-path GEMM (tests/glm_dsa/glmd_mmq_ids_test.cu; its gate for its
        # MMQ kernels is rel-L2 < 1e-4): this path rounds the activation scale and the expanded weights to f16 on top
        model = oracle.mmq_host_model(t, w_host[e], rows, cols, x[row_tok[a:b]])
        assert H.rel_l2(g, model) <= MODEL, f"expert {e}: {H.rel_l2(g, model):.3g} from the reference's MMQ host model"
        hit[dst_row[a:b]] = True
    assert np.all(got[:, rows:] == 7.0), "wrote past w_rows"
    assert np.all(got[~hit] == 7.0), "wrote a row no group owns"


@pytest.mark.parametrize("t", [H.Q4_K, H.Q8_0, H.IQ2_S, H.IQ3_S])
@pytest.mark.parametrize("limit", [H.INF, 0.75])
def test_fused_glu_equals_product_then_swiglu_bitwise(T, api, t, limit):
    n, n_ff = 4, 256
    cols = 2048 if t in (H.IQ2_S, H.IQ3_S) else 768
    counts = [5, 0, 200, 64]
    w = synth_matrices(T, api, t, n, 2 * n_ff, cols, 23)
    x = (H.rng_for("glu", t).standard_normal((sum(counts), cols)) * 2.0).astype(np.float32)
    bounds = dev(T, np.concatenate([[0], np.cumsum(counts)]).astype(np.int32))
    total = sum(counts)
    xq = api.mmq_quantize(dev(T, x), None, t)
    gu = T.zeros((total, 2 * n_ff), dtype=T.float32, device="cuda")
    api.mmq_run(api.mmq_product(w, t, 2 * n_ff, cols, w.shape[1], n, xq, bounds, None, total, gu, 2 * n_ff))
    want = api.swiglu_rows(gu, n_ff, limit)
    h = T.zeros((total, n_ff), dtype=T.float32, device="cuda")
    api.mmq_run_glu(api.mmq_product(w, t, 2 * n_ff, cols, w.shape[1], n, xq, bounds, None, total, h, n_ff), limit)
    # ... and with the q8_1 rounding of h in the write-back: the same bits as quantizing h afterwards
    hq = T.zeros(api.mmq_q8_bytes(total, n_ff), dtype=T.uint8, device="cuda")
    api.mmq_run_glu(api.mmq_product(w, t, 2 * n_ff, cols, w.shape[1], n, xq, bounds, None, total, None, n_ff, xq_out=hq), limit)
    want_hq = api.mmq_quantize(want, None, t)
    T.cuda.synchronize()
    assert np.abs(gu.cpu().numpy()).max() > 0.1
    assert T.equal(h, want)
    assert T.equal(hq, want_hq)


@pytest.mark.parametrize("t", [H.Q4_K, H.Q8_0, H.IQ2_S, H.IQ3_S])
@pytest.mark.parametrize("rows", [160, 157, 129])
def test_tall_groups_equal_short_groups_bitwise(T, api, t, rows):
    """Groups of up to 160 rows, whose finished tiles fill the rings' shared memory, on blocks that take several tiles one after
    another: the bits of the same rows in groups of half the height."""
    n, cols, w_rows, half = 40, 2048, 2048, rows // 2
    w = synth_matrices(T, api, t, n, w_rows, cols, 41)
    xq = api.mmq_quantize(dev(T, H.rng_for("tall", t, rows).standard_normal((n * rows, cols)).astype(np.float32)), None, t)
    image = xq.view(n, rows, -1)

    def run(x, c):
        out = T.zeros((n * c, w_rows), dtype=T.float32, device="cuda")
        err = T.zeros(1, dtype=T.int32, device="cuda")
        api.mmq_run(api.mmq_product(w, t, w_rows, cols, w.shape[1], n, x, dev(T, np.arange(n + 1, dtype=np.int32) * c), None, n * c, out, w_rows, error=err))
        T.cuda.synchronize()
        assert int(err.item()) == 0
        return out.view(n, c, w_rows)

    got = run(xq, rows)
    assert T.isfinite(got).all()
    assert T.equal(got[:, :half], run(image[:, :half].contiguous(), half))
    assert T.equal(got[:, half:], run(image[:, half:].contiguous(), rows - half))


@pytest.mark.parametrize("t,cols", [(H.Q4_K, 256), (H.Q4_K, 1792), (H.Q4_K, 2304), (H.Q8_0, 256), (H.Q8_0, 768), (H.IQ2_S, 4096), (H.IQ3_S, 2048)])
def test_tiles_of_every_height_one_after_another_bitwise(T, api, t, cols):
    """A tile's rows decide how tensor memory and the activation ring are divided.  Blocks that take tiles of every division in turn
    (heights at both edges of each, more tiles than SMs; K of less than a ring, and Q4_K chunks of 1, 7 and 8 + 1 blocks): the bits of
    the same rows in groups of at most 16, which all have one division."""
    w_rows, heights = 512, [1, 160, 33, 32, 129, 64, 97, 65, 128, 96, 16, 17] * 8
    w1 = synth_matrices(T, api, t, 4, w_rows, cols, 61)
    w = w1[T.arange(len(heights), device="cuda") % 4].contiguous()
    total = sum(heights)
    xq = api.mmq_quantize(dev(T, H.rng_for("heights", t, cols).standard_normal((total, cols)).astype(np.float32)), None, t)

    def run(mats, counts):
        out = T.full((total, w_rows), 7.0, dtype=T.float32, device="cuda")
        err = T.zeros(1, dtype=T.int32, device="cuda")
        bounds = dev(T, np.concatenate([[0], np.cumsum(counts)]).astype(np.int32))
        api.mmq_run(api.mmq_product(mats, t, w_rows, cols, mats.shape[1], len(counts), xq, bounds, None, total, out, w_rows, error=err))
        T.cuda.synchronize()
        assert int(err.item()) == 0
        return out

    short = [(g % 4, min(16, h - at)) for g, h in enumerate(heights) for at in range(0, h, 16)]
    want = run(w1[T.tensor([e for e, _ in short], device="cuda")].contiguous(), [n for _, n in short])
    got = run(w, heights)
    assert T.isfinite(got).all() and float(got.abs().max()) > 0.1
    assert T.equal(got, want)


@pytest.mark.parametrize("t,cols", [(H.Q4_K, 256), (H.Q4_K, 1792), (H.Q4_K, 2304), (H.Q8_0, 256), (H.Q8_0, 768), (H.IQ2_S, 4096), (H.IQ3_S, 2048)])
def test_tiles_of_every_height_behind_every_other_bitwise(T, api, t, cols):
    """A tile's rows decide how tensor memory and the activation ring are divided.  Blocks that take ten tiles and more, every division behind
    every other (heights at both edges of each; K of less than a ring, and Q4_K chunks of 1, 7 and 8 + 1 blocks), plain and with
    SwiGLU and the rounding of h in the write-back: the bits of the same rows in groups of at most 16, which all have one division."""
    w_rows, heights = 1024, [int(h) for h in H.rng_for("heights order").permutation([1, 160, 33, 32, 129, 64, 97, 65, 128, 96, 16, 17] * 31)]
    sms, per_group = T.cuda.get_device_properties(0).multi_processor_count, w_rows // 256
    division = np.repeat([(h + 31) // 32 for h in heights], per_group)               # of every tile; block b's are b, b + sms, ...
    assert len(division) >= 10 * sms and len(set(zip(division, division[sms:]))) == 25
    w1 = synth_matrices(T, api, t, 4, w_rows, cols, 61)
    w = w1[T.arange(len(heights), device="cuda") % 4].contiguous()
    total = sum(heights)
    xq = api.mmq_quantize(dev(T, H.rng_for("heights", t, cols).standard_normal((total, cols)).astype(np.float32)), None, t)

    def run(mats, counts):
        out = T.full((total, w_rows), 7.0, dtype=T.float32, device="cuda")
        err = T.zeros(1, dtype=T.int32, device="cuda")
        bounds = dev(T, np.concatenate([[0], np.cumsum(counts)]).astype(np.int32))
        api.mmq_run(api.mmq_product(mats, t, w_rows, cols, mats.shape[1], len(counts), xq, bounds, None, total, out, w_rows, error=err))
        n_ff = w_rows // 2
        hq = T.zeros(api.mmq_q8_bytes(total, n_ff), dtype=T.uint8, device="cuda")
        api.mmq_run_glu(api.mmq_product(mats, t, w_rows, cols, mats.shape[1], len(counts), xq, bounds, None, total, None, n_ff, error=err, xq_out=hq), 7.0)
        T.cuda.synchronize()
        assert int(err.item()) == 0
        return out, hq

    short = [(g % 4, min(16, h - at)) for g, h in enumerate(heights) for at in range(0, h, 16)]
    want, want_hq = run(w1[T.tensor([e for e, _ in short], device="cuda")].contiguous(), [n for _, n in short])
    got, got_hq = run(w, heights)
    assert T.isfinite(got).all() and float(got.abs().max()) > 0.1
    assert T.equal(got, want) and T.equal(got_hq, want_hq)


@pytest.mark.parametrize("t", [H.Q4_K, H.Q8_0, H.IQ2_S, H.IQ3_S])
@pytest.mark.parametrize("copies", [1, 2, 3, 4, 5])
def test_k_values_are_added_in_order(T, api, t, copies):
    """The f32 sums run over K from its start to its end, 64 values after 64, at every division of tensor memory.  Row r has X at the first of
    the 64 values r, Y at those of r + 1 and -X at those of r + 2, and all weights are one w: X w + Y w is X w in f32 (Y / X = 2^-29, of the
    same sign, so that it is lost whether the sum is rounded or cut off), and the row's result is 0.  Were r + 1 added before r or
    behind r + 2, Y w would be left."""
    cols, w_rows = 2048, 256
    if t == H.Q8_0:           # d = 0.5, q = 3
        block = np.concatenate([np.array([0.5], np.float16).view(np.uint8), np.full(32, 3, np.uint8)])
    elif t == H.Q4_K:         # d = 0.5, dmin = 0, every scale 1 and minimum 0, every q 3
        block = np.concatenate([np.array([0.5, 0.0], np.float16).view(np.uint8), np.array([1, 1, 1, 1, 0, 0, 0, 0, 1, 1, 1, 1], np.uint8), np.full(128, 0x33, np.uint8)])
    else:                     # d = 0.5, every index 0, no signs, every scale 1
        block = np.zeros(82 if t == H.IQ2_S else 110, np.uint8)
        block[:2] = np.array([0.5], np.float16).view(np.uint8)
        block[-8 if t == H.IQ2_S else -4:] = 0x11
    w = dev(T, np.tile(np.tile(block, H.row_bytes(t, cols) // len(block)), w_rows)[None])
    rows = cols // 64 - 2
    x = np.zeros((rows, cols), np.float32)
    for r in range(rows):
        x[r, 64 * r], x[r, 64 * r + 64], x[r, 64 * r + 128] = 2.0 ** 14, 2.0 ** -15, -2.0 ** 14
    x = np.tile(x, (copies, 1))
    n = len(x)

    def run(values):
        out = T.full((n, w_rows), 7.0, dtype=T.float32, device="cuda")
        xq = api.mmq_quantize(dev(T, values), None, t)
        api.mmq_run(api.mmq_product(w, t, w_rows, cols, w.shape[1], 1, xq, dev(T, np.array([0, n], np.int32)), None, n, out, w_rows))
        T.cuda.synchronize()
        return out.cpu().numpy()

    small = x.copy()
    small[np.abs(x) > 1.0] = 0.0
    assert (run(small) != 0).all()
    np.testing.assert_array_equal(run(x), 0.0)


@pytest.mark.parametrize("ta,tb,counts,n_ff", [
    (H.Q8_0, H.Q4_K, [1, 0, 161, 7, 320, 33], 256),                                       # fewer tiles than blocks, remainders of 160 rows
    (H.IQ2_S, H.IQ3_S, [5] * 24 + [0] * 3 + [170] * 3, 2048),                             # several rounds of tiles
    (H.Q4_K, H.Q8_0, [0] * 6, 256)])                                                      # no rows at all in one pair
def test_chain_equals_its_products_bitwise(T, api, ta, tb, counts, n_ff):
    """Two pairs of gate/up and down products in one chain, each down tile starting when its own rows of h are there: the bits
    of the four products run one after another - twice, on the same counters, which end at zero."""
    cols = 2048
    pairs = []
    for t, c in ((ta, counts), (tb, counts[::-1] if sum(counts) else [3, 200, 0, 9, 1, 64])):
        w, total = synth_matrices(T, api, t, len(c), 2 * n_ff, cols, 31), sum(c)
        wd = synth_matrices(T, api, t, len(c), 512, n_ff, 37)
        x = (H.rng_for("chain", t).standard_normal((max(total, 1), cols)) * 2.0).astype(np.float32)
        pairs.append(dict(t=t, n=len(c), w=w, wd=wd, total=total, xq=api.mmq_quantize(dev(T, x), None, t),
                          bounds=dev(T, np.concatenate([[0], np.cumsum(c)]).astype(np.int32))))
    err = T.zeros(1, dtype=T.int32, device="cuda")

    def products(p):
        hq = T.zeros(max(api.mmq_q8_bytes(p["total"], n_ff), 16), dtype=T.uint8, device="cuda")
        out = T.zeros((max(p["total"], 1), 512), dtype=T.float32, device="cuda")
        return (api.mmq_product(p["w"], p["t"], 2 * n_ff, cols, p["w"].shape[1], p["n"], p["xq"], p["bounds"], None, p["total"], None, n_ff,
                                error=err, xq_out=hq),
                api.mmq_product(p["wd"], p["t"], 512, n_ff, p["wd"].shape[1], p["n"], hq, p["bounds"], None, p["total"], out, 512, error=err), hq, out)

    want = [products(p) for p in pairs]
    for gu, dn, _, _ in want:
        api.mmq_run_glu(gu, 7.0)
        api.mmq_run(dn)
    counters = T.zeros(4096, dtype=T.uint8, device="cuda")
    for _ in range(2):
        got = [products(p) for p in pairs]
        api.mmq_run_chain([g[0] for g in got], [g[1] for g in got], 7.0, counters)
        T.cuda.synchronize()
        assert int(err.item()) == 0 and not counters.any()
        for a, b in zip(got, want):
            assert T.equal(a[2], b[2]) and T.equal(a[3], b[3])
    assert want[1][3].abs().max() > 0.01
    with pytest.raises(api.MayaError):                                                    # the down product reads another h
        api.mmq_run_chain([want[0][0]], [got[0][1]], 7.0, counters)


def test_chain_of_tiles_of_every_height_equals_its_products_bitwise(T, api):
    """A chain's tiles are taken as blocks get to them: ten a block and more, every division of tensor memory behind others, i-quants in one pair
    and Q4_K in the other.  The bits of the four products run one after another; the counters end at zero."""
    cols, n_ff, counts = 2048, 2048, [97, 1, 160, 33, 16, 129, 64, 32, 65, 128, 17, 96] * 4
    n, total = len(counts), sum(counts)
    assert 2 * n * (n_ff // 128 + 512 // 256) >= 10 * T.cuda.get_device_properties(0).multi_processor_count
    err = T.zeros(1, dtype=T.int32, device="cuda")
    pairs = []
    for t, c in ((H.IQ3_S, counts), (H.Q4_K, counts[::-1])):
        x = H.rng_for("chain heights", t).standard_normal((total, cols)).astype(np.float32)
        pairs.append((t, synth_matrices(T, api, t, n, 2 * n_ff, cols, 31), synth_matrices(T, api, t, n, 512, n_ff, 37),
                      api.mmq_quantize(dev(T, x), None, t), dev(T, np.concatenate([[0], np.cumsum(c)]).astype(np.int32))))

    def products(t, w, wd, xq, bounds):
        hq = T.zeros(api.mmq_q8_bytes(total, n_ff), dtype=T.uint8, device="cuda")
        out = T.zeros((total, 512), dtype=T.float32, device="cuda")
        return (api.mmq_product(w, t, 2 * n_ff, cols, w.shape[1], n, xq, bounds, None, total, None, n_ff, error=err, xq_out=hq),
                api.mmq_product(wd, t, 512, n_ff, wd.shape[1], n, hq, bounds, None, total, out, 512, error=err), hq, out)

    want = [products(*p) for p in pairs]
    for gu, dn, _, _ in want:
        api.mmq_run_glu(gu, 7.0)
        api.mmq_run(dn)
    counters = T.zeros(api._lib.load().maya_mmq_chain_bytes(2 * total, 2 * n, 2), dtype=T.uint8, device="cuda")
    got = [products(*p) for p in pairs]
    api.mmq_run_chain([g[0] for g in got], [g[1] for g in got], 7.0, counters)
    T.cuda.synchronize()
    assert int(err.item()) == 0 and not counters.any()
    for a, b in zip(got, want):
        assert T.equal(a[2], b[2]) and T.equal(a[3], b[3])
    assert min(float(p[3].abs().max()) for p in want) > 0.01


def test_refused_chain_launches_nothing_and_leaves_its_counters_alone(T, api, lib):
    """A chain with one product that cannot run is refused before its first launch, whichever product it is; the next chain on the
    same counters gives the bits of its products run one after another."""
    t, n_ff, cols, counts = H.Q8_0, 256, 256, [70, 5, 0, 200]
    n, total = len(counts), sum(counts)
    w, wd = synth_matrices(T, api, t, n, 2 * n_ff, cols, 41), synth_matrices(T, api, t, n, 256, n_ff, 43)
    bounds = dev(T, np.concatenate([[0], np.cumsum(counts)]).astype(np.int32))
    xq = api.mmq_quantize(dev(T, H.rng_for("refused-chain").standard_normal((total, cols)).astype(np.float32)), None, t)
    hq = T.zeros(api.mmq_q8_bytes(total, 2 * n_ff), dtype=T.uint8, device="cuda")         # (room for the wider h asked for below)
    out = T.zeros((total, 256), dtype=T.float32, device="cuda")
    gu = lambda **kw: api.mmq_product(**{**dict(w=w, ggml_type=t, w_rows=2 * n_ff, w_cols=cols, expert_bytes=w.shape[1], n=n, xq=xq,  # noqa: E731
                                                 bounds=bounds, ids=None, total_rows=total, dst=None, ld_dst=n_ff, xq_out=hq), **kw})
    dn = lambda **kw: api.mmq_product(**{**dict(w=wd, ggml_type=t, w_rows=256, w_cols=n_ff, expert_bytes=wd.shape[1], n=n, xq=hq,     # noqa: E731
                                                 bounds=bounds, ids=None, total_rows=total, dst=out, ld_dst=256), **kw})
    api.mmq_run_glu(gu(), H.INF)
    api.mmq_run(dn())
    want = out.clone()
    counters = T.zeros(api._lib.load().maya_mmq_chain_bytes(total, 2 * n, 2), dtype=T.uint8, device="cuda")
    T.cuda.synchronize()
    launches = lib.maya_launch_count()
    for bad in (dn(ld_dst=128), dn(dst=None), dn(ggml_type=H.Q5_K), dn(ggml_type=H.IQ3_S), dn(w_rows=200), dn(w_cols=2 * n_ff)):
        for pairs in ([(gu(), bad)], [(gu(), dn()), (gu(), bad)]):
            with pytest.raises(api.MayaError):
                api.mmq_run_chain([p[0] for p in pairs], [p[1] for p in pairs], H.INF, counters)
            T.cuda.synchronize()
            assert lib.maya_launch_count() == launches and not counters.any()
    with pytest.raises(api.MayaError):
        api.mmq_run_chain([gu(w_rows=100)], [dn()], H.INF, counters)
    assert lib.maya_launch_count() == launches
    out.zero_(), hq.zero_()
    api.mmq_run_chain([gu()], [dn()], H.INF, counters)
    T.cuda.synchronize()
    assert T.equal(out, want) and not counters.any()


def test_expert_map_selects_bounds_entries(T, api):
    """A staged group: matrix i of the product owns the rows of expert expert_map[i]."""
    t, rows, cols = H.Q4_K, 128, 256
    w = synth_matrices(T, api, t, 2, rows, cols, 5)
    counts = [4, 9, 0, 6]
    bounds = dev(T, np.concatenate([[0], np.cumsum(counts)]).astype(np.int32))
    total = sum(counts)
    x = H.rng_for("map").standard_normal((total, cols)).astype(np.float32)
    xq = api.mmq_quantize(dev(T, x), None, t)
    emap = dev(T, np.array([3, 1], np.int32))
    dst = T.zeros((total, rows), dtype=T.float32, device="cuda")
    api.mmq_run(api.mmq_product(w, t, rows, cols, w.shape[1], 2, xq, bounds, None, total, dst, rows, expert_map=emap))
    ref = T.zeros((total, rows), dtype=T.float32, device="cuda")
    for i, e in enumerate([3, 1]):
        b = np.zeros(2, np.int32)
        b[0], b[1] = sum(counts[:e]), sum(counts[: e + 1])
        api.mmq_run(api.mmq_product(w[i], t, rows, cols, w.shape[1], 1, xq, dev(T, b), None, total, ref, rows))
    T.cuda.synchronize()
    assert T.equal(dst, ref)
    assert float(dst[:4].abs().max()) == 0.0 and float(dst[13:].abs().max()) > 0.0


def test_refusals(T, api):
    t = H.Q4_K
    w = T.zeros(128 * H.row_bytes(t, 256), dtype=T.uint8, device="cuda")
    b = dev(T, np.array([0, 1], np.int32))
    xq = T.zeros(api.mmq_q8_bytes(1, 256), dtype=T.uint8, device="cuda")
    dst = T.zeros((1, 128), dtype=T.float32, device="cuda")
    ok = lambda **kw: api.mmq_product(**{**dict(w=w, ggml_type=t, w_rows=128, w_cols=256, expert_bytes=w.numel(), n=1, xq=xq,
                                                 bounds=b, ids=None, total_rows=1, dst=dst, ld_dst=128), **kw})
    api.mmq_run(ok())
    for bad in (dict(ggml_type=H.IQ2_S), dict(w_rows=100), dict(w_cols=96), dict(ld_dst=64), dict(expert_bytes=w.numel() + 8)):
        with pytest.raises(api.MayaError):
            api.mmq_run(ok(**bad))
    far = H.row_bytes(t, 256) * 128
    with pytest.raises(api.MayaError):                    # matrices further apart than a tensor map's 40-bit stride: not launched, not 0
        api.mmq_run(ok(expert_bytes=far * ((1 << 40) // far + 1)))
    with pytest.raises(api.MayaError):
        api.mmq_run_glu(ok(w_rows=128), H.INF)            # n_ff = 64 is not a multiple of 128
    assert api.mmq_q8_bytes(3, 100) == 0 and api.mmq_q8_bytes(3, 256) == 3 * xq_ld(256) * 2
    assert all(api.mmq_supported(x) for x in (H.Q8_0, H.Q4_K, H.IQ2_S, H.IQ3_S)) and not api.mmq_supported(2)


# ------------------------------------------------------------------------------------------------ the whole layer
def oracle_prefill_token(oracle, cfg, experts, ids, w, x):
    """A token as the reference's prompt path computes it: every expert by oracle.expert_mmq (the host model of the
    reference's MMQ arithmetic), combined in glmb::moe_combine's order."""
    H_, FF = cfg["n_embd"], cfg["n_ff"]
    parts = np.stack([oracle.expert_mmq(cfg["gu_type"], cfg["d_type"], experts[int(e)].cpu().numpy(), H_, FF, H.INF, x)
                      for e in ids])
    out = np.zeros(H_, np.float32)
    for j in range(len(ids)):                               # glmb::moe_combine's order: m = fma(w, o, m) from 0
        out = (np.float32(w[j]) * parts[j].astype(np.float32) + out).astype(np.float32)
    return out


@pytest.mark.parametrize("t,n_tok,E", [(H.Q4_K, 300, 16), (H.Q8_0, 77, 8), (H.IQ2_S, 200, 8), (H.IQ3_S, 90, 4)])
def test_prefill_layer_small(T, api, oracle, t, n_tok, E):
    iq = t in (H.IQ2_S, H.IQ3_S)
    cfg = dict(n_embd=2048 if iq else 512, n_ff=2048 if iq else 256, n_expert=E, k=4, gu_type=t, d_type=t)
    lc = api.MoeLayerConfig(cfg["n_embd"], cfg["n_ff"], E, cfg["k"], t, t)
    experts = T.empty((E, lc.blob_bytes), dtype=T.uint8, device="cuda")
    gu_bytes = 2 * cfg["n_ff"] * H.row_bytes(t, cfg["n_embd"])
    for e in range(E):
        api.synth_weights(t, 900 + 2 * e, 0.05, 2 * cfg["n_ff"], cfg["n_embd"], experts[e, :gu_bytes])
        api.synth_weights(t, 901 + 2 * e, 0.05, cfg["n_embd"], cfg["n_ff"], experts[e, gu_bytes:])
    logits = H.router_logits("pf", n_tok, E, None)
    x = H.activations("pf", n_tok, cfg["n_embd"], "f32")
    pf = api.MoePrefill(lc, experts, max_tokens=n_tok)
    ids, w, ffn = pf.forward(dev(T, logits), dev(T, x))
    T.cuda.synchronize()
    assert pf.error() == 0
    ids_o, w_o = oracle.router_top10(logits, cfg["k"])
    assert np.array_equal(ids.cpu().numpy(), ids_o)
    got = ffn.cpu().numpy()
    # Down rows of 256 values: the q8_1 rounding of h alone is ~2e-2 from the exact product there, and two evaluations whose
    # h differ by 1e-3 (f16 operands against the model's floats) land ~1e-2 apart through flipped roundings - hence the
    # wide bound on this small shape; each product by itself is pinned to 1e-3 in test_grouped_product_ragged_groups.
    for tok in (0, n_tok // 2, n_tok - 1):
        want = oracle_prefill_token(oracle, cfg, experts, ids_o[tok], w_o[tok], x[tok])
        assert H.rel_err(got[tok], want) <= 2.5e-2 and H.rel_l2(got[tok], want) <= 2.5e-2


def test_prefill_layer_recovers_after_a_chain_that_gave_up(T, api):
    """A chain whose bounded wait ran out leaves its counters part-way and sets the error word - the state is made here on the host;
    error() reports it and the passes after it give the right bits again."""
    cfg = api.MoeLayerConfig(512, 256, 8, 2, H.Q4_K, H.Q4_K)
    experts = T.empty((8, cfg.blob_bytes), dtype=T.uint8, device="cuda")
    api.synth_weights(H.Q4_K, 5, 0.02, experts.numel() // H.row_bytes(H.Q4_K, 256), 256, experts)
    layer = api.MoePrefill(cfg, experts, max_tokens=40)
    passes = [(dev(T, H.router_logits("recover", 40, 8, None)) * s, dev(T, H.activations("recover", 40, 512, "f32")) * s) for s in (1.0, -0.5)]
    want = [layer.forward(*p)[2].clone() for p in passes]
    assert layer.error() == 0 and not T.equal(want[0], want[1])
    layer.chain.fill_(1)
    layer.err.fill_(1)
    assert layer.error() == 1
    for p, w in zip(passes, want):
        assert T.equal(layer.forward(*p)[2], w)


def build_pools(T, api, cfg, types, seed, sigma=0.02):
    """One pool of synthetic [gate | up | down] blobs per storage type; returns (pools for MoePrefill, blob of expert e)."""
    H_, FF = cfg["n_embd"], cfg["n_ff"]
    pools, where = [], {}
    for t in sorted(set(int(v) for v in types)):
        members = [e for e in range(len(types)) if int(types[e]) == t]
        gu_bytes = 2 * FF * H.row_bytes(t, H_)
        blobs = T.empty((len(members), gu_bytes + H_ * H.row_bytes(t, FF)), dtype=T.uint8, device="cuda")
        for i, e in enumerate(members):
            api.synth_weights(t, seed + 2 * e, sigma, 2 * FF, H_, blobs[i, :gu_bytes])
            api.synth_weights(t, seed + 2 * e + 1, sigma, H_, FF, blobs[i, gu_bytes:])
            where[e] = (t, blobs, i)
        pools.append((t, blobs, members))
    T.cuda.synchronize()
    return pools, where


def test_prefill_c4_shape(T, api, oracle):
    """Configuration C4 at its full shape: 4096 tokens x top-8 over 256 experts = 32768 routed rows, bf16 activations,
    half of the experts stored as Q8_0 and half as Q4_K (seeded assignment).  Six tokens against the oracle's model of the
    reference's prompt-path arithmetic (oracle.expert_mmq); every token's expert ids; row
    conservation (every routed pair has exactly one sorted row); and a chunk's results do not depend on what else is in
    the chunk - the first 512 tokens alone give the same bits."""
    c = H.CONFIGS["C4"]
    cfg = dict(n_embd=c["n_embd"], n_ff=c["n_ff"], n_expert=c["n_expert"], k=c["k"])
    n_tok, E = c["T"], c["n_expert"]
    types = H.expert_types("C4", E, c["types"])
    assert (types == H.Q8_0).sum() == E // 2 and (types == H.Q4_K).sum() == E // 2
    pools, where = build_pools(T, api, cfg, types, 5000)
    lc = api.MoeLayerConfig(cfg["n_embd"], cfg["n_ff"], E, cfg["k"], H.Q8_0, H.Q8_0)
    logits = H.router_logits("c4", n_tok, E, None)
    x = H.activations("c4", n_tok, cfg["n_embd"], "bf16")
    x_dev = dev(T, x).to(T.bfloat16)
    pf = api.MoePrefill(lc, None, max_tokens=n_tok, pools=pools)
    ids, w, ffn = pf.forward(dev(T, logits), x_dev)
    T.cuda.synchronize()
    assert pf.error() == 0
    got = ffn.cpu().numpy().copy()
    pos = pf.pos.cpu().numpy()
    assert np.array_equal(np.sort(pos), np.arange(n_tok * cfg["k"]))
    assert int(pf.bounds[-1].item()) == n_tok * cfg["k"]
    ids_o, w_o = oracle.router_top10(logits, cfg["k"])
    assert np.array_equal(ids.cpu().numpy(), ids_o)
    for tok in (0, 1, 3, 1000, 2047, 4095):
        want = np.zeros(cfg["n_embd"], np.float32)
        seen = set()
        for j, e in enumerate(ids_o[tok]):
            t, blobs, i = where[int(e)]
            seen.add(t)
            part = oracle.expert_mmq(t, t, blobs[i].cpu().numpy(), cfg["n_embd"], cfg["n_ff"], H.INF, x[tok])
            want = (np.float32(w_o[tok][j]) * part + want).astype(np.float32)
        assert H.rel_err(got[tok], want) <= TOL and H.rel_l2(got[tok], want) <= LAYER_L2
    _, _, ffn2 = pf.forward(dev(T, logits[:512]), x_dev[:512])
    T.cuda.synchronize()
    assert np.array_equal(ffn2.cpu().numpy(), got[:512])


def test_c5_batch64_through_prompt_path_and_expert_parallel_partition(T, api, oracle):
    """Configuration C5's 64-token batch (IQ3_S experts, Zipf-skewed routing) through the prompt path: a few tokens
    against the oracle, and the expert-parallel partition - each of 4 ranks computes only its 1/4 of the experts and
    combines only their rows - adds up (rank order) to the one-rank result up to summation order."""
    c = H.CONFIGS["C5"]
    E, k, Hd, FF, n_tok = 32, c["k"], c["n_embd"], c["n_ff"], 64
    t = c["gu_type"]
    cfg = dict(n_embd=Hd, n_ff=FF, n_expert=E, k=k, gu_type=t, d_type=t)
    lc = api.MoeLayerConfig(Hd, FF, E, k, t, t)
    experts = T.empty((E, lc.blob_bytes), dtype=T.uint8, device="cuda")
    gu_bytes = 2 * FF * H.row_bytes(t, Hd)
    for e in range(E):
        api.synth_weights(t, 7700 + 2 * e, 0.02, 2 * FF, Hd, experts[e, :gu_bytes])
        api.synth_weights(t, 7701 + 2 * e, 0.02, Hd, FF, experts[e, gu_bytes:])
    T.cuda.synchronize()
    logits = H.router_logits("C5", n_tok, E, 1.1)
    x = H.activations("C5", n_tok, Hd, "bf16")
    ld, xd = dev(T, logits), dev(T, x).to(T.bfloat16)
    whole = api.MoePrefill(lc, experts, max_tokens=n_tok)
    ids, w, ffn = whole.forward(ld, xd)
    T.cuda.synchronize()
    assert whole.error() == 0
    got = ffn.cpu().numpy().copy()
    ids_o, w_o = oracle.router_top10(logits, k)
    assert np.array_equal(ids.cpu().numpy(), ids_o)
    for tok in (0, 31, 63):
        want = oracle_prefill_token(oracle, cfg, experts, ids_o[tok], w_o[tok], x[tok])
        assert H.rel_err(got[tok], want) <= TOL and H.rel_l2(got[tok], want) <= LAYER_L2
    n_ranks, per = 4, E // 4
    partial = []
    for r in range(n_ranks):
        rank = api.MoePrefill(lc, experts, max_tokens=n_tok, expert_range=(r * per, (r + 1) * per))
        partial.append(rank.forward(ld, xd)[2].cpu().numpy().copy())
        assert rank.error() == 0
    summed = np.stack([oracle.allreduce_in_order(np.stack([p[tk] for p in partial])) for tk in range(n_tok)])
    assert H.rel_err(summed, got) <= 1e-5
    assert all(np.abs(p).max() > 0 for p in partial)
    # the same partition with the cross-rank sum inside the combine launch: the four ranks run one after another on
    # this GPU, the pushes of the ranks that have not run yet placed into a rank's receive buffers beforehand
    from project_maya_b200.peer import PeerGroup
    from test_gpu_allreduce import place_peer_pushes
    ranks = PeerGroup.on_one_device(n_ranks, stride=n_tok * Hd, timeout_ms=200.0)
    vecs = [T.from_numpy(p.reshape(-1)).cuda() for p in partial]
    for mi in range(n_ranks):
        place_peer_pushes(T, ranks, mi, 1, vecs, later_only=True)
    for r in range(n_ranks):
        rank = api.MoePrefill(lc, experts, max_tokens=n_tok, expert_range=(r * per, (r + 1) * per))
        fused = rank.forward(ld, xd, peer=ranks[r])[2]
        T.cuda.synchronize()
        assert not ranks[r].poisoned()
        assert fused.cpu().numpy().tobytes() == summed.tobytes(), f"rank {r}: not the rank-ordered sum"


@pytest.mark.parametrize("n_tok,k,E", [(1, 8, 256), (37, 8, 16), (300, 4, 8), (4096, 8, 256), (129, 1, 3)])
def test_expert_group_is_the_stable_sort_by_expert(T, api, n_tok, k, E):
    """glmb::expert_count / expert_scatter (glm_batch.hpp:131-139): a pair's rank is the number of earlier pairs routed to
    the same expert, its sorted row = the expert's base + rank - numpy's stable argsort by expert id."""
    rng = H.rng_for(f"group-{n_tok}-{k}-{E}")
    ids = np.stack([rng.choice(E, size=min(k, E), replace=False) for _ in range(n_tok)]).astype(np.int32)
    k = ids.shape[1]
    counts, bounds, pos, row_tok = api.expert_group(dev(T, ids), E)
    T.cuda.synchronize()
    flat = ids.reshape(-1)
    want_counts = np.bincount(flat, minlength=E)
    order = np.argsort(flat, kind="stable")
    assert np.array_equal(counts.cpu().numpy(), want_counts)
    assert np.array_equal(bounds.cpu().numpy(), np.concatenate([[0], np.cumsum(want_counts)]))
    assert np.array_equal(row_tok.cpu().numpy(), order // k)
    want_pos = np.empty_like(order)
    want_pos[order] = np.arange(order.size)
    assert np.array_equal(pos.cpu().numpy(), want_pos)


@pytest.mark.parametrize("n_tok,k,E", [(1, 4, 8), (300, 8, 16), (512, 8, 16), (513, 8, 16)])
def test_prefill_counts_each_experts_tokens(T, api, n_tok, k, E):
    """MoePrefill.counts after a call, on both sides of the 4096 pairs up to which the rows are grouped in one launch."""
    lc = api.MoeLayerConfig(256, 256, E, k, H.Q8_0, H.Q8_0)
    layer = api.MoePrefill(lc, T.zeros((E, lc.blob_bytes), dtype=T.uint8, device="cuda"), max_tokens=n_tok)
    layer.counts.fill_(-5)
    ids = layer.forward(dev(T, H.router_logits("counts", n_tok, E, None)), dev(T, H.activations("counts", n_tok, 256, "f32")))[0]
    T.cuda.synchronize()
    assert T.equal(layer.counts, T.bincount(ids.flatten(), minlength=E).int())


@pytest.mark.parametrize("n_tok,k,E", [(1, 1, 1), (1, 8, 256), (129, 1, 3), (37, 7, 16), (300, 5, 1024), (127, 8, 1000), (4096, 8, 256)])
def test_grouping_in_one_launch_equals_three(T, api, lib, n_tok, k, E):
    """maya_expert_group against expert_count, expert_bounds and expert_scatter (the test above pins those): one warp's pairs and
    all 32 warps', remainders of 32, one expert and as many as it takes, everything routed to one of many; more are refused."""
    for spread in (E, 1):
        ids = dev(T, H.rng_for("group1", n_tok, k, E).integers(0, spread, (n_tok, k)).astype(np.int32))
        n = n_tok * k
        counts, rank, row_tok, pos = (T.full((m,), -5, dtype=T.int32, device="cuda") for m in (E, n, n, n))
        bounds = T.full((E + 1,), -5, dtype=T.int32, device="cuda")
        p = lambda *ts: [t.data_ptr() for t in ts]  # noqa: E731
        assert lib.maya_expert_count(*p(ids), n, E, *p(counts, rank), None) == 0
        assert lib.maya_expert_bounds(*p(counts), E, *p(bounds), None) == 0
        assert lib.maya_expert_scatter(*p(ids, rank, bounds), n, k, *p(row_tok, pos), None) == 0
        rank1, row_tok1, pos1 = (T.full((n,), -5, dtype=T.int32, device="cuda") for _ in range(3))
        bounds1 = T.full((E + 1,), -5, dtype=T.int32, device="cuda")
        for _ in range(2):
            assert lib.maya_expert_group(*p(ids), n, k, E, *p(rank1, bounds1, row_tok1, pos1), None) == 0
        T.cuda.synchronize()
        assert T.equal(bounds1, bounds) and T.equal(row_tok1, row_tok) and T.equal(pos1, pos)
    assert lib.maya_expert_group(*p(ids), n, k, 1025, *p(rank1, bounds1, row_tok1, pos1), None) == -4


@pytest.mark.parametrize("cols", [256, 1536, 96])
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_routed_quantizer_writes_the_gathered_image(T, api, cols, dtype):
    """maya_mmq_quantize_routed (each token rounded once, stored to its k sorted rows) against maya_mmq_quantize through
    row_tok (mmq::quantize with ids, moe_mmq.hpp:34): the same bytes."""
    n_tok, k, E = 53, 4, 7
    rng = H.rng_for(f"routedq-{cols}-{dtype}")
    ids = np.stack([rng.choice(E, size=k, replace=False) for _ in range(n_tok)]).astype(np.int32)
    x = dev(T, rng.standard_normal((n_tok, cols)).astype(np.float32))
    x[5] = 0.0                                              # an all-zero row: d = 0, every correction 0
    if dtype == "bf16":
        x = x.to(T.bfloat16)
    _, _, pos, row_tok = api.expert_group(dev(T, ids), E)
    want = api.mmq_quantize(x, row_tok, H.Q4_K)
    got = T.full_like(want, 0xA5)
    api.mmq_quantize_routed(x, pos, k, H.Q4_K, xq=got)
    T.cuda.synchronize()
    assert T.equal(got, want)


@pytest.mark.parametrize("k", [8, 3])
def test_combine_rows_four_columns_a_thread_equals_one_column_a_thread(T, api, k):
    """maya_moe_combine_rows takes four columns a thread when its rows are 16-byte aligned, one otherwise: the same
    chain m = 0, m = fma(w_j, out[pos_j], m) in plan order, + sh - bitwise."""
    n_tok, n_embd = 41, 520
    rng = H.rng_for(f"combine4-{k}")
    n = n_tok * k
    pos = dev(T, rng.permutation(n).astype(np.int32))
    w = dev(T, rng.random((n_tok, k)).astype(np.float32))
    sh = dev(T, rng.standard_normal((n_tok, n_embd)).astype(np.float32))
    buf = dev(T, rng.standard_normal(n * n_embd + 4).astype(np.float32))
    out_al = buf[:n * n_embd].view(n, n_embd)
    out_off = buf[1:1 + n * n_embd]                          # 4 bytes off a 16-byte boundary: the one-column kernel
    out_off.copy_(out_al.reshape(-1).clone())
    out_off = out_off.view(n, n_embd)
    out_al2 = out_off.clone()                                # aligned again, same values
    a = api.moe_combine_rows(out_al2, pos, w, sh, n_tok, k, n_embd)
    b = api.moe_combine_rows(out_off, pos, w, sh, n_tok, k, n_embd)
    c = api.moe_combine_rows(out_al2, pos, w, None, n_tok, k, n_embd)
    T.cuda.synchronize()
    assert T.equal(a, b)
    ref = T.zeros((n_tok, n_embd), dtype=T.float64, device="cuda")
    for j in range(k):
        ref += w[:, j:j + 1].double() * out_al2[pos.view(n_tok, k)[:, j].long()].double()
    assert float((c.double() - ref).abs().max()) <= 1e-5
    assert float((a.double() - ref - sh.double()).abs().max()) <= 1e-5
