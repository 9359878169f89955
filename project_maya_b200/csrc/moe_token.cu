// moe_token.cu - host side of the token kernel (moe_token.cuh): which layers it takes, and on which of them it is the faster kernel.
#include "maya_fused_args.cuh"
#include "maya_internal.cuh"
#include "maya_rows.cuh"
#include "maya_token_phase.cuh"

namespace maya {

template<int T> int token_by_type(const TokArgs& A, cudaStream_t s);

static int tok_tab_bytes(int type) {
#define MAYA_TOK_BYTES(TT) case TT: return RowTab<TT, true>::bytes;
    switch (type) { MAYA_TOK_TYPES(MAYA_TOK_BYTES) }
#undef MAYA_TOK_BYTES
    return 0;
}

size_t token_smem(int gu_type, TokArgs& A, int grid) {
    const bool sh = A.shared != nullptr, two = gu_type == MAYA_Q4_K || gu_type == MAYA_Q5_K;       // (a call of two q8_1 blocks)
    const int pg = row_geo(gu_type).pitch, pd = row_geo(A.d_type).pitch, tg = tok_tab_bytes(gu_type), td = tok_tab_bytes(A.d_type);
    A.stage = (4 * (pg > pd ? pg : pd) + 15) & ~15;
    A.tab = tg > td ? tg : td;
    const int x = tok_col_bytes(A.n_embd / 32) * (sh && two ? 2 : 1), h = A.k * tok_col_bytes(A.n_ff / 32) + tok_col_bytes(A.n_ff_sh / 32);
    A.cols = ((x > h ? x : h) + 15) & ~15;
    A.units = A.k * A.n_ff / 32 / grid + A.n_ff_sh / 32 / grid + 4;          // of a block, parts at both ends of both classes
    const size_t smem = (size_t) kTokWarps * 2 * A.stage + A.tab + A.cols + ((A.units * 132 + 15) & ~15) + (size_t) A.n_expert * sizeof(double);
    return smem <= kTokMostSmem ? smem : 0;
}

static TokArgs token_args(const maya_moe_layer& L, const FusedArgs& F) {
    TokArgs A{};
    (FusedArgs&) A = F;
    A.d_type = L.d_type;
    A.up_off = row_bytes(L.gu_type, L.n_embd) * (size_t) L.n_ff;
    A.down_off = 2 * A.up_off;
    return A;
}

bool token_takes(const maya_moe_layer& L, const FusedArgs& F, int sms) {
    if (sms <= 0 || F.ar.nm >= 2) return false;        // the cross-rank sum is moe_fused.cu's
    // bulk copies take aligned 16-byte windows around the rows: blobs have to start and end on 16-byte boundaries
    if ((((uintptr_t) F.experts) | F.expert_stride | (uintptr_t) F.shared) & 15u) return false;
    if (F.shared != nullptr && (L.sh_gu_type != MAYA_Q8_0 || L.sh_d_type != MAYA_Q8_0)) return false;
    if (L.n_expert > kRouteThreads * kRouterMaxPerThread || 4 * ((L.n_embd / 4 + sms - 1) / sms) > kMaxSliceRows) return false;
    TokArgs A = token_args(L, F);
    return token_smem(L.gu_type, A, sms) != 0;
}

// Layers of one core type, which the fused kernel takes too: whether this kernel is the faster one.  Its phases stream more bytes a
// second; the fused kernel is through with its set-up sooner, has 32 warps to wait for a shared expert's rows with, and handles no stages.
// So the lines lie at the routed bytes a token reads, and where rows leave stages half empty or the shared expert is much of the
// work.  From 925 timed layers of 1024 .. 8192 x 512 .. 3072, 1 to 8 experts a token, half of them with a shared expert, as three layers in
// turn and as so many that no row stays in L2: by this rule none is more than 5 % slower than on the fused kernel, 13 more than 2 %
// (seven of them IQ2_S, which out of HBM are the faster); 1.4 % (IQ2_S) to 9 % (Q4_K) faster on average.  (us fused / token kernel, 148 SMs, three layers in turn)
bool token_better(int type, const FusedArgs& A, int sms) {
    const bool sh = A.shared != nullptr;
    const int width = A.sh_hi - A.sh_lo;
    const size_t R = (size_t) A.k * (2 * (size_t) A.n_ff * row_bytes(type, A.n_embd) + (size_t) A.n_embd * row_bytes(type, A.n_ff));
    const size_t S = sh ? 2 * (size_t) width * row_bytes(MAYA_Q8_0, A.n_embd) + (size_t) A.n_embd * row_bytes(MAYA_Q8_0, width) : 0;
    const size_t MB = 1000000;
    const bool routed = 4 * S <= R;      // nearly all of the work
    switch (type) {
        case MAYA_Q4_K:              // rows of more than a segment, enough bytes, or so few units that every warp has one item
            // 1280 x 768, top 8: 15.6 / 18.0; 1536 x 1024 with a 2816-wide shared expert 0.95 times as fast; 2816 x 2816 50.5 / 40.0
            return A.n_embd > 2304 || R >= (sh ? 32 : 24) * MB || A.k * A.n_ff / 32 + width / 32 <= sms;
        case MAYA_Q8_0: {            // enough bytes; or longer rows, down rows that fill their segments of 1024 values, little beside them
            // 1312 x 1120, top 5: 17.6 / 20.1; 2528 x 1056 (a segment and one block), top 8 0.97 times as fast; 2720 x 832 with a 2816-wide
            // shared expert 0.93; 1440 x 2464 1.04; 3200 x 768, top 6 1.08; 5504 x 1568 56.4 / 51.4
            const int nsd = (A.n_ff + 1023) / 1024;
            return R >= (routed ? 105 : 120) * MB || (A.n_embd <= 1792 && R >= 80 * MB) ||
                   (A.n_embd > 2304 && 16 * A.n_ff >= 9 * 1024 * nsd && routed);
        }
        case MAYA_IQ3_S:             // 6656 x 512, top 4: 0.94 times as fast; 1536 x 768, top 8 0.94; 2560 x 768 with a 2560-wide shared expert 0.97, 2816 x 768
            // with a 512-wide one 1.09; 4096 x 2304, top 2 1.12; 6144 x 2048 67.1 / 55.4
            return (A.n_ff > 512 || (sh && A.n_embd > 6144)) &&
                   (A.n_embd > 3072 || (R >= 26 * MB && (!sh || A.n_embd > 2560)) || (R >= 20 * MB && sh && routed && A.n_embd > 2304));
        default:                     // IQ2_S.  Its rows decode fastest: beside a shared expert's 8-bit rows they wait (6144 x 2048, 2048 shared: 59.6 / 61.8,
            // 7168 x 2048 68.9 / 70.5; narrower shared experts 0.98 to 1.04 times as fast; 6144 x 2048 without one 66.3 / 54.1); 7168 x 512, top 8: 0.88
            // times as fast; 2560 x 1280, top 6 0.94; 3584 x 1024, top 5 0.99 and, out of HBM, 1.18
            return !sh && A.n_ff > 512 && ((R >= 40 * MB && A.n_embd > 2304) || (R >= 17 * MB && A.n_embd > 3072));
    }
}

int token_layer(const maya_moe_layer& L, const FusedArgs& F, unsigned* unit_count, unsigned polls, cudaStream_t s) {
    TokArgs A = token_args(L, F);
    A.unit_count = unit_count;
    A.polls = polls;
    A.drain_polls = kMbarPolls;
    switch (L.gu_type) {
        case MAYA_Q8_0: return token_by_type<MAYA_Q8_0>(A, s);
        case MAYA_Q4_K: return token_by_type<MAYA_Q4_K>(A, s);
        case MAYA_Q5_K: return token_by_type<MAYA_Q5_K>(A, s);
        case MAYA_Q6_K: return token_by_type<MAYA_Q6_K>(A, s);
        case MAYA_IQ4_XS: return token_by_type<MAYA_IQ4_XS>(A, s);
        case MAYA_IQ2_S: return token_by_type<MAYA_IQ2_S>(A, s);
        case MAYA_IQ3_S: return token_by_type<MAYA_IQ3_S>(A, s);
        case MAYA_IQ3_XXS: return token_by_type<MAYA_IQ3_XXS>(A, s);
        case MAYA_IQ2_XXS: return token_by_type<MAYA_IQ2_XXS>(A, s);
        case MAYA_IQ1_S: return token_by_type<MAYA_IQ1_S>(A, s);
        default: return kNotHere;
    }
}

}  // namespace maya
