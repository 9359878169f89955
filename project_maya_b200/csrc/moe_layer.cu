// moe_layer.cu - one decode MoE layer in one call: route -> q8_1(x) -> routed gate/up + SwiGLU -> down + combine,
// the always-on shared expert alongside.  The sequence Glm5Model::fast_moe drives in the reference
// (src/core/glm_fast_path.cu:6917-7100), without the tier plan: every expert is resident, the plan of a token is the
// blob addresses of its k routed experts (0 for experts outside [expert_lo, expert_hi): another rank's).
#include <math.h>

#include "maya_fused_args.cuh"
#include "maya_group.cuh"
#include "maya_internal.cuh"
#include "maya_router.cuh"

namespace maya {
namespace {

struct Scratch {
    uint8_t* xq;                 // [T][n_embd/32] q8_1
    unsigned long long* plan_ptr;  // [T][8]
    float* plan_w;               // [T][8]
    int* ids;                    // [T][k]
    float* weights;              // [T][k]
    uint8_t* hq;                 // [T*8][n_ff/32] q8_1
    float* part;                 // [T*8][n_embd]
    unsigned long long* grp_ptr; // [T*8]
    int* grp_start;              // [T*8 + 1]
    int* grp_ent;                // [T*8]
    int* n_groups;               // [1]
    float* sh_gu;                // [T][2 * n_ff_sh]
    uint8_t* sh_hq;              // [T][n_ff_sh/32] q8_1
    float* sh_out;               // [T][n_embd]
    float* h;                    // the fused single-token kernel's h: q8_1 image, shared-unit halves, counters
    unsigned* unit_count;        // the token kernel's counters of units that two blocks share (zero before first use)
    unsigned* sync;              // [33]: the fused and the token kernel's barrier counter, epoch, [2] error word (also the window kernels'); [3] prep_kernel's ticket;
                                 // stamps; [32] the token kernel's mark of a launch that gave up (zero before first use)
    size_t bytes;
};

size_t align_up(size_t v) { return (v + 255) & ~(size_t) 255; }

Scratch carve(const maya_moe_layer& L, int T, uint8_t* base) {
    Scratch s{};
    size_t off = 0;
    auto take = [&](size_t n) { uint8_t* p = base ? base + off : nullptr; off += align_up(n); return p; };
    // the fused kernel's words first: their place must not depend on T (a scratch sized for a window also serves
    // single tokens, and the barrier counter has to survive the calls in between)
    s.sync = (unsigned*) take((kTokMark + 1) * sizeof(unsigned));
    {
        const int ld = L.n_ff > L.n_ff_sh ? L.n_ff : L.n_ff_sh;
        // per expert and 32-value group of h: the q8_1 image (40 bytes), the f32 halves two blocks leave when a unit is
        // shared between them (128 bytes) and that unit's arrival counter
        s.h = (float*) take((size_t) (MAYA_MAX_K + 1) * (ld / 32) * (40 + 128 + 4));
        s.unit_count = (unsigned*) take((size_t) (MAYA_MAX_K + 1) * (ld / 32) * 4);
    }
    s.xq = take((size_t) T * (L.n_embd / 32) * kQ81Bytes);
    s.plan_ptr = (unsigned long long*) take((size_t) T * 8 * sizeof(unsigned long long));
    s.plan_w = (float*) take((size_t) T * 8 * sizeof(float));
    s.ids = (int*) take((size_t) T * L.k * sizeof(int));
    s.weights = (float*) take((size_t) T * L.k * sizeof(float));
    s.hq = take((size_t) T * 8 * (L.n_ff / 32) * kQ81Bytes);
    s.part = (float*) take((size_t) T * 8 * L.n_embd * sizeof(float));
    s.grp_ptr = (unsigned long long*) take((size_t) T * 8 * sizeof(unsigned long long));
    s.grp_start = (int*) take(((size_t) T * 8 + 1) * sizeof(int));
    s.grp_ent = (int*) take((size_t) T * 8 * sizeof(int));
    s.n_groups = (int*) take(sizeof(int));
    if (L.n_ff_sh > 0) {
        s.sh_gu = (float*) take((size_t) T * 2 * L.n_ff_sh * sizeof(float));
        s.sh_hq = take((size_t) T * (L.n_ff_sh / 32) * kQ81Bytes);
        s.sh_out = (float*) take((size_t) T * L.n_embd * sizeof(float));
    }
    s.bytes = off;
    return s;
}

// Everything in front of the experts in one launch: block (t, 0) routes token t and writes its plan (blob addresses, weights),
// blocks (t, 1 ..) round its activations to q8_1, and the last routing block to finish groups all the tokens' entries by
// expert.  As launches of their own - router, quantizer, plan, grouping - these took 12 to 17 us of a window.
struct PrepArgs {
    const float* logits;
    const float* bias;           // sigmoid router
    float w_scale;
    int norm_w;
    int n_expert, k;
    const void* x;
    int x_is_bf16, n_embd;
    uint8_t* xq;                 // [T][n_embd / 32] q8_1
    const uint8_t* experts;
    size_t stride;
    int lo, hi;                  // this rank's experts
    int* ids;
    float* weights;
    unsigned long long* plan_ptr;
    float* plan_w;
    GroupOut group;
    unsigned* ticket;            // zero between launches
};

template<int RT, int PER>
__global__ void __launch_bounds__(256) prep_kernel(const PrepArgs P) {
    extern __shared__ __align__(16) double s_ex[];           // n_expert doubles
    __shared__ RouterShared route;
    __shared__ GroupShared grp;
    __shared__ int s_last;
    const int t = blockIdx.x, T = gridDim.x, tid = threadIdx.x;
    grid_launch_dependents();
    grid_dependency_wait();
    if (blockIdx.y > 0) {
        const int lane = tid & 31, nblk = P.n_embd / 32, step = 8 * (gridDim.y - 1);
        for (int b0 = 8 * (blockIdx.y - 1) + (tid >> 5); b0 < nblk; b0 += 4 * step) {        // four blocks in flight a warp
            float v[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int b = b0 + i * step;
                const size_t at = (size_t) t * P.n_embd + (size_t) b * 32 + lane;
                v[i] = 0.0f;
                if (b < nblk) v[i] = P.x_is_bf16 ? __uint_as_float((uint32_t) ((const uint16_t*) P.x)[at] << 16) : ((const float*) P.x)[at];
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (b0 + i * step < nblk) q8_1_store_warp(v[i], P.xq + ((size_t) t * nblk + b0 + i * step) * kQ81Bytes, lane);
        }
        return;
    }
    const float* logits = P.logits + (size_t) t * P.n_expert;
    if constexpr (RT == 1) route_sigmoid<PER, BlockSync>(logits, P.bias, P.n_expert, P.k, P.w_scale, P.norm_w, tid, 256, s_ex, route);
    else route_softmax<PER, BlockSync>(logits, P.n_expert, P.k, tid, 256, s_ex, route);
    if (tid < 8) {
        unsigned long long p = 0ull;
        float w = 0.0f;
        if (tid < P.k) {
            const int e = route.ids[tid];
            w = route.val[tid];
            if (e >= P.lo && e < P.hi) p = (unsigned long long) (P.experts + (size_t) e * P.stride);
            P.ids[(size_t) t * P.k + tid] = e;
            P.weights[(size_t) t * P.k + tid] = w;
        }
        P.plan_ptr[t * 8 + tid] = p;
        P.plan_w[t * 8 + tid] = w;
        __threadfence();
    }
    __syncthreads();
    if (tid == 0) {
        s_last = atomicAdd(P.ticket, 1u) == (unsigned) T - 1u;
        if (s_last) *P.ticket = 0u;
        __threadfence();
    }
    __syncthreads();
    if (s_last) group_entries(tid < T * 8 ? __ldcg(P.plan_ptr + tid) : 0ull, T * 8, P.group, grp);
}

template<int RT> int launch_prep(const PrepArgs& P, int T, cudaStream_t s) {
    const int per = (P.n_expert + 255) / 256, nblk = P.n_embd / 32;
    const dim3 grid((unsigned) T, (unsigned) (1 + (nblk >= 256 ? 8 : (nblk + 31) / 32)));
    const size_t smem = (size_t) P.n_expert * sizeof(double);
    if (per <= 1) launch_dependent(prep_kernel<RT, 1>, grid, dim3(256), smem, s, P);
    else if (per <= 2) launch_dependent(prep_kernel<RT, 2>, grid, dim3(256), smem, s, P);
    else if (per <= 4) launch_dependent(prep_kernel<RT, 4>, grid, dim3(256), smem, s, P);
    else launch_dependent(prep_kernel<RT, 8>, grid, dim3(256), smem, s, P);
    return note_launch("moe_prep");
}

int check_layer(const maya_moe_layer* L) {
    if (!L || !L->experts) return MAYA_ERR_ARG;
    if (!type_qk(L->gu_type) || !type_qk(L->d_type)) return MAYA_ERR_TYPE;
    if (L->k < 1 || L->k > MAYA_MAX_K || L->n_expert < L->k) return MAYA_ERR_LIMIT;
    if (L->n_embd <= 0 || L->n_ff <= 0 || L->n_embd % type_qk(L->gu_type) || L->n_ff % type_qk(L->d_type) || L->n_ff % 32 ||
        L->n_embd % 32)
        return MAYA_ERR_ARG;
    if (L->n_ff_sh > 0) {
        if (!L->shared) return MAYA_ERR_ARG;
        if (!type_is_core(L->sh_gu_type) || !type_is_core(L->sh_d_type)) return MAYA_ERR_TYPE;
        if (L->n_embd % type_qk(L->sh_gu_type) || L->n_ff_sh % type_qk(L->sh_d_type) || L->n_ff_sh % 32) return MAYA_ERR_ARG;
    }
    if (L->expert_lo < 0 || L->expert_hi > L->n_expert || L->expert_lo > L->expert_hi) return MAYA_ERR_ARG;
    if (L->router != 0 && L->router != 1) return MAYA_ERR_ARG;
    if (L->cpu_flag != nullptr && L->cpu_part == nullptr) return MAYA_ERR_ARG;
    if (L->sh_lo != 0 || L->sh_hi != 0) {            // a slice of the shared expert's width
        if (L->sh_lo < 0 || L->sh_hi > L->n_ff_sh || L->sh_lo > L->sh_hi || L->sh_lo % 32 || L->sh_hi % 32) return MAYA_ERR_ARG;
    }
    return MAYA_OK;
}

}  // namespace
}  // namespace maya

using namespace maya;

extern "C" size_t maya_moe_layer_scratch_bytes(const maya_moe_layer* L, int n_tokens) {
    if (check_layer(L) != MAYA_OK || n_tokens < 1 || n_tokens > MAYA_MAX_WIN_TOKENS) return 0;
    return carve(*L, n_tokens, nullptr).bytes;
}

extern "C" int maya_moe_layer_error(const maya_moe_layer* L, int n_tokens, const void* scratch, void* stream) {
    if (check_layer(L) != MAYA_OK || !scratch || n_tokens < 1 || n_tokens > MAYA_MAX_WIN_TOKENS) return MAYA_ERR_ARG;
    const Scratch S = carve(*L, n_tokens, (uint8_t*) scratch);
    unsigned word = 0;
    if (cudaStreamSynchronize(as_stream(stream)) != cudaSuccess) return note_launch("layer_error sync");
    if (cudaMemcpy(&word, S.sync + 2, sizeof(word), cudaMemcpyDeviceToHost) != cudaSuccess) return note_launch("layer_error copy");
    return (int) word;
}

extern "C" int maya_moe_layer_phase_ns(const maya_moe_layer* L, const void* scratch, void* stream, unsigned long long* out6) {
    if (check_layer(L) != MAYA_OK || !scratch || !out6) return MAYA_ERR_ARG;
    const Scratch S = carve(*L, 1, (uint8_t*) scratch);
    if (cudaStreamSynchronize(as_stream(stream)) != cudaSuccess) return note_launch("phase_ns sync");
    if (cudaMemcpy(out6, S.sync + 4, 6 * sizeof(unsigned long long), cudaMemcpyDeviceToHost) != cudaSuccess)
        return note_launch("phase_ns copy");
    return MAYA_OK;
}

static int layer_decode(const maya_moe_layer* L, const float* logits, const void* x, int x_is_bf16, int n_tokens, int* ids,
                        float* weights, float* out, void* scratch, size_t scratch_bytes, const maya_peer_ar* ar, int mi,
                        unsigned seq, void* stream, const maya_hc_post_args* hc = nullptr, int kernel = MAYA_LAYER_CHOICE,
                        unsigned polls = kMbarPolls);
static int ar_args_ok(const maya_moe_layer* L, int n_tokens, float* out, const maya_peer_ar* a, int mi, unsigned seq);

extern "C" int maya_moe_layer_decode(const maya_moe_layer* L, const float* logits, const void* x, int x_is_bf16,
                                     int n_tokens, int* ids, float* weights, float* out, void* scratch,
                                     size_t scratch_bytes, void* stream) {
    return layer_decode(L, logits, x, x_is_bf16, n_tokens, ids, weights, out, scratch, scratch_bytes, nullptr, 0, 0, stream);
}

extern "C" int maya_moe_layer_decode_ar(const maya_moe_layer* L, const float* logits, const void* x, int x_is_bf16,
                                        int n_tokens, int* ids, float* weights, float* out, void* scratch,
                                        size_t scratch_bytes, const maya_peer_ar* a, int mi, unsigned seq, void* stream) {
    if (ar_args_ok(L, n_tokens, out, a, mi, seq) != MAYA_OK) return refuse(MAYA_ERR_ARG);
    return layer_decode(L, logits, x, x_is_bf16, n_tokens, ids, weights, out, scratch, scratch_bytes, a, mi, seq, stream);
}

static int ar_args_ok(const maya_moe_layer* L, int n_tokens, float* out, const maya_peer_ar* a, int mi, unsigned seq) {
    if (!a || a->nm < 2 || a->nm > MAYA_PEER_AR_MAX_RANKS || mi < 0 || mi >= a->nm || !a->recv || !a->peer_recv ||
        !a->flags || !a->peer_flags || !a->error || a->timeout_ns == 0 || a->stride % 4)
        return MAYA_ERR_ARG;
    if (L && n_tokens > 0 && (size_t) n_tokens * L->n_embd > a->stride) return MAYA_ERR_ARG;
    if (out && !aligned16(out)) return MAYA_ERR_ARG;
    // the device-side sequence number lives in the fused single-token kernel and in the window's combine launch
    if (seq == 0u && (a->seq_counter == nullptr || (n_tokens == 1 && L && (L->staged || !fused_t1_supported(*L)))))
        return MAYA_ERR_ARG;
    return MAYA_OK;
}

extern "C" int maya_moe_layer_decode_hc(const maya_moe_layer* L, const float* logits, const void* x, int x_is_bf16,
                                        int n_tokens, int* ids, float* weights, float* out, void* scratch,
                                        size_t scratch_bytes, const maya_peer_ar* a, int mi, unsigned seq,
                                        const maya_hc_post_args* hc, void* stream) {
    if (!hc || !hc->R_old || !hc->post || !hc->comb || !hc->R_new || hc->R_new == hc->R_old) return refuse(MAYA_ERR_ARG);
    if (a != nullptr && ar_args_ok(L, n_tokens, out, a, mi, seq) != MAYA_OK) return refuse(MAYA_ERR_ARG);
    return layer_decode(L, logits, x, x_is_bf16, n_tokens, ids, weights, out, scratch, scratch_bytes, a, mi, seq, stream, hc);
}

extern "C" int maya_moe_layer_kernel(const maya_moe_layer* L, int n_ranks, int n_sms) {
    const int st = check_layer(L);
    return st != MAYA_OK ? st : layer_kernel(*L, n_ranks, n_sms);
}

extern "C" int maya_moe_layer_decode_checked(const maya_moe_layer* L, const float* logits, const void* x, int x_is_bf16, int* ids,
                                             float* weights, float* out, void* scratch, size_t scratch_bytes, int kernel,
                                             unsigned polls, const maya_hc_post_args* hc, void* stream) {
    if (hc && (!hc->R_old || !hc->post || !hc->comb || !hc->R_new || hc->R_new == hc->R_old)) return refuse(MAYA_ERR_ARG);
    if (kernel < MAYA_LAYER_CHOICE || kernel > MAYA_LAYER_STAGED) return refuse(MAYA_ERR_ARG);
    return layer_decode(L, logits, x, x_is_bf16, 1, ids, weights, out, scratch, scratch_bytes, nullptr, 0, 0, stream, hc, kernel, polls);
}

// The staged paths' consumer: one hc_post launch per token, after `out` is complete.
static int hc_post_tokens(const maya_hc_post_args* hc, const float* out, int T, int n_embd, void* stream) {
    if (hc == nullptr) return MAYA_OK;
    for (int t = 0; t < T; ++t) {
        const int st = maya_hc_post(out + (size_t) t * n_embd, hc->R_old + (size_t) t * 4 * n_embd, hc->post + t * 4,
                                    hc->comb + t * 16, n_embd, hc->R_new + (size_t) t * 4 * n_embd, stream);
        if (st != MAYA_OK) return st;
    }
    return MAYA_OK;
}

static int layer_decode(const maya_moe_layer* L, const float* logits, const void* x, int x_is_bf16, int n_tokens, int* ids,
                        float* weights, float* out, void* scratch, size_t scratch_bytes, const maya_peer_ar* ar, int mi,
                        unsigned seq, void* stream, const maya_hc_post_args* hc, int kernel, unsigned polls) {
    int st = check_layer(L);
    if (st != MAYA_OK) return refuse(st);
    if (n_tokens < 1 || n_tokens > MAYA_MAX_WIN_TOKENS) return refuse(MAYA_ERR_LIMIT);
    if (!logits || !x || !out || !scratch || (((uintptr_t) scratch) & 255u)) return refuse(MAYA_ERR_ARG);
    const int T = n_tokens;
    const Scratch S = carve(*L, T, (uint8_t*) scratch);
    if (S.bytes > scratch_bytes) return refuse(MAYA_ERR_LIMIT);
    cudaStream_t s = as_stream(stream);
    int* d_ids = ids ? ids : S.ids;
    float* d_w = weights ? weights : S.weights;
    if (T == 1 && (kernel == MAYA_LAYER_CHOICE ? !L->staged : kernel != MAYA_LAYER_STAGED)) {
        st = fused_t1(*L, logits, x, x_is_bf16, d_ids, d_w, out, S.h, S.unit_count, S.sync, ar, mi, seq, hc, kernel, polls, s);
        if (st != kNotHere) return st;
        if (kernel != MAYA_LAYER_CHOICE) return refuse(MAYA_ERR_LIMIT);
    }
    if (L->n_ff_sh > 0 && L->shared_here && (L->sh_lo != 0 || (L->sh_hi != 0 && L->sh_hi != L->n_ff_sh)))
        return refuse(MAYA_ERR_ARG);                 // only the fused kernel slices the shared expert

    if (L->k > 64 || L->n_expert > 256 * kRouterMaxPerThread) return refuse(MAYA_ERR_LIMIT);
    PrepArgs P{};
    P.logits = logits; P.bias = L->router_bias; P.w_scale = L->router_w_scale; P.norm_w = L->router_norm_w;
    P.n_expert = L->n_expert; P.k = L->k; P.x = x; P.x_is_bf16 = x_is_bf16; P.n_embd = L->n_embd; P.xq = S.xq;
    P.experts = (const uint8_t*) L->experts; P.stride = L->expert_stride; P.lo = L->expert_lo; P.hi = L->expert_hi;
    P.ids = d_ids; P.weights = d_w; P.plan_ptr = S.plan_ptr; P.plan_w = S.plan_w;
    P.group = GroupOut{S.grp_ptr, S.grp_start, S.grp_ent, S.n_groups};
    P.ticket = S.sync + 3;
    st = L->router == 1 ? launch_prep<1>(P, T, s) : launch_prep<0>(P, T, s);
    if (st != MAYA_OK) return st;

    const bool shared = L->n_ff_sh > 0 && L->shared_here;
    const uint8_t* sh_blob = (const uint8_t*) L->shared;
    const size_t up_off = row_bytes(L->gu_type, L->n_embd) * (size_t) L->n_ff, down_off = 2 * up_off;
    // a Q8_0 shared expert rides in the routed experts' launches where the shapes fit them
    const bool ride = shared && L->sh_gu_type == MAYA_Q8_0 && L->sh_d_type == MAYA_Q8_0 && (((uintptr_t) sh_blob) & 15u) == 0 &&
                      window_fits(L->n_embd, L->n_ff, L->n_ff_sh);
    const SharedArgs sh{sh_blob, L->n_ff_sh, T, S.sh_hq, S.sh_out};
    if (shared && !ride) {
        const size_t sh_down_off = row_bytes(L->sh_gu_type, L->n_embd) * (size_t) L->n_ff_sh * 2;
        for (int c0 = 0; c0 < T; c0 += MAYA_MAX_COLS) {   // gate and up rows are contiguous: one GEMV of 2 * n_ff_sh rows
            const int nc = T - c0 < MAYA_MAX_COLS ? T - c0 : MAYA_MAX_COLS;
            // column-major output [c][2 * n_ff_sh] per call: offset by the columns already done
            st = maya_mmvq(L->sh_gu_type, sh_blob, S.xq + (size_t) c0 * (L->n_embd / 32) * kQ81Bytes,
                           S.sh_gu + (size_t) c0 * 2 * L->n_ff_sh, L->n_embd, 2 * L->n_ff_sh, nc, stream);
            if (st != MAYA_OK) return st;
        }
        for (int c = 0; c < T; ++c) {
            st = maya_swiglu_q8_1(S.sh_gu + (size_t) c * 2 * L->n_ff_sh, S.sh_gu + (size_t) c * 2 * L->n_ff_sh + L->n_ff_sh,
                                  L->limit, L->n_ff_sh, S.sh_hq + (size_t) c * (L->n_ff_sh / 32) * kQ81Bytes, stream);
            if (st != MAYA_OK) return st;
        }
        for (int c0 = 0; c0 < T; c0 += MAYA_MAX_COLS) {
            const int nc = T - c0 < MAYA_MAX_COLS ? T - c0 : MAYA_MAX_COLS;
            st = maya_mmvq(L->sh_d_type, sh_blob + sh_down_off, S.sh_hq + (size_t) c0 * (L->n_ff_sh / 32) * kQ81Bytes,
                           S.sh_out + (size_t) c0 * L->n_embd, L->n_ff_sh, L->n_embd, nc, stream);
            if (st != MAYA_OK) return st;
        }
    }
    maya_moe_win W{};
    W.plan_ptr = S.plan_ptr;
    W.plan_w = S.plan_w;
    W.xq = S.xq;
    W.xq_stride = (size_t) (L->n_embd / 32) * kQ81Bytes;
    W.hq = S.hq;
    W.part = S.part;
    W.cpu_part = L->cpu_flag ? L->cpu_part : nullptr;
    W.cpu_flag = L->cpu_flag;
    W.sh_out = shared ? S.sh_out : nullptr;
    W.out = out;
    W.out_stride = (size_t) L->n_embd;
    W.grp_ptr = S.grp_ptr;
    W.grp_start = S.grp_start;
    W.grp_ent = S.grp_ent;
    W.n_groups = S.n_groups;
    W.T = T;
    W.k = L->k;
    W.n_embd = L->n_embd;
    W.n_ff = L->n_ff;
    W.limit = L->limit;
    W.down_off = down_off;
    // one token: a window of one, its cross-rank sum a launch of its own; more: with `ar` the sum runs in the combine launch
    st = win_experts(L->gu_type, L->d_type, &W, true, ride ? &sh : nullptr, polls, S.sync + 2, T > 1 ? ar : nullptr, mi, seq, s);
    if (st == MAYA_OK && T == 1 && ar != nullptr) st = maya_allreduce_peer(out, L->n_embd, ar, mi, seq, stream);
    return st == MAYA_OK ? hc_post_tokens(hc, out, T, L->n_embd, stream) : st;
}
