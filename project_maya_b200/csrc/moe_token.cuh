// moe_token.cuh - one token through one MoE layer in one cooperative launch, every weight row streamed through shared memory.
//
// The form for one GPU of what moe_fused.cu does (which keeps the cross-rank sum and the layers on which it is the faster kernel: see
// token_better in moe_token.cu), for pairs of the ten block types whose ring and codebook fit shared memory together: at 6144 x 2048,
// top 8, 68 of the 100 (not IQ2_S / IQ3_S, nor either of these with Q4_K; token_smem).  Phases as there: route and round x / gate and
// up rows, SwiGLU and q8_1 of h / grid barrier / down rows and combine.
//
// What bounds it: HBM for the 4- to 8-bit types, instruction issue and the shared-memory pipe for the codebook types.  Read in
// place by 32 warps of 64 registers, a codebook type's fields cost three to four L1 lines a load (the load/store pipe was the limit,
// not issue), and the rows of the wider types had too few bytes in flight.  Here 16 warps of up to 128 registers take four
// rows at a time; every warp streams their K segments into a private ring of two stages with bulk copies, across item
// boundaries and - the routing being known - across the grid barrier.  Warps never meet inside a phase:
//   * phase 1: an item is two FFN rows of an expert (their two gate and two up rows), a block's items one contiguous share
//     of the routed experts' and one of the shared expert's.  Whichever warp brings the last of a unit's 16 items rounds its 32
//     values to one q8_1 block; a unit that two blocks share meets in the scratch, behind a counter that grows by 16 a launch.
//   * phase 2: an item is four output rows (more where a row has fewer than 32 calls) of one expert.
//   * the Q8_0 shared expert's rows are read in place - in phase 1 spread evenly among a block's other items, so that one or two
//     warps wait for them while the rest decode: as stages they would be many (a ring sized for 2-bit rows) and their handling
//     more than their dots.
// Measured beside the fused kernel on 6144 x 2048, top 8 (us, 148 SMs, rows in HBM): IQ2_S 69.6 -> 58.0, IQ3_S 71.0 -> 57.5, Q4_K
// 60.1 -> 48.0, Q8_0 73.3 -> 68.0, with a 2048-wide shared expert IQ3_S 71.8 -> 65.4, Q4_K 66.3 -> 58.0 (and IQ2_S 63.2 -> 64.4: it stays
// there); two layers of Q4_K / Q6_K, which took four launches a layer, 122.2 -> 97.8.
// The loops are kept short: with steps, rows and both row classes unrolled side by side a third of all issue slots went to
// waiting for instructions (81 us on the 6144 x 2048 IQ2_S layer with shared expert).
// The (row, expert) dots, q8_1 of h and the combine chain are rows_dot1's and the staged kernels', value for value: results are
// bit-identical to every other path's.
//
// Every wait is bounded.  A warp whose copies never land asks for nothing more; its block says so in the error word and, with the
// launch's mark, in sync[kTokMark], still meets the others at the grid barrier, and leaves after the copies in flight have had a bounded
// time.  The other blocks ask for the mark behind the barrier, where the h that they read may be incomplete, and look at it where they
// vote on their own rows (a vote of its own cost 1 %): none writes `out` or the residual stack.  The counters of split units, some of
// which stay short of a launch's 16, are set to zero by the block that gave up.
#pragma once

#include "maya_fused_args.cuh"
#include "maya_hc_post.cuh"
#include "maya_internal.cuh"
#include "maya_router.cuh"
#include "maya_rows.cuh"
#include "maya_token_phase.cuh"

#include <type_traits>

namespace maya {
namespace {

constexpr int kTokThreads = kTokWarps * 32;

// the streamed rows: gate/up [0] and down [1] of the routed experts
struct TokKind {
    int nseg, bytes, pitch;                 // segments of a row, their bytes, their distance in a stage
    int cont;                               // the item's rows come whole, in one copy, `pitch` = rb apart
    int calls, groups, rpi, nq;             // down: calls of a row; rows side by side in a warp; an item's rows; items an expert
    uint32_t rb;                            // bytes of a row
};

struct TokShared {
    RouterShared route;
    unsigned long long ptr[MAYA_MAX_K];
    float w[MAYA_MAX_K];
    float part[kMaxSliceRows][MAYA_MAX_K + 1];
    uint64_t full[kTokWarps][2];
    TokKind kind[2];
    unsigned epoch;
    int ve[MAYA_MAX_K];
    int nv;
    int bar_ok, lost;
};

static_assert(sizeof(TokShared) <= 232448 - kTokMostSmem - 1024, "with the driver's 1 KB");

// Whether ring and codebook of a pair (T: gate/up, TD: down) fit shared memory beside nothing else: a stage is the wider type's, the table
// the larger codebook's.  token_smem turns away the pairs that do not, and those that fit only narrower layers.
template<int T, int TD> constexpr bool kTokPair =
    (size_t) kTokWarps * 8 * (RowGeo<T>::pitch > RowGeo<TD>::pitch ? RowGeo<T>::pitch : RowGeo<TD>::pitch) +
        (RowTab<T, true>::bytes > RowTab<TD, true>::bytes ? RowTab<T, true>::bytes : RowTab<TD, true>::bytes) <= kTokMostSmem;

// One q8_1 block of 32 values, one a lane: its lane's quant, the scale as the f16 field holds it, and the sum a dot takes - of the
// quants, or for IQ1_S the stored f16 sum of the values (float bits).
struct TokBlock { int q; float d; int sum; };
template<bool SUM_F16> __device__ __forceinline__ TokBlock tok_round(float v) {
    const float amax = warp_max(fabsf(v)), d = fminf(__fdiv_rn(amax, 127.0f), 65504.0f);
    TokBlock t;
    t.q = amax == 0.0f ? 0 : (int) fmaxf(-127.0f, fminf(127.0f, roundf(__fdiv_rn(v, d))));
    t.d = __half2float(__float2half_rn(d));
    if constexpr (SUM_F16) t.sum = __float_as_int(__half2float(__float2half_rn(fmaxf(-65504.0f, fminf(65504.0f, warp_sum(v))))));
    else t.sum = __reduce_add_sync(0xffffffffu, t.q);
    return t;
}
// Four blocks at once: 4 consecutive values a lane, 8 lanes a block; the block's sums in warp_sum's order.
struct TokBlock4 { uint32_t q; float d; int sum; };
template<bool SUM_F16> __device__ __forceinline__ TokBlock4 tok_round4(const float (&v)[4]) {
    float amax = fmaxf(fmaxf(fabsf(v[0]), fabsf(v[1])), fmaxf(fabsf(v[2]), fabsf(v[3])));
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    const float d = fminf(__fdiv_rn(amax, 127.0f), 65504.0f);
    TokBlock4 t;
    t.q = 0u;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int q = amax == 0.0f ? 0 : (int) fmaxf(-127.0f, fminf(127.0f, roundf(__fdiv_rn(v[i], d))));
        t.q |= ((uint32_t) q & 0xFFu) << (8 * i);
    }
    t.d = __half2float(__float2half_rn(d));
    if constexpr (SUM_F16) {
        float s[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) s[i] = v[i];
#pragma unroll
        for (int o = 4; o > 0; o >>= 1)
#pragma unroll
            for (int i = 0; i < 4; ++i) s[i] += __shfl_xor_sync(0xffffffffu, s[i], o);
        const float sum = (s[0] + s[2]) + (s[1] + s[3]);
        t.sum = __float_as_int(__half2float(__float2half_rn(fmaxf(-65504.0f, fminf(65504.0f, sum)))));
    } else {
        t.sum = __dp4a((int) t.q, 0x01010101, 0);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) t.sum += __shfl_xor_sync(0xffffffffu, t.sum, o);
    }
    return t;
}
// The codebook of a type only known at run time.
__device__ __noinline__ void tok_fill(int type, uint32_t* tab, int tid) {
#define MAYA_TOK_FILL(TT) case TT: RowTab<TT, true>::fill(tab, tid, kTokThreads); break;
    switch (type) { MAYA_TOK_TYPES(MAYA_TOK_FILL) }
#undef MAYA_TOK_FILL
}
// One activation column in shared memory, planar (maya_dots.cuh): nblk q8_1 blocks, calls of XB blocks.
struct TokCol { const uint8_t* p; int nblk; };
template<int XB> __device__ __forceinline__ XQ tok_col(const TokCol& c, int j, int n) {
    const int P = c.nblk / XB;
    const int4 a = *(const int4*) (c.p + (2 * j * P + n) * 16), b = *(const int4*) (c.p + ((2 * j + 1) * P + n) * 16);
    XQ v;
    v.u[0] = a.x; v.u[1] = a.y; v.u[2] = a.z; v.u[3] = a.w;
    v.u[4] = b.x; v.u[5] = b.y; v.u[6] = b.z; v.u[7] = b.w;
    v.d = *(const float*) (c.p + c.nblk * 32 + (j * P + n) * 4);
    v.isum = *(const int*) (c.p + c.nblk * 36 + (j * P + n) * 4);
    return v;
}
// Where half `h` of block b of a column lies, and its scale (sum: nblk * 4 bytes on).
template<int XB> __device__ __forceinline__ uint32_t tok_piece(int nblk, int b, int h) { return ((2 * (b % XB) + h) * (nblk / XB) + b / XB) * 16; }
template<int XB> __device__ __forceinline__ uint32_t tok_scale(int nblk, int b) { return nblk * 32 + ((b % XB) * (nblk / XB) + b / XB) * 4; }

// Four rows in shared memory (places row[] in s) against the column: calls n + l, n + l + 32, ... below n + ncalls, in rows_dot1's order.
template<int T>
__device__ __forceinline__ void tok_dot(const uint8_t* s, const uint32_t (&row)[4], const TokCol& col, int n, int ncalls, int l,
                                        const RowLut<T, true>& lut, float (&acc)[4]) {
    constexpr int XB = Dec<T>::xblk;
    using D = SDec<T, true, true>;
    typename D::At at[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) at[r] = D::at(row[r], l);
#pragma unroll
    for (int j = 0; j < RowGeo<T>::steps; ++j) {
        if (32 * j + l >= ncalls) break;
        const XQ a = tok_col<XB>(col, 0, n + 32 * j + l);
        XQ b = a;
        if constexpr (XB == 2) b = tok_col<XB>(col, 1, n + 32 * j + l);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            D d;
            d.load(s, at[r], j, l, lut);
            acc[r] = __fadd_rn(acc[r], d.dot(a, b));
        }
    }
}
// Four Q8_0 rows in place, `calls` blocks of each from the column's first on.
__device__ __forceinline__ void tok_dot_shared(const uint8_t* r0, const uint8_t* r2, size_t rb, const TokCol& col, int calls, int lane, float (&acc)[4]) {
#pragma unroll 1
    for (int k = lane; k < calls; k += 32) {
        Dec<MAYA_Q8_0> d[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) d[r].load((r < 2 ? r0 : r2) + (r & 1) * rb + (size_t) k * 34, 0, nullptr);
        const XQ a = tok_col<1>(col, 0, k);
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[r] = __fadd_rn(acc[r], d[r].dot(a, a));
    }
}
// where segment sg of a row that starts at (the low word of) address p begins in its aligned window
template<int T> __device__ __forceinline__ uint32_t seg_off(uint32_t p, int sg) {
    if constexpr (RowGeo<T>::bytes % 16 == 0) return p & 15u;
    else return (p + (uint32_t) (sg * RowGeo<T>::bytes)) & 15u;
}
// warp_sum of four rows at once (lanes 16 apart first, then 8, 4, 2, 1): lane l's result is row 2 (l >> 4) + ((l >> 3) & 1)'s
__device__ __forceinline__ float tok_sum4(const float (&acc)[4], int lane) {
    const bool up16 = (lane & 16) != 0, up8 = (lane & 8) != 0;
    float a = up16 ? acc[2] : acc[0], b = up16 ? acc[3] : acc[1];
    a += __shfl_xor_sync(0xffffffffu, up16 ? acc[0] : acc[2], 16);
    b += __shfl_xor_sync(0xffffffffu, up16 ? acc[1] : acc[3], 16);
    float v = up8 ? b : a;
    v += __shfl_xor_sync(0xffffffffu, up8 ? a : b, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// A warp's places among n, `few` of which are special, evenly spread: place p is special where before() steps.
struct Spread {
    uint32_t q;
    __device__ __forceinline__ Spread(int few, int n) : q(n > 0 ? ((uint32_t) few * 65536u + n - 1) / (uint32_t) n : 0u) {}
    __device__ __forceinline__ int before(int p) const { return (int) (((uint32_t) p * q) >> 16); }
    __device__ __forceinline__ bool at(int p) const { return before(p + 1) > before(p); }
};

// What only a launch in which a wait ran out comes to: as functions of their own, out of the kernel's register allocation.
__device__ __noinline__ void tok_gave_up(unsigned* sync, unsigned mark) {
    atomicExch(&sync[2], 1u);
    atomicExch(&sync[kTokMark], mark);
}
// The n counters made whole for the next launch.  (Every block is past them.)
__device__ __noinline__ void tok_reset(unsigned* count, int n) {
    for (int i = threadIdx.x; i < n; i += kTokThreads) count[i] = 0u;
}

// T: gate/up type; SH: with a Q8_0 shared expert.
template<int T, bool SH>
__global__ void __launch_bounds__(kTokThreads, 1) token_kernel(const TokArgs A) {
    extern __shared__ __align__(128) uint8_t s_raw[];
    __shared__ TokShared sh;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int k = A.k, n_embd = A.n_embd, n_ff = A.n_ff;
    const bool has_sh = SH && A.shared != nullptr;
    const int ne = k + (has_sh ? 1 : 0), nblk_x = n_embd / 32, nblk_h = max(n_ff, A.n_ff_sh) / 32;
    constexpr int XB = Dec<T>::xblk;

    // [ring | codebook | columns: x, later every expert's h | h of the block's units, their counts | routing scratch]
    const uint32_t ring = warp * 2 * A.stage;
    uint32_t* const s_tab = (uint32_t*) (s_raw + kTokWarps * 2 * A.stage);
    uint8_t* const cols = (uint8_t*) s_tab + A.tab;
    float* const hb = (float*) (cols + A.cols);
    int* const hc = (int*) (hb + A.units * 32);
    double* const s_ex = (double*) (cols + A.cols + ((A.units * 132 + 15) & ~15));

    // Nothing of global memory but constants of the library is read before the wait (see moe_fused.cu)
    grid_launch_dependents();
    if (tid < kRouteThreads) {
        if (tid * 32 < A.n_expert) asm volatile("prefetch.global.L2 [%0];" ::"l"(A.logits + tid * 32));
        if (lane == 0) {
            for (int w = warp; w < kTokWarps; w += kRouteThreads / 32) {
                mbar_init(&sh.full[w][0], 4);
                mbar_init(&sh.full[w][1], 4);
            }
            mbar_fence_init();
        }
        for (int i = tid; i < A.units; i += kRouteThreads) hc[i] = 0;
    } else {
        const int t2 = tid - kRouteThreads;
        const size_t xb = (size_t) n_embd * (A.x_is_bf16 ? 2 : 4);
        for (size_t i = (size_t) t2 * 128; i < xb; i += (size_t) (kTokThreads - kRouteThreads) * 128)
            asm volatile("prefetch.global.L2 [%0];" ::"l"((const uint8_t*) A.x + i));
        RowTab<T, true>::fill(s_tab, t2, kTokThreads - kRouteThreads);
    }
    grid_dependency_wait();
    if (tid == 0) sh.epoch = *(volatile unsigned*) &A.sync[1];
    stamp(A.sync, 0);

    // ---------------------------------------------------------------- phase 0
    int o0, o1;                                          // this block's output rows: whole quads
    slice(n_embd / 4, gridDim.x, blockIdx.x, o0, o1);
    o0 *= 4;
    o1 *= 4;
    const int nrows = o1 - o0;
    if (tid < kRouteThreads) {
        if (A.router == 1) route_token<1, true>(A.logits, A.router_bias, A.n_expert, k, A.router_w_scale, A.router_norm_w, tid, s_ex, &sh.route);
        else route_token<0, true>(A.logits, nullptr, A.n_expert, k, 0.0f, 0, tid, s_ex, &sh.route);
        if (tid < k) {
            const int e = sh.route.ids[tid];
            sh.ptr[tid] = (e >= A.expert_lo && e < A.expert_hi) ? (unsigned long long) (A.experts + (size_t) e * A.expert_stride) : 0ull;
            if (blockIdx.x == 0) A.ids[tid] = e;
        }
        NamedSync<1, kRouteThreads>::sync();
        if (tid < 32) {                                  // the entries that are this rank's
            const unsigned here = __ballot_sync(0xffffffffu, tid < k && sh.ptr[tid] != 0ull);
            if (here >> tid & 1u) sh.ve[__popc(here & ((1u << tid) - 1u))] = tid;
            if (tid == 0) sh.nv = __popc(here);
        }
    } else {
        constexpr int NW2 = kTokWarps - kRouteThreads / 32;
        // x to q8_1: 128 values a warp and pass, all of six passes' loads in flight
        for (int c0 = warp - kRouteThreads / 32; c0 * 128 < n_embd; c0 += 6 * NW2) {
            float v[6][4];
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                const int at = (c0 + i * NW2) * 128 + 4 * lane;
                float4 f = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (at < n_embd) {
                    if (A.x_is_bf16) {
                        const uint16_t* x = (const uint16_t*) A.x + at;
                        f = make_float4(__uint_as_float((uint32_t) x[0] << 16), __uint_as_float((uint32_t) x[1] << 16),
                                        __uint_as_float((uint32_t) x[2] << 16), __uint_as_float((uint32_t) x[3] << 16));
                    } else {
                        const float* x = (const float*) A.x + at;
                        f = make_float4(x[0], x[1], x[2], x[3]);
                    }
                }
                v[i][0] = f.x; v[i][1] = f.y; v[i][2] = f.z; v[i][3] = f.w;
            }
#pragma unroll
            for (int i = 0; i < 6; ++i) {
                const int b = (c0 + i * NW2) * 4 + (lane >> 3);
                if ((c0 + i * NW2) * 128 >= n_embd) break;                       // the same for the whole warp
                const TokBlock4 t = tok_round4<T == MAYA_IQ1_S>(v[i]);
                if (b >= nblk_x) continue;
                const int h = (lane >> 2) & 1, w = 4 * (lane & 3);
                *(uint32_t*) (cols + tok_piece<XB>(nblk_x, b, h) + w) = t.q;
                if ((lane & 7) == 0) {
                    *(float*) (cols + tok_scale<XB>(nblk_x, b)) = t.d;
                    *(int*) (cols + tok_scale<XB>(nblk_x, b) + nblk_x * 4) = t.sum;
                }
                if constexpr (SH && XB == 2) {           // the Q8_0 rows' order of the same column, behind it
                    uint8_t* const c1 = cols + tok_col_bytes(nblk_x);
                    *(uint32_t*) (c1 + tok_piece<1>(nblk_x, b, h) + w) = t.q;
                    if ((lane & 7) == 0) *(float*) (c1 + tok_scale<1>(nblk_x, b)) = t.d;
                }
            }
        }
        if (warp == kTokWarps - 1 && lane < 2) {
            TokKind K{};
            const int type = lane == 0 ? T : A.d_type, n_in = lane == 0 ? n_embd : n_ff;
            const RowGeoRt g = row_geo(type);
            K.rb = (uint32_t) row_bytes(type, n_in);
            K.nseg = (n_in + g.vals - 1) / g.vals;
            K.bytes = g.bytes;
            K.pitch = g.pitch;
            K.calls = n_in / g.qk * g.cpb;
            K.groups = 1;
            K.rpi = 4;
            if (lane == 1 && K.nseg == 1) {
                if (K.calls < 32 && (K.calls & (K.calls - 1)) == 0) K.groups = 32 / K.calls;
                if ((int) (4 * K.groups * K.rb) + 16 <= A.stage) {
                    K.cont = 1;
                    K.pitch = (int) K.rb;
                    K.rpi = 4 * K.groups;
                } else {
                    K.groups = 1;
                }
            }
            K.nq = (nrows + K.rpi - 1) / K.rpi;
            sh.kind[lane] = K;
        }
    }
    __syncthreads();
    stamp(A.sync, 1);

    const int half = n_ff / 2, nv = sh.nv;
    int asked = 0, got = 0;                              // stages asked for and read: stage i lies in ring place i % 2
    auto wait = [&]() -> bool { return __all_sync(0xffffffffu, mbar_wait(&sh.full[warp][got & 1], (got >> 1) & 1, A.polls)); };
    // The stream.  A lane r < 4 keeps row r's next byte and how many are left of it.
    const uint8_t* a_row = nullptr;
    uint32_t a_left = 0;
    int a_seg = 0;
    auto new_row = [&](const uint8_t* row, uint32_t len) { a_row = row; a_left = len; a_seg = 0; };
    // one segment of the lane's row, in the aligned window around it.  true: that was the item's last
    auto ask = [&](int bytes, int pitch, int nseg) -> bool {
        const int p = asked & 1;
        __syncwarp();                                    // every lane has read the stage's last bytes
        if (lane < 4) {
            if (a_left > 0u) {
                const uint32_t off = (uint32_t) (uintptr_t) a_row & 15u, n = (off + min(a_left, (uint32_t) bytes) + 15u) & ~15u;
                fence_proxy_async();
                mbar_expect_tx(&sh.full[warp][p], n);
                bulk_load(s_raw + ring + p * A.stage + lane * pitch, a_row - off, n, &sh.full[warp][p]);
            } else {
                mbar_arrive_one(&sh.full[warp][p]);
            }
        }
        a_row += bytes;
        a_left -= min(a_left, (uint32_t) bytes);
        ++asked;
        return ++a_seg == nseg;
    };
    bool ok = true;

    // ---- phase 2's stream: this warp's next item to ask for, (expert a2_e, its a2_q-th), and its rows
    const TokKind& kd = sh.kind[1];
    const int n2s = has_sh ? nrows / 4 : 0, n2 = nv * kd.nq;
    struct Place { int p, e, q; };                       // place p: the q-th item of entry e
    auto next2 = [&](Place& P) {
        P.p += kTokWarps;
        P.q += kTokWarps;
        while (P.q >= kd.nq && P.e < nv) { P.q -= kd.nq; ++P.e; }
    };
    auto first2 = [&]() -> Place {
        Place P{warp, 0, warp};
        while (P.q >= kd.nq && P.e < nv) { P.q -= kd.nq; ++P.e; }
        return P;
    };
    Place a2 = first2();
    auto down_rows = [&](int ei, int q) { return (const uint8_t*) sh.ptr[sh.ve[ei]] + A.down_off + (size_t) (o0 + q * kd.rpi) * kd.rb; };
    auto open2 = [&] {
        if (a2.p >= n2) return;
        const uint8_t* row = down_rows(a2.e, a2.q);
        const int valid = min(kd.rpi, nrows - a2.q * kd.rpi);
        if (kd.cont) new_row(row, lane == 0 ? (uint32_t) valid * kd.rb : 0u);
        else new_row(row + (size_t) min(lane, valid - 1) * kd.rb, lane < valid ? kd.rb : 0u);
    };
    auto ask2 = [&] {
        if (a2.p >= n2) return;
        if (!ask(kd.cont ? A.stage : kd.bytes, kd.cont ? A.stage : kd.pitch, kd.nseg)) return;
        next2(a2);
        open2();
    };

    // ---------------------------------------------------------------- phase 1: gate / up + SwiGLU + q8_1(h)
    // the q8_1 image of h in the scratch: [unit][32] int8, [unit] f32 scales, [unit] sums; unit = expert slot * nblk_h + group
    int8_t* const gq = (int8_t*) A.h;
    float* const gd = (float*) (gq + (size_t) ne * nblk_h * 32);
    int* const gs = (int*) (gd + (size_t) ne * nblk_h);
    {
        int r0, r1, s0, s1;
        slice(nv * half, gridDim.x, blockIdx.x, r0, r1);
        slice(has_sh ? (A.sh_hi - A.sh_lo) / 2 : 0, gridDim.x, gridDim.x - 1 - blockIdx.x, s0, s1);
        const int nr = r1 - r0, ns = s1 - s0, units_r = nr > 0 ? ((r1 - 1) >> 4) - (r0 >> 4) + 1 : 0;
        const TokKind& K = sh.kind[0];
        const int n1 = nr + ns;
        const Spread sp1(ns, n1);
        // place p = warp, warp + 16, ...: (unless the shared expert's) FFN rows 2 f, 2 f + 1 of entry e
        struct Place1 { int p, i, e, f; };
        auto next1 = [&](Place1& P) {
            P.p += kTokWarps;
            const int i = P.p - (SH ? sp1.before(P.p) : 0);
            P.f += i - P.i;
            P.i = i;
            while (P.f >= half && P.e < nv) { P.f -= half; ++P.e; }
        };
        Place1 a1{warp, warp - (SH ? sp1.before(warp) : 0), 0, 0};
        if (nr > 0) {
            a1.e = (r0 + a1.i) / half;
            a1.f = r0 + a1.i - a1.e * half;
        }
        Place1 c1 = a1;
        auto open1 = [&] {
            while (SH && a1.p < n1 && sp1.at(a1.p)) next1(a1);
            if (a1.p >= n1) return;
            const uint8_t* src = (const uint8_t*) sh.ptr[sh.ve[a1.e]] + (size_t) (2 * a1.f) * K.rb;
            new_row(src + (lane & 2 ? A.up_off : 0) + (lane & 1) * K.rb, K.rb);
        };
        auto ask1 = [&] {
            if (a1.p >= n1) return;
            if (!ask(K.bytes, K.pitch, K.nseg)) return;
            next1(a1);
            open1();
        };
        open1();
        ask1();
        ask1();
        const RowLut<T, true> lut(s_tab, lane);
        const TokCol X{cols, nblk_x}, X1{SH && XB == 2 ? cols + tok_col_bytes(nblk_x) : cols, nblk_x};
        const size_t rb_sh = SH ? row_bytes(MAYA_Q8_0, n_embd) : 0;
        for (; c1.p < n1; next1(c1)) {
            float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            const bool shd = SH && sp1.at(c1.p);
            int g, lo, hi, lu;                           // the item in its class; that unit's items [lo, hi) of this block, its place here
            if (SH && shd) {
                g = s0 + sp1.before(c1.p);
                const uint8_t* row = A.shared + (size_t) (A.sh_lo + 2 * g) * rb_sh;
                tok_dot_shared(row, row + (size_t) A.n_ff_sh * rb_sh, rb_sh, X1, nblk_x, lane, acc);
                lo = max(g & ~15, s0); hi = min((g & ~15) + 16, s1); lu = units_r + (g >> 4) - (s0 >> 4);
            } else {
                g = r0 + c1.i;
                const uint32_t p0 = (uint32_t) sh.ptr[sh.ve[c1.e]] + (uint32_t) (2 * c1.f) * K.rb, up = (uint32_t) A.up_off;
                const uint32_t o[4] = {p0, p0 + K.rb, p0 + up, p0 + up + K.rb};
                for (int sg = 0; sg < K.nseg; ++sg) {
                    if (!(ok = wait())) break;
                    uint32_t row[4];
#pragma unroll
                    for (int r = 0; r < 4; ++r) row[r] = ring + (got & 1) * A.stage + r * RowGeo<T>::pitch + seg_off<T>(o[r], sg);
                    tok_dot<T>(s_raw, row, X, sg * RowGeo<T>::blocks * RowGeo<T>::cpb, min(RowGeo<T>::blocks, n_embd / RowGeo<T>::qk - sg * RowGeo<T>::blocks) * RowGeo<T>::cpb,
                               lane, lut, acc);
                    ++got;
                    ask1();
                }
                if (!ok) break;
                lo = max(g & ~15, r0); hi = min((g & ~15) + 16, r1); lu = (g >> 4) - (r0 >> 4);
            }
            const float v = tok_sum4(acc, lane), hv = swiglu(v, __shfl_xor_sync(0xffffffffu, v, 16), A.limit);
            if (lane == 0 || lane == 8) hb[lu * 32 + 2 * (g & 15) + (lane >> 3)] = hv;
            __syncwarp();
            int n = 0;
            if (lane == 0) {
                __threadfence_block();
                n = atomicAdd(&hc[lu], 1) + 1;
            }
            if (__shfl_sync(0xffffffffu, n, 0) == hi - lo) {             // the unit's last item here: its q8_1 block
                __threadfence_block();
                const int slot = shd ? k * nblk_h + (A.sh_lo + 2 * g) / 32 : sh.ve[c1.e] * nblk_h + c1.f / 16;
                float h = *(volatile float*) &hb[lu * 32 + lane];
                bool whole = true;
                if (hi - lo < 16) {                      // shared with another block: in the scratch
                    float* const hst = (float*) ((uint8_t*) A.h + (size_t) (MAYA_MAX_K + 1) * nblk_h * 40) + (size_t) slot * 32;
                    if (lane >= 2 * (lo & 15) && lane < 2 * (((hi - 1) & 15) + 1)) __stcg(&hst[lane], h);
                    __threadfence();
                    __syncwarp();
                    unsigned sum = 0u;
                    if (lane == 0) sum = atomicAdd(A.unit_count + slot, (unsigned) (hi - lo)) + (unsigned) (hi - lo);
                    whole = (__shfl_sync(0xffffffffu, sum, 0) & 15u) == 0u;
                    __threadfence();
                    if (whole) h = __ldcg(&hst[lane]);
                }
                if (whole) {
                    const TokBlock t = A.d_type == MAYA_IQ1_S && !shd ? tok_round<true>(h) : tok_round<false>(h);
                    gq[(size_t) slot * 32 + lane] = (int8_t) t.q;
                    if (lane == 0) { gd[slot] = t.d; gs[slot] = t.sum; }
                }
            }
        }
        if (ok) { open2(); ask2(); ask2(); }             // the first down rows, under the barrier
    }
    ok = __syncthreads_or(ok ? 0 : 1) == 0;              // the block agrees
    const unsigned mark = (sh.epoch + 1u) | 0x80000000u;             // this launch's, never zero
    if (!ok && tid == 0) tok_gave_up(A.sync, mark);
    if (A.d_type != T) tok_fill(A.d_type, s_tab, tid);
    stamp(A.sync, 2);
    const bool met = grid_barrier(A.sync, sh.epoch, &sh.bar_ok, [&](int i) {
        if (i >= k) return;
        sh.w[i] = A.router == 1 ? route_weight<1>(sh.route, k, i, A.router_w_scale, A.router_norm_w) : route_weight<0>(sh.route, k, i, 0.0f, 0);
        if (blockIdx.x == 0) A.weights[i] = sh.w[i];
    });
    stamp(A.sync, 3);
    bool done = ok && met;
    if (!ok && met) tok_reset(A.unit_count, (MAYA_MAX_K + 1) * nblk_h);

    // ---------------------------------------------------------------- phase 2: q8_1(h), down, combine
    if (done) {
        const unsigned lost = tid == 0 ? __ldcg(A.sync + kTokMark) : 0u;   // (asked for ahead of h: both arrive together)
        const int nb_r = n_ff / 32, total_r = nv * nb_r, b_s = has_sh ? A.sh_lo / 32 : 0, nb_s = has_sh ? (A.sh_hi - A.sh_lo) / 32 : 0;
        const int xb2 = A.d_type == MAYA_Q4_K || A.d_type == MAYA_Q5_K ? 2 : 1;
        for (int i = tid; i < 2 * (total_r + nb_s); i += kTokThreads) {          // half a block each, its scale or its sum
            const int hf = i & 1, b = i >> 1;
            const bool shd = b >= total_r;
            const int ei = shd ? 0 : b / nb_r, blk = shd ? b - total_r : b - ei * nb_r;
            const size_t src = (size_t) (shd ? k * nblk_h + b_s + blk : sh.ve[ei] * nblk_h + blk);
            const uint4 v = __ldcg((const uint4*) gq + 2 * src + hf);
            const uint32_t ds = hf ? (uint32_t) __ldcg(gs + src) : __float_as_uint(__ldcg(gd + src));
            uint8_t* const col = cols + (shd ? nv : ei) * tok_col_bytes(nb_r);
            const int n = shd ? nb_s : nb_r;
            const bool two = !shd && xb2 == 2;
            *(uint4*) (col + (two ? tok_piece<2>(n, blk, hf) : tok_piece<1>(n, blk, hf))) = v;
            *(uint32_t*) (col + (two ? tok_scale<2>(n, blk) : tok_scale<1>(n, blk)) + hf * n * 4) = ds;
        }
        if (tid == 0) sh.lost = lost == mark;            // a block gave up: looked at below, before anything is written
        __syncthreads();
        if (SH) {                                        // the shared expert's rows, by the warps that have an item less (in the loop
                                                         // below, spread among the others, this phase took 21.1 us instead of 18.6)
            const TokCol H{cols + nv * tok_col_bytes(nb_r), nb_s};
            const size_t rbs = row_bytes(MAYA_Q8_0, A.n_ff_sh);
            for (int q = (warp - n2) & (kTokWarps - 1); q < n2s; q += kTokWarps) {
                const uint8_t* row = A.shared + 2 * (size_t) A.n_ff_sh * row_bytes(MAYA_Q8_0, n_embd) + (size_t) (o0 + 4 * q) * rbs + row_bytes(MAYA_Q8_0, A.sh_lo);
                float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                tok_dot_shared(row, row + 2 * rbs, rbs, H, nb_s, lane, acc);
                const float v = tok_sum4(acc, lane);
                if ((lane & 7) == 0) sh.part[4 * q + 2 * (lane >> 4) + ((lane >> 3) & 1)][k] = v;
            }
        }
        auto down = [&](auto type_c) {
            constexpr int TD = decltype(type_c)::value;
            using G = RowGeo<TD>;
            const RowLut<TD, true> lut(s_tab, lane);
            const int l = kd.groups > 1 ? lane & (kd.calls - 1) : lane, grp = kd.groups > 1 ? lane / kd.calls : 0;
            for (Place c2 = first2(); c2.p < n2; next2(c2)) {
                float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                const uint32_t p0 = (uint32_t) (uintptr_t) down_rows(c2.e, c2.q);
                const TokCol H{cols + c2.e * tok_col_bytes(nb_r), nb_r};
                for (int sg = 0; sg < kd.nseg; ++sg) {
                    if (!(ok = wait())) return;
                    uint32_t row[4];
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        row[r] = ring + (got & 1) * A.stage + (uint32_t) ((r * kd.groups + grp) * kd.pitch) + (kd.cont ? p0 & 15u : seg_off<TD>(p0 + (uint32_t) r * kd.rb, sg));
                    tok_dot<TD>(s_raw, row, H, sg * G::blocks * G::cpb, min(G::blocks, n_ff / G::qk - sg * G::blocks) * G::cpb, l, lut, acc);
                    ++got;
                    ask2();
                }
                const int e = sh.ve[c2.e], at = c2.q * kd.rpi;
                if (kd.groups == 1) {
                    const float v = tok_sum4(acc, lane);
                    if ((lane & 7) == 0) sh.part[at + 2 * (lane >> 4) + ((lane >> 3) & 1)][e] = v;
                } else {                                 // groups of lanes side by side
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        float v = acc[r];
                        for (int o = kd.calls >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                        if (l == 0 && at + r * kd.groups + grp < nrows) sh.part[at + r * kd.groups + grp][e] = v;
                    }
                }
            }
        };
#define MAYA_TOK_DOWN(TT) case TT: if constexpr (kTokPair<T, TT>) down(std::integral_constant<int, TT>{}); break;
        switch (A.d_type) {
            MAYA_TOK_DOWN(MAYA_Q8_0) MAYA_TOK_DOWN(MAYA_Q4_K) MAYA_TOK_DOWN(MAYA_Q5_K) MAYA_TOK_DOWN(MAYA_Q6_K) MAYA_TOK_DOWN(MAYA_IQ4_XS)
            MAYA_TOK_DOWN(MAYA_IQ2_S) MAYA_TOK_DOWN(MAYA_IQ3_S) MAYA_TOK_DOWN(MAYA_IQ3_XXS) MAYA_TOK_DOWN(MAYA_IQ2_XXS) MAYA_TOK_DOWN(MAYA_IQ1_S)
        }
#undef MAYA_TOK_DOWN
        done = __syncthreads_or(ok && sh.lost == 0 ? 0 : 1) == 0;
        if (!done && tid == 0) atomicExch(&A.sync[2], 1u);
        if (done && tid < nrows) {
            float m = 0.0f;
            for (int i = 0; i < k; ++i) m = __fmaf_rn(sh.w[i], sh.ptr[i] != 0ull ? sh.part[tid][i] : 0.0f, m);
            if (A.cpu_flag != nullptr && *A.cpu_flag) m = __fadd_rn(m, A.cpu_part[o0 + tid]);    // the host lane's answer (moe_down's order)
            A.out[o0 + tid] = __fadd_rn(m, has_sh ? sh.part[tid][k] : 0.0f);
        }
    }
    // what a warp has in flight lands before the block's shared memory goes away (nothing, unless a wait ran out); A.polls may be few
    for (; got < asked; ++got) mbar_wait(&sh.full[warp][got & 1], (got >> 1) & 1, A.drain_polls);
    stamp(A.sync, 4);
    __syncthreads();
    if (A.hc.R_new != nullptr && done) hc_post_rows(A.out, A.hc, n_embd, o0, o1, tid, kTokThreads);
    stamp(A.sync, 5);
    if (blockIdx.x == 0 && tid == 0) *(volatile unsigned*) &A.sync[1] = sh.epoch + 1u;       // the next launch's epoch
}

template<int T, bool SH> int launch_token(TokArgs A, cudaStream_t s) {
    static SmemLimit smem_limit;
    const int grid = sm_count();
    const size_t smem = token_smem(T, A, grid);
    if (smem == 0) return kNotHere;
    if (!smem_limit.raise((const void*) token_kernel<T, SH>, kTokMostSmem)) return note_launch("token smem attribute");
    void* params[] = {&A};
    return launch_cooperative<token_kernel<T, SH>>(dim3(grid), dim3(kTokThreads), params, smem, s, "moe_token");
}

}  // namespace

template<int T> int token_by_type(const TokArgs& A, cudaStream_t s) { return A.shared != nullptr ? launch_token<T, true>(A, s) : launch_token<T, false>(A, s); }

}  // namespace maya
