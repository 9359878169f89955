// moe_window.cu - the routed experts of a window (2..16 tokens) or of a short plan: gate/up + SwiGLU + q8_1(h), and the down
// rows, with the weight rows streamed through shared memory.
//
// What bounds this path: on a B200 neither HBM nor the dot products but instruction issue and the shared-memory pipe - a
// 2-4 bit weight costs 60-90 instructions per 32 to decode and 14-38 per column to dot - so everything around them has to
// be cheap and no warp may wait for its loads.  One 512-thread block an SM; its warps never meet inside a row:
//   * the work is a list of jobs - a group (distinct expert) and up to `ncm` of its entries (activation columns) - times
//     chunks of 64 weight rows (32 gate + the same 32 up rows, or 64 down rows).  Every block takes one contiguous share of
//     that list, equal in estimated COST (decode + columns x dot), not in count: a chunk with eight columns costs several
//     times one with a single column.  Contiguous, so that a block stages a job's columns once for all its chunks.
//   * a warp owns four rows of a chunk and streams their K segments into a private ring with cp.async.bulk, two segments
//     ahead, across chunk and job boundaries: no block barrier stands between a warp and its next bytes, and decoding reads
//     shared memory, where a lane's 2-byte aligned fields cost one or two wavefronts a warp instead of the four to five
//     cache lines they touch in global memory.
//   * codebooks lie in several copies side by side in shared memory, lane l reading copy l % n.
// Read in place by a grid of (chunk, group) blocks (gate/up) and streamed 64 rows a stage (down), an 8-token Q4_K window took
// 318 us, a 16-token IQ3_S one 570; now 263 and 433.  (32 warps of two rows: 266 and 484, the activation reads then bind.)
//
// The arithmetic is rows_dot's (maya_dots.cuh), value for value - the same integers, the same lane order, the same sums - so
// every token's result is bit-identical to the single-token kernels'.
//
// Plain bulk copies (one destination: this block) of this GPU's own memory.  A row need not start on a 16-byte boundary: the
// aligned window around a segment is copied (expert blobs are 16-byte aligned and a whole number of 16-byte words long, so
// it stays inside).  Every wait is bounded; one that runs out makes the block skip what is left (its outputs are then
// missing) after the copies in flight were given the same bounded time to land.  A blob that is not 16-byte aligned is
// copied with ordinary loads instead.
#include "maya_dots.cuh"
#include "maya_internal.cuh"
#include "maya_stream.cuh"

#include <atomic>
#include <type_traits>

namespace maya {
namespace {

constexpr int kWNC = 8;            // most activation columns of a job
constexpr int kWStages = 2;        // segments in flight a warp
constexpr int kWMaxJobs = 128;     // T <= 16 tokens x 8 routes: a job has at least one entry
constexpr int kWChunkRows = 64;    // weight rows of a chunk

// ---- decoders: Dec<T>'s fields and dot, loaded from shared memory - byte `o` of `s` is the block's first - with fewer
//      instructions.  rep: copies of the codebook, `tab` = this lane's copy.  ONE: for a single column, where it is cheaper to
//      correct the dot for the signs (see maya_dots_t1.cuh) than to negate the weights.
__device__ __forceinline__ uint32_t s_u32(const uint8_t* s, uint32_t o) { return *(const uint32_t*) (s + o); }
// 4 bytes at an even place; sel: 0x3210 where o is a multiple of 4, else 0x5432
__device__ __forceinline__ uint32_t s_u32_a2(const uint8_t* s, uint32_t o, uint32_t sel) {
    const uint32_t a = o & ~3u;
    return prmt_raw(s_u32(s, a), s_u32(s, a + 4), sel);
}
// the selector for fields 2 bytes (and a multiple of 4) into a block at o
__device__ __forceinline__ uint32_t sel_2(uint32_t o) { return (o & 2u) ? 0x3210u : 0x5432u; }

template<int T, bool ONE> struct WDec : Dec<T> {
    static constexpr int rep = 1;
    __device__ __forceinline__ void load(const uint8_t* s, uint32_t o, int c, const uint32_t* tab) { Dec<T>::load(s + o, c, tab); }
};
// eight signed weight words (or, with ONE, codebook words XOR mask and the masks) and their dots
template<bool ONE> struct WSigned {
    int w[8];
    uint32_t mk[ONE ? 8 : 1];
    __device__ __forceinline__ void set(int i, uint32_t g, uint32_t m) {
        if constexpr (ONE) { w[i] = (int) (g ^ m); mk[i] = m; }
        else w[i] = apply_sign4(g, m);
    }
    __device__ __forceinline__ int dot4(const XQ& v, int i0, int s) const {        // words i0 .. i0 + 3
#pragma unroll
        for (int i = i0; i < i0 + 4; ++i) s = __dp4a(w[i], v.u[i], s);
        if constexpr (ONE) {
            int m = 0;
#pragma unroll
            for (int i = i0; i < i0 + 4; ++i) m = __dp4a((int) mk[i], v.u[i], m);
            s -= m;
        }
        return s;
    }
};
template<bool ONE> struct WDec<MAYA_IQ2_S, ONE> : WSigned<ONE> {
    static constexpr int rep = 8;
    int ls0, ls1;
    float d;
    __device__ __forceinline__ void load(const uint8_t* s, uint32_t o, int c, const uint32_t* tab) {
        const uint32_t sel = sel_2(o);
        d = ld_f16(s + o);
        const uint32_t qs = s_u32_a2(s, o + 2 + 4 * c, sel), sg = s_u32_a2(s, o + 34 + 4 * c, sel);
        const uint32_t qh = s[o + 66 + c], sc = s[o + 74 + c];
        ls0 = (int) (sc & 0x0F);
        ls1 = (int) (sc >> 4);
        const uint2* grid = (const uint2*) tab;
        const uint32_t hw = ((qh & 0x33u) * 0x1001u + (qh & 0xCCu) * 0x40040u) & 0x03030303u;      // see Dec1<MAYA_IQ2_S>
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            const uint2 g = grid[prmt_raw(qs, hw, 0xCC00u + ((4 + l) << 4) + l) * rep];
            const uint32_t b = byte_of(sg, l);
            this->set(2 * l, g.x, sign_mask_lo(b));
            this->set(2 * l + 1, g.y, sign_mask_hi(b));
        }
    }
    __device__ __forceinline__ float dot(const XQ& v, const XQ&) const {
        const int s0 = this->dot4(v, 0, 0), s1 = this->dot4(v, 4, 0);
        return __fmul_rn(__fmul_rn(d, v.d), (float) ((s0 * ls0 + s1 * ls1 + (s0 + s1) / 2) / 4));
    }
};
// IQ3_S: every codebook value is odd, g = 2 b + 1 with b in 0..7.  Flipping b's bits negates it: 2 ~b + 1 = -g.  So the table
// holds b, a sign is one XOR, and sum(+-g u) = 2 sum((b ^ m) u) + sum(u), the block's sum being at hand.
template<bool ONE> struct WDec<MAYA_IQ3_S, ONE> {
    static constexpr int rep = 16;
    int w[8];
    int mul;
    float d;
    __device__ __forceinline__ void load(const uint8_t* s, uint32_t o, int c, const uint32_t* tab) {
        const uint32_t sel = sel_2(o), qa = (o + 2 + 8 * c) & ~3u;
        d = ld_f16(s + o);
        const uint32_t w1 = s_u32(s, qa + 4), q0 = prmt_raw(s_u32(s, qa), w1, sel), q1 = prmt_raw(w1, s_u32(s, qa + 8), sel);
        const uint32_t qh = s[o + 66 + c], sg = s_u32_a2(s, o + 74 + 4 * c, sel);
        mul = 1 + 2 * (int) ((s[o + 106 + (c >> 1)] >> (4 * (c & 1))) & 0x0F);
        // byte l of h0 / h1: bit l / 4 + l of qh, an entry's ninth index bit
        const uint32_t h0 = ((qh & 15u) * 0x204081u) & 0x01010101u, h1 = ((qh >> 4) * 0x204081u) & 0x01010101u;
#pragma unroll
        for (int l = 0; l < 8; ++l) {
            const uint32_t b = tab[prmt_raw(l < 4 ? q0 : q1, l < 4 ? h0 : h1, 0xCC00u + ((4 + l % 4) << 4) + l % 4) * rep];
            const uint32_t sb = byte_of(sg, l >> 1);
            w[l] = (int) (b ^ ((l & 1) ? sign_mask_hi(sb) : sign_mask_lo(sb)));
        }
    }
    __device__ __forceinline__ float dot(const XQ& v, const XQ&) const {
        int s = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) s = __dp4a(w[i], v.u[i], s);
        return __fmul_rn(__fmul_rn(d, v.d), (float) ((2 * s + v.isum) * mul));
    }
};
template<bool ONE> struct WDec<MAYA_IQ3_XXS, ONE> : WSigned<ONE> {
    static constexpr int rep = 32;
    int ls;
    float d;
    __device__ __forceinline__ void load(const uint8_t* s, uint32_t o, int c, const uint32_t* tab) {
        const uint32_t sel = sel_2(o), qa = (o + 2 + 8 * c) & ~3u;
        d = ld_f16(s + o);
        const uint32_t w1 = s_u32(s, qa + 4), q0 = prmt_raw(s_u32(s, qa), w1, sel), q1 = prmt_raw(w1, s_u32(s, qa + 8), sel);
        const uint32_t aux = s_u32_a2(s, o + 66 + 4 * c, sel);
        ls = (int) (aux >> 28);
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            const uint32_t s8 = ksign8((aux >> (7 * l)) & 127u), q = l < 2 ? q0 : q1;
            this->set(2 * l, tab[byte_of(q, 2 * (l & 1)) * rep], sign_mask_lo(s8));
            this->set(2 * l + 1, tab[byte_of(q, 2 * (l & 1) + 1) * rep], sign_mask_hi(s8));
        }
    }
    __device__ __forceinline__ float dot(const XQ& v, const XQ&) const {
        const int t = this->dot4(v, 4, this->dot4(v, 0, 0));
        return __fmul_rn(__fmul_rn(d, v.d), (float) ((ls * t + t / 2) / 2));
    }
};
template<bool ONE> struct WDec<MAYA_IQ2_XXS, ONE> : WSigned<ONE> {
    static constexpr int rep = 16;
    int ls;
    float d;
    __device__ __forceinline__ void load(const uint8_t* s, uint32_t o, int c, const uint32_t* tab) {
        const uint32_t sel = sel_2(o), qa = (o + 2 + 8 * c) & ~3u;
        d = ld_f16(s + o);
        const uint32_t w1 = s_u32(s, qa + 4), qi = prmt_raw(s_u32(s, qa), w1, sel), aux = prmt_raw(w1, s_u32(s, qa + 8), sel);
        ls = (int) (aux >> 27) | 1;
        const uint2* grid = (const uint2*) tab;
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            const uint2 g = grid[byte_of(qi, l) * rep];
            const uint32_t s8 = ksign8((aux >> (7 * l)) & 127u);
            this->set(2 * l, g.x, sign_mask_lo(s8));
            this->set(2 * l + 1, g.y, sign_mask_hi(s8));
        }
    }
    __device__ __forceinline__ float dot(const XQ& v, const XQ&) const {
        const int t = this->dot4(v, 4, this->dot4(v, 0, 0));
        return __fmul_rn(__fmul_rn(d, v.d), (float) (t * ls / 8));
    }
};

// ---- the geometry of a type's stream.  A segment: kSegVals values of a row (a multiple of what 32 lanes take in one step, so
//      that a lane's calls are the same whatever the segments are).  kPitch: a segment's room in a stage, its bytes and 16 for
//      the aligned window.
template<int T> struct WGeo {
    static constexpr int warps = 16, threads = warps * 32, rw = kWChunkRows / warps;      // a warp's rows: 4
    // most columns of a job: four where a call spans two q8_1 blocks (six or eight spill 1.3 KB: 617 against 263 us on the window above)
    static constexpr int nc = Dec<T>::xblk == 2 ? 4 : kWNC;
    static constexpr int vals = T == MAYA_Q8_0 || T == MAYA_Q6_K ? 1024 : 2048;
    static constexpr int qk = Fmt<T>::qk, cpb = Dec<T>::cpb;
    static constexpr int blocks = vals / qk;                                 // weight blocks of a segment
    static constexpr int bytes = blocks * Fmt<T>::bytes;
    static constexpr int pitch = (bytes + 15 + 16) & ~15;
    static constexpr int stage = rw * pitch;                                 // a warp's stage
    static constexpr int ring = warps * kWStages * stage;
    static constexpr int tab = Fmt<T>::tab_words * 4 * WDec<T, false>::rep;
    // The cost of 32 calls of a row against nc columns, in instructions: decoding, nc dots - or, where that is more, what their
    // bytes cost at an SM's share of HBM.
    static constexpr int dec_cost = T == MAYA_Q8_0 ? 25 : T == MAYA_Q4_K || T == MAYA_IQ1_S ? 45 : T == MAYA_Q5_K ? 60 : T == MAYA_IQ3_S || T == MAYA_IQ3_XXS ? 90 : 75;
    static constexpr int col_cost = Dec<T>::xblk == 2 ? 40 : 15;
    static constexpr int byte_cost = 32 / cpb * Fmt<T>::bytes / 8;
    __device__ __forceinline__ static int cost(int nc) { return max(dec_cost + nc * col_cost, byte_cost); }
};

// What a launch works on.
struct WArgs {
    const unsigned long long* ptr;   // [groups] blob addresses (0: skipped)
    const int* start;                // [groups + 1] entry ranges, or NULL: group g has the single entry g
    const int* n_groups;             // device count, or NULL: `cap`
    const int* ent_slot;             // [entries] an entry's h / partial slot, or NULL: the entry number
    const int* skip;                 // optional "do nothing" flag
    int cap;                         // most groups (<= kWMaxJobs)
    int tok_from_slot;               // gate/up: an entry's column is slot >> 3 (a window), else column 0 (one token)
    int ncm;                         // columns of a job, <= kWNC
    int plain;                       // the rows do not start and end on 16-byte boundaries inside a blob: no bulk copies
    int n_embd, n_ff;
    size_t row_off;                  // byte offset of the rows in a blob: gate/up 0, down: the down rows
    size_t up_off;                   // gate/up: byte offset of the up rows
    float limit;
    const uint8_t* xq;               // gate/up: token columns, xq_stride apart; down: h images [slot]
    size_t xq_stride;
    uint8_t* hq;                     // gate/up out: [slot][n_ff / 32] q8_1
    float* part;                     // down out: [slot][n_embd]
};

struct WJob { unsigned long long ptr; int e0, nc; };
struct WShared {
    uint64_t full[16][kWStages];
    WJob job[kWMaxJobs];
    int cost[kWMaxJobs + 1];         // cost of a job's chunks before job j (prefix sums of the jobs' per-chunk costs)
    int njobs, fail;
    float s_g[2][kWNC][32], s_u[2][kWNC][32];
    float res[kWChunkRows][kWNC];      // a warp's sums of a chunk
};

// ---- the columns in shared memory.  A column has room for CB q8_1 blocks, a compile-time number, so that the loads of every
//      column, plane and half differ from one another by constants only (computed addresses were a sixth of the kernel's
//      instructions): the planes of 16-byte pieces of maya_dots.cuh's planar form, then as many planes of scales and of sums.
template<int CB> constexpr int kColBytes = CB * 40;
template<int XB, int CB> __device__ __forceinline__ XQ col_load(const uint8_t* cols, int c, int j, int i16, int i4) {
    constexpr int P = CB / XB;
    const uint8_t* p = cols + c * kColBytes<CB> + 2 * j * P * 16 + i16;
    const int4 a = *(const int4*) p, b = *(const int4*) (p + P * 16);
    XQ v;
    v.u[0] = a.x; v.u[1] = a.y; v.u[2] = a.z; v.u[3] = a.w;
    v.u[4] = b.x; v.u[5] = b.y; v.u[6] = b.z; v.u[7] = b.w;
    v.d = *(const float*) (cols + c * kColBytes<CB> + CB * 32 + j * P * 4 + i4);
    v.isum = *(const int*) (cols + c * kColBytes<CB> + CB * 36 + j * P * 4 + i4);
    return v;
}
// Block i of a column, a thread's: nine words in flight (word by word the columns of a job took 8 us to stage).
template<int XB, int CB, bool SUM_F16> __device__ __forceinline__ void col_store(const uint8_t* xq, uint8_t* cols, int c, int i) {
    constexpr int P = CB / XB;
    const uint32_t* src = (const uint32_t*) (xq + (size_t) i * kQ81Bytes);
    uint32_t w[9];
#pragma unroll
    for (int j = 0; j < 9; ++j) w[j] = src[j];
    uint8_t* col = cols + c * kColBytes<CB>;
    const int j = i % XB, n = i / XB;
    *(int4*) (col + (2 * j * P + n) * 16) = make_int4((int) w[1], (int) w[2], (int) w[3], (int) w[4]);
    *(int4*) (col + ((2 * j + 1) * P + n) * 16) = make_int4((int) w[5], (int) w[6], (int) w[7], (int) w[8]);
    *(float*) (col + CB * 32 + (j * P + n) * 4) = __half2float(__ushort_as_half((unsigned short) (w[0] & 0xFFFFu)));
    int s = 0;
    if constexpr (SUM_F16) s = __float_as_int(__half2float(__ushort_as_half((unsigned short) (w[0] >> 16))));
    else {
#pragma unroll
        for (int k = 1; k < 9; ++k) s = __dp4a((int) w[k], 0x01010101, s);
    }
    *(int*) (col + CB * 36 + (j * P + n) * 4) = s;
}

// One segment of a warp's rows against NC columns: rows_dot's loop (maya_dots.cuh), all four rows decoded before the
// columns, two where four would not fit the registers.  NC
// is exact (or one more than the job's columns: a column that is not there is computed from whatever lies in its place and
// dropped), so that no branch parts one column's loads from the next one's arithmetic.
template<int T, int NC, int RW, int CB>
__device__ __forceinline__ void segment_dot(const uint8_t* s, const uint32_t (&row)[RW], const uint8_t* cols, int blk0, int ncalls, int lane,
                                            const uint32_t* tab, float (&acc)[RW][NC]) {
    using G = WGeo<T>;
    constexpr int XB = Dec<T>::xblk, RP = XB == 2 || NC > 4 ? 2 : 4;
    for (int k = lane; k < ncalls; k += 32) {
        const int kb = k / G::cpb, ci = k - kb * G::cpb;
        const int n = ((blk0 + kb) * (G::qk / 32) + ci * XB) / XB;
#pragma unroll
        for (int r0 = 0; r0 < RW; r0 += RP) {
            if (r0 > 0) asm volatile("" ::: "memory");       // the second two rows' loads stay behind: their registers are the first two's
            WDec<T, NC == 1> dec[RP];
#pragma unroll
            for (int j = 0; j < RP; ++j) dec[j].load(s, row[r0 + j] + kb * Fmt<T>::bytes, ci, tab);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const XQ a = col_load<XB, CB>(cols, c, 0, n * 16, n * 4);
                XQ b = a;
                if constexpr (XB == 2) b = col_load<XB, CB>(cols, c, 1, n * 16, n * 4);
#pragma unroll
                for (int j = 0; j < RP; ++j) acc[r0 + j][c] = __fadd_rn(acc[r0 + j][c], dec[j].dot(a, b));
            }
        }
    }
}

// UP: gate/up (chunk = 32 FFN rows: a warp's rows are 2 gate + 2 up); else down (chunk = 64 rows).
template<int T, bool UP, int CB>
__global__ void __launch_bounds__(WGeo<T>::threads, 1) window_kernel(const WArgs A) {
    using G = WGeo<T>;
    using D = WDec<T, false>;
    constexpr int XB = Dec<T>::xblk, RW = G::rw, kWThreads = G::threads;
    extern __shared__ __align__(128) uint8_t s_raw[];
    __shared__ WShared sh;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n_in = UP ? A.n_embd : A.n_ff, nblk = n_in / 32;
    const size_t rb = row_bytes(T, n_in);
    const int n_rows = UP ? A.n_ff : A.n_embd;                   // rows of one output
    const int nchunk = UP ? A.n_ff / 32 : (A.n_embd + kWChunkRows - 1) / kWChunkRows;
    const uint32_t ring = warp * kWStages * G::stage;            // the warp's ring in s_raw
    uint32_t* const s_tab = (uint32_t*) (s_raw + G::ring);
    uint8_t* const cols = s_raw + G::ring + G::tab;

    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if constexpr (G::tab > 0) {                                  // the codebook's copies: constants of the library
        constexpr int W = (T == MAYA_IQ2_S || T == MAYA_IQ2_XXS) ? 2 : 1, R = D::rep;
        const uint32_t* src = tab_source<T>();
        for (int i = tid; i < G::tab / 4; i += kWThreads) {
            const uint32_t g = src[i / (W * R) * W + i % W];
            s_tab[i] = T == MAYA_IQ3_S ? (g >> 1) & 0x07070707u : g;
        }
    }
    if (lane == 0) {
        for (int s = 0; s < kWStages; ++s) mbar_init(&sh.full[warp][s], RW);
        if (warp == 0) sh.fail = 0;
    }
    mbar_fence_init();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (A.skip != nullptr && *A.skip) return;

    // ---- the jobs, by one warp: four groups a lane at most
    if (warp == 0) {
        int ng = A.n_groups ? *A.n_groups : A.cap;
        ng = min(min(ng, A.cap), kWMaxJobs);
        int base = 0;
        for (int g0 = 0; g0 < ng; g0 += 32) {
            const int g = g0 + lane;
            unsigned long long p = 0ull;
            int e0 = 0, ne = 0;
            if (g < ng) {
                p = A.ptr[g];
                e0 = A.start ? A.start[g] : g;
                ne = (A.start ? A.start[g + 1] : g + 1) - e0;
            }
            const int nj = p != 0ull && ne > 0 ? (ne + A.ncm - 1) / A.ncm : 0;
            int incl = nj;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            for (int j = 0; j < nj; ++j) {
                const int at = base + incl - nj + j;
                if (at < kWMaxJobs) sh.job[at] = WJob{p, e0 + j * A.ncm, min(A.ncm, ne - j * A.ncm)};
            }
            base += __shfl_sync(0xffffffffu, incl, 31);
        }
        const int njobs = min(base, kWMaxJobs);
        __syncwarp();
        int run = 0;
        for (int j0 = 0; j0 < njobs; j0 += 32) {
            const int j = j0 + lane, c = j < njobs ? G::cost(sh.job[j].nc) : 0;
            int incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            if (j < njobs) sh.cost[j] = run + incl - c;
            run += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) { sh.cost[njobs] = run; sh.njobs = njobs; }
    }
    __syncthreads();
    const int njobs = sh.njobs;
    // chunk c of job j starts at cost[j] * nchunk + c * (cost[j + 1] - cost[j]); this block takes those that start in [x0, x1)
    const long long total = (long long) sh.cost[njobs] * nchunk;
    auto first_at = [&](long long at, int& j, int& c) {
        j = 0;
        while (j < njobs && (long long) sh.cost[j + 1] * nchunk <= at) ++j;
        c = 0;
        if (j < njobs) {
            const int per = sh.cost[j + 1] - sh.cost[j];
            c = (int) ((at - (long long) sh.cost[j] * nchunk + per - 1) / per);
            if (c >= nchunk) { ++j; c = 0; }
        }
    };
    int job, chunk, job1, chunk1;
    first_at((long long) blockIdx.x * total / gridDim.x, job, chunk);
    first_at((long long) (blockIdx.x + 1) * total / gridDim.x, job1, chunk1);
    if (job > job1 || (job == job1 && chunk >= chunk1)) return;

    const int nseg = (n_in + G::vals - 1) / G::vals;
    // row r of this warp in (job, chunk): gate rows, then the same up rows; or down rows (the last chunk's rows past the end are
    // its last row again: read, and not written)
    auto row_ptr = [&](unsigned long long blob, int ch, int r) -> const uint8_t* {
        constexpr int H = RW / 2;
        if constexpr (UP) return (const uint8_t*) blob + A.row_off + (r / H) * A.up_off + (size_t) (ch * 32 + H * warp + r % H) * rb;
        else return (const uint8_t*) blob + A.row_off + (size_t) min(ch * kWChunkRows + RW * warp + r, n_rows - 1) * rb;
    };
    // ---- the stream: the warp's next segment to ask for
    int pj = job, pc = chunk, ps = 0, pstage = 0;
    auto ask = [&] {
        if (pj > job1 || (pj == job1 && pc >= chunk1)) return;
        const unsigned long long blob = sh.job[pj].ptr;
        __syncwarp();                                            // every lane has read the stage's last bytes
        if ((blob & 15ull) == 0 && !A.plain) {
            if (lane < RW) {
                const uint8_t* src = row_ptr(blob, pc, lane) + (size_t) ps * G::bytes;
                const uint32_t off = (uint32_t) ((uintptr_t) src & 15u), len = (uint32_t) min((size_t) G::bytes, rb - (size_t) ps * G::bytes);
                const uint32_t bytes = (off + len + 15u) & ~15u;
                fence_proxy_async();
                mbar_expect_tx(&sh.full[warp][pstage], bytes);
                bulk_load(s_raw + ring + pstage * G::stage + lane * G::pitch, src - off, bytes, &sh.full[warp][pstage]);
            }
        } else {                                                 // ordinary loads, two bytes at a time
            for (int r = 0; r < RW; ++r) {
                const uint8_t* src = row_ptr(blob, pc, r) + (size_t) ps * G::bytes;
                const uint32_t off = (uint32_t) ((uintptr_t) src & 15u), len = (uint32_t) min((size_t) G::bytes, rb - (size_t) ps * G::bytes);
                for (uint32_t i = 2 * lane; i < len; i += 64)
                    *(uint16_t*) (s_raw + ring + pstage * G::stage + r * G::pitch + off + i) = *(const uint16_t*) (src + i);
            }
            __syncwarp();
            if (lane < RW) mbar_arrive_one(&sh.full[warp][pstage]);
        }
        pstage = pstage + 1 == kWStages ? 0 : pstage + 1;
        if (++ps == nseg) {
            ps = 0;
            if (++pc == nchunk) { pc = 0; ++pj; }
        }
    };
    for (int s = 0; s < kWStages; ++s) ask();

    const uint32_t* const tab = s_tab + (lane % D::rep) * ((T == MAYA_IQ2_S || T == MAYA_IQ2_XXS) ? 2 : 1);
    int cur = -1, stage = 0, buf = 0;
    uint32_t phase = 0;
    while (job < job1 || (job == job1 && chunk < chunk1)) {
        const WJob J = sh.job[job];
        if (job != cur) {                                        // the job's columns
            __syncthreads();                                     // everyone is done with the old ones
            for (int c = 0; c < J.nc; ++c) {
                const int slot = A.ent_slot ? A.ent_slot[J.e0 + c] : J.e0 + c;
                const uint8_t* src = A.xq + (size_t) (UP ? (A.tok_from_slot ? slot >> 3 : 0) : slot) * A.xq_stride;
                for (int i = tid; i < nblk; i += kWThreads)
                    col_store<XB, CB, T == MAYA_IQ1_S>(src, cols, c, i);
            }
            cur = job;
            __syncthreads();
        }
        uint32_t rpar = 0;                                       // where the rows start in their 16-byte windows, a byte each
#pragma unroll
        for (int r = 0; r < RW; ++r) rpar |= (uint32_t) ((size_t) row_ptr(J.ptr, chunk, r) & 15) << (8 * r);
        float* const res = &sh.res[RW * warp][0];                // [row][column]
        auto chunk_dot = [&](auto nc_c) {
            constexpr int NC = decltype(nc_c)::value;
            float acc[RW][NC];
#pragma unroll
            for (int r = 0; r < RW; ++r)
#pragma unroll
                for (int c = 0; c < NC; ++c) acc[r][c] = 0.0f;
            for (int sg = 0; sg < nseg; ++sg) {
                if (!*(volatile int*) &sh.fail && !mbar_wait(&sh.full[warp][stage], phase)) *(volatile int*) &sh.fail = 1;    // bounded
                const uint32_t so = (uint32_t) (sg * G::bytes) & 15u;
                uint32_t row[RW];
#pragma unroll
                for (int r = 0; r < RW; ++r) row[r] = ring + stage * G::stage + r * G::pitch + ((((rpar >> (8 * r)) & 15u) + so) & 15u);
                const int blk0 = sg * G::blocks;
                segment_dot<T, NC, RW, CB>(s_raw, row, cols, blk0, min(G::blocks, n_in / G::qk - blk0) * G::cpb, lane, tab, acc);
                stage = stage + 1 == kWStages ? 0 : stage + 1;
                if (stage == 0) phase ^= 1u;
                ask();
            }
#pragma unroll
            for (int r = 0; r < RW; ++r)
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const float v = warp_sum(acc[r][c]);
                    if (lane == 0) res[r * kWNC + c] = v;
                }
            __syncwarp();
        };
        switch (J.nc) {
            case 1: chunk_dot(std::integral_constant<int, 1>{}); break;
            case 2: chunk_dot(std::integral_constant<int, 2>{}); break;
            case 3: chunk_dot(std::integral_constant<int, 3>{}); break;
            case 4: chunk_dot(std::integral_constant<int, 4>{}); break;
            default:
                if constexpr (G::nc > 4) {
                    if (J.nc <= 6) chunk_dot(std::integral_constant<int, 6>{});
                    else chunk_dot(std::integral_constant<int, 8>{});
                }
        }
        const bool failed = *(volatile int*) &sh.fail != 0;
        if constexpr (UP) {
            if (lane < RW * J.nc) {                              // lane = RW column + row
                const int c = lane / RW, r = lane % RW;
                (r < RW / 2 ? sh.s_g : sh.s_u)[buf][c][RW / 2 * warp + r % (RW / 2)] = res[r * kWNC + c];
            }
            __syncthreads();                                     // two buffers: one barrier a chunk
            if (warp < J.nc && !failed) {
                const int slot = A.ent_slot ? A.ent_slot[J.e0 + warp] : J.e0 + warp;
                q8_1_store_warp(swiglu(sh.s_g[buf][warp][lane], sh.s_u[buf][warp][lane], A.limit),
                                A.hq + ((size_t) slot * (A.n_ff / 32) + chunk) * kQ81Bytes, lane);
            }
            buf ^= 1;
        } else if (lane < RW * J.nc && !failed) {
            const int c = lane / RW, row = chunk * kWChunkRows + RW * warp + lane % RW;
            const int slot = A.ent_slot ? A.ent_slot[J.e0 + c] : J.e0 + c;
            if (row < n_rows) A.part[(size_t) slot * A.n_embd + row] = res[lane % RW * kWNC + c];
        }
        __syncwarp();                                            // res is written again by the next chunk
        if (++chunk == nchunk) { chunk = 0; ++job; }
    }
    if (*(volatile int*) &sh.fail) {
        // let what may still be in flight land (bounded as well) before the block's shared memory goes away
        for (int s = 0; s < kWStages; ++s) mbar_wait(&sh.full[warp][s], phase ^ (uint32_t) (s < stage));
        __syncthreads();
    }
}

template<int T, bool UP, int CB>
int launch_window_cb(WArgs A, cudaStream_t s) {
    using G = WGeo<T>;
    // columns of a job: what fits beside the ring and the codebook, eight at most (a job's rows are decoded once for them all)
    const long room = 232448l - (long) sizeof(WShared) - 256 - G::ring - G::tab;
    A.ncm = (int) (room / kColBytes<CB>);
    if (A.ncm > G::nc) A.ncm = G::nc;
    if (A.ncm == 5 || A.ncm == 7) --A.ncm;            // five columns are dotted as six, seven as eight: the room has to be there
    if (A.ncm < 1) return kWindowTooWide;
    A.plain = ((A.row_off | A.up_off | (size_t) (UP ? A.n_ff : A.n_embd) * row_bytes(T, UP ? A.n_embd : A.n_ff)) & 15) != 0;
    const size_t smem = (size_t) G::ring + G::tab + (size_t) A.ncm * kColBytes<CB>;
    static std::atomic<size_t> set_for{0};            // per instantiation: the size the attribute was last raised to
    static std::atomic<int> set_dev{-1};
    int dev = 0;
    cudaGetDevice(&dev);
    if (set_dev.load() != dev || set_for.load() < smem) {
        if (cudaFuncSetAttribute(window_kernel<T, UP, CB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem) != cudaSuccess)
            return note_launch("window smem attribute");
        set_for.store(smem);
        set_dev.store(dev);
    }
    const int sms = sm_count();
    if (sms <= 0) return refuse(MAYA_ERR_DEVICE);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned) sms);
    cfg.blockDim = dim3(G::threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, window_kernel<T, UP, CB>, A);
    return note_launch(UP ? "window_gate_up" : "window_down");
}

// The smallest column capacity that holds the row.
template<int T, bool UP> int launch_window(const WArgs& A, cudaStream_t s) {
    const int nblk = (UP ? A.n_embd : A.n_ff) / 32;
    if (nblk <= 128) return launch_window_cb<T, UP, 128>(A, s);
    if (nblk <= 256) return launch_window_cb<T, UP, 256>(A, s);
    return kWindowTooWide;
}

template<bool UP> int launch_window_type(int type, const WArgs& A, cudaStream_t s) {
#define MAYA_WIN(TT) case TT: return launch_window<TT, UP>(A, s);
    switch (type) {
        MAYA_WIN(MAYA_Q8_0) MAYA_WIN(MAYA_Q4_K) MAYA_WIN(MAYA_IQ2_S) MAYA_WIN(MAYA_IQ3_S) MAYA_WIN(MAYA_Q5_K)
        MAYA_WIN(MAYA_Q6_K) MAYA_WIN(MAYA_IQ4_XS) MAYA_WIN(MAYA_IQ3_XXS) MAYA_WIN(MAYA_IQ2_XXS) MAYA_WIN(MAYA_IQ1_S)
        default: return refuse(MAYA_ERR_TYPE);
    }
#undef MAYA_WIN
}

}  // namespace

// Gate/up + SwiGLU + q8_1(h) of the groups; kWindowTooWide (nothing launched): n_embd leaves no room for a column.
int window_gate_up(int gu_type, const GroupArgs& A, int cap_groups, int n_embd, int n_ff, size_t up_off, float limit, const void* xq,
                   size_t xq_stride, void* hq, cudaStream_t s) {
    if (cap_groups > kWMaxJobs) return kWindowTooWide;
    WArgs W{};
    W.ptr = A.ptr; W.start = A.start; W.n_groups = A.n_groups; W.ent_slot = A.ent_slot; W.skip = A.skip; W.cap = cap_groups;
    W.tok_from_slot = A.tok_from_slot; W.n_embd = n_embd; W.n_ff = n_ff; W.up_off = up_off; W.limit = limit;
    W.xq = (const uint8_t*) xq; W.xq_stride = xq_stride; W.hq = (uint8_t*) hq;
    return launch_window_type<true>(gu_type, W, s);
}
// The down rows of the groups over the h images hq [slot]: part [slot][n_embd], unweighted.
int window_down(int d_type, const GroupArgs& A, int cap_groups, int n_embd, int n_ff, size_t down_off, const void* hq, float* part,
                cudaStream_t s) {
    if (cap_groups > kWMaxJobs) return kWindowTooWide;
    WArgs W{};
    W.ptr = A.ptr; W.start = A.start; W.n_groups = A.n_groups; W.ent_slot = A.ent_slot; W.skip = A.skip; W.cap = cap_groups;
    W.n_embd = n_embd; W.n_ff = n_ff; W.row_off = down_off;
    W.xq = (const uint8_t*) hq; W.xq_stride = (size_t) (n_ff / 32) * kQ81Bytes; W.part = part;
    return launch_window_type<false>(d_type, W, s);
}

}  // namespace maya
