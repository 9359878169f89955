// moe_window.cuh - the routed experts (and the shared one) of a window (1..16 tokens): gate/up + SwiGLU + q8_1(h),
// and the down rows, with the weight rows streamed through shared memory.
//
// What bounds this path: on a B200 neither HBM nor the dot products but instruction issue and the shared-memory pipe - a
// 2-4 bit weight costs 60-90 instructions per 32 to decode and 14-38 per column to dot - so everything around them has to
// be cheap and no warp may wait for its loads.  One 512-thread block an SM; its warps never meet inside a row:
//   * the work is a list of jobs - a group (distinct expert) and up to `ncm` of its entries (activation columns) - times
//     units of weight rows.  Every block takes one contiguous share of that list, equal in measured COST, not in count: rows
//     with eight columns cost several times those with one.  Contiguous, so that a block stages a job's columns once.
//   * a warp works on four rows at a time and streams their K segments into a private ring with cp.async.bulk, two segments
//     ahead, across unit and job boundaries: no block barrier stands between a warp and its next bytes, and decoding reads
//     shared memory, where a lane's 2-byte aligned fields cost one or two wavefronts a warp instead of the four to five
//     cache lines they touch in global memory.
//   * the always-on shared expert, when it is Q8_0, is one more job list in the same launches - its rows against all the tokens -
//     so that its 40 MB hide behind an instruction-bound phase instead of taking two GEMV launches and a SwiGLU launch a token.
//   * codebooks lie in several copies side by side in shared memory, lane l reading copy l % n.
// Read in place by a grid of (rows, group) blocks (gate/up) and streamed 64 rows a stage (down), an 8-token Q4_K window took
// 318 us, a 16-token IQ3_S one 570; now 225 and 351.  (32 warps of two rows, measured when this form took 263 and 433: 266 and
// 484, the activation reads then bind.)
//
// The arithmetic is rows_dot's (maya_dots.cuh), value for value - the same integers, the same lane order, the same sums - so
// every token's result is bit-identical to the single-token kernels'.
//
// Plain bulk copies (one destination: this block) of this GPU's own memory.  A row need not start on a 16-byte boundary: the
// aligned window around a segment is copied (expert blobs are 16-byte aligned and a whole number of 16-byte words long, so
// it stays inside).  A blob that is not 16-byte aligned is copied with ordinary loads instead (types made of 2-byte fields; blocks
// of Q4_K, Q5_K and IQ4_XS are read in wider pieces and need the alignment).  Every wait is bounded.  A warp whose
// wait ran out asks for nothing more, and its block leaves - together, at the next barrier - after the copies in flight have had
// the same bounded time to land; the outputs of what was left are missing, and the error word and the group count say so.
#pragma once

#include "maya_internal.cuh"
#include "maya_rows.cuh"
#include "moe_window_args.cuh"

#include <type_traits>

namespace maya {
namespace {

constexpr int kWNC = 8;            // most activation columns of a job
constexpr int kWStages = 2;        // segments in flight a warp
constexpr int kWMaxJobs = kWMaxGroups + 16;      // a job has at least one entry; the shared expert's at least one token
constexpr int kWChunkRows = 64;    // weight rows of a block's step: 16 warps x 4

// ---- the geometry of a type's stream here
template<int T, int SPLIT = 1> struct WGeo : RowGeo<T> {
    static constexpr int split = SPLIT;          // a segment comes in this many stages, rw / SPLIT rows each
    static constexpr int warps = 16, threads = warps * 32, rw = kWChunkRows / warps;      // a warp's rows: 4
    // most columns of a job: four where a call spans two q8_1 blocks (six or eight spill 1.3 KB: 617 against 263 us on the window above)
    static constexpr int nc = Dec<T>::xblk == 2 ? 4 : kWNC;
    using RowGeo<T>::qk;
    using RowGeo<T>::cpb;
    static constexpr int stage = rw / SPLIT * RowGeo<T>::pitch;                                 // a warp's stage
    static constexpr int tab = RowTab<T, false>::bytes;
    // What a warp's four rows cost against nc columns, in units of 30 cycles, fitted to clock stamps of 16-token windows
    // (Q8_0, Q4_K, IQ2_S, IQ3_S, IQ3_XXS, IQ4_XS; the other four types' are estimates without stamps) - those of the codebook types before
    // maya_rows.cuh's decoders, with which IQ2_S and IQ3_S rows cost about a tenth less; not fitted again since: per 32
    // calls of a row the decoding (for Q8_0: waiting for its bytes) and every column's dot, and every column's sums at the end.
    // A share that is off by a tenth is a tenth of the launch: with costs counted in instructions instead the slowest of 148
    // blocks took 27 % longer than the mean.
    static constexpr int dec_cost = T == MAYA_Q8_0 ? (SPLIT > 1 ? 129 : 72) : T == MAYA_Q4_K ? 92 : T == MAYA_Q5_K ? 125 : T == MAYA_Q6_K ? 115
                                    : T == MAYA_IQ4_XS ? 92 : T == MAYA_IQ2_XXS ? 70 : T == MAYA_IQ1_S ? 58 : 77;
    static constexpr int col_cost = Dec<T>::xblk == 2 ? 24 : T == MAYA_IQ2_S || T == MAYA_Q6_K || T == MAYA_IQ3_XXS || T == MAYA_IQ2_XXS ? 11 : 8;
    static constexpr int sum_cost = 21, glu_cost = 40;       // a column's sums; gate/up: a unit's SwiGLU and barrier
    static constexpr int job_cost = 350;                     // a block's change of job: its columns, and code it has not run
    __device__ __forceinline__ static int cost(int nc, int n_in) {
        if (nc > 4) nc = (nc + 1) & ~1;          // dotted as six, as eight
        const int spilled = T == MAYA_IQ2_S && nc == 8 ? 60 : 0;     // (of the former decoder: now only beside a shared expert)
        return (dec_cost + nc * col_cost + spilled) * ((n_in / qk * cpb + 31) / 32) + nc * sum_cost;
    }
};
using WShGeo = WGeo<MAYA_Q8_0, 2>;           // the shared expert's rows: a stage no larger than the 2-bit types'

// what differs between the routed experts' jobs and the shared one's
struct WKind { int n_in, nunit, nseg, bytes, pitch; size_t rb, up, off; };
struct WJob { unsigned long long ptr; int e0, nc, shared, per; };     // per: cost of one unit
struct WShared {
    uint64_t full[16][kWStages];
    WJob job[kWMaxJobs];
    long long cost[kWMaxJobs + 1];   // cost of the jobs before job j
    int njobs;
    int gave_up[16];                 // a wait of this warp ran out
    float s_g[2][kWNC][32], s_u[2][kWNC][32];
    WKind kind[2];
};

// ---- the columns in shared memory.  A column has room for CB q8_1 blocks, a compile-time number, so that the loads of every
//      column, plane and half differ from one another by constants only: the planes of 16-byte pieces of maya_dots.cuh's planar form, then as many planes of scales and of sums.
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
// Block i of a column: its nine words are a thread's loads.
struct ColBlock { uint32_t w[9]; };
__device__ __forceinline__ void col_read(const uint8_t* xq, int i, ColBlock& v) {
    const uint32_t* src = (const uint32_t*) (xq + (size_t) i * kQ81Bytes);
#pragma unroll
    for (int j = 0; j < 9; ++j) v.w[j] = src[j];
}
template<int XB, int CB, bool SUM_F16> __device__ __forceinline__ void col_store(const ColBlock& v, uint8_t* cols, int c, int i) {
    constexpr int P = CB / XB;
    const uint32_t* w = v.w;
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
template<int T, class G, int NC, int RW, int CB>
__device__ __forceinline__ void segment_dot(const uint8_t* s, const uint32_t (&row)[RW], const uint8_t* cols, int blk0, int ncalls, int lane,
                                            const RowLut<T, false>& lut, float (&acc)[RW][NC]) {
    constexpr int XB = Dec<T>::xblk, RP = XB == 2 || NC > 4 || RW < 4 ? 2 : 4;
    using D = SDec<T, NC == 1, false>;
    for (int k = lane; k < ncalls; k += 32) {
        const int kb = k / G::cpb, ci = k - kb * G::cpb;
        // the call's place in the row, and its blocks' in a plane (the same number; written so that it costs fewest registers)
        const int n = Fmt<T>::tab_words > 0 ? blk0 * G::cpb + k : ((blk0 + kb) * (G::qk / 32) + ci * XB) / XB;
#pragma unroll
        for (int r0 = 0; r0 < RW; r0 += RP) {
            if (r0 > 0) asm volatile("" ::: "memory");       // the second two rows' loads stay behind: their registers are the first two's
            D dec[RP];
#pragma unroll
            for (int i = 0; i < RP; ++i) dec[i].load(s, D::at(row[r0 + i] + kb * Fmt<T>::bytes, ci), 0, ci, lut);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const XQ a = col_load<XB, CB>(cols, c, 0, n * 16, n * 4);
                XQ b = a;
                if constexpr (XB == 2) b = col_load<XB, CB>(cols, c, 1, n * 16, n * 4);
#pragma unroll
                for (int i = 0; i < RP; ++i) acc[r0 + i][c] = __fadd_rn(acc[r0 + i][c], dec[i].dot(a, b));
            }
        }
    }
}

// UP: gate/up - a unit of work is a block's: 32 FFN rows (one q8_1 block of h), two of them a warp with their gate and up rows.
// Else down - a unit is a warp's: four rows.  (Blocks' shares in units of 64 rows ended up to one such step apart.)
// SH: with a Q8_0 shared expert.
template<int T, bool SH, bool UP, int CB>
__global__ void __launch_bounds__(WGeo<T>::threads, 1) window_kernel(const WArgs A) {
    using G = WGeo<T>;
    using GS = WShGeo;
    constexpr int RW = G::rw, kWThreads = G::threads, kStage = SH && GS::stage > G::stage ? GS::stage : G::stage;
    constexpr int kRing = G::warps * kWStages * kStage;
    extern __shared__ __align__(128) uint8_t s_raw[];
    __shared__ WShared sh;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t ring = warp * kWStages * kStage;              // the warp's ring in s_raw
    uint32_t* const s_tab = (uint32_t*) (s_raw + kRing);
    uint8_t* const cols = s_raw + kRing + G::tab;

    grid_launch_dependents();
    if (lane == 0) {
        for (int s = 0; s < kWStages; ++s) mbar_init(&sh.full[warp][s], RW);
        sh.gave_up[warp] = 0;
        if (warp < 2) {
            WKind& k = sh.kind[warp];
            const int ff = warp ? A.n_ff_sh : A.n_ff;
            k.n_in = UP ? A.n_embd : ff;
            k.nunit = UP ? ff / 32 : A.n_embd / RW;
            k.nseg = warp ? (k.n_in + GS::vals - 1) / GS::vals : (k.n_in + G::vals - 1) / G::vals;
            k.bytes = warp ? GS::bytes : G::bytes;
            k.pitch = warp ? GS::pitch : G::pitch;
            k.rb = row_bytes(warp ? (int) MAYA_Q8_0 : T, k.n_in);
            k.up = warp ? (size_t) A.n_ff_sh * k.rb : A.up_off;
            k.off = warp ? 0 : A.row_off;
        }
    }
    mbar_fence_init();
    __syncthreads();
    grid_dependency_wait();

    // ---- the jobs, by one warp; the codebook's copies, by the others
    if (warp > 0) {
        RowTab<T, false>::fill(s_tab, tid - 32, kWThreads - 32);
    } else {
        int ng = *A.n_groups;
        const bool lost = ng < 0;                                // a wait of the launch in front ran out: no work
        ng = max(0, min(min(ng, A.cap), kWMaxGroups));
        int base = 0;
        long long run = 0;
        const int nsh = SH && A.sh != nullptr && !lost ? (A.n_tok + A.ncm - 1) / A.ncm : 0;
        const WKind &kr = sh.kind[0], &ks = sh.kind[1];
        for (int g0 = 0; g0 < ng + nsh; g0 += 32) {              // a lane: one group, or one of the shared expert's jobs
            const int g = g0 + lane;
            WJob J{0ull, 0, 0, 0, 0};
            int ne = 0;
            if (g < ng) {
                J.ptr = A.ptr[g];
                J.e0 = A.start[g];
                ne = A.start[g + 1] - J.e0;
            } else if (g < ng + nsh) {
                J.ptr = (unsigned long long) A.sh;
                J.e0 = (g - ng) * A.ncm;
                ne = min(A.ncm, A.n_tok - J.e0);
                J.shared = 1;
            }
            const int nj = J.ptr != 0ull && ne > 0 ? (ne + A.ncm - 1) / A.ncm : 0;
            auto job_of = [&](int j) {
                WJob r = J;
                r.e0 = J.e0 + j * A.ncm;
                r.nc = min(A.ncm, ne - j * A.ncm);
                r.per = (J.shared ? GS::cost(r.nc, ks.n_in) : G::cost(r.nc, kr.n_in)) + (UP ? G::glu_cost : 0);
                return r;
            };
            constexpr int kStart = G::job_cost * (UP ? 1 : G::warps);        // (down: in units of a warp's work)
            long long mine = 0;
            for (int j = 0; j < nj; ++j) mine += kStart + (long long) job_of(j).per * (J.shared ? ks.nunit : kr.nunit);
            int incl = nj;
            long long cost = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, incl, o);
                const long long w = __shfl_up_sync(0xffffffffu, cost, o);
                if (lane >= o) { incl += v; cost += w; }
            }
            int at = base + incl - nj;
            long long before = run + cost - mine;
            for (int j = 0; j < nj; ++j, ++at) {
                const WJob r = job_of(j);
                if (at < kWMaxJobs) { sh.job[at] = r; sh.cost[at] = before; }
                before += kStart + (long long) r.per * (J.shared ? ks.nunit : kr.nunit);
            }
            base += __shfl_sync(0xffffffffu, incl, 31);
            run += __shfl_sync(0xffffffffu, cost, 31);
        }
        if (lane == 0) { sh.njobs = min(base, kWMaxJobs); sh.cost[min(base, kWMaxJobs)] = run; }
    }
    __syncthreads();
    const int njobs = sh.njobs;
    // unit c of job j starts at cost[j] + job_cost + c * per; this block takes those that start in its share of the whole
    const long long total = sh.cost[njobs];
    auto first_at = [&](long long at, int& j, int& c) {
        j = 0;
        while (j < njobs && sh.cost[j + 1] <= at) ++j;
        c = 0;
        if (j < njobs) {
            const int per = sh.job[j].per;
            const long long in = at - sh.cost[j] - G::job_cost * (UP ? 1 : G::warps);
            c = in > 0 ? (int) ((in + per - 1) / per) : 0;
            if (c >= sh.kind[SH ? sh.job[j].shared : 0].nunit) { ++j; c = 0; }
        }
    };
    int job, unit0, job1, unit1;
    first_at((long long) blockIdx.x * total / gridDim.x, job, unit0);
    first_at((long long) (blockIdx.x + 1) * total / gridDim.x, job1, unit1);
    if (job > job1 || (job == job1 && unit0 >= unit1)) return;
    constexpr int kStep = UP ? 1 : G::warps;                     // a warp's next unit
    const int off = UP ? 0 : warp;
    auto limit_of = [&](int j) { return j == job1 ? unit1 : sh.kind[SH ? sh.job[j].shared : 0].nunit; };     // j <= job1, j < njobs

    // row r of this warp in a unit: gate rows, then the same up rows; or down rows
    auto row_ptr = [&](unsigned long long blob, const WKind& k, int unit, int r) -> const uint8_t* {
        constexpr int H = RW / 2;
        const uint8_t* base = (const uint8_t*) blob + k.off;
        if constexpr (UP) return base + (r / H) * k.up + (size_t) (unit * 32 + H * warp + r % H) * k.rb;
        else return base + (size_t) (RW * unit + r) * k.rb;
    };
    // ---- the stream: what the warp asks for next - job, unit, segment, and which of the segment's stages
    int pj = job, pc = unit0 + off, ps = 0, pq = 0;
    uint32_t asked = 0;                                          // stages asked for, modulo 2 kWStages: the next one's place is asked % kWStages
    static_assert(kWStages == 2, "a stage is a bit of `asked`");
    auto ask = [&] {
        while (pj < njobs && pj <= job1 && pc >= limit_of(pj)) { ++pj; pc = off; }
        if (pj >= njobs || pj > job1) return;
        const WJob& J = sh.job[pj];
        const WKind& k = sh.kind[SH ? J.shared : 0];
        __syncwarp();                                            // every lane has read the stage's last bytes
        // Beside a shared expert which of two constants each: looked up, and with a division for the rows of a stage, they cost two-token windows
        // 2 to 6 % (6144 x 2048 IQ2_S with 2048 shared 130.0 / 124.4 us).  Without one they are looked up, each where it is used: as constants
        // 4 % slower on Q8_0, looked up ahead of the branches below 1 % on IQ2_S (six tokens of 6400 x 3072 246.7 / 243.5 us): a register each.
        const bool js = SH && J.shared;
        auto seg_bytes = [&]() -> int { if constexpr (SH) return js ? GS::bytes : G::bytes; else return k.bytes; };
        auto pitch = [&]() -> int { if constexpr (SH) return js ? GS::pitch : G::pitch; else return k.pitch; };
        const int split = js ? GS::split : 1;
        const uint32_t at = (uint32_t) (ps * seg_bytes()), len = min((uint32_t) seg_bytes(), (uint32_t) k.rb - at);
        const uint32_t pstage = asked & 1u, dst = ring + pstage * kStage;
        const int rows = js ? RW / GS::split : RW, first = js ? pq * rows : 0;      // the stage's rows
        if ((J.ptr & 15ull) == 0 && (!A.plain || js)) {
            if (lane < rows) {
                const uint8_t* src = row_ptr(J.ptr, k, pc, first + lane) + at;
                const uint32_t off = (uint32_t) (uintptr_t) src & 15u, bytes = (off + len + 15u) & ~15u;
                fence_proxy_async();
                mbar_expect_tx(&sh.full[warp][pstage], bytes);
                bulk_load(s_raw + dst + lane * pitch(), src - off, bytes, &sh.full[warp][pstage]);
            } else if (SH && lane < RW) {
                mbar_arrive_one(&sh.full[warp][pstage]);
            }
        } else {                                                 // ordinary loads, two bytes at a time
            for (int r = 0; r < rows; ++r) {
                const uint8_t* src = row_ptr(J.ptr, k, pc, first + r) + at;
                const uint32_t off = (uint32_t) (uintptr_t) src & 15u;
                for (uint32_t i = 2 * lane; i < len; i += 64) *(uint16_t*) (s_raw + dst + r * pitch() + off + i) = *(const uint16_t*) (src + i);
            }
            __syncwarp();
            if (lane < RW) mbar_arrive_one(&sh.full[warp][pstage]);
        }
        asked = (asked + 1) & 3u;
        if (SH && ++pq < split) return;
        pq = 0;
        if (++ps == k.nseg) {
            ps = 0;
            pc += kStep;
        }
    };
    for (int s = 0; s < kWStages; ++s) ask();

    const RowLut<T, false> lut(s_tab, lane);
    const RowLut<MAYA_Q8_0, false> lut_sh(s_tab, lane);          // (no codebook)
    int stage = 0, buf = 0;
    uint32_t phase = 0;
    auto gave_up = [&](int w) { return *(volatile int*) &sh.gave_up[w]; };
    for (int first_unit = unit0; job <= job1 && job < njobs; ++job, first_unit = 0) {
        const int limit = limit_of(job);
        if (first_unit >= limit) continue;
        const WJob& J = sh.job[job];
        const bool shd = SH && J.shared;
        const WKind& K = sh.kind[shd ? 1 : 0];
        const int nc = J.nc, n_in = K.n_in;
        auto slot_of = [&](int c) { return shd ? J.e0 + c : A.ent_slot[J.e0 + c]; };     // shared: the token
        if (__syncthreads_or(gave_up(warp))) goto leave;         // everyone is done with the old columns; or has to leave
        {
            const int nblk = n_in / 32, items = nc * nblk;
            for (int i0 = tid; i0 < items; i0 += 2 * kWThreads) {                // two q8_1 blocks a thread in flight
                ColBlock v[2];
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int i = i0 + u * kWThreads;
                    if (i >= items) continue;
                    const int c = i / nblk, slot = slot_of(c);
                    const uint8_t* src;
                    if constexpr (UP) src = A.xq + (size_t) (shd ? slot : slot >> 3) * A.xq_stride;
                    else src = shd ? A.sh_hq + (size_t) slot * nblk * kQ81Bytes : A.xq + (size_t) slot * A.xq_stride;
                    col_read(src, i - c * nblk, v[u]);
                }
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int i = i0 + u * kWThreads;
                    if (i >= items) continue;
                    const int c = i / nblk;
                    if (SH && shd) col_store<1, CB, false>(v[u], cols, c, i - c * nblk);
                    else col_store<Dec<T>::xblk, CB, T == MAYA_IQ1_S>(v[u], cols, c, i - c * nblk);
                }
            }
        }
        __syncthreads();
        for (int unit = first_unit + off; unit < limit; unit += kStep) {
        // where the warp's rows start in their 16-byte windows
        const uint32_t p0 = (uint32_t) (uintptr_t) row_ptr(J.ptr, K, unit, 0), rb16 = (uint32_t) K.rb & 15u, up16b = (uint32_t) K.up & 15u;
        const uint32_t start[RW] = {p0, p0 + rb16, UP ? p0 + up16b : p0 + 2 * rb16, UP ? p0 + up16b + rb16 : p0 + 3 * rb16};
        static_assert(RW == 4, "four rows a warp");
        // a sum's row is its place in the reduction below: bits 4 and 3 of the lane
        const int my_row = 2 * (lane >> 4) + ((lane >> 3) & 1);
        auto unit_dot = [&](auto type_c, auto geo, auto nc_c) {
            constexpr int TY = decltype(type_c)::value, NC = decltype(nc_c)::value;
            using GT = decltype(geo);
            float acc[RW][NC];
#pragma unroll
            for (int r = 0; r < RW; ++r)
#pragma unroll
                for (int c = 0; c < NC; ++c) acc[r][c] = 0.0f;
            constexpr int RS = RW / GT::split;                   // rows of a stage
            for (int sg = 0; sg < K.nseg; ++sg) {
                const uint32_t so = (uint32_t) (sg * GT::bytes);            // (a row's segments can start anywhere, too)
                const int blk0 = sg * GT::blocks, ncalls = min(GT::blocks, n_in / GT::qk - blk0) * GT::cpb;
#pragma unroll
                for (int p = 0; p < GT::split; ++p) {
                    if (!__all_sync(0xffffffffu, mbar_wait(&sh.full[warp][stage], phase, A.polls))) {
                        *(volatile int*) &sh.gave_up[warp] = 1;
                        return;
                    }
                    uint32_t row[RS];
#pragma unroll
                    for (int r = 0; r < RS; ++r) row[r] = ring + stage * kStage + r * GT::pitch + ((start[p * RS + r] + so) & 15u);
                    if constexpr (TY == T) segment_dot<TY, GT, NC, RS, CB>(s_raw, row, cols, blk0, ncalls, lane, lut, *(float(*)[RS][NC]) &acc[p * RS]);
                    else segment_dot<TY, GT, NC, RS, CB>(s_raw, row, cols, blk0, ncalls, lane, lut_sh, *(float(*)[RS][NC]) &acc[p * RS]);
                    stage = stage + 1 == kWStages ? 0 : stage + 1;
                    if (stage == 0) phase ^= 1u;
                    ask();
                }
            }
            // warp_sum's tree (lanes 16 apart first, then 8, 4, 2, 1) on four rows at once: after the first exchange a lane keeps two
            // of them, after the second one - six shuffles a column instead of twenty, the same additions
            const bool up16 = (lane & 16) != 0, up8 = (lane & 8) != 0;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                float a = up16 ? acc[2][c] : acc[0][c], b = up16 ? acc[3][c] : acc[1][c];
                a += __shfl_xor_sync(0xffffffffu, up16 ? acc[0][c] : acc[2][c], 16);
                b += __shfl_xor_sync(0xffffffffu, up16 ? acc[1][c] : acc[3][c], 16);
                float v = up8 ? b : a;
                v += __shfl_xor_sync(0xffffffffu, up8 ? a : b, 8);
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if ((lane & 7) == 0 && c < nc) {
                    if constexpr (UP) {
                        (my_row < 2 ? sh.s_g : sh.s_u)[buf][c][2 * warp + (my_row & 1)] = v;
                    } else {
                        (shd ? A.sh_out : A.part)[(size_t) slot_of(c) * A.n_embd + RW * unit + my_row] = v;
                    }
                }
            }
        };
        auto unit_any = [&](auto type_c, auto geo) {
            switch (nc) {
                case 1: unit_dot(type_c, geo, std::integral_constant<int, 1>{}); break;
                case 2: unit_dot(type_c, geo, std::integral_constant<int, 2>{}); break;
                case 3: unit_dot(type_c, geo, std::integral_constant<int, 3>{}); break;
                case 4: unit_dot(type_c, geo, std::integral_constant<int, 4>{}); break;
                default:
                    if constexpr (G::nc > 4) {
                        if (nc <= 6) unit_dot(type_c, geo, std::integral_constant<int, 6>{});
                        else unit_dot(type_c, geo, std::integral_constant<int, 8>{});
                    }
            }
        };
        if constexpr (SH) {
            if (shd) unit_any(std::integral_constant<int, MAYA_Q8_0>{}, GS{});
            else unit_any(std::integral_constant<int, T>{}, G{});
        } else {
            unit_any(std::integral_constant<int, T>{}, G{});
        }
        if constexpr (UP) {
            if (__syncthreads_or(gave_up(warp))) goto leave;     // two buffers: one barrier a unit
            if (warp < nc)
                q8_1_store_warp(swiglu(sh.s_g[buf][warp][lane], sh.s_u[buf][warp][lane], A.limit),
                                (shd ? A.sh_hq : A.hq) + ((size_t) slot_of(warp) * K.nunit + unit) * kQ81Bytes, lane);
            buf ^= 1;
        } else if (gave_up(warp)) {
            break;                                               // (the warps meet again at the change of job)
        }
        }
    }
    if (!gave_up(warp)) return;
leave:
    // let what this warp has in flight land - the stages asked for and not yet read - before the block's shared memory goes away
    for (uint32_t i = 2 * phase + stage; i != asked; i = (i + 1) & 3u) mbar_wait(&sh.full[warp][i & 1u], i >> 1);     // modulo 4, as `asked`
    if (gave_up(warp) && lane == 0) {
        if (A.error != nullptr) atomicExch(A.error, 1u);
        atomicExch(A.n_groups, -1);
    }
}

template<int T, bool SH, bool UP, int CB>
int launch_window_cb(WArgs A, cudaStream_t s) {
    using G = WGeo<T>;
    constexpr int kStage = SH && WShGeo::stage > G::stage ? WShGeo::stage : G::stage, kRing = G::warps * kWStages * kStage;
    // columns of a job: what fits beside the ring and the codebook, eight at most (a job's rows are decoded once for them all)
    constexpr long room = 232448l - (long) sizeof(WShared) - 256 - kRing - G::tab;
    static_assert(room >= kColBytes<CB>, "a column has to fit");
    A.ncm = (int) (room / kColBytes<CB>);
    if (A.ncm > G::nc) A.ncm = G::nc;
    if (A.ncm == 5 || A.ncm == 7) --A.ncm;            // five columns are dotted as six, seven as eight: the room has to be there
    A.plain = ((A.row_off | A.up_off | (size_t) (UP ? A.n_ff : A.n_embd) * row_bytes(T, UP ? A.n_embd : A.n_ff)) & 15) != 0;
    const size_t smem = (size_t) kRing + G::tab + (size_t) A.ncm * kColBytes<CB>;
    static SmemLimit smem_limit;                           // (smem is the same in every call of an instantiation)
    if (!smem_limit.raise((const void*) window_kernel<T, SH, UP, CB>, smem)) return note_launch("window smem attribute");
    const int sms = sm_count();
    if (sms <= 0) return refuse(MAYA_ERR_DEVICE);
    launch_dependent(window_kernel<T, SH, UP, CB>, dim3((unsigned) sms), dim3(G::threads), smem, s, A);
    return note_launch(UP ? "window_gate_up" : "window_down");
}

// The smallest column capacity that holds the row.
template<int T, bool SH, bool UP> int launch_window(const WArgs& A, cudaStream_t s) {
    int n_in = UP ? A.n_embd : A.n_ff;
    if (!UP && SH && A.n_ff_sh > n_in) n_in = A.n_ff_sh;
    if (n_in <= 128 * 32) return launch_window_cb<T, SH, UP, 128>(A, s);
    if (n_in <= 256 * 32) return launch_window_cb<T, SH, UP, 256>(A, s);
    return kWindowTooWide;
}

}  // namespace

// Instantiated in moe_window_{up,down}[_sh]_{k,i}.cu - GROUP 0: Q8_0, the K-quants and IQ4_XS, 1: the codebook types - a
// translation unit each, so that they compile side by side.
template<bool SH, bool UP, int GROUP> int launch_window_group(int type, const WArgs& A, cudaStream_t s) {
#define MAYA_WIN(TT) case TT: return launch_window<TT, SH, UP>(A, s);
    if constexpr (GROUP == 0) {
        switch (type) {
            MAYA_WIN(MAYA_Q8_0) MAYA_WIN(MAYA_Q4_K) MAYA_WIN(MAYA_Q5_K) MAYA_WIN(MAYA_Q6_K) MAYA_WIN(MAYA_IQ4_XS)
        }
    } else {
        switch (type) {
            MAYA_WIN(MAYA_IQ2_S) MAYA_WIN(MAYA_IQ3_S) MAYA_WIN(MAYA_IQ3_XXS) MAYA_WIN(MAYA_IQ2_XXS) MAYA_WIN(MAYA_IQ1_S)
        }
    }
#undef MAYA_WIN
    return refuse(MAYA_ERR_TYPE);
}

}  // namespace maya
