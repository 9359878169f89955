// mmq_tc.cu - the prompt path's grouped-by-expert GEMM over quantized expert matrices on the 5th-generation tensor
// cores: for every expert e, the activation rows [bounds[e], bounds[e+1]) times its [w_rows, w_cols] quantized matrix.
//
// Replaces mmq::quantize / mmq::Context::run / run_glu (include/strata/prefill/moe_mmq.hpp:34-81, src/prefill/
// moe_mmq.cu:114-228), which wrap llama.cpp's int8 `mma.sync` MMQ kernels (not part of the reference tree).  The
// reference rounds activations to q8_1 and multiplies integers with per-32 scales; an integer tcgen05 contraction
// would have to leave tensor memory every 32 values of K to apply those scales, so here both operands are f16:
// activations are stored once as d * q of their q8_1 image (the reference's rounding of x, kept so that results stay
// within its tolerance), weights are expanded from their GGUF blocks in shared memory, and `tcgen05.mma.kind::f16`
// accumulates in f32 in tensor memory.
//
// One block = a slab of 256 weight rows (128 gate + 128 up rows for the fused SwiGLU form) x up to 160 activation
// rows of one expert: two M = 128 accumulators of N = rows (rounded up to 16) columns in tensor memory.  The expanded
// weights are the A operand and live in tensor memory too (lane = weight row, the layout a thread-per-row expansion
// produces by itself), so shared memory carries only raw blocks and activations: an SM's 128 bytes/clock of shared
// memory cannot feed two f16 operands of M = N = 128 products at the tensor core's rate.  Warp roles:
//   warp 16     TMA loads of raw weight blocks, 64 rows x 256 K-values a "unit", into a ring of units;
//   warp 18     TMA loads of activation tiles, 128 (+ 32) or 32 rows x 64 K-values, in the 128-byte swizzle layout
//               the tensor core reads at full rate;
//   warps 0..15 two teams of 8 warps that take alternate K steps (i-quants: alternate blocks of 256 K-values); in a team one thread
//               per weight row expands 32 K-values of the row per step (packed half2 arithmetic:
//               Q8_0 w = q * d; Q4_K w = fma(q, d * sc, -(dmin * m))) and tcgen05.st-s them into the row's lane;
//   warps 17,19 one accumulator each: two tcgen05.mma per step (2 K = 16 halves, A from tensor memory, B from shared
//               memory), one commit per two steps -> the steps' buffers are free (the warp cannot issue products as fast as
//               the tensor core retires them unless their operands stay in uniform registers: see there);
//   warps 0..15 afterwards: the epilogue - tcgen05.ld (lane = weight row, column = activation row), SwiGLU, optional
//               q8_1 rounding of h for the next product; f32 results leave through shared memory, one bulk copy per activation row.
// Which expert and which 160-row group of it a block handles is found on the device from `bounds`; no count travels
// to the host.
//
// What bounds it: for groups of many rows the board's power limit and the expansion, for groups of few rows the expansion alone,
// 4 instructions a weight.  That holds only while no waiting role is in the way: clock stamps of 64 tokens of IQ3_S showed finished
// weights waiting 3000 cycles - the activation loader, one lane in a divergent branch, took 540 cycles a tile (every operand of a copy
// crossed into a uniform register), longer than the expansion.  Now both loaders walk their loops as whole warps and an elected lane
// copies, the role's number is warp-uniform to the compiler (an issuing warp's products 137 -> 47 cycles), the stages fill tensor
// memory, and a stage is asked for before the expansion that goes there.  Then the
// expansions themselves: Q4_K's header two sub-blocks at a time, IQ2_S's codebook of byte selectors.  us a layer, without and with all of
// it, in turn on one board: 64 tokens of IQ3_S 437 / 367, 777 of IQ2_S with a shared expert 1309 / 1161, 4096 of Q8_0 / Q4_K 3580 / 3284,
// 90 of Q8_0 with a shared expert 134 / 110, 363 of IQ3_S 2040 / 1667.
//
// Every mbarrier wait is bounded: a wait that runs out sets the error word, the roles stop, copies in
// flight are waited for (bounded), tensor memory is freed and the block returns.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_fp16.h>

#include <cstdio>
#include <cstring>
#include <type_traits>
#include <utility>

#include "maya_internal.cuh"
#include "maya_rows.cuh"
#include "maya_tcgen05.cuh"

namespace maya {
namespace {

constexpr int TM = 256;                 // weight rows of a block
constexpr int TN = 160;                 // most activation rows of a block
constexpr int BK = 32;                  // K values of one step
constexpr int kMaxSt = 7;               // most stages of expanded weights (the A operand, in tensor memory), 64 K-values each
constexpr int kMaxBSt = 8;              // most activation tiles (64 K-values) in flight
constexpr int kUnitRows = 64;           // weight rows of one raw unit
constexpr int kDqWarps = 16;            // two teams of 8
constexpr int kMmqThreads = (kDqWarps + 4) * 32;   // + raw-unit loader, issuer of accumulator 0, activation loader, issuer of accumulator 1
constexpr int kBBox = 128 * 64 * 2;     // 16 KB: 128 activation rows x 64 K-values, 128-byte swizzle
constexpr int kBStage = kBBox + 32 * 64 * 2;   // + the 32-row box of a block with more than 128 rows: 20 KB
constexpr int kMaxUnits = 16;
constexpr int kDone = 16;               // ring of "pair of K steps consumed" barriers (one tcgen05.commit per pair: a commit
                                        // costs the tensor pipe about as much as a product)
// Raw weight units, one tiled TMA box of 64 rows each.  Q8_0 / Q4_K: a row's 256 K-values are 272 / 144 bytes, a
// multiple of 16.  IQ2_S / IQ3_S blocks are 82 / 110 bytes: the box is the 16-byte aligned window around the rows' block
// (96 / 128 bytes used) taken 112 / 144 bytes wide, so that rows are an odd number of 16-byte words apart in shared
// memory (a warp's 16-byte reads of 32 rows fall in different banks).
template<int T> constexpr bool kIq = T == MAYA_IQ2_S || T == MAYA_IQ3_S;
template<int T> constexpr int kBlkBytes = T == MAYA_IQ2_S ? 82 : T == MAYA_IQ3_S ? 110 : 0;
template<int T> constexpr int kWin = T == MAYA_IQ2_S ? 96 : 128;
template<int T> constexpr int kRawRow = T == MAYA_Q4_K ? 144 : T == MAYA_Q8_0 ? 272 : T == MAYA_IQ2_S ? 112 : 144;
template<int T> constexpr int kUnitBytes = kUnitRows * kRawRow<T>;
// Raw units in flight: whole rounds of what the expanding warps take - 4 a block of K, i-quants 8, two blocks - so that a place of the ring is
// always the same warps' and each of them waits for every one of its phases.  A wait names a phase by its parity alone: a warp that came
// to a place other warps had filled the round before (rings of 9, 10 and 11 units) and was a block ahead of them, as seven stages let it be, took a unit
// that had not even been asked for.  A load that came 2.6 us late was enough.
template<int T> constexpr int kUnits = T == MAYA_Q4_K ? 12 : 8;
template<int T> constexpr int kBRing = (T == MAYA_Q4_K ? 5 : 4) * kBStage;    // activation tiles (64 K-values) in flight
// i-quants: the codebook, 64 KB of it, in kCopies copies that lie side by side in every entry - lane l reads copy l % kCopies - so that a warp's
// random entries spread over the banks.  Both have 8-byte entries: IQ3_S's 512 are four values as f16, sixteen copies, free of conflicts; IQ2_S's 1024 are
// byte selectors of eight values, eight copies (see iq_lookup).  (As f16, 16 bytes in four copies, IQ2_S's look-ups held the shared-memory pipe for
// eight wavefronts each, nine tenths of the time.  As bytes a codebook takes one byte permute more for every two weights, and the expansion is bound by
// instructions: 64 tokens of IQ3_S 553 -> 475 us.)
template<int T> constexpr int kCopies = T == MAYA_IQ2_S ? 8 : T == MAYA_IQ3_S ? 16 : 0;
template<int T> constexpr int kTabBytes = T == MAYA_IQ2_S ? 1024 * 8 * kCopies<T> : T == MAYA_IQ3_S ? 512 * 8 * kCopies<T> : 0;
// the codebook lies behind the rings - and behind a finished tile, which takes their place: 160 rows of 256 f32 values
template<int T> constexpr int kTabOff = kBRing<T> + kUnits<T> * kUnitBytes<T> > TN * TM * 4 ? kBRing<T> + kUnits<T> * kUnitBytes<T> : TN * TM * 4;
template<int T> constexpr size_t kSmemBytes = (size_t) kTabOff<T> + kTabBytes<T>;
template<int T> constexpr bool kUnitsFit = kUnits<T> <= kMaxUnits && kUnits<T> % (kIq<T> ? 8 : 4) == 0 && kSmemBytes<T> <= 227 * 1024 - 1024;
static_assert(kUnitsFit<MAYA_Q4_K> && kUnitsFit<MAYA_Q8_0> && kUnitsFit<MAYA_IQ2_S> && kUnitsFit<MAYA_IQ3_S>, "the ring of raw units");

// The activation image: a row is its w_cols f16 values d * q, then one f16 per 32 values - the group's SUM CORRECTION
// xa = f16(sum of the unquantized values) - sum of the row's stored d * q values - padded with zeros to a multiple of 64.  llama.cpp's
// MMQ keeps that unquantized sum beside the block (the "ds4" q8_1 layout) and a type with a constant term per group
// (Q4_K: -dmin * m) multiplies the term by it, not by the sum of the rounded values; here the same result comes from
// extra K steps inside a Q4_K product: A = -dmin * m of a row's groups, B = xa.  Other types do not read the tail.
// Optional clock stamps of a tile's phases (built only with -DMAYA_MMQ_STAMPS, see build.py --stamps and
// mmq_tile_phases.py): 16 slots per tile for the first 4096 tiles of each of the four (type class, fused) kernels.
#ifdef MAYA_MMQ_STAMPS
__device__ long long g_stamps[4 * 4096 * 16];
#endif
__host__ __device__ constexpr int64_t xq_tail(int64_t cols) { return ((cols / 32) + 63) & ~(int64_t) 63; }
__host__ __device__ constexpr int64_t xq_ld(int64_t cols) { return cols + xq_tail(cols); }

struct MmqArgs {
    int w_rows, w_cols;          // rows of one output (n_ff for the fused form: gate rows, then up rows), K
    int n;                       // matrices of this product
    const int* expert_map;       // optional: matrix i owns the rows of bounds entry expert_map[i]
    const int* bounds;
    const int* ids;              // optional dst row of a sorted row
    float* dst;                  // optional for the fused form
    int64_t ld_dst;
    __half* xq_out;              // fused form, optional: q8_1-rounded h as f16, [sorted row][w_rows]
    float limit;
    unsigned* error;             // optional sticky error word
    // In a chain of products (maya_mmq_run_chain), else NULL.  claim: [0] the next tile to be taken, [1] blocks that found none
    // left.  ready: per group of rows [0] how often one of its h rows has left a gate/up tile, [1] down tiles that have waited for
    // it; the down product of the group starts when [0] reaches its rows times ready_slabs.  All zero between chains.
    unsigned* claim;
    unsigned* ready;
    int ready_slabs;             // down: gate/up tiles of a group; gate/up: unused
    int alone;                   // not behind another product of its chain: everything in front has to be done first
};

__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *(uint32_t*) &h; }
__device__ __forceinline__ __half2 bits_h2(uint32_t u) { return *(__half2*) &u; }
// bytes (lo, hi) of x -> the half2 (1024 + lo, 1024 + hi): 0x64 is the high byte of 1024.0 in f16
__device__ __forceinline__ __half2 bytes01_plus1024(uint32_t x) { return bits_h2(__byte_perm(x, 0x64646464u, 0x4140)); }
__device__ __forceinline__ __half2 bytes23_plus1024(uint32_t x) { return bits_h2(__byte_perm(x, 0x64646464u, 0x4342)); }

// The q8_1 rounding of maya_mmq_quantize for a thread that holds 8 consecutive values of a 32-value group (the group's
// four threads are four consecutive lanes; every lane of the warp must call): llama.cpp's quantize_mmq_q8_1 as the
// reference's host model states it - d_inv = 127 / amax, q = round(v * d_inv) clamped to +-127, d = min(1 / d_inv, 65504)
// kept as f16, stored f16(d) * q.  o = the 8 stored values; the return value is the group's sum correction
// f16(S) - sum of the stored values, with S added in quantize_mmq_q8_1's order: four consecutive values left to right
// (this thread holds partial sums 2j and 2j + 1 of the group's eight), then the tree at distances 4, 2, 1.
__device__ __forceinline__ __half q8_1_round8(const float (&v)[8], uint32_t (&o)[4]) {
    float amax = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
    amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 2));
    const float d_inv = __fdiv_rn(127.0f, amax);
    const float dh = amax == 0.0f ? 0.0f : __half2float(__float2half_rn(fminf(__fdiv_rn(1.0f, d_inv), 65504.0f)));
    float bsum = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float q0 = 0.0f, q1 = 0.0f;
        if (amax != 0.0f) {
            q0 = fmaxf(-127.0f, fminf(127.0f, roundf(__fmul_rn(v[2 * i], d_inv))));
            q1 = fmaxf(-127.0f, fminf(127.0f, roundf(__fmul_rn(v[2 * i + 1], d_inv))));
        }
        const __half2 r = __floats2half2_rn(dh * q0, dh * q1);
        o[i] = h2_bits(r);
        bsum += __low2float(r) + __high2float(r);     // the stored values: multiples of one power of two, 24 bits in all - exact
    }
    float s0 = __fadd_rn(__fadd_rn(__fadd_rn(v[0], v[1]), v[2]), v[3]), s1 = __fadd_rn(__fadd_rn(__fadd_rn(v[4], v[5]), v[6]), v[7]);
    s0 = __fadd_rn(s0, __shfl_xor_sync(0xFFFFFFFFu, s0, 2));
    s1 = __fadd_rn(s1, __shfl_xor_sync(0xFFFFFFFFu, s1, 2));
    s0 = __fadd_rn(s0, __shfl_xor_sync(0xFFFFFFFFu, s0, 1));
    s1 = __fadd_rn(s1, __shfl_xor_sync(0xFFFFFFFFu, s1, 1));
    bsum += __shfl_xor_sync(0xFFFFFFFFu, bsum, 1);
    bsum += __shfl_xor_sync(0xFFFFFFFFu, bsum, 2);
    return __float2half_rn(__half2float(__float2half_rn(__fadd_rn(s0, s1))) - bsum);
}

// ---- Q4_K: of a 144-byte block's 16-byte header, d * sc and -(dmin * m) of sub-blocks 2 (2 i + t) and 2 (2 i + t) + 1, i = 0 or 1, as a half2
// each.  y, z, w: the header's scale words, shifted so that their low 16 bits are columns 2 t and 2 t + 1.  (Two sub-blocks at a time and only those a
// team expands: all eight one by one, in an array the team indexed, took four times the instructions and local memory.)
__device__ __forceinline__ __half2 q4k_pair(uint32_t two_bytes, __half2 factor) {
    return __hmul2(factor, __hsub2(bytes01_plus1024(two_bytes), __float2half2_rn(1024.0f)));      // the difference is exact
}
__device__ __forceinline__ __half2 q4k_scale(int i, uint32_t y, uint32_t w, __half2 d2) {
    return q4k_pair(i == 0 ? y & 0x3F3Fu : (w & 0x0F0Fu) | ((y >> 2) & 0x3030u), d2);
}
__device__ __forceinline__ __half2 q4k_min(int i, uint32_t z, uint32_t w, __half2 m2) {
    return __hneg2(q4k_pair(i == 0 ? z & 0x3F3Fu : ((w >> 4) & 0x0F0Fu) | ((z >> 2) & 0x3030u), m2));
}
// 32 weights of sub-block (2p + hi) from the 32 quant bytes of pair p
__device__ __forceinline__ void q4k_stage(const uint4 qa, const uint4 qb, int hi, __half2 dl, __half2 nml, uint32_t* r) {
    const uint32_t w[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
    const __half2 k1024 = __float2half2_rn(1024.0f);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t x = (hi ? (w[i] >> 4) : w[i]) & 0x0F0F0F0Fu;
        r[2 * i] = h2_bits(__hfma2(__hsub2(bytes01_plus1024(x), k1024), dl, nml));
        r[2 * i + 1] = h2_bits(__hfma2(__hsub2(bytes23_plus1024(x), k1024), dl, nml));
    }
}
// ---- Q8_0: block J (34 bytes) of a 272-byte raw row, read as three aligned 16-byte words
template<int J>
__device__ __forceinline__ void q80_stage(const uint8_t* rrow, uint32_t* r) {
    constexpr int kBase = (34 * J) / 16 * 16, kOff = 34 * J - kBase;     // kOff = 0, 2, ..., 14
    const uint4 a = *(const uint4*) (rrow + kBase), b = *(const uint4*) (rrow + kBase + 16), c = *(const uint4*) (rrow + kBase + 32);
    const uint32_t w[12] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, c.y, c.z, c.w};
    const uint32_t dw = w[kOff / 4];
    const __half dh = __ushort_as_half((unsigned short) ((kOff % 4) ? (dw >> 16) : (dw & 0xFFFF)));
    const __half2 d2 = __half2half2(dh), k1152 = __float2half2_rn(1152.0f);
    constexpr int kQ = kOff + 2;
    if constexpr (kQ % 4 != 0) {
        // the quants start two bytes into a word: values (4i, 4i + 1) are bytes 2, 3 of word i and values (4i + 2, 4i + 3)
        // bytes 0, 1 of word i + 1 - picked by the same byte permutes that widen them, no aligning permute
        uint32_t u[9];
#pragma unroll
        for (int i = 0; i < 9; ++i) u[i] = w[kQ / 4 + i] ^ 0x80808080u;     // q + 128 as unsigned bytes
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            r[2 * i] = h2_bits(__hmul2(__hsub2(bytes23_plus1024(u[i]), k1152), d2));
            r[2 * i + 1] = h2_bits(__hmul2(__hsub2(bytes01_plus1024(u[i + 1]), k1152), d2));
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t x = w[kQ / 4 + i] ^ 0x80808080u;
            r[2 * i] = h2_bits(__hmul2(__hsub2(bytes01_plus1024(x), k1152), d2));
            r[2 * i + 1] = h2_bits(__hmul2(__hsub2(bytes23_plus1024(x), k1152), d2));
        }
    }
}

// ---- i-quants.  `w` = the row's window as 32-bit words; the block starts OFF bytes into it (OFF is even and the same
// for all rows of a K block).  Only the FIELDS are taken apart by code that knows OFF (eight small variants, every position a
// compile-time constant); the expansion works on the taken-out fields, so there is one copy of it.  Expanding straight from
// the window in eight variants made the loop too long for the instruction cache: half of all warp cycles waited for a fetch.
template<int BYTE> __device__ __forceinline__ uint32_t win_u32(const uint32_t* w) {
    constexpr int i = BYTE / 4, r = BYTE % 4;
    static_assert(r % 2 == 0, "fields start on even bytes");
    if constexpr (r == 0) return w[i];
    else return __byte_perm(w[i], w[i + 1], 0x5432);
}
// the words at BYTE, BYTE + 4, ...
template<int BYTE, int... I> __device__ __forceinline__ void win_words(const uint32_t* w, uint32_t* dst, std::integer_sequence<int, I...>) {
    ((dst[I] = win_u32<BYTE + 4 * I>(w)), ...);
}
// A block's fields.  q: codebook index bytes (a word a sub-block of 32 values for IQ2_S, two for IQ3_S); sg: a word of sign bits
// a sub-block; byte j of qh: sub-block j's high index bits; sc: scales, IQ2_S byte j = sub-block j's two, IQ3_S nibble j = sub-block j's.
template<int T> struct IqFields {
    uint32_t q[T == MAYA_IQ2_S ? 8 : 16], sg[8], qh[2], sc[T == MAYA_IQ2_S ? 2 : 1], d2;     // d2: the block's scale, twice
};
template<int T, int OFF> __device__ __forceinline__ void iq_fields(const uint32_t* w, IqFields<T>& F) {
    F.d2 = __byte_perm(w[OFF / 4], 0, OFF % 4 == 0 ? 0x1010 : 0x3232);
    win_words<OFF + 2>(w, F.q, std::make_integer_sequence<int, T == MAYA_IQ2_S ? 8 : 16>{});
    win_words<OFF + (T == MAYA_IQ2_S ? 34 : 74)>(w, F.sg, std::make_integer_sequence<int, 8>{});
    win_words<OFF + 66>(w, F.qh, std::make_integer_sequence<int, 2>{});
    win_words<OFF + (T == MAYA_IQ2_S ? 74 : 106)>(w, F.sc, std::make_integer_sequence<int, T == MAYA_IQ2_S ? 2 : 1>{});
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
    uint2 v;
    asm("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
// Sub-block J's look-ups -> o[16], 8 bytes an entry.  tab: shared-memory address of this lane's copy of the codebook; f: the entries' distance
// twice, as dp2a takes it (an index's 16 bits times the distance plus the base are one instruction).
// IQ2_S: the magnitudes are 8, 25 and 43, so a sub-block's half has three weights but for the signs, and an entry is four byte selectors of 16 bits,
// two to a word, each picking two of them: o[2 l], o[2 l + 1] the words of entry l.
template<int J> __device__ __forceinline__ void iq_lookup(const IqFields<MAYA_IQ2_S>& F, uint32_t tab, uint32_t f, uint32_t* o) {
    const uint32_t qh = byte_of(F.qh[J / 4], J % 4);
    // byte l of hw = bits 2l, 2l + 1 of qh: an entry's high index bits
    const uint32_t hw = ((qh & 0x33u) * 0x1001u + (qh & 0xCCu) * 0x40040u) & 0x03030303u;
    const uint32_t p0 = prmt_raw(F.q[J], hw, 0x5140u), p1 = prmt_raw(F.q[J], hw, 0x7362u);      // the indices, two to a word
#pragma unroll
    for (int l = 0; l < 4; ++l) {
        const uint2 g = lds64((l & 1) ? dp2a_high(l < 2 ? p0 : p1, f, tab) : dp2a_low(l < 2 ? p0 : p1, f, tab));
        o[2 * l] = g.x; o[2 * l + 1] = g.y;
    }
}
__device__ __forceinline__ uint32_t iq2s_select(uint32_t four) {             // four codebook bytes, 0x08, 0x19 or 0x2b: value i's bytes 2 c, 2 c + 1
    const uint32_t c = (four >> 4) & 0x03030303u;
    return c << 1 | c << 5 | 0x10101010u;
}
// IQ3_S: the entry's four values as f16.
template<int J> __device__ __forceinline__ void iq_lookup(const IqFields<MAYA_IQ3_S>& F, uint32_t tab, uint32_t f, uint32_t* o) {
    const uint32_t qh = byte_of(F.qh[J / 4], J % 4);
    // byte l of h0 / h1 = bit l / 4 + l of qh, the ninth index bit of entry l / 4 + l
    const uint32_t h0 = ((qh & 15u) * 0x204081u) & 0x01010101u, h1 = ((qh >> 4) * 0x204081u) & 0x01010101u;
    const uint32_t p[4] = {prmt_raw(F.q[2 * J], h0, 0x5140u), prmt_raw(F.q[2 * J], h0, 0x7362u), prmt_raw(F.q[2 * J + 1], h1, 0x5140u),
                           prmt_raw(F.q[2 * J + 1], h1, 0x7362u)};
#pragma unroll
    for (int l = 0; l < 8; ++l) {
        const uint2 g = lds64((l & 1) ? dp2a_high(p[l / 2], f, tab) : dp2a_low(p[l / 2], f, tab));
        o[2 * l] = g.x; o[2 * l + 1] = g.y;
    }
}
// Pair p's signs from sign byte s: s * (2^(15 - 2p) + 2^(30 - 2p)) has them at bits 15 and 31 (the two shifted copies of the 8 bits do not meet);
// masked out and the signs flipped by one three-input operation.
__device__ __forceinline__ uint32_t iq_signs(uint32_t s, int p) { return (s * ((1u << (15 - 2 * p)) + (1u << (30 - 2 * p)))) & 0x80008000u; }
// Eight values in place: times dl (one f16 rounding), then the signs.
__device__ __forceinline__ void iq_eight(uint32_t s, __half2 dl, uint32_t* r) {
#pragma unroll
    for (int p = 0; p < 4; ++p) r[p] = h2_bits(__hmul2(bits_h2(r[p]), dl)) ^ iq_signs(s, p);
}
// A byte's two scale nibbles (n0 low) -> (f16 scale times a (2 n0 + 1), and times a (2 n1 + 1)), a a power of two: the factors are exact
// and each product is rounded once, as f16 of the f32 product is.
template<int T> __device__ __forceinline__ __half2 iq_scales(uint32_t word, int byte, uint32_t d2) {
    const uint32_t z = (__byte_perm(word, 0, byte | 0x40 | byte << 8 | 0x4000) & 0x00F0000Fu) | 0x64006400u;     // 1024 + n0, 1024 + 16 n1
    const __half2 n = T == MAYA_IQ2_S ? __hfma2(bits_h2(z), __floats2half2_rn(0.25f, 0.015625f), __floats2half2_rn(-255.875f, -15.875f))
                                      : __hfma2(bits_h2(z), __floats2half2_rn(2.0f, 0.125f), __floats2half2_rn(-2047.0f, -127.0f));
    return __hmul2(bits_h2(d2), n);
}
// Sub-blocks J and J + 1 (J even): look-ups -> weights, in place; `mid` runs when the first is done.
// IQ2_S (ggml dequantize_row_iq2_s): y = d (0.5 + ls) 0.25 * grid[qs | qh bits] * sign; the factor is f16(d (2 ls + 1) / 8), and the three
// products by it are rounded once, as every weight's own would be.  (A selector's upper half is brought down by a dp2a: the byte permutes fill the integer pipe,
// and with a shift there 3000 tokens of 4096 x 2048 took 1.02 times, with f16 entries 1.10 times as long; 777 of 6144 x 2048 1.03 and 1.07 times.)
template<int J, class Mid> __device__ __forceinline__ void iq_finish2(const IqFields<MAYA_IQ2_S>& F, uint32_t* o, Mid mid) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const __half2 dl = iq_scales<MAYA_IQ2_S>(F.sc[J / 4], (J + h) % 4, F.d2);
        uint32_t* const r = o + 16 * h;
        uint32_t sel[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) sel[i] = r[i];
#pragma unroll
        for (int l = 0; l < 4; ++l) {
            const __half2 d = l < 2 ? __low2half2(dl) : __high2half2(dl);
            const uint32_t a = h2_bits(__hmul2(d, __floats2half2_rn(8.0f, 25.0f))), b = h2_bits(__hmul2(d, __floats2half2_rn(43.0f, 43.0f)));
            const uint32_t s = byte_of(F.sg[J + h], l);
#pragma unroll
            for (int p = 0; p < 4; ++p)
                r[4 * l + p] = prmt_raw(a, b, (p & 1) ? dp2a_high(sel[2 * l + p / 2], 1u << 24, 0u) : sel[2 * l + p / 2]) ^ iq_signs(s, p);
        }
        if (h == 0) mid();
    }
}
// IQ3_S (ggml dequantize_row_iq3_s): y = d (1 + 2 scale) * grid[qs | qh bit] * sign.
template<int J, class Mid> __device__ __forceinline__ void iq_finish2(const IqFields<MAYA_IQ3_S>& F, uint32_t* o, Mid mid) {
    const __half2 db = iq_scales<MAYA_IQ3_S>(F.sc[0], J / 2, F.d2);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const __half2 dl = h == 0 ? __low2half2(db) : __high2half2(db);
#pragma unroll
        for (int l = 0; l < 4; ++l) iq_eight(byte_of(F.sg[J + h], l), dl, o + 16 * h + 4 * l);
        if (h == 0) mid();
    }
}

// A block works on tile after tile (see mmq_kernel): what the roles share of one of them.  e < 0: no tile left.
struct TileInfo { int e, row0, nrows, m0, lin; };     // lin: its place in the list
constexpr int kTiles = 8;            // ring of tile entries: the raw-unit loader, which makes them, is at most kMaxUnits / 4 + 1
                                     // tiles ahead of the slowest reader (it waits for every unit to be read)

// How a tile of `nrows` activation rows divides tensor memory and the activation ring.  Two accumulators of as many columns as
// there are rows, in steps of 32; what is left of the 512 holds stages of expanded weights, 32 columns for each accumulator - three
// beside 160 rows, seven beside 32: with three, the two teams of expanding warps waited for each other, since a team takes a block's
// fields out of its window (400 to 600 cycles) while the other one's pairs need the stages in between.  An activation tile is a 128-row
// box (and a 32-row box behind it), or just the latter.
struct TileGeo {
    uint32_t acc;                    // columns of an accumulator: accumulator 0 at 0, accumulator 1 at acc, the stages from 2 acc
    int st, bst;                     // stages of expanded weights, of activations
    uint32_t bbytes;                 // bytes of the latter
};
template<int T> __device__ __forceinline__ TileGeo tile_geo(int nrows) {
    const int q = (max(nrows, 1) + 31) >> 5;
    TileGeo g;
    g.acc = 32u * (uint32_t) q;
    g.st = kMaxSt + 1 - q;
    g.bbytes = q == 1 ? 32 * 128 : q <= 4 ? kBBox : kBStage;
    g.bst = q == 1 ? kMaxBSt : min(kMaxBSt, q <= 4 ? kBRing<T> / kBBox : kBRing<T> / kBStage);
    return g;
}
static_assert(2 * TN + 64 * (kMaxSt + 1 - TN / 32) <= 512 && 64 + 64 * kMaxSt <= 512 && kMaxBSt * 32 * 128 <= kBRing<MAYA_Q8_0>, "tile_geo");

struct Pipe {                       // static shared memory of a block
    uint64_t a_full[kMaxSt], b_full[kMaxBSt];
    uint64_t done[kDone];            // done[p % kDone]: the products of K-step pair p (64 K-values) have completed
    uint64_t raw_full[kMaxUnits], raw_empty[kMaxUnits];
    uint64_t tile_full[kTiles];      // tile entry written
    uint64_t final;                  // a tile's products have completed
    uint64_t acc_free;               // its accumulators have been read: the next tile's products may overwrite them
    uint64_t stg_free[2];            // the write-back of an even / odd tile has left shared memory: loads may overwrite it
    TileInfo tile[kTiles];
    uint32_t tmem;
    int fail;
};

__device__ __forceinline__ bool failed(const Pipe& P) { return *(volatile const int*) &P.fail != 0; }
// Bounded wait of a whole warp; false when it ran out (the block's failure flag is then set) or another role has failed.  The lanes
// vote on every look - a look may find a barrier's phase ended for some of them and not yet for the others - so that they leave
// together: what follows (tensor-memory stores, elected copies and products) needs the warp converged.
// (try_wait with a suspend-time hint, so that the waiting roles poll less: 1 to 7 % slower, longest when all roles used it; four looks
// between two counts of the loop 5 to 10 % slower.)
__device__ __forceinline__ bool wait_or_fail(Pipe& P, uint64_t* bar, uint32_t parity) {
    for (unsigned i = 0; i < (1u << 21); ++i) {
        if (__all_sync(0xFFFFFFFFu, mbar_try_wait(bar, parity))) return true;
        if (i > 4096) {                          // try_wait itself suspends the thread for a while; back off only late
            __nanosleep(64);
            if ((i & 255) == 0 && __any_sync(0xFFFFFFFFu, failed(P))) return false;
        }
    }
    *(volatile int*) &P.fail = 1;
    return false;
}

// A group's activation rows as the write-back leaves them in shared memory: rows rounded up to 8, and the bytes of the whole
__device__ __forceinline__ int rows_up8(int nrows) { return (nrows + 7) & ~7; }
template<bool GLU> __device__ __forceinline__ int staging_bytes(int nrows) { return rows_up8(nrows) * (GLU ? 128 * 4 : TM * 4); }

// A tile's rows of h are written by threads this one has met at a barrier since: count them for the down product ...
__device__ __forceinline__ void red_release(unsigned* counter, unsigned n) {
    fence_proxy_async_all();                         // they are read by tensor copies
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(counter), "r"(n) : "memory");
}
// ... whose activation loader waits here (a second at most).  false: the wait ran out or another role has failed.
__device__ __forceinline__ bool wait_rows(Pipe& P, const unsigned* counter, unsigned want) {
    unsigned long long t0 = 0, now;
    for (unsigned i = 0;; ++i) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
        if (v >= want) break;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        if (i == 0) t0 = now;
        if (now - t0 > 1000000000ull) { *(volatile int*) &P.fail = 1; return false; }
        if (failed(P)) return false;
        __nanosleep(200);
    }
    fence_proxy_async_all();                         // the tensor copies that follow read what the counter vouches for
    return true;
}

// Persistent: one block an SM takes tiles blockIdx.x, blockIdx.x + gridDim.x, ... of the list (group-major, a group's slabs
// of weight rows side by side, so that the blocks at work share its activation rows in L2).  How many groups there are is
// known only on the device; a grid sized for the most there can be cost 20 to 30 us a launch in blocks that found no tile
// (64 tokens over 256 experts: 259 group rows launched, 55 in use), and every tile paid the block's set-up - tensor-memory
// allocation, codebook, barriers - and its first loads' latency behind the previous block's write-back.  Here the barriers'
// phases run on from tile to tile, and the raw loader starts the next tile's units while the last one is written back.
template<int T, bool GLU>
__global__ void __launch_bounds__(kMmqThreads, 1)
mmq_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x,
           const __grid_constant__ CUtensorMap tm_x32, const MmqArgs A) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ Pipe P;
    const int tid = threadIdx.x, warp = __shfl_sync(0xFFFFFFFFu, tid >> 5, 0), lane = tid & 31;
    constexpr int NU = kUnits<T>;
    const int nkt = A.w_cols / BK, nkb = A.w_cols / 256;
    // Q4_K: after every 8 blocks of K (32 pairs of K steps) one more pair carries the sum correction of those blocks' 64
    // groups - A = the groups' constant terms -dmin * m, B = the tail of the activation image (see xq_tail); the last pair
    // of a K that is not a multiple of 2048 is padded with zeros.  ntp = how many such pairs.
    const int ntp = T == MAYA_Q4_K ? (nkb + 7) / 8 : 0;
    const int npairs = nkt / 2 + ntp;               // pairs of K steps of a tile
    constexpr int kSlab = GLU ? 128 : TM;
    const int nslab = (A.w_rows + kSlab - 1) / kSlab;
#ifdef MAYA_MMQ_STAMPS
    auto stamps_of = [&](int lin) -> long long* {
        return lin < 4096 ? g_stamps + ((size_t) ((T == MAYA_Q4_K || T == MAYA_IQ3_S ? 2 : 0) + (GLU ? 1 : 0)) * 4096 + lin) * 16 : nullptr;
    };
#endif

    uint8_t* const raw = smem + kBRing<T>;
    if (tid == 0) {
        for (int s = 0; s < kMaxSt; ++s) mbar_init(&P.a_full[s], 8);
        for (int s = 0; s < kMaxBSt; ++s) mbar_init(&P.b_full[s], 1);
        for (int s = 0; s < kDone; ++s) mbar_init(&P.done[s], 2);      // both issuers commit
        for (int u = 0; u < NU; ++u) { mbar_init(&P.raw_full[u], 1); mbar_init(&P.raw_empty[u], kIq<T> ? 2 : 4); }
        for (int i = 0; i < kTiles; ++i) mbar_init(&P.tile_full[i], 1);
        mbar_init(&P.final, 2);
        mbar_init(&P.acc_free, kDqWarps);
        mbar_init(&P.stg_free[0], kDqWarps);
        mbar_init(&P.stg_free[1], kDqWarps);
        P.fail = 0;
        mbar_fence_init();
    }
    if (warp == kDqWarps && lane < 3)
        asm volatile("prefetch.tensormap [%0];" ::"l"(lane == 0 ? &tm_w : lane == 1 ? &tm_x : &tm_x32) : "memory");
    if (warp == 0) tmem_alloc(&P.tmem, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = P.tmem;
    if (A.alone) grid_dependency_wait();             // (its set-up overlaps the launch in front)
    // In a chain the next product's blocks may start from here on, where this one's have ended: after the wait, since they do not
    // wait for what is in front of this one.  What they do wait for is in `ready`.
    grid_launch_dependents();
    // the block's t-th tile, for a role that waits for its entry; false: the wait ran out or another role has failed
    auto tile_of = [&](int t, TileInfo& ti) -> bool {
        if (!wait_or_fail(P, &P.tile_full[t % kTiles], (t / kTiles) & 1)) return false;
        ti = P.tile[t % kTiles];
        return true;
    };

    if (warp < kDqWarps) {
        // ------------------------------------------------------------ weight expansion
        // Two teams of 8 warps; in each, thread = one of the slab's 256 rows.  Team t expands the K steps kt with
        // kt % 2 == t, so that a step's latency (shared-memory reads, the packed-half chain, the tensor-memory store
        // and its wait) overlaps the other team's step.
        if constexpr (kIq<T>) {                     // the codebook's copies, once per block, under the first loads' latency
            const __half2 k1024 = __float2half2_rn(1024.0f);
            auto wide = [&](uint32_t g) {           // four codebook bytes as f16
                return make_uint2(h2_bits(__hsub2(bytes01_plus1024(g), k1024)), h2_bits(__hsub2(bytes23_plus1024(g), k1024)));
            };
            uint2* const grid = (uint2*) (smem + kTabOff<T>);
            for (int i = tid; i < kTabBytes<T> / 8; i += kDqWarps * 32) {
                const int e = i / kCopies<T>;
                if constexpr (T == MAYA_IQ2_S) {
                    const uint2 g = ((const uint2*) g_iq2s_grid)[e];
                    grid[i] = make_uint2(iq2s_select(g.x), iq2s_select(g.y));
                } else {
                    grid[i] = wide(g_iq3s_grid[e]);
                }
            }
            named_bar_sync(2, kDqWarps * 32);
        }
        const int team = warp >> 3, row = tid & 255, w8 = warp & 7;
        const int slab = row >> 6;
        const uint8_t* const rbase = raw + (size_t) (row & 63) * kRawRow<T>;
        // rows 0..127 feed accumulator 0, rows 128..255 accumulator 1; a warp reaches the 32 lanes of its quadrant
        const uint32_t a_lane = tmem + ((uint32_t) (32 * (w8 & 3)) << 16) + (w8 >> 2) * 32;
        const uint32_t afull0 = smem_u32(&P.a_full[0]), done0 = smem_u32(&P.done[0]);
        // The team's next pair of the tile, its stage and that stage's place in tensor memory.  (A tile's stages start at 0: every product
        // of the tile before it has completed.)
        int seq = 0, st = 0, n_st = 0, kp0 = 0;          // kp0: pairs of the tiles before this one
        uint32_t a_at = 0;
        auto ahead = [&](int d) {                        // d <= 4
            seq += d;
            st += d;
            if (st >= n_st) st -= n_st;
            if (kIq<T> && st >= n_st) st -= n_st;        // there are at least three
        };
        // The stage is free when pair seq - n_st, which read it last, has completed.  look(): whether it is, asked before the expansion so
        // that the answer is there behind it; acquire(): now (the warp is then converged, as the stores need it).
        auto look = [&]() -> bool {
            if (seq < n_st) return true;
            const unsigned pp = (unsigned) (kp0 + seq - n_st);
            return mbar_test_wait_addr(done0 + 8 * (pp & (kDone - 1)), (pp / kDone) & 1u);
        };
        auto acquire = [&](bool seen) -> bool {
            if (!__all_sync(0xFFFFFFFFu, seen)) {
                const unsigned pp = (unsigned) (kp0 + seq - n_st);
                if (!wait_or_fail(P, &P.done[pp & (kDone - 1)], (pp / kDone) & 1u)) return false;
            }
            tc_fence_after();
            __syncwarp();
            return true;
        };
        auto release = [&] {
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_addr(afull0 + 8 * st);
        };
        // i-quants: this lane's copy of the codebook, and the entries' distance
        constexpr uint32_t kEnt = kCopies<T> * 8;
        [[maybe_unused]] const uint32_t tab = smem_u32(smem + kTabOff<T>) + (kIq<T> ? lane % (kIq<T> ? kCopies<T> : 1) * 8 : 0);
        [[maybe_unused]] const uint32_t tab_f = kEnt | kEnt << 24;
        [[maybe_unused]] uint4 corr[8];      // Q4_K: the constant terms of the current 8-block chunk (indexed by kb: local memory)
        // A pair's two halves of 32 K-values: the first half's tensor-memory store is under way while the second half is
        // expanded (the store, its wait and the hand-off were a serial tail of every pair).
        auto st_half = [&](int h, const uint32_t* o16) { tmem_st16(a_at + 64 * st + 16 * h, *(const uint32_t(*)[16]) o16); };
        // the place of the raw unit of this warp's rows in the next block it expands (i-quants: always the same), and its barrier's phase
        int slot = slab + (kIq<T> ? 4 * team : 0);
        uint32_t raw_phase = 0;
        for (int t = 0;; ++t, kp0 += npairs) {
        TileInfo ti;
        bool ok = tile_of(t, ti);
        if (named_bar_or(3, kDqWarps * 32, !ok) || ti.e < 0) break;      // the same for every expanding warp
        const int nrows = ti.nrows, row0 = ti.row0, m0 = ti.m0;
        const TileGeo geo = tile_geo<T>(nrows);
        seq = st = 0;
        n_st = geo.st;
        ahead(kIq<T> ? 4 * team : team);
        a_at = a_lane + 2 * geo.acc;
#ifdef MAYA_MMQ_STAMPS
        long long* const stamps = tid == 0 && ok ? stamps_of(ti.lin) : nullptr;
        if (stamps) { stamps[0] = clock64(); stamps[14] = nrows; stamps[15] = npairs; }
#endif
        // i-quants: a team expands every other block whole - its fields are taken out of the window once.  The products take the pairs in
        // K's order all the same (the accumulator's sums are f32: another order is another result): a team's four pairs wait in the stages
        // while the other team's are taken.  The other types: both teams work on a block, on alternate pairs.
        for (int kb = kIq<T> ? team : 0; kb < nkb && ok; kb += kIq<T> ? 2 : 1) {
            if (!wait_or_fail(P, &P.raw_full[slot], raw_phase)) { ok = false; break; }
            const uint8_t* rrow = rbase + (size_t) slot * kUnitBytes<T>;
            uint32_t o[32];
            if constexpr (kIq<T>) {
                constexpr int NWD = kWin<T> / 4;
                uint32_t wv[NWD];
#pragma unroll
                for (int i = 0; i < NWD / 4; ++i) {
                    const uint4 v = *(const uint4*) (rrow + 16 * i);
                    wv[4 * i] = v.x; wv[4 * i + 1] = v.y; wv[4 * i + 2] = v.z; wv[4 * i + 3] = v.w;
                }
                IqFields<T> F;
                // where the block starts in its window: period 8 in kb, a multiple of 4 for every other block
                switch ((kb * kBlkBytes<T>) & 15) {
                    case 0: iq_fields<T, 0>(wv, F); break;
                    case 2: iq_fields<T, 2>(wv, F); break;
                    case 4: iq_fields<T, 4>(wv, F); break;
                    case 6: iq_fields<T, 6>(wv, F); break;
                    case 8: iq_fields<T, 8>(wv, F); break;
                    case 10: iq_fields<T, 10>(wv, F); break;
                    case 12: iq_fields<T, 12>(wv, F); break;
                    default: iq_fields<T, 14>(wv, F);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&P.raw_empty[slot]);      // its two warps have read the unit
                // Both sub-blocks' look-ups are under way before the first is finished, and the next pair's before this one's stores
                // are waited for.
                iq_lookup<0>(F, tab, tab_f, o);
                iq_lookup<1>(F, tab, tab_f, o + 16);
                auto pair = [&](auto i) {
                    constexpr int J = 2 * decltype(i)::value;
                    const bool seen = look();
                    bool got = true;
                    iq_finish2<J>(F, o, [&] {
                        got = acquire(seen);
                        if (got) st_half(0, o);
                    });
                    if (!got) return false;
                    st_half(1, o + 16);
                    if constexpr (J < 6) {
                        iq_lookup<J + 2>(F, tab, tab_f, o);
                        iq_lookup<J + 3>(F, tab, tab_f, o + 16);
                    }
                    release();
                    ahead(1);
                    return true;
                };
                ok = pair(std::integral_constant<int, 0>{}) && pair(std::integral_constant<int, 1>{}) && pair(std::integral_constant<int, 2>{}) &&
                     pair(std::integral_constant<int, 3>{});
                ahead(4);
            } else if constexpr (T == MAYA_Q4_K) {
                const uint4 hdr = *(const uint4*) rrow;
                const __half2 d2 = __low2half2(bits_h2(hdr.x)), m2 = __high2half2(bits_h2(hdr.x));
                const int mine = 16 * team, chunk = kb >> 3;     // the team that owns the chunk's correction pair keeps the constant terms
                __half2 nml[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) nml[i] = q4k_min(i, hdr.z >> mine, hdr.w >> mine, m2);
                if ((chunk & 1) == team) {
                    const int other = 16 - mine;
                    uint32_t own[2], oth[2];
#pragma unroll
                    for (int i = 0; i < 2; ++i) { own[i] = h2_bits(nml[i]); oth[i] = h2_bits(q4k_min(i, hdr.z >> other, hdr.w >> other, m2)); }
                    corr[kb & 7] = team == 0 ? make_uint4(own[0], oth[0], own[1], oth[1]) : make_uint4(oth[0], own[0], oth[1], own[1]);
                }
#pragma unroll
                for (int i = 0; i < 2; ++i) {        // the 64 values of quant pair p: low nibbles, then high nibbles
                    const int p = 2 * i + team;
                    const uint4 qa = *(const uint4*) (rrow + 16 + 32 * p), qb = *(const uint4*) (rrow + 32 + 32 * p);
                    const __half2 dl = q4k_scale(i, hdr.y >> mine, hdr.w >> mine, d2);
                    const bool seen = look();
                    q4k_stage(qa, qb, 0, __low2half2(dl), __low2half2(nml[i]), o);
                    if (!acquire(seen)) { ok = false; break; }
                    st_half(0, o);
                    q4k_stage(qa, qb, 1, __high2half2(dl), __high2half2(nml[i]), o + 16);
                    st_half(1, o + 16);
                    release();
                    if (i == 0) ahead(2);
                }
                // the chunk's correction pair stands behind its last pair, team 1's
                const bool last = (kb & 7) == 7 || kb == nkb - 1;
                if (!last) {
                    ahead(2);
                } else if (ok && (chunk & 1) == team) {
                    ahead(2 - team);
#pragma unroll
                    for (int b = 0; b < 8; ++b) {
                        const uint4 c = b <= (kb & 7) ? corr[b] : make_uint4(0u, 0u, 0u, 0u);
                        o[4 * b] = c.x; o[4 * b + 1] = c.y; o[4 * b + 2] = c.z; o[4 * b + 3] = c.w;
                    }
                    ok = acquire(look());
                    if (ok) {
                        tmem_st32(a_at + 64 * st, o);
                        release();
                    }
                    ahead(1 + team);
                } else {
                    ahead(3);
                }
            } else {
#define MAYA_Q80_PAIR(PP)                                                                      \
    if (ok) {                                                                                  \
        const bool seen = look();                                                              \
        q80_stage<2 * (PP)>(rrow, o);                                                          \
        ok = acquire(seen);                                                                    \
        if (ok) {                                                                              \
            st_half(0, o);                                                                     \
            q80_stage<2 * (PP) + 1>(rrow, o + 16);                                             \
            st_half(1, o + 16);                                                                \
            release();                                                                         \
            ahead(2);                                                                          \
        }                                                                                      \
    }
                if (team == 0) { MAYA_Q80_PAIR(0) MAYA_Q80_PAIR(2) }
                else { MAYA_Q80_PAIR(1) MAYA_Q80_PAIR(3) }
#undef MAYA_Q80_PAIR
            }
            if (!ok) break;
            if constexpr (!kIq<T>) {
                __syncwarp();
                if (lane == 0) mbar_arrive(&P.raw_empty[slot]);      // 4 warps read a unit; after the 4th it may be overwritten
            }
            if constexpr (!kIq<T>) slot += 4;
            if (kIq<T> || slot >= NU) { if constexpr (!kIq<T>) slot -= NU; raw_phase ^= 1u; }
        }
        // ------------------------------------------------------------ write-back
        if (ok && !wait_or_fail(P, &P.final, t & 1)) ok = false;
        tc_fence_after();
        // every expansion warp gets here (all waits are bounded) and they agree: what follows has barriers that need them all
        if (named_bar_or(3, kDqWarps * 32, !ok)) break;
#ifdef MAYA_MMQ_STAMPS
        if (stamps) stamps[4] = clock64();               // accumulators complete, expanding warps met
#endif
        {
            // The tile leaves through shared memory (the activation ring, and the raw ring behind it where the group is large:
            // the loaders know, and wait for stg_free before they write there): the warps drop their lanes' values into
            // [activation row][weight row] order, then one bulk copy per activation row writes it out.
            const int q = warp & 3, hs = warp >> 2;                      // hs = 0..3
            const uint32_t lane_base = tmem + ((uint32_t) (32 * q) << 16);
            uint8_t* const stg = smem;
            constexpr int kThreadsEpi = kDqWarps * 32;
            auto accumulators_read = [&] {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&P.acc_free);
            };
            if constexpr (GLU) {
                // Two passes.  First the tile goes from tensor memory to shared memory as h = SwiGLU(gate, up) in f32,
                // [activation row][128]: 16 warps = 4 lane quadrants x 4 groups, a group takes every 4th chunk of 8
                // activation rows.  Then, for the f16 image, every thread rounds 8 consecutive values of a row at a time
                // (4 threads a 32-value group, as maya_mmq_quantize does: the same function, the same bytes) - the groups' amax
                // and sums cost two shuffles each instead of a warp-wide reduction per value - and stores them from its
                // registers, 256 bytes a half warp.  (Through shared memory and one bulk copy a row the block waited for
                // the copies' reads, and in a chain for their completion.)
                float* b32 = (float*) stg;                               // [rows][128] h
                const int nchunk = (nrows + 7) >> 3;
                const int mcol = 32 * q + lane;
                for (int c = hs; c < nchunk; c += 4) {
                    const int col0 = 8 * c;
                    float v[8], up[8];
                    tmem_ld8(lane_base + col0, v);
                    tmem_ld8(lane_base + geo.acc + col0, up);
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (col0 + j < nrows) b32[(col0 + j) * 128 + mcol] = swiglu(v[j], up[j], A.limit);   // uniform in the warp
                }
                accumulators_read();
#ifdef MAYA_MMQ_STAMPS
                if (stamps) stamps[5] = clock64();       // SwiGLU tile in shared memory
#endif
                if (A.xq_out) {
                    named_bar_sync(2, kThreadsEpi);
                    const int ch = tid & 15;                             // the row's 8-value chunk; a warp covers two rows
                    const int64_t ldq = xq_ld(A.w_rows);
                    for (int r0 = 0; r0 < nrows; r0 += kThreadsEpi / 16) {
                        const int r = r0 + (tid >> 4);
                        const bool live = r < nrows;                     // the same for a group's four threads
                        const float* src = b32 + (live ? r : 0) * 128 + 8 * ch;
                        const float4 lo = *(const float4*) src, hi = *(const float4*) (src + 4);
                        const float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
                        uint32_t o[4];
                        const __half xa = q8_1_round8(v, o);
                        if (live) {
                            __half* const dst = A.xq_out + (int64_t) (row0 + r) * ldq;
                            *(uint4*) (dst + m0 + 8 * ch) = make_uint4(o[0], o[1], o[2], o[3]);
                            if ((ch & 3) == 0) dst[A.w_rows + (m0 >> 5) + (ch >> 2)] = xa;
                            if (m0 == 0)                                 // the zero padding behind the row's corrections
                                for (int64_t c = A.w_rows + A.w_rows / 32 + ch; c < ldq; c += 16) dst[c] = __float2half_rn(0.0f);
                        }
                    }
                }
#ifdef MAYA_MMQ_STAMPS
                if (stamps) stamps[6] = clock64();       // tile rounded
#endif
                if (A.dst) {                                             // h itself, a bulk copy a row
                    fence_proxy_async();
                    named_bar_sync(1, kThreadsEpi);
                    if (tid < nrows) {
                        const int64_t row_g = row0 + tid;
                        bulk_store(A.dst + (int64_t) (A.ids ? A.ids[row_g] : row_g) * A.ld_dst + m0, b32 + tid * 128, 128 * 4);
                        bulk_commit();
                    }
                }
            } else {
                // 16 warps = 4 lane quadrants x 2 accumulators x 2 groups that take alternate chunks of 16 activation rows
                const int acc = hs & 1, grp = hs >> 1;
                const bool have = m0 + 128 * acc < A.w_rows;             // this warp's accumulator exists
                const uint32_t row_bytes_out = (uint32_t) min(TM, A.w_rows - m0) * 4;
                float* buf = (float*) stg;                               // [rows][256] f32
                const int nchunk = (nrows + 15) >> 4;
                const int mcol = 128 * acc + 32 * q + lane;
                if (have) {
                    for (int c = grp; c < nchunk; c += 2) {
                        const int col0 = 16 * c;
                        float v[16];
                        tmem_ld16(lane_base + acc * geo.acc + col0, v);
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (col0 + j < nrows) buf[(col0 + j) * TM + mcol] = v[j];
                    }
                }
                accumulators_read();
                fence_proxy_async();
                named_bar_sync(1, kThreadsEpi);
                if (tid < nrows) {
                    const int row_g = row0 + tid;
                    bulk_store(A.dst + (int64_t) (A.ids ? A.ids[row_g] : row_g) * A.ld_dst + m0, buf + tid * TM, row_bytes_out);
                    bulk_commit();
                }
            }
            if (tid < nrows) bulk_wait_read<0>();                        // the copies have read shared memory ...
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&P.stg_free[t & 1]);              // ... which the next tile's loads may overwrite
        }
#ifdef MAYA_MMQ_STAMPS
        if (stamps) stamps[7] = clock64();               // written back
#endif
        }
    } else if (warp == kDqWarps) {
        // ------------------------------------------------------------ the tile list, and raw weight units (one warp)
        const uint32_t raw0 = smem_u32(raw), rawfull0 = smem_u32(&P.raw_full[0]);
        int slot = 0, prev_rows = 0;         // the next raw unit's place; rows of the tile before this one
        uint32_t raw_phase = 1;              // of the barrier that says the place is free: at once the first time round
        // In a chain the tiles are taken as blocks get to them (blocks of the next product start where this one's have run out of
        // tiles), a tile ahead of its use; else block b's are b, b + grid, ...
        int claimed = (int) blockIdx.x;
        if (A.claim != nullptr && lane == 0) claimed = (int) atomicAdd(A.claim, 1u);
        for (int t = 0;; ++t) {
            // Which (matrix, 160-row group) is this tile's: the warp scans the per-matrix group counts - each lane the counts
            // of a run of consecutive matrices, an exclusive warp scan of the runs' sums, then the lane whose run holds the
            // wanted group walks it - 1024 matrices a round.
            const int lin = __shfl_sync(0xFFFFFFFFu, claimed, 0), want_all = lin / nslab;
            int found_e = -1, row0 = 0, nrows = 0, base = 0;
            for (int e0 = 0; e0 < A.n; e0 += 1024) {
                const int per = (min(A.n - e0, 1024) + 31) >> 5;          // matrices a lane (<= 32)
                const int lo = e0 + lane * per, hi = min(lo + per, min(A.n, e0 + 1024));
                int mine = 0;
                for (int e = lo; e < hi; ++e) {
                    const int be = A.expert_map ? A.expert_map[e] : e;
                    mine += (A.bounds[be + 1] - A.bounds[be] + TN - 1) / TN;
                }
                int incl = mine;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                    if (lane >= o) incl += v;
                }
                const int total = __shfl_sync(0xFFFFFFFFu, incl, 31);
                const int want = want_all - base;
                const bool mine_is_it = want >= incl - mine && want < incl;
                if (mine_is_it) {
                    int g = want - (incl - mine);
                    for (int e = lo; e < hi; ++e) {
                        const int be = A.expert_map ? A.expert_map[e] : e;
                        const int b0 = A.bounds[be], b1 = A.bounds[be + 1], cnt = (b1 - b0 + TN - 1) / TN;
                        if (g < cnt) { found_e = e; row0 = b0 + g * TN; nrows = min(TN, b1 - row0); break; }
                        g -= cnt;
                    }
                }
                const unsigned holds = __ballot_sync(0xFFFFFFFFu, mine_is_it);
                if (holds != 0u) {
                    const int src = __ffs(holds) - 1;
                    found_e = __shfl_sync(0xFFFFFFFFu, found_e, src);
                    row0 = __shfl_sync(0xFFFFFFFFu, row0, src);
                    nrows = __shfl_sync(0xFFFFFFFFu, nrows, src);
                    break;
                }
                base += total;
            }
            const int m0 = (lin % nslab) * kSlab;
            bool ok = true;
            {
                claimed = lin + (int) gridDim.x;
                if (A.claim != nullptr && found_e >= 0 && lane == 0) claimed = (int) atomicAdd(A.claim, 1u);
                // Entry t % kTiles was read by every role before tile t - kTiles ended.  The write-back of the tile two before
                // this one has to be over in any case (so that a barrier's phase is never two behind), that of the tile before
                // only where it stretches into the raw ring.
                if (t >= 2) ok = wait_or_fail(P, &P.stg_free[t & 1], ((t - 2) >> 1) & 1);
                if (lane == 0) {
                    P.tile[t % kTiles] = TileInfo{found_e, row0, nrows, m0, lin};
                    mbar_arrive(&P.tile_full[t % kTiles]);
                }
                __syncwarp();
                if (found_e >= 0) {
                    if (ok && t >= 1 && staging_bytes<GLU>(prev_rows) > kBRing<T>)
                        ok = wait_or_fail(P, &P.stg_free[(t - 1) & 1], ((t - 1) >> 1) & 1);
                    for (int kb = 0; kb < nkb && ok; ++kb) {
                        for (int sl = 0; sl < 4; ++sl) {
                            if (!wait_or_fail(P, &P.raw_empty[slot], raw_phase)) { ok = false; break; }
                            const int wrow = GLU ? (sl < 2 ? m0 + 64 * sl : A.w_rows + m0 + 64 * (sl - 2)) : m0 + 64 * sl;
                            // x: the block's 32-bit words (k-quants), or the 16-byte aligned byte offset of the window around the
                            // i-quant block (the box is then 112 / 144 bytes of each row; past the row's end it reads as zeros)
                            const int x0 = kIq<T> ? (int) (((size_t) kb * kBlkBytes<T>) & ~(size_t) 15) : kb * (kRawRow<T> / 4);
                            tma_expect_load_3d(raw0 + slot * kUnitBytes<T>, &tm_w, rawfull0 + 8 * slot, kUnitBytes<T>, x0, wrow, found_e);
                            if (++slot == NU) { slot = 0; raw_phase ^= 1u; }
                        }
                    }
                }
            }
            if (!ok || found_e < 0) break;
            prev_rows = nrows;
        }
        // Let the copies in flight land before the block ends: a place's last one.  Also when all went well so far - the roles that
        // would wait for them may still give up.
        for (int i = 0; i < NU; ++i) wait_or_fail(P, &P.raw_full[i], i < slot ? raw_phase ^ 1u : raw_phase);
        if (A.claim != nullptr && lane == 0 && atomicAdd(A.claim + 1, 1u) == gridDim.x - 1u) {       // no block will claim again
            A.claim[0] = 0u;
            A.claim[1] = 0u;
        }
    } else if (warp == kDqWarps + 1 || warp == kDqWarps + 3) {
        // ------------------------------------------------------------ tensor-core issue (two warps, one accumulator each, on
        //                                                              different schedulers)
        // One product of N = rows rounded up to 16 per accumulator and K = 16: an M = 128 product occupies the tensor core
        // for N / 2 cycles, but only if this warp can issue one that often.  The whole warp walks the loop, converged, and
        // one elected lane issues: everything the products take is warp-uniform and stays in uniform registers.  (With a
        // single lane inside a divergent branch every operand of every product crossed from a vector register first, and
        // issuing was the longest stage of the pipeline.)
        const int my = warp == kDqWarps + 1 ? 0 : 1;
        const uint32_t tm = __shfl_sync(0xFFFFFFFFu, tmem, 0);
        const uint64_t bdesc0 = smem_desc_sw128(smem_u32(smem));
        const uint32_t b_hi = (uint32_t) (bdesc0 >> 32), b_lo0 = (uint32_t) bdesc0;
        const uint32_t bfull0 = smem_u32(&P.b_full[0]), afull0 = smem_u32(&P.a_full[0]), done0 = smem_u32(&P.done[0]);
        uint32_t ph_a = 0, ph_b = 0, done_at = 0;    // the barriers' phases, a bit each; the next pair's place in the ring of done barriers
        for (int t = 0;; ++t) {
            TileInfo ti;
            bool ok = tile_of(t, ti);
            if (!ok) break;
            const int n_rows = __shfl_sync(0xFFFFFFFFu, ti.nrows, 0);
            if (__shfl_sync(0xFFFFFFFFu, ti.e, 0) < 0) break;
            if (t > 0) {                             // the accumulators still hold the tile before until its write-back has read them
                ok = wait_or_fail(P, &P.acc_free, (t - 1) & 1);
                if (!ok) break;
                tc_fence_after();
            }
            const int n_mma = max(16, (n_rows + 15) & ~15);
            const uint32_t idesc = (1u << 4) | ((uint32_t) (n_mma >> 3) << 17) | ((uint32_t) (128 >> 4) << 24);
            const TileGeo geo = tile_geo<T>(n_rows);
            const uint32_t a0 = tm + 2 * geo.acc + my * 32, d0 = tm + my * geo.acc, b_step = geo.bbytes >> 4;
            uint32_t first = 0;                      // 0: the first product overwrites
            uint32_t b_lo = b_lo0, at = a0, sa = 0, sb = 0;       // the next pair's place in the activation ring and in tensor memory, its stages
            for (int kp = 0; kp < npairs; ++kp) {
                const uint32_t pa = (ph_a >> sa) & 1u, pb = (ph_b >> sb) & 1u;
                const bool rb = mbar_test_wait_addr(bfull0 + 8 * sb, pb), ra = mbar_test_wait_addr(afull0 + 8 * sa, pa);
                if (!__all_sync(0xFFFFFFFFu, rb && ra)) {        // not there yet: the bounded waits
                    if (!wait_or_fail(P, &P.b_full[sb], pb) || !wait_or_fail(P, &P.a_full[sa], pa)) { ok = false; break; }
                }
                tc_fence_after();
#ifdef MAYA_MMQ_STAMPS
                if (my == 0 && kp == 0 && lane == 0 && stamps_of(ti.lin)) stamps_of(ti.lin)[2] = clock64();       // the first product
#endif
                mma_f16_ts_x4_commit(d0, at, b_lo, b_hi, idesc, first, done0 + done_at);
                first = 1;
                done_at = (done_at + 8) & (8 * kDone - 1);
                ph_a ^= 1u << sa;
                ph_b ^= 1u << sb;
                at += 64;
                if (++sa == (uint32_t) geo.st) { sa = 0; at = a0; }
                b_lo += b_step;
                if (++sb == (uint32_t) geo.bst) { sb = 0; b_lo = b_lo0; }
            }
#ifdef MAYA_MMQ_STAMPS
            if (my == 0 && lane == 0 && stamps_of(ti.lin)) stamps_of(ti.lin)[3] = clock64();                      // the last product issued
#endif
            if (!ok) break;
            mma_commit_elect(smem_u32(&P.final));
        }
    } else if (warp == kDqWarps + 2) {
        // ------------------------------------------------------------ activation tiles (one warp)
        const int nmain = nkt / 2;
        const uint32_t ring0 = smem_u32(smem), bfull0 = smem_u32(&P.b_full[0]);
        int p0 = 0;                                  // pairs of the tiles before this one
        uint32_t phases = 0;                         // a bit a place of the ring: the phase its next load ends
        bool ok = true;
        unsigned* counter = nullptr;                 // gate/up in a chain: the counter of the tile before's rows, not counted yet
        unsigned written = 0;
        auto count_rows = [&] {
            if (counter != nullptr && lane == 0) red_release(counter, written);
            counter = nullptr;
            __syncwarp();
        };
        for (int t = 0;; ++t, p0 += npairs) {
            TileInfo ti;
            ok = tile_of(t, ti);
            // the write-back of the tile before uses the activation ring
            if (ok && t > 0) ok = wait_or_fail(P, &P.stg_free[(t - 1) & 1], ((t - 1) >> 1) & 1);
            const int e = __shfl_sync(0xFFFFFFFFu, ti.e, 0), nrows = __shfl_sync(0xFFFFFFFFu, ti.nrows, 0);
            const int row0 = __shfl_sync(0xFFFFFFFFu, ti.row0, 0), lin = __shfl_sync(0xFFFFFFFFu, ti.lin, 0);
            if (!ok || e < 0) {
                if (ok) count_rows();
                break;
            }
            if (!GLU && A.ready != nullptr) {
                unsigned* const r = A.ready + 2 * (lin / nslab);
                ok = __all_sync(0xFFFFFFFFu, wait_rows(P, r, (unsigned) (nrows * A.ready_slabs)));
                if (!ok) break;
                if (lane == 0 && atomicAdd(r + 1, 1u) == (unsigned) nslab - 1u) { r[0] = 0u; r[1] = 0u; }      // the group's last tile to wait
                __syncwarp();
            }
            const TileGeo geo = tile_geo<T>(nrows);
            int sb = 0;
            for (int kb2 = 0; kb2 < npairs; ++kb2) {
                // the pair's 64 K-values in the image: K values in order, and after every 32 pairs (or at the end) the
                // chunk's 64 corrections from the tail behind the row's K values
                int xcol;
                if (ntp == 0) {
                    xcol = kb2 * 64;
                } else {
                    const int c = kb2 / 33, r = kb2 - c * 33;
                    const bool is_corr = r == 32 || kb2 == nmain + ntp - 1;
                    xcol = is_corr ? A.w_cols + 64 * c : (kb2 - c) * 64;
                }
                if (kb2 >= geo.bst) {                // the place was last read by pair kb2 - bst
                    const unsigned pp = (unsigned) (p0 + kb2 - geo.bst);
                    if (!wait_or_fail(P, &P.done[pp % kDone], (pp / kDone) & 1u)) { ok = false; break; }
                }
                const uint32_t dst = ring0 + (uint32_t) sb * geo.bbytes, bar = bfull0 + 8 * sb;
                tma_expect_load_2d(dst, geo.bbytes < kBBox ? &tm_x32 : &tm_x, bar, geo.bbytes, xcol, row0);
                if (geo.bbytes > kBBox) tma_load_2d_elect(dst + kBBox, &tm_x32, bar, xcol, row0 + 128);
                phases ^= 1u << sb;
                if (++sb == geo.bst) sb = 0;
                if (kb2 == min(geo.bst, npairs) - 1) count_rows();       // behind the loads the expansion waits for
            }
            if (!ok) break;
            if (GLU && A.ready != nullptr) { counter = A.ready + 2 * (lin / nslab); written = (unsigned) nrows; }
        }
        if (!ok)                                     // let the copies in flight land before the block ends: a place's last one
            for (int i = 0; i < kMaxBSt; ++i) wait_or_fail(P, &P.b_full[i], ((phases >> i) & 1u) ^ 1u);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 512);
    grid_dependency_wait();                          // a block ends after the products in front of its own
    if (tid == 0 && failed(P) && A.error != nullptr) atomicExch(A.error, 1u);
}

// x rows -> f16 rows of their q8_1 image.  A thread owns 8 consecutive values (one 16-byte store), the 4 threads of a
// 32-value block find its amax with two shuffles.  blockIdx.x is the row, blockIdx.y * 256 + threadIdx.x the 8-value chunk.
// ROUTED = false: image row r is x row ids[r] (ids == nullptr: r).  ROUTED = true: x row t is rounded once and its image
// stored to the k rows pos[t * k + j] (the sorted rows of the token's k routes) - the same bytes as the gathered form
// writes through row_tok, at one eighth of the arithmetic for k = 8.
template<typename X, bool ROUTED>
__global__ void __launch_bounds__(256) mmq_quantize_kernel(const X* __restrict__ x, const int* __restrict__ ids,
                                                           __half* __restrict__ xq, int cols, int64_t ld, int k) {
    const int64_t row = blockIdx.x;
    grid_launch_dependents();
    grid_dependency_wait();
    const int cpr = cols >> 3, c = (int) blockIdx.y * 256 + (int) threadIdx.x;
    const bool live = c < cpr;                       // cpr is a multiple of 4: a block's 4 threads live together
    const int64_t src = (!ROUTED && ids) ? ids[row] : row;
    float v[8];
    if (live) {
        if constexpr (sizeof(X) == 2) {              // bf16 bits, widened exactly
            const uint4 u = *(const uint4*) (x + src * ld + c * 8);
            const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) { v[2 * i] = __uint_as_float(w[i] << 16); v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u); }
        } else {
            const float4 a = *(const float4*) (x + src * ld + c * 8), b = *(const float4*) (x + src * ld + c * 8 + 4);
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = 0.0f;
    }
    uint32_t o[4];
    const __half xa = q8_1_round8(v, o);
    // a warp's eight groups: their corrections leave as one 16-byte store when a row is a whole number of warps
    const bool packed = (cols & 255) == 0;
    uint4 cw = make_uint4(0u, 0u, 0u, 0u);
    if (packed) {
        const uint32_t mine = (uint32_t) __half_as_ushort(xa);
        const uint32_t pair = mine | (__shfl_down_sync(0xFFFFFFFFu, mine, 4) << 16);        // lanes 0, 8, 16, 24: groups (2i, 2i + 1)
        const uint32_t p1 = __shfl_sync(0xFFFFFFFFu, pair, 8), p2 = __shfl_sync(0xFFFFFFFFu, pair, 16), p3 = __shfl_sync(0xFFFFFFFFu, pair, 24);
        cw = make_uint4(pair, p1, p2, p3);
    }
    if (!live) return;
    const int64_t ldq = xq_ld(cols);
    const int nd = ROUTED ? k : 1;
    for (int j = 0; j < nd; ++j) {
        const int64_t dr = ROUTED ? (int64_t) ids[row * k + j] : row;
        __half* d = xq + dr * ldq;
        *(uint4*) (d + c * 8) = make_uint4(o[0], o[1], o[2], o[3]);
        if (packed) { if ((threadIdx.x & 31) == 0) *(uint4*) (d + cols + (c >> 2)) = cw; }
        else if ((c & 3) == 0) d[cols + (c >> 2)] = xa;
        if (c == 0)                                   // the zero padding behind the row's corrections
            for (int64_t t = cols + cols / 32; t < ldq; ++t) d[t] = __float2half_rn(0.0f);
    }
}

template<typename X>
int launch_quantize(const X* x, const int32_t* ids, void* xq, int type, int64_t cols, int64_t ld, int64_t rows, int k, void* stream) {
    if (!maya_mmq_supported(type)) return refuse(MAYA_ERR_TYPE);
    if (rows <= 0) return MAYA_OK;
    if (!x || !xq || cols <= 0 || cols % 32 || ld < cols || cols > 0x7FFFFFF0ll) return refuse(MAYA_ERR_ARG);
    if (k < 0 || (k > 0 && !ids)) return refuse(MAYA_ERR_ARG);
    if (!aligned16(x) || !aligned16(xq) || (ld * sizeof(X)) % 16) return refuse(MAYA_ERR_ARG);   // 16-byte loads and stores
    const int64_t by = (cols / 8 + 255) / 256;
    if (rows > 0x7FFFFFFFll || by > 65535) return refuse(MAYA_ERR_LIMIT);
    const dim3 grid((unsigned) rows, (unsigned) by);
    launch_dependent(k > 0 ? mmq_quantize_kernel<X, true> : mmq_quantize_kernel<X, false>, grid, dim3(256), 0, as_stream(stream), x, ids,
                     (__half*) xq, (int) cols, ld, k > 0 ? k : 0);
    return note_launch(k > 0 ? "mmq_quantize_routed" : "mmq_quantize");
}

// ---- tensor maps (driver entry point looked up once; the library does not link libcuda)
PFN_cuTensorMapEncodeTiled encode_fn() {
    static PFN_cuTensorMapEncodeTiled fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return (PFN_cuTensorMapEncodeTiled) p;
    }();
    return fn;
}
// The driver refused a tensor map (a stride or an extent beyond what a map can hold): nothing is launched.
int no_map(const char* what) {
    std::fprintf(stderr, "maya_moe: %s tensor map refused\n", what);
    return refuse(MAYA_ERR_LAUNCH);
}
bool make_map(CUtensorMap* m, CUtensorMapDataType dt, int rank, const void* base, const cuuint64_t* dim, const cuuint64_t* stride,
              const cuuint32_t* box, CUtensorMapSwizzle swizzle) {
    PFN_cuTensorMapEncodeTiled fn = encode_fn();
    if (!fn) return false;
    const cuuint32_t es[3] = {1, 1, 1};
    return fn(m, dt, (cuuint32_t) rank, const_cast<void*>(base), dim, stride, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// An upper bound of sum(ceil(rows_e / 160)), known without the counts.
int64_t most_groups(const maya_mmq_product* p) { return (p->total_rows > 0 ? p->total_rows / TN : 0) + p->n; }

template<int T, bool GLU>
int launch_mmq(const maya_mmq_product* p, const MmqArgs& A, cudaStream_t s) {
    const int64_t mat_rows = p->w_rows, K = p->w_cols;
    const size_t rbw = row_bytes(T, K);
    CUtensorMap tw, tx, tx32;
    std::memset(&tw, 0, sizeof(tw));
    if constexpr (!kIq<T>) {   // weights as 32-bit words: (word in row, row in matrix, matrix); a box = 256 K-values of 64 rows
        const cuuint64_t dim[3] = {(cuuint64_t) (rbw / 4), (cuuint64_t) mat_rows, (cuuint64_t) p->n};
        const cuuint64_t st[2] = {(cuuint64_t) rbw, (cuuint64_t) p->expert_bytes};
        const cuuint32_t box[3] = {(cuuint32_t) (kRawRow<T> / 4), kUnitRows, 1};
        if (!make_map(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT32, 3, p->w, dim, st, box, CU_TENSOR_MAP_SWIZZLE_NONE))
            return no_map("mmq weight");
    } else {                   // i-quants as bytes: a box = the 112 / 144 bytes of 64 rows that hold the block's window;
                               // a row is a multiple of 16 bytes (K a multiple of 2048) and so is every window's start
        const cuuint64_t dim[3] = {(cuuint64_t) rbw, (cuuint64_t) mat_rows, (cuuint64_t) p->n};
        const cuuint64_t st[2] = {(cuuint64_t) rbw, (cuuint64_t) p->expert_bytes};
        const cuuint32_t box[3] = {(cuuint32_t) kRawRow<T>, kUnitRows, 1};
        if (!make_map(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, p->w, dim, st, box, CU_TENSOR_MAP_SWIZZLE_NONE))
            return no_map("mmq weight");
    }
    {   // activations: f16 [row][K + tail] (xq_ld); a box = 64 K-values (128 bytes) of 128 or 32 rows, written with the 128-byte swizzle
        const cuuint64_t dim[2] = {(cuuint64_t) xq_ld(K), (cuuint64_t) p->total_rows};
        const cuuint64_t st[1] = {(cuuint64_t) xq_ld(K) * 2};
        const cuuint32_t box[2] = {64, 128}, box32[2] = {64, 32};
        if (!make_map(&tx, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, p->xq, dim, st, box, CU_TENSOR_MAP_SWIZZLE_128B) ||
            !make_map(&tx32, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, p->xq, dim, st, box32, CU_TENSOR_MAP_SWIZZLE_128B))
            return no_map("mmq activation");
    }
    constexpr size_t smem = kSmemBytes<T>;
    if (cudaFuncSetAttribute(mmq_kernel<T, GLU>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem) != cudaSuccess)
        return note_launch("mmq smem attribute");
    const int64_t groups = most_groups(p);
    const int slab = GLU ? 128 : TM, sms = sm_count();
    if (sms <= 0) return refuse(MAYA_ERR_DEVICE);
    const int64_t most = (int64_t) ((A.w_rows + slab - 1) / slab) * groups;      // tiles there can be
    const dim3 grid((unsigned) (most < sms ? most : sms));
    launch_dependent(mmq_kernel<T, GLU>, grid, dim3(kMmqThreads), smem, s, tw, tx, tx32, A);
    return note_launch("mmq");
}

// Everything about a product that can be refused, before anything is launched.
int check_product(const maya_mmq_product* p, bool glu) {
    if (!p || !p->w || !p->xq || !p->bounds) return MAYA_ERR_ARG;
    if (!p->dst && !(glu && p->xq_out)) return MAYA_ERR_ARG;
    if (!maya_mmq_supported(p->type)) return MAYA_ERR_TYPE;
    if ((p->type == MAYA_IQ2_S || p->type == MAYA_IQ3_S) && p->w_cols % 2048) return MAYA_ERR_ARG;   // 16-byte aligned rows
    if (p->n <= 0 || p->total_rows <= 0) return MAYA_OK;
    const int64_t out_rows = glu ? p->w_rows / 2 : p->w_rows;
    if (p->w_cols <= 0 || p->w_cols % 256 || out_rows <= 0 || out_rows % 128 || (glu && p->w_rows % 2)) return MAYA_ERR_ARG;
    if (p->expert_bytes % (size_t) type_bytes(p->type) || p->expert_bytes % 16 || (p->dst && p->ld_dst < out_rows)) {
        std::fprintf(stderr, "maya_mmq_run: expert_bytes %zu is not a whole number of blocks and of 16 bytes, or ld_dst too small\n",
                     p->expert_bytes);
        return MAYA_ERR_ARG;
    }
    if (!aligned16(p->w) || !aligned16(p->xq) || (p->xq_out && !aligned16(p->xq_out))) return MAYA_ERR_ARG;
    if (p->dst && (!aligned16(p->dst) || p->ld_dst % 4)) return MAYA_ERR_ARG;      // rows leave as 16-byte aligned bulk copies
    if (most_groups(p) > 65535) return MAYA_ERR_LIMIT;
    return MAYA_OK;
}

struct Chain { unsigned *claim, *ready; int ready_slabs; bool first; };

int run_product(const maya_mmq_product* p, bool glu, float limit, const Chain* chain, cudaStream_t s) {
    const int st = check_product(p, glu);
    if (st != MAYA_OK) return refuse(st);
    if (p->n <= 0 || p->total_rows <= 0) return MAYA_OK;
    const int64_t out_rows = glu ? p->w_rows / 2 : p->w_rows;
    MmqArgs A{};
    A.w_rows = (int) out_rows; A.w_cols = (int) p->w_cols; A.n = p->n; A.expert_map = p->expert_map; A.bounds = p->bounds;
    A.ids = p->ids; A.dst = p->dst; A.ld_dst = p->ld_dst; A.xq_out = glu ? (__half*) p->xq_out : nullptr; A.limit = limit;
    A.error = p->error;
    A.alone = chain == nullptr || chain->first;
    if (chain != nullptr) { A.claim = chain->claim; A.ready = chain->ready; A.ready_slabs = chain->ready_slabs; }
    switch (p->type) {
        case MAYA_Q4_K: return glu ? launch_mmq<MAYA_Q4_K, true>(p, A, s) : launch_mmq<MAYA_Q4_K, false>(p, A, s);
        case MAYA_Q8_0: return glu ? launch_mmq<MAYA_Q8_0, true>(p, A, s) : launch_mmq<MAYA_Q8_0, false>(p, A, s);
        case MAYA_IQ2_S: return glu ? launch_mmq<MAYA_IQ2_S, true>(p, A, s) : launch_mmq<MAYA_IQ2_S, false>(p, A, s);
        default: return glu ? launch_mmq<MAYA_IQ3_S, true>(p, A, s) : launch_mmq<MAYA_IQ3_S, false>(p, A, s);
    }
}

}  // namespace
}  // namespace maya

using namespace maya;

#ifdef MAYA_MMQ_STAMPS
// 4 x 4096 x 16 int64: [Q8_0/IQ2_S down, gate/up, Q4_K/IQ3_S down, gate/up][tile][stamp]; slots 14, 15 = rows, K-step pairs
extern "C" __attribute__((visibility("default"))) int maya_mmq_stamps_read(long long* host) {
    return (int) cudaMemcpyFromSymbol(host, g_stamps, sizeof(g_stamps));
}
#endif
extern "C" int maya_mmq_supported(int type) {
    return type == MAYA_Q4_K || type == MAYA_Q8_0 || type == MAYA_IQ2_S || type == MAYA_IQ3_S;
}
extern "C" size_t maya_mmq_q8_bytes(int64_t rows, int64_t cols) {
    if (rows <= 0 || cols <= 0 || cols % 32) return 0;
    return (size_t) rows * (size_t) xq_ld(cols) * sizeof(__half);
}
extern "C" int maya_mmq_quantize(const float* x, const int32_t* ids, void* xq, int type, int64_t cols, int64_t ld,
                                 int64_t rows, void* stream) {
    return launch_quantize<float>(x, ids, xq, type, cols, ld, rows, 0, stream);
}
extern "C" int maya_mmq_quantize_bf16(const uint16_t* x, const int32_t* ids, void* xq, int type, int64_t cols, int64_t ld,
                                      int64_t rows, void* stream) {
    return launch_quantize<uint16_t>(x, ids, xq, type, cols, ld, rows, 0, stream);
}
extern "C" int maya_mmq_quantize_routed(const float* x, const int32_t* pos, int k, void* xq, int type, int64_t cols, int64_t ld,
                                        int64_t tokens, void* stream) {
    if (k <= 0) return refuse(MAYA_ERR_ARG);
    return launch_quantize<float>(x, pos, xq, type, cols, ld, tokens, k, stream);
}
extern "C" int maya_mmq_quantize_routed_bf16(const uint16_t* x, const int32_t* pos, int k, void* xq, int type, int64_t cols,
                                             int64_t ld, int64_t tokens, void* stream) {
    if (k <= 0) return refuse(MAYA_ERR_ARG);
    return launch_quantize<uint16_t>(x, pos, xq, type, cols, ld, tokens, k, stream);
}
extern "C" int maya_mmq_run(const maya_mmq_product* p, void* stream) { return run_product(p, false, 0.0f, nullptr, as_stream(stream)); }
extern "C" int maya_mmq_run_glu(const maya_mmq_product* p, float limit, void* stream) {
    return run_product(p, true, limit, nullptr, as_stream(stream));
}
// Words of a chain's counters: two claim words a product, two ready words a group of a pair (an upper bound of the groups).
extern "C" size_t maya_mmq_chain_bytes(int64_t total_rows, int n_matrices, int n_pairs) {
    if (total_rows <= 0 || n_matrices <= 0 || n_pairs <= 0) return 0;
    return sizeof(unsigned) * (4 * (size_t) n_pairs + 2 * ((size_t) n_pairs * (size_t) (total_rows / TN) + (size_t) n_matrices));
}
extern "C" int maya_mmq_run_chain(const maya_mmq_product* gate_up, const maya_mmq_product* down, int n_pairs, float limit, void* counters,
                                  size_t counter_bytes, void* stream) {
    if (n_pairs <= 0) return MAYA_OK;
    if (!gate_up || !down || !counters || ((uintptr_t) counters & 3u)) return refuse(MAYA_ERR_ARG);
    // Nothing is launched before every product has been looked at: a gate/up product without its down product would leave its
    // rows counted, and the next chain on these counters would take them for its own.
    size_t need = 4 * (size_t) n_pairs;
    auto empty = [&](int i) { return gate_up[i].n == 0 || gate_up[i].total_rows <= 0; };
    for (int i = 0; i < n_pairs; ++i) {
        const maya_mmq_product &g = gate_up[i], &d = down[i];
        if (g.n != d.n || g.bounds != d.bounds || g.expert_map != d.expert_map || g.total_rows != d.total_rows || g.xq_out != d.xq ||
            !g.xq_out || g.n < 0)
            return refuse(MAYA_ERR_ARG);
        need += 2 * (size_t) most_groups(&g);
        if (empty(i)) continue;
        int st = check_product(&g, true);
        if (st == MAYA_OK) st = check_product(&d, false);
        if (st == MAYA_OK && d.w_cols != g.w_rows / 2) st = MAYA_ERR_ARG;          // the rows of h it reads are n_ff values long
        if (st != MAYA_OK) return refuse(st);
    }
    if (need * sizeof(unsigned) > counter_bytes) return refuse(MAYA_ERR_LIMIT);
    unsigned* const words = (unsigned*) counters;
    bool first = true;
    for (int pass = 0; pass < 2; ++pass) {
        unsigned* ready = words + 4 * n_pairs;
        for (int i = 0; i < n_pairs; ++i) {
            const maya_mmq_product& p = pass ? down[i] : gate_up[i];
            const Chain c{words + 4 * i + 2 * pass, ready, (int) (gate_up[i].w_rows / 256), first};
            ready += 2 * most_groups(&p);
            if (empty(i)) continue;
            const int st = run_product(&p, pass == 0, limit, &c, as_stream(stream));
            if (st != MAYA_OK) {                     // the launch itself failed: the products before it leave counts behind
                cudaMemsetAsync(counters, 0, need * sizeof(unsigned), as_stream(stream));
                return st;
            }
            first = false;
        }
    }
    return MAYA_OK;
}
