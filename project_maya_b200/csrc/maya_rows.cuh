// maya_rows.cuh - decoding quantized weight rows that lie in shared memory: what the window kernel (moe_window.cuh) and the token
// kernel (moe_token.cuh) share.
//
// What bounds it (throughputs measured one instruction at a time, cycles a warp instruction holds a scheduler's pipe): the
// integer pipe takes a LOP3, PRMT, SHF or I2F every 2 cycles, the multiply pipe an IMAD, IDP (dp4a, dp2a) or HFMA2 every 2, the
// shared-memory pipe one wavefront a cycle for all four schedulers, issue 1.  The two arithmetic pipes run side by side, so a
// decoder is written to load the three evenly:
//   * a codebook index becomes an address in ONE dp2a - its 16 bits times the entries' distance plus the table's base - and a
//     sign byte in one dp4a, instead of a byte permute and a shift-add on the busier integer pipe;
//   * where a magnitude takes one of few values (IQ2_S: 8, 25, 43) the codebook holds selectors: a nibble a value, two bits
//     of magnitude and room for the sign bit, which a second table spreads from the sign byte.  One OR, and a byte
//     permute of {8, 25, 43, -, -8, -25, -43, -} by four of the nibbles IS the four signed weights: no masks and no
//     correction, and a look-up moves 4 bytes instead of 8;
//   * a lane's place in a step of 32 calls is the same in every step, so a row's addresses and alignments are found once.
// GEMV of 131072 rows of 6144, one column, 16 warps streaming: IQ2_S 107 -> 96 us, IQ3_S 107 -> 96 (read in place by 32 warps: 130, 143).
#pragma once

#include "maya_stream.cuh"

namespace maya {

__device__ __forceinline__ uint32_t s_u32(const uint8_t* s, uint32_t o) { return *(const uint32_t*) (s + o); }
// 4 bytes at an even place; sel: 0x3210 where o is a multiple of 4, else 0x5432
__device__ __forceinline__ uint32_t s_u32_a2(const uint8_t* s, uint32_t o, uint32_t sel) {
    const uint32_t a = o & ~3u;
    return prmt_raw(s_u32(s, a), s_u32(s, a + 4), sel);
}
// the selector for fields 2 bytes (and a multiple of 4) into a block at o
__device__ __forceinline__ uint32_t sel_2(uint32_t o) { return (o & 2u) ? 0x3210u : 0x5432u; }
// c + a's low or high 16 bits times f, b = f | f << 24, f < 256
__device__ __forceinline__ uint32_t dp2a_low(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("dp2a.lo.u32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ uint32_t dp2a_high(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("dp2a.hi.u32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
// c + byte l of a times f (b = f << 8 l), f < 256
__device__ __forceinline__ uint32_t dp4a_u(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("dp4a.u32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ uint32_t lds_u32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}

// ---- the geometry of a type's stream.  A segment: `vals` values of a row (a multiple of what 32 lanes take in one step, so that a
//      lane's calls are the same whatever the segments are).  pitch: a segment's room in a stage, its bytes and 16 for the aligned
//      window around it.
template<int T> struct RowGeo {
    static constexpr int vals = T == MAYA_Q8_0 || T == MAYA_Q6_K ? 1024 : 2048;
    static constexpr int qk = Fmt<T>::qk, cpb = Dec<T>::cpb;
    static constexpr int blocks = vals / qk;                     // weight blocks of a segment
    static constexpr int steps = blocks * cpb / 32;              // and steps of 32 calls
    static constexpr int bytes = blocks * Fmt<T>::bytes;
    static constexpr int pitch = (bytes + 15 + 16) & ~15;
};
struct RowGeoRt { int vals, qk, cpb, bytes, pitch; };
template<int T> __host__ __device__ inline RowGeoRt row_geo_of() { return {RowGeo<T>::vals, RowGeo<T>::qk, RowGeo<T>::cpb, RowGeo<T>::bytes, RowGeo<T>::pitch}; }
__host__ __device__ inline RowGeoRt row_geo(int type) {
    switch (type) {
        case MAYA_Q8_0: return row_geo_of<MAYA_Q8_0>();
        case MAYA_Q4_K: return row_geo_of<MAYA_Q4_K>();
        case MAYA_Q5_K: return row_geo_of<MAYA_Q5_K>();
        case MAYA_Q6_K: return row_geo_of<MAYA_Q6_K>();
        case MAYA_IQ4_XS: return row_geo_of<MAYA_IQ4_XS>();
        case MAYA_IQ2_S: return row_geo_of<MAYA_IQ2_S>();
        case MAYA_IQ3_S: return row_geo_of<MAYA_IQ3_S>();
        case MAYA_IQ3_XXS: return row_geo_of<MAYA_IQ3_XXS>();
        case MAYA_IQ2_XXS: return row_geo_of<MAYA_IQ2_XXS>();
        default: return row_geo_of<MAYA_IQ1_S>();
    }
}

// ---- the codebook in shared memory: copies of every entry side by side, lane l reading copy l % copies, so that a warp's
//      random look-ups spread over the banks.  MANY: as many as help (one activation column leaves the room); else half.
template<int T, bool MANY> struct RowTab {
    static constexpr int W = T == MAYA_IQ2_XXS ? 2 : 1;                        // words of an entry
    static constexpr int copies = T == MAYA_IQ2_S ? (MANY ? 16 : 8) : T == MAYA_IQ3_S ? (MANY ? 32 : 16) : T == MAYA_IQ3_XXS ? 32
                                  : T == MAYA_IQ2_XXS ? 16 : T == MAYA_IQ1_S && MANY ? 8 : 1;
    static constexpr int signs = T == MAYA_IQ2_S ? (MANY ? 32 : 16) : 0;       // copies of the sign words, behind the codebook
    static constexpr int words = T == MAYA_IQ2_S ? 1024 : Fmt<T>::tab_words;   // of one copy
    static constexpr int sign_off = words * 4 * copies, bytes = sign_off + 256 * 4 * signs;

    // by threads tid of nt, 16 bytes a store: consecutive threads to consecutive places
    __device__ __forceinline__ static void fill(uint32_t* tab, int tid, int nt) {
        if constexpr (bytes > 0) {
            const uint32_t* src = tab_source<T>();
            if constexpr (W == 2) {                                              // two words an entry: two copies a store
                constexpr int P = copies / 2;
#pragma unroll 4
                for (int i = tid; i < words / 2 * P; i += nt) {
                    const uint2 g = ((const uint2*) src)[i / P];
                    ((uint4*) tab)[i] = make_uint4(g.x, g.y, g.x, g.y);
                }
            } else if constexpr (copies == 1) {
                for (int i = tid; i < words; i += nt) tab[i] = src[i];
            } else {
                constexpr int P = copies / 4;
#pragma unroll 4
                for (int i = tid; i < words * P; i += nt) {
                    uint32_t g;
                    if constexpr (T == MAYA_IQ2_S) {                             // eight nibbles: 0, 1, 2 for 8, 25, 43
                        const uint2 v = ((const uint2*) src)[i / P];
                        auto pack = [](uint32_t c) {                             // 0x08, 0x19, 0x2b
                            c = (c >> 4) & 0x03030303u;
                            c = (c | c >> 4) & 0x00FF00FFu;
                            return (c | c >> 8) & 0xFFFFu;
                        };
                        g = pack(v.x) | pack(v.y) << 16;
                    } else {
                        g = src[i / P];
                        if constexpr (T == MAYA_IQ3_S) g = (g >> 1) & 0x07070707u;       // see SDec<MAYA_IQ3_S>
                    }
                    ((uint4*) tab)[i] = make_uint4(g, g, g, g);
                }
            }
            if constexpr (signs > 0) {
                constexpr int P = signs / 4;
#pragma unroll 2
                for (int i = tid; i < 256 * P; i += nt) {                        // bit j of the byte at bit 4 j + 2
                    const uint32_t e = (uint32_t) (i / P);
                    uint32_t g = (e & 0x0Fu) | (e & 0xF0u) << 12;                // bits 0..3 and 16..19
                    g = (g & 0x00030003u) | (g & 0x000C000Cu) << 6;              // two to a byte
                    g = ((g & 0x01010101u) | (g & 0x02020202u) << 3) << 2;
                    ((uint4*) (tab + sign_off / 4))[i] = make_uint4(g, g, g, g);
                }
            }
        }
    }
};
// this lane's copy of it
template<int T, bool MANY> struct RowLut {
    const uint32_t* p;
    uint32_t a, s;               // shared-memory addresses of the codebook and of the sign words
    uint32_t fa, fs;             // the entries' distances, as dp2a takes them
    __device__ __forceinline__ RowLut(const uint32_t* tab, int lane) {
        using R = RowTab<T, MANY>;
        p = tab + (lane % R::copies) * R::W;
        a = smem_u32(p);
        constexpr uint32_t ca = R::copies * R::W * 4, cs = R::signs * 4;
        asm volatile("mov.u32 %0, %1;" : "=r"(fa) : "n"(ca | ca << 24));      // (opaque: kept in registers)
        asm volatile("mov.u32 %0, %1;" : "=r"(fs) : "n"(cs | cs << 24));
        s = smem_u32(tab) + R::sign_off + (R::signs > 0 ? lane % (R::signs > 0 ? R::signs : 1) * 4 : 0);
    }
};

// ---- decoders: Dec<T>'s fields and dot for a call whose block lies in shared memory.  at(): what a lane needs of a row, `row`
//      the row's place in `s`, call `l` (0..31) of a step of 32; load(): step j.  Blocks of a step's end lie kStep bytes
//      behind those of the step before, a multiple of 4 for every type.  ONE: for a single column, where it is cheaper to
//      correct the dot for the signs (see maya_dots_t1.cuh) than to negate the weights.
template<int T> struct RowStep {
    static constexpr int cpb = Dec<T>::cpb, bytes = 32 / cpb * Fmt<T>::bytes;
    static_assert(32 % cpb == 0 && bytes % 4 == 0, "a step's alignment is every step's");
};
template<int T, bool ONE, bool MANY> struct SDec : Dec<T> {
    struct At { uint32_t o; };
    __device__ __forceinline__ static At at(uint32_t row, int l) { return {row + l / RowStep<T>::cpb * Fmt<T>::bytes}; }
    __device__ __forceinline__ void load(const uint8_t* s, const At& A, int j, int l, const RowLut<T, MANY>& L) {
        if constexpr (T == MAYA_IQ1_S) load_iq1(s + A.o + j * RowStep<T>::bytes, l % 8, L.p);
        else Dec<T>::load(s + A.o + j * RowStep<T>::bytes, l % RowStep<T>::cpb, L.p);
    }
private:
    __device__ __forceinline__ void load_iq1(const uint8_t* blk, int c, const uint32_t* tab) {        // Dec<MAYA_IQ1_S>::load, the entries apart
        if constexpr (T == MAYA_IQ1_S) {
            const uint32_t qs = ld_u32_a2(blk + 2 + 4 * c), qh = ld_u16(blk + 34 + 2 * c);
            this->d1q = ld_f16(blk) * (float) (2 * ((qh >> 12) & 7) + 1);
            this->delta = (qh & 0x8000u) ? -1.125f : -0.875f;
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                const uint32_t g = tab[(((qs >> (8 * l)) & 0xFF) | (((qh >> (3 * l)) & 7) << 8)) * RowTab<T, MANY>::copies];
                this->w[2 * l] = (int) (g & 0x0F0F0F0Fu);
                this->w[2 * l + 1] = (int) ((g >> 4) & 0x0F0F0F0Fu);
            }
        }
    }
};
// IQ2_S: the weights as nibble selectors (see the head of the file).
template<bool ONE, bool MANY> struct SDec<MAYA_IQ2_S, ONE, MANY> {
    struct At { uint32_t q, o, c, sel; };        // the index bytes' aligned word, the block, its byte `call`
    int w[8];
    int ls0, ls1;
    float d;
    __device__ __forceinline__ static At at(uint32_t row, int l) {
        const uint32_t o = row + (l >> 3) * 82;
        return {(o + 2 + 4 * (l & 7)) & ~3u, o, o + (l & 7), sel_2(o)};
    }
    __device__ __forceinline__ void load(const uint8_t* s, const At& A, int j, int, const RowLut<MAYA_IQ2_S, MANY>& L) {
        const uint8_t *q = s + A.q + j * 328, *c = s + A.c + j * 328;
        const uint32_t qs = prmt_raw(s_u32(q, 0), s_u32(q, 4), A.sel), sg = prmt_raw(s_u32(q, 32), s_u32(q, 36), A.sel);
        const uint32_t qh = c[66], sc = c[74];
        d = ld_f16(s + A.o + j * 328);
        ls0 = (int) (sc & 0x0F);
        ls1 = (int) (sc >> 4);
        const uint32_t hw = ((qh & 0x33u) * 0x1001u + (qh & 0xCCu) * 0x40040u) & 0x03030303u;      // see Dec1<MAYA_IQ2_S>
        const uint32_t p0 = prmt_raw(qs, hw, 0x5140u), p1 = prmt_raw(qs, hw, 0x7362u);             // the indices, two to a word
        const uint32_t g0 = __byte_perm(sg, 0, 0x4140), g1 = __byte_perm(sg, 0, 0x4342);           // and the sign bytes
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t p = i < 2 ? p0 : p1, q = i < 2 ? g0 : g1;
            const uint32_t n = lds_u32((i & 1) ? dp2a_high(p, L.fa, L.a) : dp2a_low(p, L.fa, L.a)) | lds_u32((i & 1) ? dp2a_high(q, L.fs, L.s) : dp2a_low(q, L.fs, L.s));
            w[2 * i] = (int) prmt_raw(0x002B1908u, 0x00D5E7F8u, n);
            w[2 * i + 1] = (int) prmt_raw(0x002B1908u, 0x00D5E7F8u, n >> 16);
        }
    }
    __device__ __forceinline__ float dot(const XQ& v, const XQ&) const {
        int s0 = 0, s1 = 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) { s0 = __dp4a(w[i], v.u[i], s0); s1 = __dp4a(w[4 + i], v.u[4 + i], s1); }
        return __fmul_rn(__fmul_rn(d, v.d), (float) ((s0 * ls0 + s1 * ls1 + (s0 + s1) / 2) / 4));
    }
};
// IQ3_S: every codebook value is odd, g = 2 b + 1 with b in 0..7.  Flipping b's bits negates it: 2 ~b + 1 = -g.  So the table
// holds b, a sign is one XOR, and sum(+-g u) = 2 sum((b ^ m) u) + sum(u), the block's sum being at hand.
template<bool ONE, bool MANY> struct SDec<MAYA_IQ3_S, ONE, MANY> {
    struct At { uint32_t q, g, o, c, n, sel; };  // the aligned words of the index and of the sign bytes, the block, its bytes `call` and `call` / 2
    int w[8];
    int mul;
    float d;
    __device__ __forceinline__ static At at(uint32_t row, int l) {
        const uint32_t o = row + (l >> 3) * 110;
        return {(o + 2 + 8 * (l & 7)) & ~3u, (o + 74 + 4 * (l & 7)) & ~3u, o, o + (l & 7), o + ((l & 7) >> 1), sel_2(o)};
    }
    __device__ __forceinline__ void load(const uint8_t* s, const At& A, int j, int l, const RowLut<MAYA_IQ3_S, MANY>& L) {
        const uint8_t *q = s + A.q + j * 440, *g = s + A.g + j * 440;
        const uint32_t w1 = s_u32(q, 4), q0 = prmt_raw(s_u32(q, 0), w1, A.sel), q1 = prmt_raw(w1, s_u32(q, 8), A.sel);
        const uint32_t sg = prmt_raw(s_u32(g, 0), s_u32(g, 4), A.sel), qh = s[A.c + j * 440 + 66];
        d = ld_f16(s + A.o + j * 440);
        mul = 1 + 2 * (int) ((s[A.n + j * 440 + 106] >> (4 * (l & 1))) & 0x0F);
        // byte i of h0 / h1: bit i / 4 + i of qh, an entry's ninth index bit
        const uint32_t h0 = ((qh & 15u) * 0x204081u) & 0x01010101u, h1 = ((qh >> 4) * 0x204081u) & 0x01010101u;
        const uint32_t p[4] = {prmt_raw(q0, h0, 0x5140u), prmt_raw(q0, h0, 0x7362u), prmt_raw(q1, h1, 0x5140u), prmt_raw(q1, h1, 0x7362u)};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t sb = byte_of(sg, i);
            w[2 * i] = (int) (lds_u32(dp2a_low(p[i], L.fa, L.a)) ^ sign_mask_lo(sb));
            w[2 * i + 1] = (int) (lds_u32(dp2a_high(p[i], L.fa, L.a)) ^ sign_mask_hi(sb));
        }
    }
    __device__ __forceinline__ float dot(const XQ& v, const XQ&) const {
        int s = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) s = __dp4a(w[i], v.u[i], s);
        return __fmul_rn(__fmul_rn(d, v.d), (float) ((2 * s + v.isum) * mul));
    }
};
// eight signed weight words (or, with ONE, codebook words XOR mask and the masks) and their dots
template<bool ONE> struct SSigned {
    int w[8];
    uint32_t mk[ONE ? 8 : 1];
    __device__ __forceinline__ void set(int i, uint32_t g, uint32_t m) {
        if constexpr (ONE) { w[i] = (int) (g ^ m); mk[i] = m; }
        else w[i] = apply_sign4(g, m);
    }
    __device__ __forceinline__ int dot(const XQ& v) const {
        int s = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) s = __dp4a(w[i], v.u[i], s);
        if constexpr (ONE) {
            int m = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) m = __dp4a((int) mk[i], v.u[i], m);
            s -= m;
        }
        return s;
    }
};
template<bool ONE, bool MANY> struct SDec<MAYA_IQ3_XXS, ONE, MANY> : SSigned<ONE> {
    struct At { uint32_t q, g, o, sel; };
    int ls;
    float d;
    __device__ __forceinline__ static At at(uint32_t row, int l) {
        const uint32_t o = row + (l >> 3) * 98;
        return {(o + 2 + 8 * (l & 7)) & ~3u, (o + 66 + 4 * (l & 7)) & ~3u, o, sel_2(o)};
    }
    __device__ __forceinline__ void load(const uint8_t* s, const At& A, int j, int, const RowLut<MAYA_IQ3_XXS, MANY>& L) {
        constexpr int R = RowTab<MAYA_IQ3_XXS, MANY>::copies * 4;
        const uint8_t *q = s + A.q + j * 392, *g = s + A.g + j * 392;
        d = ld_f16(s + A.o + j * 392);
        const uint32_t w1 = s_u32(q, 4), q0 = prmt_raw(s_u32(q, 0), w1, A.sel), q1 = prmt_raw(w1, s_u32(q, 8), A.sel);
        const uint32_t aux = prmt_raw(s_u32(g, 0), s_u32(g, 4), A.sel);
        ls = (int) (aux >> 28);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t s8 = ksign8((aux >> (7 * i)) & 127u), qw = i < 2 ? q0 : q1;
            this->set(2 * i, lds_u32(dp4a_u(qw, (uint32_t) R << (16 * (i & 1)), L.a)), sign_mask_lo(s8));
            this->set(2 * i + 1, lds_u32(dp4a_u(qw, (uint32_t) R << (16 * (i & 1) + 8), L.a)), sign_mask_hi(s8));
        }
    }
    __device__ __forceinline__ float dot(const XQ& v, const XQ&) const {
        const int t = SSigned<ONE>::dot(v);
        return __fmul_rn(__fmul_rn(d, v.d), (float) ((ls * t + t / 2) / 2));
    }
};
template<bool ONE, bool MANY> struct SDec<MAYA_IQ2_XXS, ONE, MANY> : SSigned<ONE> {
    struct At { uint32_t q, o, sel; };
    int ls;
    float d;
    __device__ __forceinline__ static At at(uint32_t row, int l) {
        const uint32_t o = row + (l >> 3) * 66;
        return {(o + 2 + 8 * (l & 7)) & ~3u, o, sel_2(o)};
    }
    __device__ __forceinline__ void load(const uint8_t* s, const At& A, int j, int, const RowLut<MAYA_IQ2_XXS, MANY>& L) {
        constexpr int R = RowTab<MAYA_IQ2_XXS, MANY>::copies;
        const uint8_t* q = s + A.q + j * 264;
        d = ld_f16(s + A.o + j * 264);
        const uint32_t w1 = s_u32(q, 4), qi = prmt_raw(s_u32(q, 0), w1, A.sel), aux = prmt_raw(w1, s_u32(q, 8), A.sel);
        ls = (int) (aux >> 27) | 1;
        const uint2* grid = (const uint2*) L.p;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint2 g = grid[byte_of(qi, i) * R];
            const uint32_t s8 = ksign8((aux >> (7 * i)) & 127u);
            this->set(2 * i, g.x, sign_mask_lo(s8));
            this->set(2 * i + 1, g.y, sign_mask_hi(s8));
        }
    }
    __device__ __forceinline__ float dot(const XQ& v, const XQ&) const {
        const int t = SSigned<ONE>::dot(v);
        return __fmul_rn(__fmul_rn(d, v.d), (float) (t * ls / 8));
    }
};

}  // namespace maya
