// rms_router.cu - the producer in front of the expert FFN: residual add, RMS norm and the router's logits in one launch,
// so that a decode layer is two launches end to end (this one, then the fused layer kernel).
//
// Reference counterparts: glmf::rms_q8 (include/strata/kernels/glm_fast.hpp:534, src/kernels/cuda/glm_fast.cu:5669-5697:
// h += add; x = h * rsqrt(mean(h^2) + eps) * w) and the router job of the multi-GEMV that Glm5Model::fast_moe issues
// next (src/core/glm_fast_path.cu:6925: logits = router_w . x with x in f32; router_w is F32 or BF16).  The q8_1 image
// of x that rms_q8 also writes is made by the layer kernel itself here.
//
// Every block recomputes the norm of the (small) hidden state - no grid-wide step - and then owns a few experts' router
// rows; block 0 also writes x and the updated residual stream.  The residual goes to h_out, which must not alias h when
// add is given (other blocks may still be reading h).
//
// What bounds it is latency, not bytes (3.1 MB of router rows at 256 experts of 6144 bf16 = 0.5 us): one wait for the
// launch, one round trip for h, one for the router rows.  So the rows are asked into L2 before the wait on the launch in
// front and into registers before the norm's reduction, 16 bytes a lane; and a block takes only as many experts as leave
// one block an SM (its eight warps split between them), where one warp per expert kept 32 of 148 SMs busy with a chain
// of dependent 2-byte loads: 19.7 us a call at that size, 5.4 so.  The norm's weights come with the same round trip as h, in registers, where
// they were a third one behind the reduction: 4.4 us (64 experts of 2048 3.1 / 2.7, 512 of 7168 8.8 / 7.4; calls in a row in a graph).
//
// A logit is an f32 sum whose order - and with it its last bits - depends on how many warps share a row (8, 4, 2 or 1, by the
// number of experts and SMs) and on whether the 16-byte form runs (alignment): equal to rounding, not bit for bit, between calls
// that differ in these.  The same call gives the same bits.
#include "maya_common.cuh"

namespace maya {
namespace {

constexpr int kRmsThreads = 256;
constexpr int kRmsWarps = kRmsThreads / 32;
constexpr int kAhead = 8;              // 16-byte pieces of a router row a lane holds before the norm is known

// Dot of 16 bytes of a router row with the values of x they meet.
template<bool BF16> __device__ __forceinline__ float dot16(const uint4 r, const float* xv, float acc) {
    if constexpr (BF16) {
        const float4 a = *(const float4*) xv, b = *(const float4*) (xv + 4);
        acc = __fmaf_rn(__uint_as_float(r.x << 16), a.x, acc); acc = __fmaf_rn(__uint_as_float(r.x & 0xFFFF0000u), a.y, acc);
        acc = __fmaf_rn(__uint_as_float(r.y << 16), a.z, acc); acc = __fmaf_rn(__uint_as_float(r.y & 0xFFFF0000u), a.w, acc);
        acc = __fmaf_rn(__uint_as_float(r.z << 16), b.x, acc); acc = __fmaf_rn(__uint_as_float(r.z & 0xFFFF0000u), b.y, acc);
        acc = __fmaf_rn(__uint_as_float(r.w << 16), b.z, acc); acc = __fmaf_rn(__uint_as_float(r.w & 0xFFFF0000u), b.w, acc);
    } else {
        const float4 a = *(const float4*) xv;
        acc = __fmaf_rn(__uint_as_float(r.x), a.x, acc); acc = __fmaf_rn(__uint_as_float(r.y), a.y, acc);
        acc = __fmaf_rn(__uint_as_float(r.z), a.z, acc); acc = __fmaf_rn(__uint_as_float(r.w), a.w, acc);
    }
    return acc;
}

// VEC: rows and vectors are 16-byte aligned and whole 16-byte pieces; else one element at a time.
template<bool BF16, bool VEC>
__global__ void __launch_bounds__(kRmsThreads) rms_router_kernel(const float* __restrict__ h, const float* __restrict__ add,
                                                                 const float* __restrict__ w, float eps, int n,
                                                                 const uint8_t* __restrict__ router, int n_expert, int epb,
                                                                 float* __restrict__ h_out, float* __restrict__ x_out,
                                                                 float* __restrict__ logits) {
    extern __shared__ __align__(16) float xs[];
    __shared__ float sred[kRmsWarps], sdot[kRmsWarps];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const size_t rb = (size_t) n * (BF16 ? 2 : 4);
    const int e0 = blockIdx.x * epb, ne = min(epb, n_expert - e0);
    // Programmatic dependent launch: nothing is read or written before the wait; a prefetch into L2 is neither.
    grid_launch_dependents();
    for (size_t b = (size_t) tid * 128; b < ne * rb; b += kRmsThreads * 128)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(router + (size_t) e0 * rb + b));
    for (int e = tid * 32; e < n; e += kRmsThreads * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(w + e));
    grid_dependency_wait();

    // the block's warps split evenly over its experts (epb divides kRmsWarps): expert e0 + warp / wpe, part warp % wpe
    const int wpe = kRmsWarps / epb, ex = e0 + warp / wpe, first = (warp % wpe) * 32 + lane, step = 32 * wpe;
    constexpr int kVals = BF16 ? 8 : 4;                   // values in 16 bytes
    const int pieces = n / kVals;
    const uint4* row = (const uint4*) (router + (size_t) ex * rb);
    uint4 r[kAhead];
    if constexpr (VEC) {
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
            r[i] = make_uint4(0u, 0u, 0u, 0u);
            if (ex < n_expert && first + i * step < pieces) r[i] = row[first + i * step];
        }
    }
    float ss = 0.0f;
    float4 wr[kAhead];
    if constexpr (VEC) {
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
            const int e = (tid + i * kRmsThreads) * 4;
            wr[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (e < n) wr[i] = *(const float4*) (w + e);
        }
#pragma unroll 4
        for (int e = tid * 4; e < n; e += kRmsThreads * 4) {
            float4 t = *(const float4*) (h + e);
            if (add != nullptr) {
                const float4 a = *(const float4*) (add + e);
                t.x += a.x; t.y += a.y; t.z += a.z; t.w += a.w;
            }
            *(float4*) (xs + e) = t;
            ss += t.x * t.x + t.y * t.y + t.z * t.z + t.w * t.w;
        }
    } else {
        for (int e = tid; e < n; e += kRmsThreads) {
            float t = h[e];
            if (add != nullptr) t += add[e];
            xs[e] = t;
            ss += t * t;
        }
    }
    ss = warp_sum(ss);
    if (lane == 0) sred[warp] = ss;
    __syncthreads();
    float tot = 0.0f;
#pragma unroll
    for (int i = 0; i < kRmsWarps; ++i) tot += sred[i];
    const float inv = rsqrtf(tot / (float) n + eps);
    if constexpr (VEC) {                                  // a thread scales the values it added itself
        auto scale = [&](int e, const float4 wv) {
            const float4 t = *(const float4*) (xs + e);
            const float4 xv = make_float4(t.x * inv * wv.x, t.y * inv * wv.y, t.z * inv * wv.z, t.w * inv * wv.w);
            *(float4*) (xs + e) = xv;
            if (blockIdx.x == 0) {
                *(float4*) (x_out + e) = xv;
                if (h_out != nullptr) *(float4*) (h_out + e) = t;
            }
        };
#pragma unroll
        for (int i = 0; i < kAhead; ++i)
            if ((tid + i * kRmsThreads) * 4 < n) scale((tid + i * kRmsThreads) * 4, wr[i]);
        for (int e = (tid + kAhead * kRmsThreads) * 4; e < n; e += kRmsThreads * 4) scale(e, *(const float4*) (w + e));
    } else {
        for (int e = tid; e < n; e += kRmsThreads) {
            const float t = xs[e], xv = t * inv * w[e];
            xs[e] = xv;
            if (blockIdx.x == 0) {
                x_out[e] = xv;
                if (h_out != nullptr) h_out[e] = t;
            }
        }
    }
    __syncthreads();
    float acc = 0.0f;
    if (ex < n_expert) {
        if constexpr (VEC) {
#pragma unroll
            for (int i = 0; i < kAhead; ++i)
                if (first + i * step < pieces) acc = dot16<BF16>(r[i], xs + (size_t) (first + i * step) * kVals, acc);
#pragma unroll 4
            for (int p = first + kAhead * step; p < pieces; p += step) acc = dot16<BF16>(row[p], xs + (size_t) p * kVals, acc);
        } else {
            for (int e = first; e < n; e += step) {
                const float v = BF16 ? __uint_as_float((uint32_t) ((const uint16_t*) row)[e] << 16) : ((const float*) row)[e];
                acc = __fmaf_rn(v, xs[e], acc);
            }
        }
    }
    acc = warp_sum(acc);
    if (lane == 0) sdot[warp] = acc;
    __syncthreads();
    if (tid < ne) {
        float v = sdot[tid * wpe];
        for (int i = 1; i < wpe; ++i) v += sdot[tid * wpe + i];
        logits[e0 + tid] = v;
    }
}

template<bool BF16, bool VEC>
int launch(const float* h, const float* add, const float* w, float eps, int n, const void* router, int n_expert, float* h_out,
           float* x_out, float* logits, cudaStream_t s) {
    const size_t smem = (size_t) n * sizeof(float);
    static SmemLimit smem_limit;
    if (smem > kSmemNoLimit && !smem_limit.raise((const void*) rms_router_kernel<BF16, VEC>, kSmemMost)) return note_launch("rms_router smem attribute");
    // experts a block: the fewest (1, 2, 4 or 8) that leave at most one block an SM, so that a small router spreads over the
    // chip (beyond 8 experts an SM blocks share SMs)
    const int sms = sm_count();
    int epb = 1;
    while (epb < kRmsWarps && (n_expert + epb - 1) / epb > sms) epb *= 2;
    launch_dependent(rms_router_kernel<BF16, VEC>, dim3((unsigned) ((n_expert + epb - 1) / epb)), dim3(kRmsThreads), smem, s, h, add, w, eps,
                     n, (const uint8_t*) router, n_expert, epb, h_out, x_out, logits);
    return note_launch("rms_router");
}

}  // namespace
}  // namespace maya

using namespace maya;

extern "C" int maya_rms_router(const float* h, const float* add, const float* norm_w, float eps, int n_embd,
                               const void* router_w, int router_is_bf16, int n_expert, float* h_out, float* x_out,
                               float* logits, void* stream) {
    if (!h || !norm_w || !router_w || !x_out || !logits || n_embd <= 0 || n_expert <= 0) return refuse(MAYA_ERR_ARG);
    if (add != nullptr && h_out == h) return refuse(MAYA_ERR_ARG);       // other blocks still read h
    if ((size_t) n_embd * sizeof(float) > kSmemMost) return refuse(MAYA_ERR_LIMIT);
    const bool vec = n_embd % 8 == 0 && aligned16(h) && (!add || aligned16(add)) && aligned16(norm_w) && aligned16(router_w) &&
                     (!h_out || aligned16(h_out)) && aligned16(x_out);
    cudaStream_t s = as_stream(stream);
#define RMS_CASE(B, V) launch<B, V>(h, add, norm_w, eps, n_embd, router_w, n_expert, h_out, x_out, logits, s)
    if (router_is_bf16) return vec ? RMS_CASE(true, true) : RMS_CASE(true, false);
    return vec ? RMS_CASE(false, true) : RMS_CASE(false, false);
#undef RMS_CASE
}
