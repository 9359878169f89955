// maya_token_phase.cuh - what the two single-token layer kernels (moe_fused.cu, moe_token.cuh) share: the routing phase, the grid
// barrier, phase stamps and the cooperative launch.
#pragma once

#include "maya_common.cuh"
#include "maya_router.cuh"

namespace maya {
namespace {

constexpr int kRouteThreads = 256;
constexpr int kMaxSliceRows = 96;          // output rows a block may own (n_embd / grid rounded up)
constexpr unsigned long long kBarrierTimeoutNs = 1000000000ull;   // the grid barrier gives up after a second

// balanced contiguous split of n rows over nb blocks
__device__ __forceinline__ void slice(int n, int nb, int b, int& r0, int& r1) {
    const int base = n / nb, rem = n % nb;
    r0 = b * base + min(b, rem);
    r1 = r0 + base + (b < rem ? 1 : 0);
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// block 0's wall-clock stamp of a phase boundary (a 64-bit ns count in two scratch words)
__device__ __forceinline__ void stamp(unsigned* sync, int i) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *(volatile unsigned long long*) &sync[4 + 2 * i] = global_ns();
}

// All blocks of the (cooperative) grid meet here.  false in EVERY thread of the block when the wait ran out: thread 0
// leaves the outcome in shared memory before the closing barrier.  meanwhile(lane): what the second warp does while the first one's thread 0 waits.
template<class Meanwhile> __device__ __forceinline__ bool grid_barrier(unsigned* sync, unsigned epoch, int* s_ok, Meanwhile meanwhile) {
    __syncthreads();
    if (threadIdx.x >= 32 && threadIdx.x < 64) meanwhile((int) threadIdx.x - 32);
    if (threadIdx.x == 0) {
        int ok = 1;
        __threadfence();
        atomicAdd(&sync[0], 1u);
        const unsigned target = (epoch + 1u) * gridDim.x;
        const unsigned long long t0 = global_ns();
        while ((int) (*(volatile unsigned*) &sync[0] - target) < 0) {
            if (global_ns() - t0 > kBarrierTimeoutNs) { ok = 0; atomicExch(&sync[2], 1u); break; }
            __nanosleep(20);
        }
        __threadfence();
        *s_ok = ok;
    }
    __syncthreads();
    return *s_ok != 0;
}

// The token's routing by the block's first kRouteThreads threads, as a function of its own: run once a launch, it is
// kept out of the kernel's register allocation and instruction scheduling (which proved sensitive to what phase 0 holds).
// LATER: which experts, and only the values their weights are made of.  The token kernel makes the weights (route_weight: a sum and a
// division in double) while the grid barrier is waited for; made here its first rows waited for them (us a token in a graph, here / there:
// 2048 x 1024 Q4_K 16.97 / 16.49, 2048 x 2048 24.12 / 23.69).  The fused kernel, whose body has no register to spare, has them made
// here: there they cost it 0.3 us (6144 x 2048 IQ2_S with 2048 shared 59.54 / 59.86).
template<int RT, bool LATER>
__device__ __noinline__ void route_token(const float* logits, const float* bias, int n_expert, int k, float w_scale, int norm_w,
                                         int tid, double* s_ex, RouterShared* route) {
    using RS = NamedSync<1, kRouteThreads>;
    const int per = (n_expert + kRouteThreads - 1) / kRouteThreads;
    if constexpr (RT == 1) {
        if (per <= 1) route_sigmoid<1, RS, LATER>(logits, bias, n_expert, k, w_scale, norm_w, tid, kRouteThreads, s_ex, *route);
        else if (per <= 2) route_sigmoid<2, RS, LATER>(logits, bias, n_expert, k, w_scale, norm_w, tid, kRouteThreads, s_ex, *route);
        else if (per <= 4) route_sigmoid<4, RS, LATER>(logits, bias, n_expert, k, w_scale, norm_w, tid, kRouteThreads, s_ex, *route);
        else route_sigmoid<8, RS, LATER>(logits, bias, n_expert, k, w_scale, norm_w, tid, kRouteThreads, s_ex, *route);
    } else {
        if (per <= 1) route_softmax<1, RS, LATER>(logits, n_expert, k, tid, kRouteThreads, s_ex, *route);
        else if (per <= 2) route_softmax<2, RS, LATER>(logits, n_expert, k, tid, kRouteThreads, s_ex, *route);
        else if (per <= 4) route_softmax<4, RS, LATER>(logits, n_expert, k, tid, kRouteThreads, s_ex, *route);
        else route_softmax<8, RS, LATER>(logits, n_expert, k, tid, kRouteThreads, s_ex, *route);
    }
}

// A cooperative launch (the grid barrier needs every block resident) and, where the driver accepts the attribute,
// programmatically serialized after the launch in front of it: its set-up then overlaps that launch's tail.  (In a stream a cooperative
// launch gives up the overlap - it starts 2 to 3 us after the launch in front has ended - in a graph it keeps it.  An ordinary
// launch would keep it there too, but starts with the blocks that fit: they hold their SMs and wait, and a launch on another stream whose
// own blocks wait for one another, NCCL's say, may have the others and wait for these.)
template<auto Kernel>
int launch_cooperative(dim3 grid, dim3 block, void** params, size_t smem, cudaStream_t s, const char* what) {
    static std::atomic<int> pdl{-1};           // for this kernel: the attribute is in use (1), was refused by the driver (0), has not been tried (-1)
    const void* const kernel = (const void*) Kernel;
    if (pdl.load() != 0) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = grid;
        cfg.blockDim = block;
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        cudaLaunchAttribute at[2];
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
        at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = 2;
        const cudaError_t e = cudaLaunchKernelExC(&cfg, kernel, params);
        if (e == cudaSuccess) { pdl.store(1); return note_launch(what); }
        // only "this attribute / combination is not supported" turns the attribute off; any other failure is the launch's
        if (e != cudaErrorNotSupported && e != cudaErrorInvalidValue) return note_launch(what);
        cudaGetLastError();
        pdl.store(0);
    }
    cudaLaunchCooperativeKernel(kernel, grid, block, params, smem, s);
    return note_launch(what);
}

}  // namespace
}  // namespace maya
