// maya_tcgen05.cuh - thin wrappers over the Blackwell tensor-core instructions used by the prefill GEMM: tensor
// memory allocation, tcgen05.mma (kind::f16, operands in shared memory), tcgen05.commit onto an mbarrier, tcgen05.ld.
//
// Shared-memory operand layout used here (K-major, no swizzle): an operand tile of R rows x 64 K-values of f16 is
// stored as 8 "K chunks" of 8 values (16 bytes): byte offset of (row r, chunk c) = c * (R * 16) + r * 16.  The 8 x 16-byte
// core matrices the tensor core reads are then contiguous 128-byte pieces: consecutive 8-row groups are 128 bytes
// apart (stride byte offset) and the two chunks one K = 16 instruction reads are R * 16 bytes apart (leading byte offset).
#pragma once

#include "maya_stream.cuh"

namespace maya {

__device__ __forceinline__ void tmem_alloc(uint32_t* smem_dst, uint32_t ncols) {   // one whole warp
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {      // the same warp
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// the same for 16 and for 8 consecutive columns
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

// matrix descriptor of a K-major operand in the 128-byte swizzle layout (rows of 64 f16 = 128 bytes, 8-row groups 1024
// bytes apart, 16-byte chunks XOR-ed with the row number modulo 8 - what a TMA load with CU_TENSOR_MAP_SWIZZLE_128B
// writes).  The tile must start on a 1024-byte boundary; a K = 16 step further along the row is +32 bytes on `addr`.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr) {
    return (uint64_t) ((addr & 0x3FFFFu) >> 4) | (1ull << 16) | ((uint64_t) (1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// Tiled TMA load of a 3-d box (plain: this block only, no multicast) from the tensor described by `map` (a CUtensorMap in
// kernel-parameter or global memory) into shared memory; `bytes` are expected on `bar`, where completion is counted.
// c0 * element size must be a multiple of 16 bytes.  Called by a converged warp with warp-uniform operands, one elected lane
// copies: the operands stay in the uniform registers that the copy wants (a lane of its own in a divergent branch took 400 to 500
// cycles a tile).
__device__ __forceinline__ void tma_expect_load_3d(uint32_t dst_smem, const void* map, uint32_t bar, uint32_t bytes, int c0, int c1, int c2) {
    __syncwarp();
    asm volatile(
        "{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
        "@e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%2], %6;\n\t"
        "@e cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n\t}"
        ::"r"(dst_smem), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(bytes)
        : "memory");
}
__device__ __forceinline__ void tma_expect_load_2d(uint32_t dst_smem, const void* map, uint32_t bar, uint32_t bytes, int c0, int c1) {
    __syncwarp();
    asm volatile(
        "{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
        "@e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%2], %5;\n\t"
        "@e cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n\t}"
        ::"r"(dst_smem), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(bytes)
        : "memory");
}
// the same without the expectation, for a second box on the same barrier
__device__ __forceinline__ void tma_load_2d_elect(uint32_t dst_smem, const void* map, uint32_t bar, int c0, int c1) {
    __syncwarp();
    asm volatile(
        "{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
        "@e cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n\t}"
        ::"r"(dst_smem), "l"(map), "r"(bar), "r"(c0), "r"(c1)
        : "memory");
}
// shared -> global bulk copy (16-byte aligned, size % 16 == 0), tracked by this thread's bulk groups
__device__ __forceinline__ void bulk_store(void* dst_gmem, const void* src_smem, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst_gmem), "r"(smem_u32(src_smem)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template<int N> __device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void named_bar_sync(int id, int nthreads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory"); }
// the same, with the OR over the threads of a condition as its result in every one of them
__device__ __forceinline__ bool named_bar_or(int id, int nthreads, bool cond) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %3, 0;\n\tbar.red.or.pred p, %1, %2, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(r) : "r"(id), "r"(nthreads), "r"((uint32_t) cond) : "memory");
    return r != 0;
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_arrive_addr(uint32_t bar_smem) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_smem) : "memory");
}

// The products of 64 K-values (four K = 16 steps) into one accumulator and the commit that follows them, issued by one elected
// lane of a CONVERGED warp.  Every operand must be warp-uniform and the caller's control flow too: then the operands live in
// uniform registers, where the instruction wants them.  The four B descriptors are the address word `b_lo`, + 2 per step (32
// bytes inside the 128-byte swizzle row), under the constant upper word `b_hi`; the A column advances 8 per step.
// `first` = 0 makes the first product overwrite the accumulator.
__device__ __forceinline__ void mma_f16_ts_x4_commit(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                                     uint32_t first, uint32_t bar_smem) {
    asm volatile(
        "{\n\t.reg .pred e, p, t;\n\t.reg .b32 a1, a2, a3, b1, b2, b3;\n\t.reg .b64 d0, d1, d2, d3;\n\t"
        "setp.ne.b32 p, %5, 0;\n\tsetp.eq.b32 t, 0, 0;\n\t"
        "add.u32 a1, %1, 8;\n\tadd.u32 a2, %1, 16;\n\tadd.u32 a3, %1, 24;\n\t"
        "add.u32 b1, %2, 2;\n\tadd.u32 b2, %2, 4;\n\tadd.u32 b3, %2, 6;\n\t"
        "mov.b64 d0, {%2, %3};\n\tmov.b64 d1, {b1, %3};\n\tmov.b64 d2, {b2, %3};\n\tmov.b64 d3, {b3, %3};\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], d0, %4, p;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a1], d1, %4, t;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a2], d2, %4, t;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [a3], d3, %4, t;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%6];\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(first), "r"(bar_smem)
        : "memory");
}
// one look at the barrier at shared address `bar_smem`
__device__ __forceinline__ bool mbar_test_wait_addr(uint32_t bar_smem, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar_smem), "r"(parity)
        : "memory");
    return ok != 0;
}
// 16 consecutive 32-bit columns of this thread's lane (lane = 32 * (warp % 4) + lane id): register j -> column + j
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
          "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
          "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
          "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// arrive on `bar` when every tcgen05.mma the elected lane of this (converged) warp issued so far has completed
__device__ __forceinline__ void mma_commit_elect(uint32_t bar_smem) {
    asm volatile(
        "{\n\t.reg .pred e;\n\telect.sync _|e, 0xffffffff;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar_smem) : "memory");
}

}  // namespace maya
