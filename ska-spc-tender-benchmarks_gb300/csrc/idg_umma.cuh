// idg_umma.cuh -- tcgen05 building blocks: tensor memory, fp16 matrix
// multiply-accumulate with the A operand in tensor memory, descriptors.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "idg_ptx.cuh"

namespace idg {

// Tensor memory: 128 lanes x 512 columns of 32 bits per SM.  One warp allocates
// (the address lands in shared memory) and the same warp frees.
__device__ __forceinline__ void tmem_alloc(uint32_t *slot, uint32_t columns) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(slot)), "r"(columns)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t addr, uint32_t columns) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr), "r"(columns) : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Instruction descriptor of kind::f16: fp16 x fp16 -> fp32, A and B K-major.
__host__ __device__ constexpr uint32_t umma_idesc_f16(int M, int N) {
    return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
constexpr uint32_t kUmmaNegateA = 1u << 13; // or-ed in: D -= A B
// One lane of a converged warp, the same one on every call: 1 there, 0 elsewhere.
__device__ __forceinline__ uint32_t elect_lane() {
    uint32_t r;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(r));
    return r;
}
// Shared-memory descriptor, no swizzle, K-major: 8 x 16-byte core matrices of
// 128 contiguous bytes; `k_stride` bytes between core matrices along K and
// `mn_stride` bytes between groups of eight rows.  Upper and lower half.
__host__ __device__ constexpr uint32_t umma_desc_hi(uint32_t mn_stride) {
    return ((mn_stride >> 4) & 0x3fffu) | (1u << 14);
}
__device__ __forceinline__ uint32_t umma_desc_lo(uint32_t addr, uint32_t k_stride) {
    return ((addr >> 4) & 0x3fffu) | ((k_stride >> 4) << 16);
}
// A value that is the same in every lane, for the compiler to see as such.
__device__ __forceinline__ uint32_t warp_uniform(uint32_t v) { return __shfl_sync(0xffffffffu, v, 0); }
// D[tmem] (+)= A[tmem] B[smem]; one thread issues.  Operands that are uniform
// over its warp and constant descriptor parts keep this to a few instructions; a
// loop on run-time descriptors took 126 cycles per product (the tensor core
// needs 32 for N = 64).
template <bool ACC, uint32_t IDESC, uint32_t DESC_HI>
__device__ __forceinline__ void umma_f16_ts(uint32_t d, uint32_t a, uint32_t b_lo) {
    asm volatile(
        "{\n .reg .pred p;\n .reg .b64 b;\n setp.ne.u32 p, %3, 0;\n mov.b64 b, {%2, %5};\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %4, p;\n}\n" ::"r"(d),
        "r"(a), "r"(b_lo), "n"(ACC ? 1 : 0), "r"(IDESC), "r"(DESC_HI)
        : "memory");
}
// The same with the choice at run time.
template <uint32_t IDESC, uint32_t DESC_HI>
__device__ __forceinline__ void umma_f16_ts_if(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t acc) {
    asm volatile(
        "{\n .reg .pred p;\n .reg .b64 b;\n setp.ne.u32 p, %3, 0;\n mov.b64 b, {%2, %5};\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %4, p;\n}\n" ::"r"(d),
        "r"(a), "r"(b_lo), "r"(acc), "r"(IDESC), "r"(DESC_HI)
        : "memory");
}
// The mbarrier completes a phase when every MMA issued so far by this thread has finished.
__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
                 : "memory");
}

// One warp's 32 lanes x 4 / 16 columns between registers and tensor memory
// (thread i of the warp <-> lane 32 * (warp % 4) + i; `addr` names that lane
// quarter's first lane).  Volatile keeps these in order with the waits and
// fences around them; they name no memory, so ordinary loads and stores may
// move past them.
__device__ __forceinline__ void tmem_st4(uint32_t addr, const uint32_t (&r)[4]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(r[0]), "r"(r[1]),
                 "r"(r[2]), "r"(r[3]));
}
// 16 columns, arrived when this returns.
__device__ __forceinline__ void tmem_ld16(uint32_t addr, f2 (&v)[8]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];\n"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr));
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = (f2)r[2 * i] | ((f2)r[2 * i + 1] << 32);
}
// Two runs of 16 columns, arrived when this returns (the wait is part of the
// statement, so nothing that uses the registers can move before it).
__device__ __forceinline__ void tmem_ld16x2(uint32_t a0, uint32_t a1, f2 (&v)[8], f2 (&w)[8]) {
    uint32_t r[16], q[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%32];\n"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, "
        "%29, %30, %31}, [%33];\n"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(q[0]),
          "=r"(q[1]), "=r"(q[2]), "=r"(q[3]), "=r"(q[4]), "=r"(q[5]), "=r"(q[6]), "=r"(q[7]), "=r"(q[8]), "=r"(q[9]),
          "=r"(q[10]), "=r"(q[11]), "=r"(q[12]), "=r"(q[13]), "=r"(q[14]), "=r"(q[15])
        : "r"(a0), "r"(a1));
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        v[i] = (f2)r[2 * i] | ((f2)r[2 * i + 1] << 32);
        w[i] = (f2)q[2 * i] | ((f2)q[2 * i + 1] << 32);
    }
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

} // namespace idg
