// Warp-level tensor-core building blocks: asynchronous copies into shared memory, ldmatrix, mma.sync.
#pragma once
#include "dtype.cuh"

namespace djv {

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void cp_async16_zfill(uint32_t dst_smem, const void *src, int src_bytes) {
  asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16, %2;" ::"r"(dst_smem), "l"(src), "r"(src_bytes)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
// four 8x8 fp16 matrices: lane (g, t) gets elements [g][2t], [g][2t+1] of each ...
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr_smem) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr_smem)
               : "memory");
}
// ... or, transposed on the way, elements [2t][g], [2t+1][g]
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr_smem) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr_smem)
               : "memory");
}

__device__ __forceinline__ void mma_m16n8k16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                             uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// the same product in the element type of the operands
template <typename T>
__device__ __forceinline__ void mma_m16n8k16_t(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                               uint32_t b0, uint32_t b1);
template <>
__device__ __forceinline__ void mma_m16n8k16_t<__half>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                                       uint32_t a3, uint32_t b0, uint32_t b1) {
  mma_m16n8k16(d, a0, a1, a2, a3, b0, b1);
}
template <>
__device__ __forceinline__ void mma_m16n8k16_t<bf16>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                                     uint32_t a3, uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// acc += s in fp32. The tensor cores cut off what does not fit beside the accumulator that they are given, always towards
// zero, so a long chain of products in one accumulator drifts: a few products start from zero and join the rest here.
__device__ __forceinline__ void add_sums(float (&acc)[4], const float (&s)[4]) {
#pragma unroll
  for (int e = 0; e < 4; ++e) acc[e] += s[e];
}

}  // namespace djv
