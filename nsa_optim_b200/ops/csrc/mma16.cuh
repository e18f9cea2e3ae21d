// Warp-level bf16 matrix products (mma.sync m16n8k16, fp32 accumulation) on padded shared-memory tiles.
//
// For per-chunk products of 64-row tiles, of which a tcgen05 tile of 128 rows would be half empty.  The kernels that use
// them are chains of dependent phases with products of a few thousand cycles at most between them; accumulators in
// registers go straight into the next phase's arithmetic, without a trip through tensor memory.
// Tiles are row-major with a pitch that is an odd multiple of 16 bytes, so ldmatrix is free of bank conflicts.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

namespace mma16 {
typedef __nv_bfloat16 bf16;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const bf16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_addr(p)) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], const bf16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_addr(p)) : "memory");
}
// A fragment of rows m0.., columns k0..:  from a tile stored [m][k] / [k][m].
__device__ __forceinline__ void load_a(uint32_t (&r)[4], const bf16* tile, int pitch, int m0, int k0) {
  const int l = threadIdx.x & 31;
  ldsm4(r, tile + (m0 + (l & 15)) * pitch + k0 + (l >> 4) * 8);
}
__device__ __forceinline__ void load_a_t(uint32_t (&r)[4], const bf16* tile, int pitch, int m0, int k0) {
  const int l = threadIdx.x & 31, i = l >> 3;
  ldsm4_t(r, tile + (k0 + (i >> 1) * 8 + (l & 7)) * pitch + m0 + (i & 1) * 8);
}
// B fragments of 16 columns n0.. (registers 0-1: the first eight, 2-3: the next), reduction k0..:
// from a tile stored [n][k] / [k][n].
__device__ __forceinline__ void load_b(uint32_t (&r)[4], const bf16* tile, int pitch, int n0, int k0) {
  const int l = threadIdx.x & 31, i = l >> 3;
  ldsm4(r, tile + (n0 + (i >> 1) * 8 + (l & 7)) * pitch + k0 + (i & 1) * 8);
}
__device__ __forceinline__ void load_b_t(uint32_t (&r)[4], const bf16* tile, int pitch, int n0, int k0) {
  const int l = threadIdx.x & 31, i = l >> 3;
  ldsm4_t(r, tile + (k0 + (i & 1) * 8 + (l & 7)) * pitch + n0 + (i >> 1) * 8);
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Two accumulators (16 columns) from one B fragment pair.
__device__ __forceinline__ void mma2(float (&c0)[4], float (&c1)[4], const uint32_t (&a)[4], const uint32_t (&b)[4]) {
  mma(c0, a, b[0], b[1]);
  mma(c1, a, b[2], b[3]);
}
// Accumulator element e of a lane: row (lane >> 2) + 8 * (e >> 1), column 2 * (lane & 3) + (e & 1).
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool pred) {   // zero fill when !pred
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(smem)), "l"(gmem), "r"(pred ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
}  // namespace mma16
