// Warp-level tensor-core and async-copy helpers (mma.sync m16n8k16 bfloat16, ldmatrix, cp.async).
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

namespace hb {

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool pred) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  const int bytes = pred ? 16 : 0;   // src-size 0: the 16 bytes are filled with zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}
__device__ __forceinline__ void ldmatrix_x4(unsigned (&r)[4], const void* smem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(s));
}
__device__ __forceinline__ void ldmatrix_x4_trans(unsigned (&r)[4], const void* smem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(s));
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<unsigned*>(&v);
}
// the same held to bfloat16's largest finite value (a NaN stays one)
__device__ __forceinline__ unsigned pack_bf16_sat(float lo, float hi) {
  unsigned r;
  asm("cvt.rn.satfinite.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// Two floats as three pairs of bfloat16 that sum to them exactly (8 + 8 + 8 bits): the six products of pieces down to
// 2^-24 of the whole, on the tensor cores with float32 sums, are a float32 product's. Floats above bfloat16's largest value
// (3.39e38) would round to infinity: the first piece stops at that value and the other two hold the rest, so any finite
// float has finite pieces. Of what is not finite at least one piece is NaN, and so is every product of it.
__device__ __forceinline__ void split3(float x, float y, unsigned (&p)[3]) {
  p[0] = pack_bf16_sat(x, y);
  x -= __uint_as_float(p[0] << 16);
  y -= __uint_as_float(p[0] & 0xffff0000u);
  p[1] = pack_bf16(x, y);
  x -= __uint_as_float(p[1] << 16);
  y -= __uint_as_float(p[1] & 0xffff0000u);
  p[2] = pack_bf16(x, y);
}

}  // namespace hb
