// Shared by the recurrences that run over chunks of tokens on the tensor cores
// (lightning.cu, decay_chunks.cu, delta_chunks.cu): matrix fragments from shared memory, the
// product of a warp, and 32-bit numbers as sums of bfloat16 parts.
#pragma once

#include "common.cuh"

namespace le {

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const __nv_bfloat16 *p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_addr(p)));
}
__device__ __forceinline__ void ldsm4_trans(uint32_t (&r)[4], const __nv_bfloat16 *p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_addr(p)));
}
// d += a b of one warp: a 16 x 16, b 16 x 8, bfloat16 in, 32-bit sums.
__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// d = a b: the first product of a sum.
__device__ __forceinline__ void mma_first(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
}
__device__ __forceinline__ void add4(float (&d)[4], const float (&x)[4]) {
  d[0] += x[0], d[1] += x[1], d[2] += x[2], d[3] += x[3];
}
// d += (a[0] + a[1] + a[2]) b with a in three parts, largest first.  The tensor cores cut the sums they add a product
// to (they do not round to the nearest), so a long chain of products into one accumulator leans towards zero; the
// three parts' products meet in an accumulator of their own, smallest first, and join `d` by a rounded addition.
__device__ __forceinline__ void mma_split3(float (&d)[4], const uint32_t (&a)[3][4], uint32_t b0, uint32_t b1) {
  float x[4];
  mma_first(x, a[2], b0, b1);
  mma(x, a[1], b0, b1);
  mma(x, a[0], b0, b1);
  add4(d, x);
}
// Two floats as two bfloat16 pairs whose sum keeps 16 bits of each.
__device__ __forceinline__ void split_pair(float x, float y, uint32_t &high, uint32_t &low) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
  const __nv_bfloat162 l = __floats2bfloat162_rn(x - __low2float(h), y - __high2float(h));
  high = *reinterpret_cast<const uint32_t *>(&h);
  low = *reinterpret_cast<const uint32_t *>(&l);
}
__device__ __forceinline__ float low_of(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float high_of(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }
// Two floats as three bfloat16 pairs whose sum is all 24 bits of each (down to the smallest bfloat16).
__device__ __forceinline__ void split_pair3(float x, float y, uint32_t &high, uint32_t &mid, uint32_t &low) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
  high = *reinterpret_cast<const uint32_t *>(&h);
  split_pair(x - low_of(high), y - high_of(high), mid, low);
}
// The same for a state, which may have overflown: an infinity is its first part, and the others are finite (inf - inf would
// make the sum NaN; the minimum takes the bound, which lies above all rests).  What is within 2^-9 of the largest number
// counts as overflown.
__device__ __forceinline__ void split_state3(float x, float y, uint32_t &high, uint32_t &mid, uint32_t &low) {
  constexpr float BOUND = 5.3e36f;         // 2^122
  const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
  high = *reinterpret_cast<const uint32_t *>(&h);
  split_pair(fminf(x - low_of(high), BOUND), fminf(y - high_of(high), BOUND), mid, low);
}
__device__ __forceinline__ void copy16_async(void *dst, const void *src, bool live) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_addr(dst)), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void commit_copies() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void wait_for_copies() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

}  // namespace le
