// Warp-level products on the tensor cores (mma.sync m16n8k16, bfloat16 operands, float32 sums) for the recurrences that are walked in
// chunks: fragments, swizzled tiles in shared memory, and a float32 number as the sum of three bfloat16 numbers.
//
// Fragments of a lane, with g = lane / 4 and c = lane % 4: A (16 x 16): rows g and g + 8 at k 2c, 2c+1, then the same rows at k 2c+8, 2c+9;
// B (16 x 8): k 2c, 2c+1, then 2c+8, 2c+9, of column g; sums (16 x 8): row g at columns 2c, 2c+1, then row g + 8.
#pragma once

#include "common.cuh"

namespace roost {

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// The same from zero. The tensor cores cut their sums off (towards zero), so a long chain of products onto one sum leans that way: 27 of them left
// outputs five times as far from 64 bits as a chain of FMAs does. A few products from zero whose sum then joins a float32 sum by an addition that
// rounds to nearest do not.
__device__ __forceinline__ void mma_bf16_zero(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}

// Byte offset of 16-byte piece `piece` of row `row` in a tile of rows of ROW_BYTES (a multiple of 128): eight rows' pieces of one column
// fall in different banks.
template <int ROW_BYTES>
__device__ __forceinline__ uint32_t swizzled(int row, int piece) {
  return (uint32_t)(row * ROW_BYTES + ((piece ^ (row & 7)) << 4));
}

__device__ __forceinline__ void copy16_async(uint32_t smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem), "l"(gmem) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }
__device__ __forceinline__ void zero16(uint32_t smem) { asm volatile("st.shared.v4.b32 [%0], {%1,%1,%1,%1};\n" ::"r"(smem), "r"(0) : "memory"); }

// Two float32 numbers as pairs of bfloat16 numbers (the first in the lower half) whose sums they are: each pair takes the leading eight bits
// of what the ones before left over, so nothing of the 24 bits is lost.
__device__ __forceinline__ void split3(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  const uint32_t xb = __float_as_uint(x), yb = __float_as_uint(y);
  hi = __byte_perm(xb, yb, 0x7632);
  const float x1 = x - __uint_as_float(xb & 0xffff0000u), y1 = y - __uint_as_float(yb & 0xffff0000u);
  const uint32_t xb1 = __float_as_uint(x1), yb1 = __float_as_uint(y1);
  mid = __byte_perm(xb1, yb1, 0x7632);
  const float x2 = x1 - __uint_as_float(xb1 & 0xffff0000u), y2 = y1 - __uint_as_float(yb1 & 0xffff0000u);
  lo = __byte_perm(__float_as_uint(x2), __float_as_uint(y2), 0x7632);
}

// The same parts rounded to nearest, for products of two such numbers: what is left out of them (the middle part of one times the last of the other)
// is then a quarter as large and of either sign.
__device__ __forceinline__ void split3_nearest(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  auto pack = [](float u, float v) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(u, v);
    return *reinterpret_cast<const uint32_t*>(&p);
  };
  hi = pack(x, y);
  const float x1 = x - __uint_as_float(hi << 16), y1 = y - __uint_as_float(hi & 0xffff0000u);
  mid = pack(x1, y1);
  lo = pack(x1 - __uint_as_float(mid << 16), y1 - __uint_as_float(mid & 0xffff0000u));
}

}  // namespace roost
