// Warp-level tensor-core pieces shared by the chunked scans: ldmatrix, bf16 mma.sync, and float32 operands as sums of
// three bf16 numbers.
//
// A float32 x is x1 + x2 + x3 with x1 = bf16(x), x2 = bf16(x - x1), x3 = bf16(x - x1 - x2): 24 significant bits, all
// of float32's.  A product of such an operand with an exact bf16 one is three bf16 products accumulated in float32; of
// two such operands six (the three terms below 2^-24 are dropped).  That keeps float32 precision on the bf16 tensor
// pipe: mma.sync m16n8k16 bf16 runs 1024 multiply-adds per clock and SM (measured), 340 or 170 of them float32-exact,
// against 128 on the CUDA cores.
#pragma once

#include <cuda_bf16.h>
#include <stdint.h>

namespace dr {
namespace mma {

__device__ __forceinline__ void bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
// Addresses for the fragments of a row-major bf16 array in shared memory (row stride `ld` elements, a multiple of 8
// whose 16-byte count is odd, so that the eight rows of a matrix start on distinct banks); r0, c0: corner of the block.
//   frag_a:  16 x 16 block as an A operand (m = row, k = column), with ldsm4
//   frag_at: 16 x 16 block as an A operand with m = column, k = row, with ldsm4t
//   frag_b:  16 rows x 16 columns as B operands with n = row, k = column, with ldsm4: {r0,r1} rows 0-7, {r2,r3} rows 8-15
//   frag_bt: the same with k = row, n = column, with ldsm4t: {r0,r1} columns 0-7, {r2,r3} columns 8-15
__device__ __forceinline__ uint32_t frag_a(uint32_t base, int ld, int r0, int c0, int lane) {
  return base + 2u * (uint32_t)((r0 + (lane & 15)) * ld + c0 + (lane >> 4) * 8);
}
__device__ __forceinline__ uint32_t frag_at(uint32_t base, int ld, int r0, int c0, int lane) {
  return base + 2u * (uint32_t)((r0 + (lane & 7) + (lane >> 4) * 8) * ld + c0 + ((lane >> 3) & 1) * 8);
}
__device__ __forceinline__ uint32_t frag_b(uint32_t base, int ld, int r0, int c0, int lane) {
  return base + 2u * (uint32_t)((r0 + (lane & 7) + (lane >> 4) * 8) * ld + c0 + ((lane >> 3) & 1) * 8);
}
__device__ __forceinline__ uint32_t frag_bt(uint32_t base, int ld, int r0, int c0, int lane) {
  return base + 2u * (uint32_t)((r0 + (lane & 15)) * ld + c0 + (lane >> 4) * 8);
}

__device__ __forceinline__ uint32_t pack(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ float lo_f(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float hi_f(uint32_t u) { return __uint_as_float(u & 0xffff0000u); }
// a pair of floats as three packed bf16 pairs
__device__ __forceinline__ void split3(float x, float y, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
  p1 = pack(x, y);
  x -= lo_f(p1); y -= hi_f(p1);
  p2 = pack(x, y);
  x -= lo_f(p2); y -= hi_f(p2);
  p3 = pack(x, y);
}

// The same by truncation: 8 + 8 + 8 bits, so the three terms add up to the float exactly (rounding needs the terms' signs for
// that); eleven instructions either way, these without a conversion.  Infinities come out as inf, NaN, NaN.
__device__ __forceinline__ void split3_exact(float x, float y, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
  uint32_t a = __float_as_uint(x), b = __float_as_uint(y);
  p1 = __byte_perm(a, b, 0x7632);
  x -= __uint_as_float(a & 0xffff0000u); y -= __uint_as_float(b & 0xffff0000u);
  a = __float_as_uint(x); b = __float_as_uint(y);
  p2 = __byte_perm(a, b, 0x7632);
  x -= __uint_as_float(a & 0xffff0000u); y -= __uint_as_float(b & 0xffff0000u);
  p3 = __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
}

}  // namespace mma
}  // namespace dr
