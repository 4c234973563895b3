// float32 products on the warp-level tensor cores: tf32 operands, one product (operands cut to 11 significant bits) or
// three (float32 precision); prefix sums of the log decay shared by the kernels built on them.
//
// mma.sync m16n8k8 tf32 runs 512 multiply-adds per clock and SM (measured: 8 cycles per instruction and scheduler), so
// three products leave 170 float32-precision multiply-adds per clock, against 128 on the CUDA cores, without their
// shared-memory fetch per multiply-add.
#pragma once

#include <stdint.h>

namespace dr {
namespace mma {

__device__ __forceinline__ void tf32(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// One operand of a tf32 product; X3: as hi + lo, hi = x rounded to tf32's 11 significant bits, lo = x - hi (exact, cut to 11
// bits by the tensor core: 23 bits in all); the product then is hi hi + hi lo + lo hi.
template <bool X3>
struct AFrag {
  uint32_t h[4], l[X3 ? 4 : 1];
  __device__ __forceinline__ void set(float a0, float a1, float a2, float a3) {
    const float a[4] = {a0, a1, a2, a3};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      h[i] = __float_as_uint(a[i]);
      if constexpr (X3) {
        h[i] = (h[i] + 0x1000u) & 0xffffe000u;
        l[i] = __float_as_uint(a[i] - __uint_as_float(h[i]));
      }
    }
  }
};
template <bool X3>
struct BFrag {
  uint32_t h[2], l[X3 ? 2 : 1];
  __device__ __forceinline__ void set(float b0, float b1) {
    h[0] = __float_as_uint(b0); h[1] = __float_as_uint(b1);
    if constexpr (X3) {
      h[0] = (h[0] + 0x1000u) & 0xffffe000u;
      h[1] = (h[1] + 0x1000u) & 0xffffe000u;
      l[0] = __float_as_uint(b0 - __uint_as_float(h[0]));
      l[1] = __float_as_uint(b1 - __uint_as_float(h[1]));
    }
  }
};
template <bool X3>
__device__ __forceinline__ void fma(float (&d)[4], const AFrag<X3>& a, const BFrag<X3>& b) {
  if constexpr (X3) {
    tf32(d, a.l, b.h);
    tf32(d, a.h, b.l);
  }
  tf32(d, a.h, b.h);
}
// A operand of 16 rows and 8 columns of a float32 array (row-major, row stride 4 mod 32 words: no bank conflicts) in one instruction:
// ldmatrix moves pairs of 16-bit entries, i.e. whole words.  lda_at: the lane's address, to be advanced by columns.
__device__ __forceinline__ uint32_t lda_at(uint32_t base, int ld, int r0, int lane) {
  return base + 4u * (uint32_t)((r0 + (lane & 15)) * ld + (lane >> 4) * 4);
}
template <bool X3>
__device__ __forceinline__ void lda(AFrag<X3>& a, uint32_t addr) {
  uint32_t x[4];
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]) : "r"(addr) : "memory");
  a.set(__uint_as_float(x[0]), __uint_as_float(x[1]), __uint_as_float(x[2]), __uint_as_float(x[3]));
}
// products with one operand that is exact in a single term (a bf16 value)
template <bool X3>
__device__ __forceinline__ void fma_a1(float (&d)[4], const AFrag<false>& a, const BFrag<X3>& b) {
  if constexpr (X3) tf32(d, a.h, b.l);
  tf32(d, a.h, b.h);
}
template <bool X3>
__device__ __forceinline__ void fma_b1(float (&d)[4], const AFrag<X3>& a, const BFrag<false>& b) {
  if constexpr (X3) tf32(d, a.l, b.h);
  tf32(d, a.h, b.h);
}

// In-place inclusive prefix sum over the 64 rows of sG [64][LD] per channel; NTHR threads, `seg`: scratch of
// NTHR / (D / 4) rows of D floats.  Ends with a barrier.
template <int NTHR, int D, int LD = D + 4>
__device__ __forceinline__ void scan_channels(float* sG, float* seg, int tid) {
  constexpr int NSEG = NTHR / (D / 4), R = 64 / NSEG;   // rows per segment
  const int s = tid / (D / 4), c4 = 4 * (tid % (D / 4));
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f), loc[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const float4 x = *reinterpret_cast<const float4*>(sG + (R * s + r) * LD + c4);
    acc.x += x.x; acc.y += x.y; acc.z += x.z; acc.w += x.w;
    loc[r] = acc;
  }
  *reinterpret_cast<float4*>(seg + s * D + c4) = acc;
  __syncthreads();
  float4 pre = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int s2 = 0; s2 < s; ++s2) {
    const float4 x = *reinterpret_cast<const float4*>(seg + s2 * D + c4);
    pre.x += x.x; pre.y += x.y; pre.z += x.z; pre.w += x.w;
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
    *reinterpret_cast<float4*>(sG + (R * s + r) * LD + c4) =
        make_float4(loc[r].x + pre.x, loc[r].y + pre.y, loc[r].z + pre.z, loc[r].w + pre.w);
  __syncthreads();
}
// inclusive sums of 64 scalars, rows lane and lane + 32
__device__ __forceinline__ void scan_scalars(float& lo, float& hi, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const float a = __shfl_up_sync(0xffffffffu, lo, o), b = __shfl_up_sync(0xffffffffu, hi, o);
    if (lane >= o) { lo += a; hi += b; }
  }
  hi += __shfl_sync(0xffffffffu, lo, 31);
}

}  // namespace mma
}  // namespace dr
