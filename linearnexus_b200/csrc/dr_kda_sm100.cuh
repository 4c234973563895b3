// Chunkwise forward with PER-CHANNEL decay (KDA) for Blackwell, as two kernels:
//
//   (1) intra_kernel   all chunks in parallel, persistent CTAs: everything that does not
//                      depend on the running state.  Cumulative log decay G, the decayed chunk-local
//                      products A_kk, A_qk, the unit-lower inverse T = (I + diag(beta) A_kk)^-1 and the
//                      bf16 operand tiles of the state pass, written to a workspace record per chunk in
//                      exactly the swizzled order the tensor cores read, so that the state kernel
//                      fetches each tile with ONE 1-d bulk copy (no tensor map).
//   (2) state_kernel   one CTA per sequence walks the chunks; the fp32 state lives transposed in tensor
//                      memory (lane = value column) and every product is a tcgen05.mma:
//                          U^T      = V^T (T diag(beta))^T                   128x64x64   smem x smem
//                          Vn^T     = U^T - S^T W^T                          128x64x128  tmem x smem
//                          Dq       = S^T Qg^T                               128x64x128
//                          Do       = Vn^T A_qk^T                            128x64x64
//                          S^T      = S^T diag(e^{G_L}) + Vn^T Kd            128x128x64
//                      with W = T diag(beta) (k^ e^G), Qg = scale q^ e^G, Kd = k^ e^{G_L - G}.
//
// Per-channel decay cannot be folded into row/column factors of a plain K K^T product the way a scalar
// decay can, and e^{-G} alone overflows for strong decay.  A chunk that decays by at most 2^64 takes one product of decayed rows (see
// intra_kernel); for the others the chunk-local products use 16-row
// sub-blocks: rows of sub-block bi against earlier columns are the bf16 tensor-core product of
// x_i e^{G_i - G_n}  and  k_j e^{G_n - G_j}  with n the first row of bi, so both exponents are <= 0; the four diagonal
// 16x16 blocks use the same form while their decay range stays below 2^64 and are summed exactly in fp32 otherwise.
//
// Shape: K = V = 128, chunk 64, bf16 q/k/v, g bf16 or fp32 ([.., K] for KDA; the scalar-decay and
// decay-free variants are served too, by broadcasting), fp32 beta/state, bf16 or fp32 output.
#pragma once

#include <algorithm>

#include "dr_chunk_sm100.cuh"
#include "dr_launch.h"
#include "dr_mma.cuh"

namespace dr {
namespace kda {

using sm100::LDT;

constexpr int kC = 64, kD = 128;
constexpr int kThreads = 256;

// workspace record of one chunk (bytes); tiles in the 128-byte swizzle, panels of 64 columns one after the other
constexpr int WS_W = 0;                    // W^T [128][64] bf16
constexpr int WS_QG = WS_W + 16384;        // Qg  [64][128] bf16
constexpr int WS_KD = WS_QG + 16384;       // Kd  [64][128] bf16
constexpr int WS_TB = WS_KD + 16384;       // T diag(beta) [64][64] bf16
constexpr int WS_AQK = WS_TB + 8192;       // A_qk         [64][64] bf16
constexpr int WS_EGL = WS_AQK + 8192;      // e^{G_L}[128] fp32
constexpr int WS_REC = WS_EGL + 512;       // 66048

// What callers are asked for per record: the size the ABI has announced from the start (records once carried V, too).
constexpr int WS_ASKED = 82432;
static_assert(WS_REC <= WS_ASKED, "records fit what callers provide");
inline int64_t workspace_bytes(int64_t units, int T) { return units * ((T + kC - 1) / kC) * (int64_t)WS_ASKED; }

// ---- the general products, for chunks past the line -----------------------------------------------------------------
// The inputs lie as raw bf16 with their l2-norm factors on the side, and the decayed bf16 operands of the tensor-core products are formed in
// registers from them (no scaled copies in shared memory).
constexpr int LDF = 136;   // row stride (floats) of G: the products read pairs of eight rows without bank conflicts
constexpr int LDH = 136;   // row stride (bf16) of the raw q, k rows and of the W staging tile
constexpr int LDQ = 72;    // row stride (bf16) of A_qk
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float2 bf2(uint32_t u) {
  return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u));
}

// two bf16 products in one instruction (operands and result packed in 32 bits)
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
  uint32_t d;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}

// packed pairs: one instruction per two products
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 d;
  asm("mul.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)));
  return d;
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  float2 d;
  asm("fma.rn.f32x2 %0, %2, %3, %1;"
      : "=l"(reinterpret_cast<unsigned long long&>(d))
      : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)),
        "l"(0xbf800000bf800000ull));
  return d;
}
__device__ __forceinline__ float2 ex2x2(float2 a) { return make_float2(ex2(a.x), ex2(a.y)); }

// four consecutive elements starting at element index i (a multiple of 4)
__device__ __forceinline__ void ld4(const void* p, int64_t i, int dt, float (&x)[4]) {
  if (dt == DR_BF16) {
    const uint2 u = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(p) + i);
    const float2 a = bf2(u.x), b = bf2(u.y);
    x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
  } else {
    const float4 f = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p) + i);
    x[0] = f.x; x[1] = f.y; x[2] = f.z; x[3] = f.w;
  }
}

// 16-byte piece number `piece` of a [64][64] tile in core-matrix order -> (row, first column)
__device__ __forceinline__ void piece64(int piece, int& row, int& col) {
  row = (piece >> 6) * 8 + (piece & 7);
  col = ((piece >> 3) & 7) * 8;
}

// Kernel parameters of the intra pass; a packed batch adds the table of its sequences (p then describes the packed
// arrays: B = 1, T = all tokens, token-major).
struct IntraParams {
  CUtensorMap tq, tk, tg;   // panels of q and k; g as boxes of 64 rows
  FwdParams p;
  WideMarks marks;
  uint8_t* ws;
  int chunks, use_tma;
};
struct IntraPackedParams : IntraParams {
  SeqTable seqs;
};
// The pass in transition form (see "few sequences" below): fragments instead of records.
struct IntraTransParams {
  CUtensorMap tq, tk, tv, tg;   // panels of q, k and v; g as boxes of 64 rows
  FwdParams p;
  uint4 *nf, *yf;     // [chunks][8 | 4 row tiles][8 k-steps][32 lanes]: A operands of m16n8k16
  float4 *zf, *of;    // [chunks][8 | 4 row tiles][16 column tiles][32 lanes]: addends
  float* el;          // [chunks][128] e^{G_L}
  int64_t chunks;
};

// eight channels of one row: scale q^ e^G, k^ e^{G_L - G}, k^ e^G (G of the row and of the chunk's last row in log2 units)
__device__ __forceinline__ void decayed_piece(const float* gr, const float* gl, uint4 q, uint4 k, float rq, float rk,
                                              uint4& qg, uint4& kd, uint4& kg) {
  float4 g4[2], l4[2];
  g4[0] = *reinterpret_cast<const float4*>(gr); g4[1] = *reinterpret_cast<const float4*>(gr + 4);
  l4[0] = *reinterpret_cast<const float4*>(gl); l4[1] = *reinterpret_cast<const float4*>(gl + 4);
  const float2 q2 = make_float2(rq, rq), k2 = make_float2(rk, rk);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 gg = reinterpret_cast<const float2*>(g4)[e], ll = reinterpret_cast<const float2*>(l4)[e];
    const float2 eg = ex2x2(gg), kk = mul2(bf2(reinterpret_cast<const uint32_t*>(&k)[e]), k2);
    const float2 x = mul2(mul2(bf2(reinterpret_cast<const uint32_t*>(&q)[e]), q2), eg), y = mul2(kk, ex2x2(sub2(ll, gg))), z = mul2(kk, eg);
    reinterpret_cast<uint32_t*>(&qg)[e] = tc::pack_bf16(x.x, x.y);
    reinterpret_cast<uint32_t*>(&kd)[e] = tc::pack_bf16(y.x, y.y);
    reinterpret_cast<uint32_t*>(&kg)[e] = tc::pack_bf16(z.x, z.y);
  }
}

// The chunk-local products for any decay: A_kk (below the diagonal) and A_qk (bf16; above the diagonal of its 16-row blocks scratch) from G
// and the raw rows.  256 threads (named barrier 1); G, rows and norm factors in shared memory behind a barrier; ends with one.
__device__ __forceinline__ void general_products(const float* sG, const __nv_bfloat16* sK, const __nv_bfloat16* sQ, float* sAkk, float* sT,
                                                 __nv_bfloat16* sAqk, const float* sRk, const float* sRq, int tid) {
  const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  // ---- chunk-local products on mma.sync (bf16) -------------------------------------------------------------------
  // Rows of sub-block bi against the columns of blocks 0..bi; operands  x_i e^{G_i - G_n}  and  k_j e^{G_n - G_j}
  // (n = first row of bi) are formed in registers; the k and q rows share their decay factors and the column
  // operand.  For columns of EARLIER blocks both exponents are <= 0.  For the columns of bi itself the second
  // exponent is positive, at most the decay accumulated over the block; when that exceeds 2^64 in some channel
  // (never with trained gates, but legal input) the block is redone exactly below.
  // Eight warp tasks: (bi; 8-column tiles)  3;0-2  3;3-5  3;6-7  2;0-2  2;3-5  1;0-1  1;2-3  0;0-1
  auto block_unsafe = [&](int blk) -> bool {   // warp-uniform
    const float4 ga = *reinterpret_cast<const float4*>(sG + (16 * blk) * LDF + 4 * lane);
    const float4 gb = *reinterpret_cast<const float4*>(sG + (16 * blk + 15) * LDF + 4 * lane);
    float m = fmaxf(fmaxf(ga.x - gb.x, ga.y - gb.y), fmaxf(ga.z - gb.z, ga.w - gb.w));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    return !(m <= 64.f);
  };
  {
    const int bi = warp < 3 ? 3 : warp < 5 ? 2 : warp < 7 ? 1 : 0;
    const int nt0 = warp < 3 ? 3 * warp : warp < 5 ? 3 * (warp - 3) : warp < 7 ? 2 * (warp - 5) : 0;
    const int ntn = (warp == 2 || warp >= 5) ? 2 : 3;
    const bool skip_diag = block_unsafe(bi);
    const int r0 = 16 * bi + g, r1 = r0 + 8, nrow = 16 * bi;
    float dk[3][4], dq[3][4];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      dk[i][0] = dk[i][1] = dk[i][2] = dk[i][3] = 0.f;
      dq[i][0] = dq[i][1] = dq[i][2] = dq[i][3] = 0.f;
    }
#pragma unroll 2
    for (int ks = 0; ks < 8; ++ks) {
      const int k0 = ks * 16 + 2 * t;
      const float2 gn0 = *reinterpret_cast<const float2*>(sG + nrow * LDF + k0);
      const float2 gn1 = *reinterpret_cast<const float2*>(sG + nrow * LDF + k0 + 8);
      uint32_t ak[4], aq[4];
      {
        const float2 ga = *reinterpret_cast<const float2*>(sG + r0 * LDF + k0);
        const float2 gb = *reinterpret_cast<const float2*>(sG + r1 * LDF + k0);
        const float2 gc = *reinterpret_cast<const float2*>(sG + r0 * LDF + k0 + 8);
        const float2 gd = *reinterpret_cast<const float2*>(sG + r1 * LDF + k0 + 8);
        // decay factors as bf16 pairs, shared by the k and the q row; the products are packed bf16 multiplies (the
        // operands of the tensor-core product are bf16 either way: one rounding of the factor, one of the product)
        const uint32_t ea = tc::pack_bf16(ex2(ga.x - gn0.x), ex2(ga.y - gn0.y)), eb = tc::pack_bf16(ex2(gb.x - gn0.x), ex2(gb.y - gn0.y));
        const uint32_t ec = tc::pack_bf16(ex2(gc.x - gn1.x), ex2(gc.y - gn1.y)), ed = tc::pack_bf16(ex2(gd.x - gn1.x), ex2(gd.y - gn1.y));
        ak[0] = mul_bf16x2(*reinterpret_cast<const uint32_t*>(sK + r0 * LDH + k0), ea);
        ak[1] = mul_bf16x2(*reinterpret_cast<const uint32_t*>(sK + r1 * LDH + k0), eb);
        ak[2] = mul_bf16x2(*reinterpret_cast<const uint32_t*>(sK + r0 * LDH + k0 + 8), ec);
        ak[3] = mul_bf16x2(*reinterpret_cast<const uint32_t*>(sK + r1 * LDH + k0 + 8), ed);
        aq[0] = mul_bf16x2(*reinterpret_cast<const uint32_t*>(sQ + r0 * LDH + k0), ea);
        aq[1] = mul_bf16x2(*reinterpret_cast<const uint32_t*>(sQ + r1 * LDH + k0), eb);
        aq[2] = mul_bf16x2(*reinterpret_cast<const uint32_t*>(sQ + r0 * LDH + k0 + 8), ec);
        aq[3] = mul_bf16x2(*reinterpret_cast<const uint32_t*>(sQ + r1 * LDH + k0 + 8), ed);
      }
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        if (i < ntn && !(skip_diag && nt0 + i >= 2 * bi)) {
          const int j = 8 * (nt0 + i) + g;
          const float2 gj0 = *reinterpret_cast<const float2*>(sG + j * LDF + k0);
          const float2 gj1 = *reinterpret_cast<const float2*>(sG + j * LDF + k0 + 8);
          uint32_t bb[2];
          bb[0] = mul_bf16x2(*reinterpret_cast<const uint32_t*>(sK + j * LDH + k0),
                             tc::pack_bf16(ex2(gn0.x - gj0.x), ex2(gn0.y - gj0.y)));
          bb[1] = mul_bf16x2(*reinterpret_cast<const uint32_t*>(sK + j * LDH + k0 + 8),
                             tc::pack_bf16(ex2(gn1.x - gj1.x), ex2(gn1.y - gj1.y)));
          mma_bf16(dk[i], ak, bb);
          mma_bf16(dq[i], aq, bb);
        }
      }
    }
    const float fk0 = sRk[r0], fk1 = sRk[r1], fq0 = sRq[r0], fq1 = sRq[r1];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      if (i < ntn) {
        const int c = 8 * (nt0 + i) + 2 * t;
        const float c0 = sRk[c], c1 = sRk[c + 1];
        *reinterpret_cast<uint32_t*>(sAqk + r0 * LDQ + c) = tc::pack_bf16(dq[i][0] * fq0 * c0, dq[i][1] * fq0 * c1);
        *reinterpret_cast<uint32_t*>(sAqk + r1 * LDQ + c) = tc::pack_bf16(dq[i][2] * fq1 * c0, dq[i][3] * fq1 * c1);
        *reinterpret_cast<float2*>(sAkk + r0 * LDT + c) = make_float2(dk[i][0] * fk0 * c0, dk[i][1] * fk0 * c1);
        *reinterpret_cast<float2*>(sAkk + r1 * LDT + c) = make_float2(dk[i][2] * fk1 * c0, dk[i][3] * fk1 * c1);
      }
    }
  }
  // ---- diagonal 16x16 blocks exactly (fp32), only for blocks whose decay range is too wide for the product form ----
  // Two warps per block, 64 channels each, two channels per lane; the 16 rows of k and the per-row decay
  // d_r = e^{G_r - G_{r-1}} stay in registers, so e^{G_i - G_j} is a running product (no exponentials per pair).
  // Partial sums of the two channel halves meet in a scratch array (the T array, not yet in use).
  sm100::group_sync(1);   // the tensor-core tasks have written their (possibly non-finite) entries of these blocks
  if (block_unsafe(warp >> 1)) {
    const int blk = warp >> 1, half = warp & 1, ch0 = 64 * half + 2 * lane;
    float2 kr[16], dd[16];
    {
      float2 gprev = make_float2(0.f, 0.f);
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const int row = 16 * blk + r;
        kr[r] = bf2(*reinterpret_cast<const uint32_t*>(sK + row * LDH + ch0));
        const float2 gg = *reinterpret_cast<const float2*>(sG + row * LDF + ch0);
        dd[r] = make_float2(ex2(gg.x - gprev.x), ex2(gg.y - gprev.y));   // dd[0] is never used
        gprev = gg;
      }
    }
    float* part = sT + (half * 4 + blk) * 512;   // [i][j][kk,qk]
    const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
    const int idx = (b4 ? 4 : 0) + (b3 ? 2 : 0) + (b2 ? 1 : 0);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const float2 qi = bf2(*reinterpret_cast<const uint32_t*>(sQ + (16 * blk + i) * LDH + ch0));
      const float2 ki = kr[i];
      float2 P = make_float2(1.f, 1.f);
#pragma unroll
      for (int jg = (i & ~3); jg >= 0; jg -= 4) {
        float v[8];
#pragma unroll
        for (int u = 3; u >= 0; --u) {
          const int j = jg + u;
          if (j <= i) {
            const float w0 = kr[j].x * P.x, w1 = kr[j].y * P.y;
            v[u] = ki.x * w0 + ki.y * w1;
            v[u + 4] = qi.x * w0 + qi.y * w1;
            if (j > 0) { P.x *= dd[j].x; P.y *= dd[j].y; }
          } else {
            v[u] = 0.f; v[u + 4] = 0.f;
          }
        }
        // eight sums over the 32 lanes in nine shuffles: each level halves the number of live values
        float x4[4], y2[2];
#pragma unroll
        for (int k4 = 0; k4 < 4; ++k4) {
          const float keep = b4 ? v[k4 + 4] : v[k4], send = b4 ? v[k4] : v[k4 + 4];
          x4[k4] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
        }
#pragma unroll
        for (int k2 = 0; k2 < 2; ++k2) {
          const float keep = b3 ? x4[k2 + 2] : x4[k2], send = b3 ? x4[k2] : x4[k2 + 2];
          y2[k2] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
        }
        float z = (b2 ? y2[1] : y2[0]) + __shfl_xor_sync(0xffffffffu, b2 ? y2[0] : y2[1], 4);
        z += __shfl_xor_sync(0xffffffffu, z, 2);
        z += __shfl_xor_sync(0xffffffffu, z, 1);
        if (t == 0) {
          const int j = jg + (idx & 3);
          if (j <= i) part[(i * 16 + j) * 2 + (idx >> 2)] = z;
        }
      }
    }
    asm volatile("bar.sync %0, 64;" ::"r"(8 + blk) : "memory");   // the two warps of this block
    const float* p0 = sT + blk * 512;
    const float* p1 = sT + (4 + blk) * 512;
    for (int e = lane; e < 256; e += 32) {
      const int i = e >> 4, j = e & 15, gi = 16 * blk + i, gj = 16 * blk + j;
      if (half == 0) {
        if (j < i) sAkk[gi * LDT + gj] = (p0[2 * e] + p1[2 * e]) * sRk[gi] * sRk[gj];
      } else if (j <= i) {
        sAqk[gi * LDQ + gj] = __float2bfloat16_rn((p0[2 * e + 1] + p1[2 * e + 1]) * sRq[gi] * sRk[gj]);
      }
    }
  }
  sm100::group_sync(1);
}
// ---- intra-chunk kernel, records ------------------------------------------------------------------------------------------------
// Two persistent CTAs per SM: eight warps that work, one that issues copies and products.  A worker warp owns eight rows of the chunk, a lane
// four channels of them, from the prefix sums to the tiles.
//
// With G summed from the chunk's start, e^{G_i - G_j} = e^{G_i} e^{-G_j}: while no channel decays by more than 2^64 over the chunk and no log decay is
// positive, the factors fit bf16's exponents, and both chunk-local products are one tcgen05 product, [k^ e^G; q^ e^G] (k^ e^{-G})^T, of tiles
// of which the record and W need the first two anyway.  An entry above the diagonal may be as large as 2^64 |k|^2; none is used.
// Chunks with a wider range (never with trained gates, but legal input) take general_products, which refers the decays to 16-row blocks.
//
// Rows arrive by TMA a chunk ahead: k and q into the tiles that their decayed forms are written over, q where q^ e^G of the chunk
// before has left for its record, k where Kd has.  So Kd takes k^ e^G's place of the chunk before and the two change places every
// chunk.  Tiles are in the 128-byte swizzle, rows of 128 bytes, panels of 64 columns (W^T: [128 channels][64 tokens], one panel); they go to
// the record by bulk copies.
//
// What bounds it: B=4 T=8192 H=32 (16384 chunks): 820 us with the general products for every chunk and rows loaded by the warps -> 448, the whole
// forward 1076 -> 723; 2.1 GB of rows and records are 327 us at the copy rate.  16.5 K cycles per chunk, two chunks at a time (24 K): 1.2 K
// waiting for rows, 2.0 K prefix sums and norms, 2.0 K tiles, 1.4 K for the product, 3.8 K inverse, 0.9 K for W^T; issue slots 51 %.  With loads by
// the warps into registers a chunk ahead they wait 6 K cycles for room in what the tiles leave of the L1 (690 us).  Fewer instructions in the
// prefix sums and norms (packed adds, one barrier with a vote) made it 2 to 7 % slower.  Output error against float64 (2-norm, 64 heads,
// T=500): 4.3e-3 -> 3.8e-3, one rounding per operand instead of two; without any decay, where the general form's factors are 1,
// 2.9e-3 -> 3.4e-3.  A sequence of one token (2.8e-3 -> 4.1e-3) keeps the general form.
constexpr int kIntraThreads = kThreads + 32;
constexpr int IS_A = 0, IS_Q = 8192, IS_B = 16384, IS_PANEL = 24576;   // k^ e^G | q^ e^G | Kd of 64 channels, then of the other 64; A and B by turns
constexpr int IS_G = 2 * IS_PANEL;         // log decay as it arrives [64][128]
constexpr int IS_AQK = IS_G + 32768;
constexpr int IS_TOT = IS_AQK + 8192;      // decay of each eight rows [8][128]
constexpr int IS_X = 96256;                // k^ e^{-G}, then A_kk and its inverse [64][68] fp32, then T diag(beta), two terms
constexpr int IS_BETA = IS_X + 64 * LDT * 4;
struct IntraCtl {
  float beta[64], rk[64], rq[64];
  uint64_t bar[2], full, free;
  alignas(16) int up[8];   // per warp: a log decay of its rows is positive
  uint32_t tmem_base;
  int wide, abort;
};
constexpr int IS_TOTAL = IS_BETA + sizeof(IntraCtl);
// the arrays of the general products: A_kk where the inverse expects it
constexpr int IG_K = 64 * LDF * 4, IG_Q = IG_K + 64 * LDH * 2, IG_T = IG_Q + 64 * LDH * 2, IG_AQK = IG_T + 64 * LDT * 4;
static_assert(IS_TOT + 4096 <= IS_X && IS_X % 1024 == 0 && IG_AQK + 64 * LDQ * 2 <= IS_X, "shared memory");
static_assert(2 * (IS_TOTAL + 1024) <= 233472, "two CTAs per SM");

static __device__ __noinline__ void general_products_call(uint8_t* smem, const float* rk, const float* rq, int tid) {   // the rare way
  general_products(reinterpret_cast<const float*>(smem), reinterpret_cast<const __nv_bfloat16*>(smem + IG_K),
                   reinterpret_cast<const __nv_bfloat16*>(smem + IG_Q), reinterpret_cast<float*>(smem + IS_X), reinterpret_cast<float*>(smem + IG_T),
                   reinterpret_cast<__nv_bfloat16*>(smem + IG_AQK), rk, rq, tid);
}

// Whether the chunk takes the general products, the same in every warp: a channel decays by more than 2^64 (run: this lane's four, whole chunk;
// not a number counts), or a log decay is positive -- sums of others fall from row to row, so that e^G and e^{-G} of every row lie within 2^64.
__device__ __forceinline__ bool any_wide(float4 run, const int (&up)[8], float limit = 64.f) {
  const int4 a = *reinterpret_cast<const int4*>(up), b = *reinterpret_cast<const int4*>(up + 4);
  const bool rise = (a.x | a.y | a.z | a.w) | (b.x | b.y | b.z | b.w);
  return __any_sync(0xffffffffu, rise || !(run.x >= -limit && run.y >= -limit && run.z >= -limit && run.w >= -limit));
}

template <class Params>
__global__ void __launch_bounds__(kIntraThreads, 2) intra_kernel(const __grid_constant__ Params P) {
  constexpr bool kPacked = std::is_same<Params, IntraPackedParams>::value;
  const FwdParams& p = P.p;
  extern __shared__ __align__(1024) uint8_t smem[];
  IntraCtl& ctl = *reinterpret_cast<IntraCtl*>(smem + IS_BETA);
  float* sX = reinterpret_cast<float*>(smem + IS_X);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  if (warp == 8) {
    tc::tmem_alloc(tc::smem_u32(&ctl.tmem_base), 128);
    tc::tmem_relinquish();
  }
  if (tid == 0) {
    tc::mbar_init(tc::smem_u32(&ctl.bar[0]), 1);
    tc::mbar_init(tc::smem_u32(&ctl.bar[1]), 1);
    tc::mbar_init(tc::smem_u32(&ctl.full), 1);
    tc::mbar_init(tc::smem_u32(&ctl.free), 1);
    tc::fence_mbar_init();
    ctl.abort = 0;
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  pdl_entry();
  if constexpr (!kPacked)
    if (P.marks.at && blockIdx.x == 0 && tid < 3) P.marks.at[2 + tid] = 0.f;
  const uint32_t tb = ctl.tmem_base, sb = tc::smem_u32(smem);
  auto wait_bar = [&](uint64_t& bar, uint32_t parity) {
    const uint32_t at = tc::smem_u32(&bar);
    sm100::wait_inline(at, parity, &ctl.abort, at - tc::smem_u32(&ctl), warp == 8);
  };
  // chunk number -> batch, head, first token, rows of it that exist, number of its record
  struct At { int b, h, tok, rows, one; int64_t rec; };   // one: packed, a sequence of one token
  auto place = [&](int c) -> At {
    At x;
    if constexpr (kPacked) {   // heads outermost in the grid, innermost but one in the records
      x.b = 0;
      x.h = c / P.seqs.chunks;
      c -= x.h * P.seqs.chunks;
      int lo = 0, hi = P.seqs.n - 1;   // the last sequence that starts at or before chunk c
      while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (P.seqs.first[mid] <= c) lo = mid; else hi = mid - 1;
      }
      const int n = c - P.seqs.first[lo], T = P.seqs.len[lo];
      x.tok = P.seqs.start[lo] + n * kC;
      x.rows = min(kC, T - n * kC);
      x.one = T == 1;
      x.rec = (int64_t)P.seqs.first[lo] * p.map.H + (int64_t)x.h * ((T + kC - 1) / kC) + n;
    } else {
      const int nchunks = (p.map.T + kC - 1) / kC, unit = c / nchunks, n = c - unit * nchunks;
      x.b = unit / p.map.H; x.h = unit - x.b * p.map.H;
      x.tok = n * kC;
      x.rows = min(kC, p.map.T - n * kC);
      x.rec = c;
    }
    return x;
  };

  if (warp == 8) {
    // =========================== ISSUING WARP (one thread) ==================================================================
    auto adv = [](uint64_t d, uint32_t bytes) { return d + (uint64_t)(bytes >> 4); };
    auto load_g = [&](const At& x) {
      const uint32_t bar = tc::smem_u32(&ctl.full), bytes = p.g_dt == DR_BF16 ? 16384 : 32768;
      tc::mbar_arrive_expect_tx(bar, 32768 + bytes);
      tc::tma_load_4d(sb + IS_G, &P.tg, 0, x.tok, x.h, x.b, bar);
    };
    auto load_qk = [&](const At& x, int k_at) {
      const uint32_t bar = tc::smem_u32(&ctl.full);
      const int hq = p.map.hq(x.h);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        tc::tma_load_4d(sb + e * IS_PANEL + k_at, &P.tk, 64 * e, hq, x.tok, x.b, bar);
        tc::tma_load_4d(sb + e * IS_PANEL + IS_Q, &P.tq, 64 * e, hq, x.tok, x.b, bar);
      }
    };
    if (P.use_tma && tc::elect_one()) {
      const At x = place(blockIdx.x);
      load_g(x);
      load_qk(x, IS_A);
    }
    __syncwarp();
    uint32_t ph = 0, ph0 = 0;   // ph: chunks so far; also which of the two places has k^ e^G
#pragma unroll 1
    for (int c = blockIdx.x; c < P.chunks; c += gridDim.x, ph ^= 1) {
      const At x = place(c);
      uint8_t* rec = P.ws + x.rec * WS_REC;
      const int next = c + gridDim.x;
      const uint32_t kg = ph ? IS_B : IS_A, kd = ph ? IS_A : IS_B;
      asm volatile("bar.sync 2, 288;" ::: "memory");
      tc::tc_fence_after();
      const bool wide = ctl.wide;
      if (tc::elect_one()) {
        if (!wide) {   // rows: k^ e^G, q^ e^G or the other way round
          const uint64_t ad = tc::smem_desc_sw128(sb + (ph ? IS_Q : IS_A), 128, 1024), bd = tc::smem_desc_sw128(sb + IS_X, 128, 1024);
#pragma unroll
          for (int ks = 0; ks < 8; ++ks)
            tc::mma_ss(tb, adv(ad, (ks >> 2) * IS_PANEL + (ks & 3) * 32), adv(bd, (ks >> 2) * 8192 + (ks & 3) * 32), tc::idesc_bf16(128, 64, 0, 0), ks > 0);
          tc::mma_commit(tc::smem_u32(&ctl.bar[0]));
        }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          tc::bulk_s2g(rec + WS_KD + 8192 * e, sb + e * IS_PANEL + kd, 8192);
          tc::bulk_s2g(rec + WS_QG + 8192 * e, sb + e * IS_PANEL + IS_Q, 8192);
        }
        if (wide) tc::bulk_s2g(rec + WS_AQK, sb + IS_AQK, 8192);
        tc::bulk_commit();
        if (P.use_tma && next < P.chunks) {
          const At y = place(next);
          load_g(y);
          if (!wide) wait_bar(ctl.bar[0], ph0);
          tc::bulk_wait_read_all();
          load_qk(y, kd);
        }
      }
      __syncwarp();
      if (!wide) {
        ph0 ^= 1;
        asm volatile("bar.sync 3, 288;" ::: "memory");
        if (tc::elect_one()) tc::bulk_s2g(rec + WS_AQK, sb + IS_AQK, 8192);
        __syncwarp();
      }
      asm volatile("bar.sync 4, 288;" ::: "memory");
      tc::tc_fence_after();
      if (tc::elect_one()) {
        // W^T = (k^ e^G)^T (T diag(beta))^T: sixteen tokens at a time, N = the rows that they reach
        const uint64_t ad = tc::smem_desc_sw128(sb + kg, IS_PANEL, 1024), bd = tc::smem_desc_sw128(sb + IS_X, 128, 1024);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          const uint32_t id = tc::idesc_bf16(128, 64 - 16 * ks, 1, 0);
          tc::mma_ss(tb + 64 + 16 * ks, adv(ad, ks * 2048), adv(bd, ks * (2048 + 32)), id, ks > 0);
          tc::mma_ss(tb + 64 + 16 * ks, adv(ad, ks * 2048), adv(bd, 8192 + ks * (2048 + 32)), id, 1);
        }
        tc::mma_commit(tc::smem_u32(&ctl.bar[1]));
        tc::bulk_s2g(rec + WS_TB, sb + IS_X, 8192);
      }
      __syncwarp();
      asm volatile("bar.sync 5, 288;" ::: "memory");
      if (tc::elect_one()) {
#pragma unroll
        for (int e = 0; e < 2; ++e) tc::bulk_s2g(rec + WS_W + 8192 * e, sb + e * IS_PANEL + kg, 8192);
        tc::bulk_commit();
        tc::bulk_wait_read_all();
        sm100::mbar_arrive(tc::smem_u32(&ctl.free));   // everything but the next chunk's rows may be written over
      }
      __syncwarp();
    }
    tc::bulk_wait_all();
  } else {
    // =========================== WORKERS ====================================================================================
    auto sync = []() { sm100::group_sync(1); };
    auto hand_over = [](int id) {
      tc::fence_async_smem();
      tc::tc_fence_before();
      asm volatile("bar.arrive %0, 288;" ::"r"(id) : "memory");
    };
    constexpr float kLog2e = 1.4426950408889634f;
    uint32_t ph = 0, ph0 = 0;
#pragma unroll 1
    for (int c = blockIdx.x; c < P.chunks; c += gridDim.x, ph ^= 1) {
      const int kg = ph ? IS_B : IS_A, kd = ph ? IS_A : IS_B;
      // byte of this lane's four channels in row 8 warp + r of a panel: + 128 r, piece ^ r
      const int piece = (lane & 15) >> 1, own = (lane >> 4) * IS_PANEL + warp * 1024 + (lane & 1) * 8;
      auto entry = [&](int base, int r) { return reinterpret_cast<uint2*>(smem + base + own + r * 128 + ((piece ^ r) << 4)); };
      // ---- the warp's rows, prefix sums over them, norm factors ------------------------------------------------------------------------
      float4 G[8];
      {
        const At x = place(c);
        const int rows = x.rows - 8 * warp, tok = x.tok + 8 * warp;
        const int64_t s_tok = p.map.tok(1), s_at = p.map.base(x.b, x.h, 1) + tok * s_tok;
        const float bt = lane < 8 && lane < rows && in_bounds(p.status, s_at + lane * s_tok, p.n_tok) ? p.beta[s_at + lane * s_tok] : 0.f;
        if (P.use_tma) {
          wait_bar(ctl.full, ph);
          if (p.g_dt == DR_BF16) {
#pragma unroll
            for (int r = 0; r < 8; ++r) {
              const uint2 u = *reinterpret_cast<const uint2*>(smem + IS_G + (8 * warp + r) * 256 + lane * 8);
              const float2 y = bf2(u.x), z = bf2(u.y);
              G[r] = make_float4(y.x, y.y, z.x, z.y);
            }
          } else {
#pragma unroll
            for (int r = 0; r < 8; ++r) G[r] = *reinterpret_cast<const float4*>(smem + IS_G + (8 * warp + r) * 512 + lane * 16);
          }
          if (kPacked && rows < 8) {   // rows of the next sequence
#pragma unroll
            for (int r = 0; r < 8; ++r)
              if (r >= rows) { *entry(IS_Q, r) = *entry(kg, r) = make_uint2(0u, 0u); G[r] = make_float4(0.f, 0.f, 0.f, 0.f); }
          }
        } else {   // arrays that TMA does not take, and one decay per token
          wait_bar(ctl.free, ph ^ 1);
          const int64_t st = p.map.tok_qk(kD), gst = p.map.tok(kD);
          const int64_t at = p.map.base_qk(x.b, x.h, kD) + tok * st + 4 * lane, g_at = p.map.base(x.b, x.h, kD) + tok * gst + 4 * lane;
#pragma unroll
          for (int r = 0; r < 8; ++r) {
            uint2 q = make_uint2(0u, 0u), k = q;
            float y[4] = {0.f, 0.f, 0.f, 0.f};
            if (r < rows && in_bounds_run(p.status, at + r * st, 4, p.n_qk)) {
              q = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(p.q) + at + r * st);
              k = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(p.k) + at + r * st);
              if (p.variant == DR_KDA && in_bounds_run(p.status, g_at + r * gst, 4, p.n_gk)) ld4(p.g, g_at + r * gst, p.g_dt, y);
              else if (p.variant == DR_GATED && in_bounds(p.status, s_at + r * s_tok, p.n_tok)) y[0] = y[1] = y[2] = y[3] = ld_elem(p.g, s_at + r * s_tok, p.g_dt);
            }
            G[r] = make_float4(y[0], y[1], y[2], y[3]);
            *entry(IS_Q, r) = q;
            *entry(kg, r) = k;
          }
        }
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        // (a sequence of one token counts as a rise: the 16-row form's operands are its rows as they are, which the tiles' rounding is worse than)
        float up = (kPacked ? x.one : p.map.T == 1) ? 1.f : 0.f;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          up = fmaxf(up, fmaxf(fmaxf(G[r].x, G[r].y), fmaxf(G[r].z, G[r].w)));
          acc.x += G[r].x * kLog2e; acc.y += G[r].y * kLog2e; acc.z += G[r].z * kLog2e; acc.w += G[r].w * kLog2e;
          G[r] = acc;
        }
        *reinterpret_cast<float4*>(smem + IS_TOT + warp * 512 + lane * 16) = acc;
        const int rise = __any_sync(0xffffffffu, up > 0.f);
        if (lane == 0) ctl.up[warp] = rise;
        // the sums are scattered over the lanes as they are reduced (16 shuffles), so that each lane takes one square root and one quotient
        float ss[16];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const uint2 q = *entry(IS_Q, r), k = *entry(kg, r);
          const float2 q0 = bf2(q.x), q1 = bf2(q.y), k0 = bf2(k.x), k1 = bf2(k.y);
          ss[r] = q0.x * q0.x + q0.y * q0.y + q1.x * q1.x + q1.y * q1.y;
          ss[8 + r] = k0.x * k0.x + k0.y * k0.y + k1.x * k1.x + k1.y * k1.y;
        }
#pragma unroll
        for (int o = 16, m = 8; o > 1; o >>= 1, m >>= 1) {
#pragma unroll
          for (int i = 0; i < m; ++i) {
            const bool up = lane & o;
            const float send = up ? ss[i] : ss[i + m], keep = up ? ss[i + m] : ss[i];
            ss[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
          }
        }
        ss[0] += __shfl_xor_sync(0xffffffffu, ss[0], 1);
        if (!(lane & 1)) {   // lanes 0, 2 .. 14: q rows, 16 .. 30: k rows
          const float top = lane < 16 ? p.scale : 1.f;
          (lane < 16 ? ctl.rq : ctl.rk)[8 * warp + ((lane >> 1) & 7)] = p.l2norm ? top / (sqrtf(ss[0]) + 1e-6f) : top;
        }
        if (lane < 8) ctl.beta[8 * warp + lane] = bt;
        if (warp == 0) {   // (the record's tail; its address is not worth keeping)
          sync();
          float4 run = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
          for (int s = 0; s < 8; ++s) {
            const float4 y = *reinterpret_cast<const float4*>(smem + IS_TOT + s * 512 + lane * 16);
            run.x += y.x; run.y += y.y; run.z += y.z; run.w += y.w;
          }
          if (in_bounds(p.status, x.rec, P.chunks))
            *reinterpret_cast<float4*>(P.ws + x.rec * WS_REC + WS_EGL + 16 * lane) = make_float4(ex2(run.x), ex2(run.y), ex2(run.z), ex2(run.w));
          if (!kPacked && P.marks.at) {
            const bool mark = any_wide(run, ctl.up, P.marks.limit);
            if (lane == 0 && in_bounds(p.status, x.rec, P.chunks)) P.marks.at[x.rec * P.marks.stride] = mark ? 1.f : 0.f;
          }
        } else {
          sync();
        }
      }
      bool wide;   // the same in every warp: each sees all channels
      float4 el;   // e^{G_L}
      {
        float4 pre = make_float4(0.f, 0.f, 0.f, 0.f), run = pre;
#pragma unroll
        for (int s = 0; s < 8; ++s) {
          if (s == warp) pre = run;
          const float4 y = *reinterpret_cast<const float4*>(smem + IS_TOT + s * 512 + lane * 16);
          run.x += y.x; run.y += y.y; run.z += y.z; run.w += y.w;
        }
        wide = any_wide(run, ctl.up);
        el = make_float4(ex2(run.x), ex2(run.y), ex2(run.z), ex2(run.w));
#pragma unroll
        for (int r = 0; r < 8; ++r) G[r] = make_float4(G[r].x + pre.x, G[r].y + pre.y, G[r].z + pre.z, G[r].w + pre.w);
      }
      if (tid == 0) ctl.wide = wide;
      wait_bar(ctl.free, ph ^ 1);   // the chunk before has left
      if (!wide) {
        // ---- the tiles ------------------------------------------------------------------------------------------------------------------
        const float2 el0 = make_float2(el.x, el.y), el1 = make_float2(el.z, el.w);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const float2 g0 = make_float2(G[r].x, G[r].y), g1 = make_float2(G[r].z, G[r].w);
          const float2 e0 = ex2x2(g0), e1 = ex2x2(g1), i0 = make_float2(ex2(-g0.x), ex2(-g0.y)), i1 = make_float2(ex2(-g1.x), ex2(-g1.y));
          const float fk = ctl.rk[8 * warp + r], fq = ctl.rq[8 * warp + r];
          const float2 rk = make_float2(fk, fk), rq = make_float2(fq, fq);
          const uint2 q = *entry(IS_Q, r), k = *entry(kg, r);
          const float2 k0 = mul2(bf2(k.x), rk), k1 = mul2(bf2(k.y), rk);
          const float2 x0 = mul2(k0, i0), x1 = mul2(k1, i1);
          const float2 a0 = mul2(k0, e0), a1 = mul2(k1, e1), b0 = mul2(mul2(bf2(q.x), rq), e0), b1 = mul2(mul2(bf2(q.y), rq), e1);
          const float2 d0 = mul2(x0, el0), d1 = mul2(x1, el1);
          *entry(kg, r) = make_uint2(tc::pack_bf16(a0.x, a0.y), tc::pack_bf16(a1.x, a1.y));
          *entry(IS_Q, r) = make_uint2(tc::pack_bf16(b0.x, b0.y), tc::pack_bf16(b1.x, b1.y));
          *entry(kd, r) = make_uint2(tc::pack_bf16(d0.x, d0.y), tc::pack_bf16(d1.x, d1.y));
          *reinterpret_cast<uint2*>(smem + IS_X + (lane >> 4) * 8192 + warp * 1024 + (lane & 1) * 8 + r * 128 + ((piece ^ r) << 4)) =
              make_uint2(tc::pack_bf16(x0.x, x0.y), tc::pack_bf16(x1.x, x1.y));
        }
      } else {
        // ---- any decay: through the arrays of the general products ---------------------------------------------------------------------------
        uint2 q[8], k[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          q[r] = *entry(IS_Q, r);
          k[r] = *entry(kg, r);
        }
        sync();   // every warp has its rows and the decays
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const int row = 8 * warp + r;
          *reinterpret_cast<float4*>(smem + (row * LDF + 4 * lane) * 4) = G[r];
          *reinterpret_cast<uint2*>(smem + IG_K + (row * LDH + 4 * lane) * 2) = k[r];
          *reinterpret_cast<uint2*>(smem + IG_Q + (row * LDH + 4 * lane) * 2) = q[r];
        }
        sync();
        general_products_call(smem, ctl.rk, ctl.rq, tid);
        uint4 tq[4], td[4], tk[4], aq[2];
        const float* sG = reinterpret_cast<const float*>(smem);
#pragma unroll
        for (int it = 0; it < 4; ++it) {
          const int i = tid + kThreads * it, row = i >> 4, col = (i & 15) * 8;
          decayed_piece(sG + row * LDF + col, sG + 63 * LDF + col, *reinterpret_cast<const uint4*>(smem + IG_Q + (row * LDH + col) * 2),
                        *reinterpret_cast<const uint4*>(smem + IG_K + (row * LDH + col) * 2), ctl.rq[row], ctl.rk[row], tq[it], td[it], tk[it]);
        }
#pragma unroll
        for (int it = 0; it < 2; ++it) {
          const int i = tid + kThreads * it, row = i >> 3, col = (i & 7) * 8;
          aq[it] = *reinterpret_cast<const uint4*>(smem + IG_AQK + (row * LDQ + col) * 2);
          uint32_t* w = reinterpret_cast<uint32_t*>(&aq[it]);
#pragma unroll
          for (int e = 0; e < 4; ++e) {   // keep j <= row
            const int j = col + 2 * e;
            if (j > row) w[e] = 0u;
            else if (j + 1 > row) w[e] &= 0x0000ffffu;
          }
        }
        sync();
#pragma unroll
        for (int it = 0; it < 4; ++it) {
          const int i = tid + kThreads * it, row = i >> 4, col = (i & 15) * 8, off = (col >> 6) * IS_PANEL + row * 128 + ((((col & 63) >> 3) ^ (row & 7)) << 4);
          *reinterpret_cast<uint4*>(smem + kg + off) = tk[it];
          *reinterpret_cast<uint4*>(smem + IS_Q + off) = tq[it];
          *reinterpret_cast<uint4*>(smem + kd + off) = td[it];
        }
#pragma unroll
        for (int it = 0; it < 2; ++it) {
          const int i = tid + kThreads * it, row = i >> 3, col = (i & 7) * 8;
          *reinterpret_cast<uint4*>(smem + IS_AQK + row * 128 + (((col >> 3) ^ (row & 7)) << 4)) = aq[it];
        }
      }
      hand_over(2);
      const int row = 32 * (warp & 3) + lane, hf = warp >> 2;   // this thread's row of the products, half of their columns
      const uint32_t ta = tb + ((uint32_t)(32 * (warp & 3)) << 16) + 32 * hf;
      if (!wide) {
        // ---- A_kk, A_qk (rows 0 .. 63 and 64 .., by turns) ------------------------------------------------------------------------------------
        wait_bar(ctl.bar[0], ph0);
        ph0 ^= 1;
        tc::tc_fence_after();
        uint32_t x[32];
        tc::tmem_ld32(ta, x);
        tc::tc_wait_ld();
        const int i = row & 63, last = i - 32 * hf;
        if ((uint32_t)(row >> 6) == ph) {   // over k^ e^{-G}, which has been read; what is above the diagonal is not used
#pragma unroll
          for (int e = 0; e < 8; ++e)
            *reinterpret_cast<uint4*>(sX + i * LDT + 32 * hf + 4 * e) = make_uint4(x[4 * e], x[4 * e + 1], x[4 * e + 2], x[4 * e + 3]);
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            uint32_t w[4];
#pragma unroll
            for (int f = 0; f < 4; ++f) {
              const int j = 8 * e + 2 * f;
              w[f] = tc::pack_bf16(j <= last ? __uint_as_float(x[j]) : 0.f, j + 1 <= last ? __uint_as_float(x[j + 1]) : 0.f);
            }
            *reinterpret_cast<uint4*>(smem + IS_AQK + i * 128 + (((4 * hf + e) ^ (i & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
        hand_over(3);
        sync();
      }
      // ---- T = (I + diag(beta) A_kk)^-1 in place, then T diag(beta) as two terms ---------------------------------------------------------------
      sm100::block_inverse_64(sX, ctl.beta, sX, tid);
      {
        uint4 hi[2], lo[2];
#pragma unroll
        for (int it = 0; it < 2; ++it) {
          int r, col;
          piece64(tid + kThreads * it, r, col);   // eight rows to a quarter warp: the 16-byte reads are free of bank conflicts
          float a[8], bb[8];
          *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(sX + r * LDT + col);
          *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(sX + r * LDT + col + 4);
          *reinterpret_cast<float4*>(bb) = *reinterpret_cast<const float4*>(ctl.beta + col);
          *reinterpret_cast<float4*>(bb + 4) = *reinterpret_cast<const float4*>(ctl.beta + col + 4);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float x = col + 2 * e <= r ? a[2 * e] * bb[2 * e] : 0.f, y = col + 2 * e + 1 <= r ? a[2 * e + 1] * bb[2 * e + 1] : 0.f;
            const uint32_t u = tc::pack_bf16(x, y);
            const float2 f = bf2(u);
            reinterpret_cast<uint32_t*>(&hi[it])[e] = u;
            reinterpret_cast<uint32_t*>(&lo[it])[e] = tc::pack_bf16(x - f.x, y - f.y);
          }
        }
        sync();
#pragma unroll
        for (int it = 0; it < 2; ++it) {
          int r, col;
          piece64(tid + kThreads * it, r, col);
          const int off = r * 128 + (((col >> 3) ^ (r & 7)) << 4);
          *reinterpret_cast<uint4*>(smem + IS_X + off) = hi[it];
          *reinterpret_cast<uint4*>(smem + IS_X + 8192 + off) = lo[it];
        }
      }
      hand_over(4);
      // ---- W^T, over k^ e^G ------------------------------------------------------------------------------------------------------------------
      wait_bar(ctl.bar[1], ph);
      tc::tc_fence_after();
      {
        uint32_t x[32];
        tc::tmem_ld32(ta + 64, x);
        tc::tc_wait_ld();
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          uint32_t w[4];
#pragma unroll
          for (int f = 0; f < 4; ++f) w[f] = tc::pack_bf16(__uint_as_float(x[8 * e + 2 * f]), __uint_as_float(x[8 * e + 2 * f + 1]));
          *reinterpret_cast<uint4*>(smem + kg + (row >> 6) * IS_PANEL + (row & 63) * 128 + (((4 * hf + e) ^ (row & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
      hand_over(5);
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 8) {
    sm100::settle(ctl.abort);
    tc::tmem_dealloc(tb, 128);
  }
  if (tid == 0) sm100::report_wait(p.status, ctl.abort);
}

// ---- intra-chunk kernel, transition form ------------------------------------------------------------------------------------------
// The chunk's effect on the state and on its own output, as fragments of trans_state_kernel:
//   N = -Kd^T W, Z = Kd^T U, Y = Qg - A_qk W, A_qk U   with W = T diag(beta) k^ e^G, U = T diag(beta) V
// One CTA of eight warps per chunk, two per SM; up to T as intra_kernel, with one place for each tile.  The four products have bf16 operands as
// in the other forwards; their accumulators are read in the shape of mma.sync's, which is what the fragments are, so nothing passes through
// shared memory on its way out.  A_qk's products have M = 128 rows, of which the lower 64 are V's bits and nobody reads them.
//
// What bounds it: B=1, T=1777, H=16 (448 chunks, one and a half waves): 48 us with the general products and everything on mma.sync -> 32.5, the
// layer around it 95 -> 82; the phases of a chunk follow each other, two chunks to an SM.  Errors against float64 (2-norm, output / state, T=1024, H=4):
// Gated 4.7e-3 / 3.0e-3 -> 3.9e-3 / 2.4e-3, KDA (T=1100) 4.4e-3 / 3.0e-3 -> 3.5e-3 / 2.5e-3: one rounding per decayed operand instead of two,
// and T diag(beta) as two terms.
constexpr int IT_KG = 0, IT_QG = 16384, IT_AQK = 32768, IT_V = IT_AQK + 8192, IT_TOT = IT_V + 16384;   // k^ e^G, later U^T; ..; V
constexpr int IT_KD = IS_X - 16384;        // Kd; the log decay arrives over Kd and X
struct TransCtl {
  float beta[64], rk[64], rq[64];
  uint64_t bar[4], full, full_v;
  alignas(16) int up[8];   // see IntraCtl
  uint32_t tmem_base;
  int abort;
};
constexpr int IT_TOTAL = IS_BETA + sizeof(TransCtl);
static_assert(IT_TOT + 4096 <= IT_KD && IT_KD % 1024 == 0 && IT_V % 1024 == 0 && 2 * (IT_TOTAL + 1024) <= 233472, "two CTAs per SM");

static __global__ void __launch_bounds__(kThreads, 2) intra_trans_kernel(const __grid_constant__ IntraTransParams P) {
  const FwdParams& p = P.p;
  extern __shared__ __align__(1024) uint8_t smem[];
  TransCtl& ctl = *reinterpret_cast<TransCtl*>(smem + IS_BETA);
  float* sX = reinterpret_cast<float*>(smem + IS_X);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int T = p.map.T, nchunks = (T + kC - 1) / kC, unit = blockIdx.x / nchunks, t0 = (blockIdx.x - unit * nchunks) * kC;
  const int b = unit / p.map.H, h = unit - b * p.map.H, rows = min(kC, T - t0) - 8 * warp;   // rows of this warp (may be none)
  const int64_t chunk = blockIdx.x;
  if (warp == 0) {
    tc::tmem_alloc(tc::smem_u32(&ctl.tmem_base), 256);
    tc::tmem_relinquish();
  }
  if (tid == 0) {
    for (int i = 0; i < 4; ++i) tc::mbar_init(tc::smem_u32(&ctl.bar[i]), 1);
    tc::mbar_init(tc::smem_u32(&ctl.full), 1);
    tc::mbar_init(tc::smem_u32(&ctl.full_v), 1);
    tc::fence_mbar_init();
    ctl.abort = 0;
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  pdl_entry();
  const uint32_t tb = ctl.tmem_base, sb = tc::smem_u32(smem);
  auto wait_bar = [&](uint64_t& bar, uint32_t parity) {
    const uint32_t at = tc::smem_u32(&bar);
    sm100::wait_inline(at, parity, &ctl.abort, at - tc::smem_u32(&ctl), 0);
  };
  auto adv = [](uint64_t d, uint32_t bytes) { return d + (uint64_t)(bytes >> 4); };
  auto tiles_sync = [&]() {
    tc::fence_async_smem();
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
  };
  auto load_v = [&]() {
    const uint32_t bar = tc::smem_u32(&ctl.full_v);
    tc::mbar_arrive_expect_tx(bar, 16384);
    tc::tma_load_4d(sb + IT_V, &P.tv, 0, h, t0, b, bar);
    tc::tma_load_4d(sb + IT_V + 8192, &P.tv, 64, h, t0, b, bar);
  };
  if (tid == 0) {
    const uint32_t bar = tc::smem_u32(&ctl.full);
    const int hq = p.map.hq(h);
    tc::mbar_arrive_expect_tx(bar, 32768 + (p.variant == DR_KDA ? (p.g_dt == DR_BF16 ? 16384 : 32768) : 0));
    if (p.variant == DR_KDA) tc::tma_load_4d(sb + IT_KD, &P.tg, 0, t0, h, b, bar);
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      tc::tma_load_4d(sb + IT_KG + 8192 * e, &P.tk, 64 * e, hq, t0, b, bar);
      tc::tma_load_4d(sb + IT_QG + 8192 * e, &P.tq, 64 * e, hq, t0, b, bar);
    }
    load_v();
  }
  constexpr float kLog2e = 1.4426950408889634f;
  // byte of this lane's four channels in row 8 warp + r of a panel: + 128 r, piece ^ r
  const int piece = (lane & 15) >> 1, own = (lane >> 4) * 8192 + warp * 1024 + (lane & 1) * 8;
  auto entry = [&](int base, int r) { return reinterpret_cast<uint2*>(smem + base + own + r * 128 + ((piece ^ r) << 4)); };
  // ---- the warp's rows, prefix sums over them, norm factors ----------------------------------------------------------------------------
  float4 G[8];
  {
    const int64_t s_tok = p.map.tok(1), s_at = p.map.base(b, h, 1) + (t0 + 8 * warp) * s_tok;
    const float bt = lane < 8 && lane < rows && in_bounds(p.status, s_at + lane * s_tok, p.n_tok) ? p.beta[s_at + lane * s_tok] : 0.f;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      float x = 0.f;
      if (p.variant == DR_GATED && r < rows && in_bounds(p.status, s_at + r * s_tok, p.n_tok)) x = ld_elem(p.g, s_at + r * s_tok, p.g_dt);
      G[r] = make_float4(x, x, x, x);
    }
    wait_bar(ctl.full, 0);
    if (p.variant == DR_KDA) {
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        if (p.g_dt == DR_BF16) {
          const uint2 u = *reinterpret_cast<const uint2*>(smem + IT_KD + (8 * warp + r) * 256 + lane * 8);
          const float2 y = bf2(u.x), z = bf2(u.y);
          G[r] = make_float4(y.x, y.y, z.x, z.y);
        } else {
          G[r] = *reinterpret_cast<const float4*>(smem + IT_KD + (8 * warp + r) * 512 + lane * 16);
        }
      }
    }
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float up = T == 1 ? 1.f : 0.f;   // (see intra_kernel)
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      up = fmaxf(up, fmaxf(fmaxf(G[r].x, G[r].y), fmaxf(G[r].z, G[r].w)));
      acc.x += G[r].x * kLog2e; acc.y += G[r].y * kLog2e; acc.z += G[r].z * kLog2e; acc.w += G[r].w * kLog2e;
      G[r] = acc;
    }
    *reinterpret_cast<float4*>(smem + IT_TOT + warp * 512 + lane * 16) = acc;
    const int rise = __any_sync(0xffffffffu, up > 0.f);
    if (lane == 0) ctl.up[warp] = rise;
    // the sums are scattered over the lanes as they are reduced (16 shuffles), so that each lane takes one square root and one quotient
    float ss[16];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const uint2 q = *entry(IT_QG, r), k = *entry(IT_KG, r);
      const float2 q0 = bf2(q.x), q1 = bf2(q.y), k0 = bf2(k.x), k1 = bf2(k.y);
      ss[r] = q0.x * q0.x + q0.y * q0.y + q1.x * q1.x + q1.y * q1.y;
      ss[8 + r] = k0.x * k0.x + k0.y * k0.y + k1.x * k1.x + k1.y * k1.y;
    }
#pragma unroll
    for (int o = 16, m = 8; o > 1; o >>= 1, m >>= 1) {
#pragma unroll
      for (int i = 0; i < m; ++i) {
        const bool up = lane & o;
        const float send = up ? ss[i] : ss[i + m], keep = up ? ss[i + m] : ss[i];
        ss[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
    ss[0] += __shfl_xor_sync(0xffffffffu, ss[0], 1);
    if (!(lane & 1)) {   // lanes 0, 2 .. 14: q rows, 16 .. 30: k rows
      const float top = lane < 16 ? p.scale : 1.f;
      (lane < 16 ? ctl.rq : ctl.rk)[8 * warp + ((lane >> 1) & 7)] = p.l2norm ? top / (sqrtf(ss[0]) + 1e-6f) : top;
    }
    if (lane < 8) ctl.beta[8 * warp + lane] = bt;
  }
  __syncthreads();   // the log decay, where Kd and k^ e^{-G} go, has been read, too
  bool wide;   // the same in every warp: each sees all channels
  float4 el;   // e^{G_L}
  {
    float4 pre = make_float4(0.f, 0.f, 0.f, 0.f), run = pre;
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      if (s == warp) pre = run;
      const float4 y = *reinterpret_cast<const float4*>(smem + IT_TOT + s * 512 + lane * 16);
      run.x += y.x; run.y += y.y; run.z += y.z; run.w += y.w;
    }
    wide = any_wide(run, ctl.up);
    el = make_float4(ex2(run.x), ex2(run.y), ex2(run.z), ex2(run.w));
    if (warp == 0 && in_bounds_run(p.status, chunk * kD + 4 * lane, 4, P.chunks * kD)) *reinterpret_cast<float4*>(P.el + chunk * kD + 4 * lane) = el;
#pragma unroll
    for (int r = 0; r < 8; ++r) G[r] = make_float4(G[r].x + pre.x, G[r].y + pre.y, G[r].z + pre.z, G[r].w + pre.w);
  }
  const int row = 32 * (warp & 3) + lane, hf = warp >> 2;   // this thread's row of a product, half of its columns
  const uint32_t ta = tb + ((uint32_t)(32 * (warp & 3)) << 16);
  if (!wide) {
    // ---- the tiles; A_kk, A_qk -------------------------------------------------------------------------------------------------------------
    const float2 el0 = make_float2(el.x, el.y), el1 = make_float2(el.z, el.w);
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const float2 g0 = make_float2(G[r].x, G[r].y), g1 = make_float2(G[r].z, G[r].w);
      const float2 e0 = ex2x2(g0), e1 = ex2x2(g1), i0 = make_float2(ex2(-g0.x), ex2(-g0.y)), i1 = make_float2(ex2(-g1.x), ex2(-g1.y));
      const float fk = ctl.rk[8 * warp + r], fq = ctl.rq[8 * warp + r];
      const float2 rk = make_float2(fk, fk), rq = make_float2(fq, fq);
      const uint2 q = *entry(IT_QG, r), k = *entry(IT_KG, r);
      const float2 k0 = mul2(bf2(k.x), rk), k1 = mul2(bf2(k.y), rk);
      const float2 x0 = mul2(k0, i0), x1 = mul2(k1, i1);
      const float2 a0 = mul2(k0, e0), a1 = mul2(k1, e1), b0 = mul2(mul2(bf2(q.x), rq), e0), b1 = mul2(mul2(bf2(q.y), rq), e1);
      const float2 d0 = mul2(x0, el0), d1 = mul2(x1, el1);
      *entry(IT_KG, r) = make_uint2(tc::pack_bf16(a0.x, a0.y), tc::pack_bf16(a1.x, a1.y));
      *entry(IT_QG, r) = make_uint2(tc::pack_bf16(b0.x, b0.y), tc::pack_bf16(b1.x, b1.y));
      *entry(IT_KD, r) = make_uint2(tc::pack_bf16(d0.x, d0.y), tc::pack_bf16(d1.x, d1.y));
      *entry(IS_X, r) = make_uint2(tc::pack_bf16(x0.x, x0.y), tc::pack_bf16(x1.x, x1.y));
    }
    tiles_sync();
    if (warp == 0) {
      if (tc::elect_one()) {
        const uint64_t kg = tc::smem_desc_sw128(sb + IT_KG, 128, 1024), qg = tc::smem_desc_sw128(sb + IT_QG, 128, 1024), bd = tc::smem_desc_sw128(sb + IS_X, 128, 1024);
        // rows 64 .. of the first product and of the second are the tile that follows, and not read
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
          tc::mma_ss(tb, adv(kg, (ks >> 2) * 8192 + (ks & 3) * 32), adv(bd, (ks >> 2) * 8192 + (ks & 3) * 32), tc::idesc_bf16(128, 64, 0, 0), ks > 0);
          tc::mma_ss(tb + 64, adv(qg, (ks >> 2) * 8192 + (ks & 3) * 32), adv(bd, (ks >> 2) * 8192 + (ks & 3) * 32), tc::idesc_bf16(128, 64, 0, 0), ks > 0);
        }
        tc::mma_commit(tc::smem_u32(&ctl.bar[0]));
      }
      __syncwarp();
    }
    wait_bar(ctl.bar[0], 0);
    tc::tc_fence_after();
    if (row < 64) {   // what is above the diagonal of A_kk is not used
      uint32_t x[32];
      tc::tmem_ld32(ta + 32 * hf, x);
      tc::tc_wait_ld();
#pragma unroll
      for (int e = 0; e < 8; ++e)
        *reinterpret_cast<uint4*>(sX + row * LDT + 32 * hf + 4 * e) = make_uint4(x[4 * e], x[4 * e + 1], x[4 * e + 2], x[4 * e + 3]);
      tc::tmem_ld32(ta + 64 + 32 * hf, x);
      tc::tc_wait_ld();
      const int last = row - 32 * hf;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        uint32_t w[4];
#pragma unroll
        for (int f = 0; f < 4; ++f) {
          const int j = 8 * e + 2 * f;
          w[f] = tc::pack_bf16(j <= last ? __uint_as_float(x[j]) : 0.f, j + 1 <= last ? __uint_as_float(x[j + 1]) : 0.f);
        }
        *reinterpret_cast<uint4*>(smem + IT_AQK + row * 128 + (((4 * hf + e) ^ (row & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
  } else {
    // ---- any decay: through the arrays of the general products, over V, which arrives once more ------------------------------------------------
    uint2 q[8], k[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      q[r] = *entry(IT_QG, r);
      k[r] = *entry(IT_KG, r);
    }
    wait_bar(ctl.full_v, 0);
    __syncthreads();   // every warp has its rows and the decays
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int i = 8 * warp + r;
      *reinterpret_cast<float4*>(smem + (i * LDF + 4 * lane) * 4) = G[r];
      *reinterpret_cast<uint2*>(smem + IG_K + (i * LDH + 4 * lane) * 2) = k[r];
      *reinterpret_cast<uint2*>(smem + IG_Q + (i * LDH + 4 * lane) * 2) = q[r];
    }
    __syncthreads();
    general_products_call(smem, ctl.rk, ctl.rq, tid);
    uint4 tq[4], td[4], tk[4], aq[2];
    const float* sG = reinterpret_cast<const float*>(smem);
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int i = tid + kThreads * it, r = i >> 4, col = (i & 15) * 8;
      decayed_piece(sG + r * LDF + col, sG + 63 * LDF + col, *reinterpret_cast<const uint4*>(smem + IG_Q + (r * LDH + col) * 2),
                    *reinterpret_cast<const uint4*>(smem + IG_K + (r * LDH + col) * 2), ctl.rq[r], ctl.rk[r], tq[it], td[it], tk[it]);
    }
#pragma unroll
    for (int it = 0; it < 2; ++it) {
      const int i = tid + kThreads * it, r = i >> 3, col = (i & 7) * 8;
      aq[it] = *reinterpret_cast<const uint4*>(smem + IG_AQK + (r * LDQ + col) * 2);
      uint32_t* w = reinterpret_cast<uint32_t*>(&aq[it]);
#pragma unroll
      for (int e = 0; e < 4; ++e) {   // keep j <= r
        const int j = col + 2 * e;
        if (j > r) w[e] = 0u;
        else if (j + 1 > r) w[e] &= 0x0000ffffu;
      }
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int i = tid + kThreads * it, r = i >> 4, col = (i & 15) * 8, off = (col >> 6) * 8192 + r * 128 + ((((col & 63) >> 3) ^ (r & 7)) << 4);
      *reinterpret_cast<uint4*>(smem + IT_KG + off) = tk[it];
      *reinterpret_cast<uint4*>(smem + IT_QG + off) = tq[it];
      *reinterpret_cast<uint4*>(smem + IT_KD + off) = td[it];
    }
#pragma unroll
    for (int it = 0; it < 2; ++it) {
      const int i = tid + kThreads * it, r = i >> 3, col = (i & 7) * 8;
      *reinterpret_cast<uint4*>(smem + IT_AQK + r * 128 + (((col >> 3) ^ (r & 7)) << 4)) = aq[it];
    }
    tiles_sync();
    if (tid == 0) load_v();
  }
  __syncthreads();
  // ---- T = (I + diag(beta) A_kk)^-1 in place, then T diag(beta) as two terms -----------------------------------------------------------------
  sm100::block_inverse_64(sX, ctl.beta, sX, tid);
  {
    uint4 hi[2], lo[2];
#pragma unroll
    for (int it = 0; it < 2; ++it) {
      int r, col;
      piece64(tid + kThreads * it, r, col);   // eight rows to a quarter warp: the 16-byte reads are free of bank conflicts
      float a[8], bb[8];
      *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(sX + r * LDT + col);
      *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(sX + r * LDT + col + 4);
      *reinterpret_cast<float4*>(bb) = *reinterpret_cast<const float4*>(ctl.beta + col);
      *reinterpret_cast<float4*>(bb + 4) = *reinterpret_cast<const float4*>(ctl.beta + col + 4);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float x = col + 2 * e <= r ? a[2 * e] * bb[2 * e] : 0.f, y = col + 2 * e + 1 <= r ? a[2 * e + 1] * bb[2 * e + 1] : 0.f;
        const uint32_t u = tc::pack_bf16(x, y);
        const float2 f = bf2(u);
        reinterpret_cast<uint32_t*>(&hi[it])[e] = u;
        reinterpret_cast<uint32_t*>(&lo[it])[e] = tc::pack_bf16(x - f.x, y - f.y);
      }
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < 2; ++it) {
      int r, col;
      piece64(tid + kThreads * it, r, col);
      const int off = r * 128 + (((col >> 3) ^ (r & 7)) << 4);
      *reinterpret_cast<uint4*>(smem + IS_X + off) = hi[it];
      *reinterpret_cast<uint4*>(smem + IS_X + 8192 + off) = lo[it];
    }
  }
  tiles_sync();
  // ---- W^T, U^T: sixteen tokens at a time, N = the rows that they reach; then as tiles [128 channels][64 tokens] ----------------------------------
  wait_bar(ctl.full_v, wide);
  if (warp == 0) {
    if (tc::elect_one()) {
      const uint64_t kg = tc::smem_desc_sw128(sb + IT_KG, 8192, 1024), vd = tc::smem_desc_sw128(sb + IT_V, 8192, 1024), bd = tc::smem_desc_sw128(sb + IS_X, 128, 1024);
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        const uint32_t id = tc::idesc_bf16(128, 64 - 16 * ks, 1, 0);
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          tc::mma_ss(tb + 16 * ks, adv(kg, ks * 2048), adv(bd, 8192 * x + ks * (2048 + 32)), id, ks + x > 0);
          tc::mma_ss(tb + 64 + 16 * ks, adv(vd, ks * 2048), adv(bd, 8192 * x + ks * (2048 + 32)), id, ks + x > 0);
        }
      }
      tc::mma_commit(tc::smem_u32(&ctl.bar[1]));
    }
    __syncwarp();
  }
  wait_bar(ctl.bar[1], 0);
  tc::tc_fence_after();
#pragma unroll
  for (int y = 0; y < 2; ++y) {
    uint32_t x[32];
    tc::tmem_ld32(ta + 64 * y + 32 * hf, x);
    tc::tc_wait_ld();
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      uint32_t w[4];
#pragma unroll
      for (int f = 0; f < 4; ++f) w[f] = tc::pack_bf16(__uint_as_float(x[8 * e + 2 * f]), __uint_as_float(x[8 * e + 2 * f + 1]));
      *reinterpret_cast<uint4*>(smem + (y ? IT_KG : IS_X) + row * 128 + (((4 * hf + e) ^ (row & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
  tiles_sync();
  const int g = lane >> 2, t = lane & 3;
  const uint64_t wd = tc::smem_desc_sw128(sb + IS_X, 128, 1024), ud = tc::smem_desc_sw128(sb + IT_KG, 128, 1024);
  // ---- N, Z -> fragments ---------------------------------------------------------------------------------------------------------------------
  if (warp == 0) {
    if (tc::elect_one()) {
      const uint64_t kd = tc::smem_desc_sw128(sb + IT_KD, 8192, 1024);
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) tc::mma_ss(tb, adv(kd, ks * 2048), adv(wd, ks * 32), tc::idesc_bf16(128, 128, 1, 0), ks > 0);
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) tc::mma_ss(tb + 128, adv(kd, ks * 2048), adv(ud, ks * 32), tc::idesc_bf16(128, 128, 1, 0), ks > 0);
      tc::mma_commit(tc::smem_u32(&ctl.bar[2]));
    }
    __syncwarp();
  }
  wait_bar(ctl.bar[2], 0);
  tc::tc_fence_after();
#pragma unroll
  for (int m = 0; m < 2; ++m) {   // sixteen rows at a time, 64 columns
    const int mt = 2 * (warp & 3) + m;
    uint32_t x[32];
    tc::tmem_ld_frag(ta + ((uint32_t)(16 * m) << 16) + 64 * hf, x);
    tc::tc_wait_ld();
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      uint32_t w[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) w[e] = mma::pack(-__uint_as_float(x[8 * ks + 2 * e]), -__uint_as_float(x[8 * ks + 2 * e + 1]));
      const int64_t at = ((chunk * 8 + mt) * 8 + 4 * hf + ks) * 32 + lane;
      if (in_bounds(p.status, at, P.chunks * (8 * 8 * 32))) P.nf[at] = make_uint4(w[0], w[1], w[2], w[3]);
    }
    tc::tmem_ld_frag(ta + ((uint32_t)(16 * m) << 16) + 128 + 64 * hf, x);
    tc::tc_wait_ld();
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
      const int64_t at = ((chunk * 8 + mt) * 16 + 8 * hf + nt) * 32 + lane;
      if (in_bounds(p.status, at, P.chunks * (8 * 16 * 32)))
        P.zf[at] = make_float4(__uint_as_float(x[4 * nt]), __uint_as_float(x[4 * nt + 1]), __uint_as_float(x[4 * nt + 2]), __uint_as_float(x[4 * nt + 3]));
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  // ---- Y = Qg - A_qk W, A_qk U -> fragments -------------------------------------------------------------------------------------------------------
  if (warp == 0) {
    if (tc::elect_one()) {
      const uint64_t ad = tc::smem_desc_sw128(sb + IT_AQK, 128, 1024);
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) tc::mma_ss(tb, adv(ad, ks * 32), adv(wd, ks * 32), tc::idesc_bf16(128, 128, 0, 0), ks > 0);
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) tc::mma_ss(tb + 128, adv(ad, ks * 32), adv(ud, ks * 32), tc::idesc_bf16(128, 128, 0, 0), ks > 0);
      tc::mma_commit(tc::smem_u32(&ctl.bar[3]));
    }
    __syncwarp();
  }
  wait_bar(ctl.bar[3], 0);
  tc::tc_fence_after();
  if ((warp & 3) < 2) {
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int mt = 2 * (warp & 3) + m;
      uint32_t x[32];
      tc::tmem_ld_frag(ta + ((uint32_t)(16 * m) << 16) + 64 * hf, x);
      tc::tc_wait_ld();
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {   // e & 1: row half, e >> 1: column half
          const int r = 16 * mt + g + 8 * (e & 1);   // (r & 7 is g)
          const float2 q = bf2(*reinterpret_cast<const uint32_t*>(smem + IT_QG + hf * 8192 + r * 128 + (((2 * ks + (e >> 1)) ^ g) << 4) + 4 * t));
          const int i = 8 * ks + 4 * (e >> 1) + 2 * (e & 1);
          w[e] = mma::pack(q.x - __uint_as_float(x[i]), q.y - __uint_as_float(x[i + 1]));
        }
        const int64_t at = ((chunk * 4 + mt) * 8 + 4 * hf + ks) * 32 + lane;
        if (in_bounds(p.status, at, P.chunks * (4 * 8 * 32))) P.yf[at] = make_uint4(w[0], w[1], w[2], w[3]);
      }
      tc::tmem_ld_frag(ta + ((uint32_t)(16 * m) << 16) + 128 + 64 * hf, x);
      tc::tc_wait_ld();
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) {
        const int64_t at = ((chunk * 4 + mt) * 16 + 8 * hf + nt) * 32 + lane;
        if (in_bounds(p.status, at, P.chunks * (4 * 16 * 32)))
          P.of[at] = make_float4(__uint_as_float(x[4 * nt]), __uint_as_float(x[4 * nt + 1]), __uint_as_float(x[4 * nt + 2]), __uint_as_float(x[4 * nt + 3]));
      }
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    sm100::settle(ctl.abort);
    tc::tmem_dealloc(tb, 256);
  }
  if (tid == 0) sm100::report_wait(p.status, ctl.abort);
}

// ---- state kernel ----------------------------------------------------------------------------------------------
// tensor-memory columns
constexpr uint32_t TM_S = 0;      // S^T fp32                        128
constexpr uint32_t TM_SB = 128;   // bf16 copy of S^T (A operand)      64
constexpr uint32_t TM_DU = 192;   // 2 x 64: U^T -> Vn^T -> Do
constexpr uint32_t TM_DQ = 320;   // S^T Qg^T                          64
constexpr uint32_t TM_VA = 384;   // Vn^T bf16                         32
constexpr uint32_t TM_COLS = 512;
// shared memory: two record buffers, two V tiles (two swizzled panels of 64 columns each, straight from the input by
// TMA), then the fp32 output staging tile [64][128]
constexpr int V_PANEL = 64 * 128, V_TILE = 2 * V_PANEL;
constexpr int ST_REC = (WS_REC + 1023) / 1024 * 1024;
constexpr int ST_V = 2 * ST_REC;
constexpr int ST_O = ST_V + 2 * V_TILE;
static_assert(ST_V % 1024 == 0, "swizzled tiles");
constexpr int ST_TOTAL = ST_O + 64 * 128 * 4;

static_assert(sizeof(IntraPackedParams) <= 4096, "kernel parameters");
struct StateCtl {
  uint64_t full[2], go1, go2, go3, bar1, bar2;
  uint32_t tmem_base;
  int abort;
};

// Nine warps.  Warps 0-7 (256 threads; two warps per 32-lane quarter of tensor memory, each taking half of the
// columns) do everything that touches data; warp 8 only issues: the bulk copies of the records and every
// tcgen05.mma.  Issuing one product costs its thread ~100 cycles, 28 products per chunk: on a worker warp that
// time would sit on the serial chain of the chunk, on the issuing warp it overlaps the workers' epilogues.
// Hand-offs are mbarriers: go1 (bf16 state copy written), go2 (the previous chunk's Dq has been read),
// go3 (bf16 V_new written) from the workers; bar1, bar2 (products complete) from tcgen05.commit.
constexpr int kStateThreads = kThreads + 32;

// Kernel parameters of the state pass: the forward parameters plus the output tensor map ({128, T, H, B} view of
// o in its own dtype; one box {128, 64, 1, 1} stores a chunk's rows and clips the ragged tail).
struct StateParams {
  CUtensorMap to;
  CUtensorMap tv;   // panels of v (see sm100::make_panel_map)
  FwdParams p;
  const uint8_t* ws;
  int use_tma_out;
};
struct StatePackedParams : StateParams {
  SeqTable seqs;
};
static_assert(sizeof(StatePackedParams) <= 4096, "kernel parameters");

template <class Params>
__global__ void __launch_bounds__(kStateThreads, 1) state_kernel(const __grid_constant__ Params P) {
  constexpr bool kPacked = std::is_same<Params, StatePackedParams>::value;
  const FwdParams& p = P.p;
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(8) StateCtl ctl;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int hs = (tid >> 7) & 1, l128 = tid & 127;
  int T = p.map.T, unit = blockIdx.x, tok0 = 0;
  int b = unit / p.map.H;
  const int h = unit % p.map.H;
  int64_t rec0;
  if constexpr (kPacked) {
    T = P.seqs.len[b];
    tok0 = P.seqs.start[b];
    unit = P.seqs.index[b] * p.map.H + h;
    rec0 = (int64_t)P.seqs.first[b] * p.map.H + (int64_t)h * ((T + kC - 1) / kC);
    b = 0;
  }
  const int nchunks = (T + kC - 1) / kC;
  if constexpr (!kPacked) rec0 = (int64_t)unit * nchunks;
  const int64_t o_tok = p.map.tok(kD), o_base = p.map.base(b, h, kD) + tok0 * o_tok;
  const uint8_t* recs = P.ws + rec0 * WS_REC;
  // the last chunk of a packed sequence: its V tile ends in rows of the next sequence, which the workers clear
  auto packed_tail = [&](int n) { return kPacked && T - n * kC < kC; };

  if (warp == 0) {
    tc::tmem_alloc(tc::smem_u32(&ctl.tmem_base), TM_COLS);
    tc::tmem_relinquish();
  }
  if (tid == 0) {
    tc::mbar_init(tc::smem_u32(&ctl.full[0]), 1);
    tc::mbar_init(tc::smem_u32(&ctl.full[1]), 1);
    tc::mbar_init(tc::smem_u32(&ctl.go1), kThreads);
    tc::mbar_init(tc::smem_u32(&ctl.go2), kThreads);
    tc::mbar_init(tc::smem_u32(&ctl.go3), kThreads);
    tc::mbar_init(tc::smem_u32(&ctl.bar1), 1);
    tc::mbar_init(tc::smem_u32(&ctl.bar2), 1);
    tc::fence_mbar_init();
    ctl.abort = 0;
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  pdl_entry();
  const uint32_t tbase = ctl.tmem_base;
  const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
  auto wait_bar = [&](uint64_t* bar, uint32_t parity) {
    if (tc::mbar_try(tc::smem_u32(bar), parity)) return;
    sm100::wait_more(tc::smem_u32(bar), parity, p.status, &ctl.abort, (uint32_t)((const char*)bar - (const char*)&ctl),
                     (uint32_t)(warp == 8 ? 1 : 0));
  };
  auto arrive = [&](uint64_t* bar) { sm100::mbar_arrive(tc::smem_u32(bar)); };
  auto workers_sync = [&]() { asm volatile("bar.sync 1, 256;" ::: "memory"); };

  if (warp == 8) {
    // =========================== ISSUING WARP (one thread) ======================================================
    if (tc::elect_one()) {
      // the record of chunk m -> buffer m & 1, the V rows straight from the input
      auto issue_load = [&](int m) {
        const uint32_t bar = tc::smem_u32(&ctl.full[m & 1]);
        tc::mbar_arrive_expect_tx(bar, WS_REC + V_TILE);
        const uint32_t dst = tc::smem_u32(smem + (m & 1) * ST_REC), dv = tc::smem_u32(smem + ST_V + (m & 1) * V_TILE);
        const uint8_t* src = recs + (int64_t)m * WS_REC;
        tc::tma_load_4d(dv, &P.tv, 0, h, tok0 + m * kC, b, bar);
        tc::tma_load_4d(dv + V_PANEL, &P.tv, 64, h, tok0 + m * kC, b, bar);
#pragma unroll
        for (int i = 0; i < 3; ++i) tc::bulk_g2s(dst + i * 16384, src + i * 16384, 16384, bar);   // W, Qg, Kd
        tc::bulk_g2s(dst + WS_TB, src + WS_TB, WS_REC - WS_TB, bar);                                   // Tb, A_qk, e^{G_L}
      };
      if (nchunks > 0) issue_load(0);
      if (nchunks > 1) issue_load(1);
      const uint32_t id_n64 = tc::idesc_bf16(128, 64, 0, 0);
      const uint32_t id_n64_amn = tc::idesc_bf16(128, 64, 1, 0);
      const uint32_t id_n64_neg = tc::idesc_bf16(128, 64, 0, 1) | (1u << 13);
      const uint32_t id_n128_bmn = tc::idesc_bf16(128, 128, 0, 1);
      for (int n = 0; n < nchunks; ++n) {
        const int s = n & 1;
        const uint8_t* st = smem + s * ST_REC;
        const uint32_t aW = tc::smem_u32(st + WS_W), aQg = tc::smem_u32(st + WS_QG), aKd = tc::smem_u32(st + WS_KD);
        const uint32_t aV = tc::smem_u32(smem + ST_V + s * V_TILE), aTb = tc::smem_u32(st + WS_TB), aAqk = tc::smem_u32(st + WS_AQK);
        wait_bar(&ctl.full[s], (n >> 1) & 1);
        // U^T = V^T Tb^T needs no state: issue it before the workers' state pass has finished
        if (packed_tail(n)) wait_bar(&ctl.go1, n & 1);
        tc::tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          const uint64_t ad = tc::smem_desc_sw128(aV + ks * 2048, V_PANEL, 1024);   // MN-major, 16 chunk rows per step
          const uint64_t bd = tc::smem_desc_sw128(aTb + ks * 32, 128, 1024);
          tc::mma_ss(tbase + TM_DU + 64 * s, ad, bd, id_n64_amn, ks > 0);
        }
        wait_bar(&ctl.go1, n & 1);
        tc::tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {   // Vn^T = U^T - S^T W^T
          const uint64_t bd = tc::smem_desc_sw128(aW + ks * 2048, 16384, 1024);   // MN-major
          tc::mma_ts(tbase + TM_DU + 64 * s, tbase + TM_SB + ks * 8, bd, id_n64_neg, 1);
        }
        tc::mma_commit(tc::smem_u32(&ctl.bar1));
        if (n > 0) wait_bar(&ctl.go2, (n - 1) & 1);   // the previous chunk's Dq has been read
        tc::tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {   // Dq = S^T Qg^T
          const uint64_t bd = tc::smem_desc_sw128(aQg + (ks >> 2) * 8192 + (ks & 3) * 32, 128, 1024);
          tc::mma_ts(tbase + TM_DQ, tbase + TM_SB + ks * 8, bd, id_n64, ks > 0);
        }
        wait_bar(&ctl.go3, n & 1);
        tc::tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {   // S^T += Vn^T Kd   (Kd MN-major)
          const uint64_t bd = tc::smem_desc_sw128(aKd + ks * 2048, 8192, 1024);
          tc::mma_ts(tbase + TM_S, tbase + TM_VA + ks * 8, bd, id_n128_bmn, 1);
        }
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {   // Do = Vn^T A_qk^T
          const uint64_t bd = tc::smem_desc_sw128(aAqk + ks * 32, 128, 1024);
          tc::mma_ts(tbase + TM_DU + 64 * s, tbase + TM_VA + ks * 8, bd, id_n64, ks > 0);
        }
        tc::mma_commit(tc::smem_u32(&ctl.bar2));
        // every product that reads this buffer has completed once bar2 flips: fetch the record of chunk n + 2
        if (n + 2 < nchunks) {
          wait_bar(&ctl.bar2, n & 1);
          tc::fence_async_smem();
          issue_load(n + 2);
        }
      }
    }
  } else {
    // =========================== WORKERS ===========================================================================
    // initial state: S^T[v][k] = h0[k][v]
    {
      const float* h0 = p.h0 ? p.h0 + (int64_t)unit * kD * kD : nullptr;
#pragma unroll
      for (int cc = 0; cc < 2; ++cc) {
        const int c0 = 64 * hs + 32 * cc;
        uint32_t r[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) r[j] = h0 ? __float_as_uint(h0[(c0 + j) * kD + l128]) : 0u;
        tc::tmem_st32(tbase + TM_S + lane_addr + c0, r);
      }
      tc::tc_wait_st();
    }
    float* sO = reinterpret_cast<float*>(smem + ST_O);
    __nv_bfloat16* sOh = reinterpret_cast<__nv_bfloat16*>(smem + ST_O);
    // O^T of chunk m = Dq + Do -> staging tile [64][128] in the output dtype -> one tiled TMA store (or, without a
    // tensor map, row copies by the threads)
    auto output_epilogue = [&](int m) {
      const int t0m = m * kC, rowsm = min(kC, T - t0m);
      const bool tma_out = P.use_tma_out && !packed_tail(m);   // (a box would run into the next sequence)
      if (P.use_tma_out && tid == 0) tc::bulk_wait_read_all();   // the previous store has read the staging tile
      workers_sync();
      {
        const int c0 = 32 * hs;
        uint32_t rq[32], ro[32];
        tc::tmem_ld32(tbase + TM_DQ + lane_addr + c0, rq);
        tc::tmem_ld32(tbase + TM_DU + 64 * (m & 1) + lane_addr + c0, ro);
        tc::tc_wait_ld();
        tc::tc_fence_before();
        arrive(&ctl.go2);   // Dq (and this accumulator) may be overwritten
        if (p.out_dt == DR_BF16) {
#pragma unroll
          for (int j = 0; j < 32; ++j)
            sOh[(c0 + j) * kD + l128] = __float2bfloat16_rn(__uint_as_float(rq[j]) + __uint_as_float(ro[j]));
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) sO[(c0 + j) * kD + l128] = __uint_as_float(rq[j]) + __uint_as_float(ro[j]);
        }
      }
      if (!p.o) return;
      if (tma_out) {
        tc::fence_async_smem();
        workers_sync();
        if (tid == 0) {
          tc::tma_store_4d(&P.to, tc::smem_u32(sO), 0, tok0 + t0m, h, b);
          tc::bulk_commit();
        }
        return;
      }
      workers_sync();
      const int r = tid >> 2, qtr = tid & 3;
      if (r < rowsm) {
        const int64_t at = o_base + (int64_t)(t0m + r) * o_tok + 32 * qtr;
        if (p.out_dt == DR_BF16) {
          __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(p.o) + at;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            reinterpret_cast<uint4*>(dst)[j] = reinterpret_cast<const uint4*>(sOh + r * kD + 32 * qtr)[j];
        } else {
          float* dst = reinterpret_cast<float*>(p.o) + at;
#pragma unroll
          for (int j = 0; j < 8; ++j)
            reinterpret_cast<float4*>(dst)[j] = reinterpret_cast<const float4*>(sO + r * kD + 32 * qtr)[j];
        }
      }
    };

    for (int n = 0; n < nchunks; ++n) {
      const int s = n & 1;
      const float* sEGL = reinterpret_cast<const float*>(smem + s * ST_REC + WS_EGL);
      wait_bar(&ctl.full[s], (n >> 1) & 1);
      if (n > 0) {
        wait_bar(&ctl.bar2, (n - 1) & 1);   // the previous chunk's state update and Do have completed
        tc::tc_fence_after();
      }
      // ---- state pass: bf16 copy of S^T for the products; fp32 master decayed per key channel -------------------
      {
#pragma unroll
        for (int cc = 0; cc < 2; ++cc) {
          const int c0 = 64 * hs + 32 * cc;
          uint32_t r[32], pk[16];
          tc::tmem_ld32(tbase + TM_S + lane_addr + c0, r);
          tc::tc_wait_ld();
#pragma unroll
          for (int j = 0; j < 16; ++j) pk[j] = tc::pack_bf16(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
          if (p.ckpt) {
            float* ck = p.ckpt + ((int64_t)unit * nchunks + n) * kD * kD;
#pragma unroll
            for (int j = 0; j < 32; ++j) ck[(c0 + j) * kD + l128] = __uint_as_float(r[j]);
          }
#pragma unroll
          for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) * sEGL[c0 + j]);
          tc::tmem_st16(tbase + TM_SB + lane_addr + c0 / 2, pk);
          tc::tmem_st32(tbase + TM_S + lane_addr + c0, r);
        }
        tc::tc_wait_st();
      }
      if (packed_tail(n)) {   // nothing of the next sequence, not even a NaN times 0, may reach this one
        const int rowsn = T - n * kC;
        for (int i = tid; i < (kC - rowsn) * 16; i += kThreads)
          *reinterpret_cast<uint4*>(smem + ST_V + s * V_TILE + (i & 8) / 8 * V_PANEL + (rowsn + (i >> 4)) * 128 + (i & 7) * 16) =
              make_uint4(0u, 0u, 0u, 0u);
        tc::fence_async_smem();
      }
      tc::tc_fence_before();
      arrive(&ctl.go1);
      if (n > 0) output_epilogue(n - 1);   // overlaps the products of this chunk
      wait_bar(&ctl.bar1, n & 1);
      tc::tc_fence_after();
      // ---- Vn^T -> bf16 -------------------------------------------------------------------------------------------
      {
        const int c0 = 32 * hs;
        uint32_t r[32], pa[16];
        tc::tmem_ld32(tbase + TM_DU + 64 * s + lane_addr + c0, r);
        tc::tc_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; ++j) pa[j] = tc::pack_bf16(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
        tc::tmem_st16(tbase + TM_VA + lane_addr + c0 / 2, pa);
      }
      tc::tc_wait_st();
      tc::tc_fence_before();
      arrive(&ctl.go3);
    }
    if (nchunks > 0) {
      wait_bar(&ctl.bar2, (nchunks - 1) & 1);
      tc::tc_fence_after();
      output_epilogue(nchunks - 1);
      if (P.use_tma_out && tid == 0) tc::bulk_wait_all();
    }
    if (p.hT) {
      float* hT = p.hT + (int64_t)unit * kD * kD;
#pragma unroll
      for (int cc = 0; cc < 2; ++cc) {
        const int c0 = 64 * hs + 32 * cc;
        uint32_t r[32];
        tc::tmem_ld32(tbase + TM_S + lane_addr + c0, r);
        tc::tc_wait_ld();
#pragma unroll
        for (int j = 0; j < 32; ++j) hT[(c0 + j) * kD + l128] = __uint_as_float(r[j]);
      }
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    sm100::settle(ctl.abort);
    tc::tmem_dealloc(tbase, TM_COLS);
  }
}

// ---- few sequences: the state pass in transition form ------------------------------------------------------------------------
// The state kernel above has one CTA per sequence and ~2 us of dependent tensor-memory round trips per chunk, the fused kernel
// ~3.7 us: with a handful of sequences most SMs idle.  Here a chunk's whole effect on the state is one product,
//     S' = e^{G_L} S + N S + Z,    O = Y S + A_qk U,
// with N, Z, Y, A_qk U from the intra pass, and the value columns are cut into slices of 8 NT per CTA.  Warps 0-7 keep 16 state
// rows each in registers, their bf16 copy in shared memory is the B operand; warps 8-11 compute the output beside the chain.
// Operands are bf16 where the other forwards have bf16 operands (N, Y and the copy of S), the state, Z and the sums fp32.
//
// STAGED: a chunk's operands (60 KB with 16 columns) arrive by bulk copies of a thirteenth warp, two or three chunks ahead, and each lane
// reads its fragments from shared memory as they lie, one chunk ahead.  Loaded from memory one chunk ahead, they were what the chain of
// many CTAs waited for (1.2 us a chunk, first stall the loads; 8 sequences, T=4096, whole forward: 129 -> 101 us; 16, T=1777: a layer 103 ->
// 96), while with six sequences or fewer memory answers within a chunk and the copy is a detour (four, T=3000: 60.6 against 64.0;
// six, T=2000: 49.6 against 52.5).
constexpr int kTrWorkers = 12 * 32;
template <bool STAGED> constexpr int kTrThreads = kTrWorkers + (STAGED ? 32 : 0);
template <int NT>
struct TrSmem {
  static constexpr int kStages = NT == 2 ? 3 : 2;
  static constexpr int kN = 0, kY = kN + 128 * 128 * 2, kZ = kY + 64 * 128 * 2, kO = kZ + 8 * NT * 512, kE = kO + 4 * NT * 512;
  static constexpr int kStage = kE + 512, kTotal = kStages * kStage;
};

template <int NT, bool STAGED>
__global__ void __launch_bounds__(kTrThreads<STAGED>, 1) trans_state_kernel(const __grid_constant__ IntraTransParams P) {
  using L = TrSmem<NT>;
  constexpr int VS = 8 * NT, LDS = VS + 8, SL = kD / VS, ST = L::kStages;
  const FwdParams& p = P.p;
  extern __shared__ __align__(128) uint8_t trans_smem[];   // a name of its own: see chain_kernel
  __shared__ __align__(16) __nv_bfloat16 sS[2][kD * LDS];
  __shared__ __align__(8) struct { uint64_t full[ST], empty[ST]; int abort; } ctl;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  if constexpr (STAGED) {
    if (tid == 0) {
      for (int i = 0; i < ST; ++i) {
        tc::mbar_init(tc::smem_u32(&ctl.full[i]), 1);
        tc::mbar_init(tc::smem_u32(&ctl.empty[i]), kTrWorkers / 32);
      }
      tc::fence_mbar_init();
      ctl.abort = 0;
    }
    __syncthreads();
  }
  pdl_entry();
  auto wait_bar = [&](uint64_t& bar, uint32_t parity) {
    const uint32_t at = tc::smem_u32(&bar);
    sm100::wait_inline(at, parity, &ctl.abort, at - tc::smem_u32(&ctl), warp == 12);
  };
  const int unit = blockIdx.x / SL, v0 = (blockIdx.x % SL) * VS;
  const int b = unit / p.map.H, h = unit % p.map.H, T = p.map.T, N = (T + kC - 1) / kC;
  const int64_t chunk0 = (int64_t)unit * N;
  const bool state = warp < 8;
  const int mt = state ? warp : warp - 8, r0 = 16 * mt + g, r1 = r0 + 8;
  if (STAGED && warp == 12) {
    // copies of a chunk: lane 0 N, 1 Y, 2 e^{G_L}, 3-10 the row tiles of Z, 11-14 those of A_qk U
    for (int n = 0; n < N; ++n) {
      const int st = n % ST;
      if (n >= ST) wait_bar(ctl.empty[st], (n / ST - 1) & 1);
      const uint32_t bar = tc::smem_u32(&ctl.full[st]), dst = tc::smem_u32(trans_smem) + st * L::kStage;
      if (lane == 0) tc::mbar_arrive_expect_tx(bar, L::kStage);
      __syncwarp();
      const int64_t c = chunk0 + n;
      if (lane == 0) tc::bulk_g2s(dst + L::kN, P.nf + c * 8 * 8 * 32, 128 * 128 * 2, bar);
      if (lane == 1) tc::bulk_g2s(dst + L::kY, P.yf + c * 4 * 8 * 32, 64 * 128 * 2, bar);
      if (lane == 2) tc::bulk_g2s(dst + L::kE, P.el + c * kD, 512, bar);
      if (lane >= 3 && lane < 11) tc::bulk_g2s(dst + L::kZ + (lane - 3) * NT * 512, P.zf + ((c * 8 + lane - 3) * 16 + v0 / 8) * 32, NT * 512, bar);
      if (lane >= 11 && lane < 15) tc::bulk_g2s(dst + L::kO + (lane - 11) * NT * 512, P.of + ((c * 4 + lane - 11) * 16 + v0 / 8) * 32, NT * 512, bar);
    }
    sm100::settle(ctl.abort);
    return;
  }
  uint4 a[8];
  float4 c[NT];
  float S[NT][4], el0 = 0.f, el1 = 0.f;
  // this lane's fragments of chunk n
  struct Source { const uint4* a; const float4* c; const float* el; };
  auto source = [&](int n) {
    if constexpr (STAGED) {
      const uint8_t* stage = trans_smem + n % ST * L::kStage;
      return Source{reinterpret_cast<const uint4*>(stage + (state ? L::kN : L::kY)) + mt * 8 * 32 + lane,
                    reinterpret_cast<const float4*>(stage + (state ? L::kZ : L::kO)) + mt * NT * 32 + lane, reinterpret_cast<const float*>(stage + L::kE)};
    } else {
      const int64_t at = (chunk0 + n) * (state ? 8 : 4) + mt;
      return Source{(state ? P.nf : P.yf) + at * 8 * 32 + lane, (state ? P.zf : P.of) + (at * 16 + v0 / 8) * 32 + lane, P.el + (chunk0 + n) * kD};
    }
  };
  auto arrived = [&](int n) { if constexpr (STAGED) wait_bar(ctl.full[n % ST], (n / ST) & 1); };
  auto done = [&](int n) {   // the warp has read its part of the stage
    if constexpr (STAGED) {
      __syncwarp();
      if (lane == 0) sm100::mbar_arrive(tc::smem_u32(&ctl.empty[n % ST]));
    }
  };
  auto s_at = [&](int r, int nt) { return ((int64_t)unit * kD + r) * kD + v0 + 8 * nt + 2 * t; };
  {
    arrived(0);
    const Source f = source(0);
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) a[ks] = f.a[ks * 32];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) c[nt] = f.c[nt * 32];
    if (state) { el0 = f.el[r0]; el1 = f.el[r1]; }
    done(0);
  }
  if (state) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      float2 lo = make_float2(0.f, 0.f), hi = lo;
      if (p.h0 && in_bounds_run(p.status, s_at(r0, nt), 2, p.n_state) && in_bounds_run(p.status, s_at(r1, nt), 2, p.n_state)) {
        lo = *reinterpret_cast<const float2*>(p.h0 + s_at(r0, nt));
        hi = *reinterpret_cast<const float2*>(p.h0 + s_at(r1, nt));
      }
      S[nt][0] = lo.x; S[nt][1] = lo.y; S[nt][2] = hi.x; S[nt][3] = hi.y;
    }
  }
  const int64_t o_tok = p.map.tok(kD), o_base = p.map.base(b, h, kD) + v0;
  for (int n = 0; n < N; ++n) {
    __nv_bfloat16* cS = sS[n & 1];
    if (state) {
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        *reinterpret_cast<uint32_t*>(cS + r0 * LDS + 8 * nt + 2 * t) = mma::pack(S[nt][0], S[nt][1]);
        *reinterpret_cast<uint32_t*>(cS + r1 * LDS + 8 * nt + 2 * t) = mma::pack(S[nt][2], S[nt][3]);
      }
    }
    if constexpr (STAGED) asm volatile("bar.sync 1, %0;" ::"n"(kTrWorkers) : "memory");
    else __syncthreads();
    float d[NT][4], e[NT][4];   // two accumulators: shorter chains
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      d[nt][0] = c[nt].x; d[nt][1] = c[nt].y; d[nt][2] = c[nt].z; d[nt][3] = c[nt].w;
      e[nt][0] = e[nt][1] = e[nt][2] = e[nt][3] = 0.f;
    }
    // the next chunk's fragments replace this one's as they are used
    const bool more = n + 1 < N;
    if (more) arrived(n + 1);
    const Source f = source(more ? n + 1 : n);
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) c[nt] = f.c[nt * 32];
    const uint32_t base = tc::smem_u32(cS);
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      const uint32_t ar[4] = {a[ks].x, a[ks].y, a[ks].z, a[ks].w};
      a[ks] = f.a[ks * 32];
#pragma unroll
      for (int n2 = 0; n2 < NT / 2; ++n2) {
        uint32_t bb[4];
        mma::ldsm4t(bb, mma::frag_bt(base, LDS, 16 * ks, 16 * n2, lane));
        mma::bf16((ks & 1) ? e[2 * n2] : d[2 * n2], ar, bb[0], bb[1]);
        mma::bf16((ks & 1) ? e[2 * n2 + 1] : d[2 * n2 + 1], ar, bb[2], bb[3]);
      }
    }
    float x0 = 0.f, x1 = 0.f;
    if (STAGED && state) { x0 = f.el[r0]; x1 = f.el[r1]; }
    if (more) done(n + 1);
    if (state) {
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        S[nt][0] = el0 * S[nt][0] + (d[nt][0] + e[nt][0]); S[nt][1] = el0 * S[nt][1] + (d[nt][1] + e[nt][1]);
        S[nt][2] = el1 * S[nt][2] + (d[nt][2] + e[nt][2]); S[nt][3] = el1 * S[nt][3] + (d[nt][3] + e[nt][3]);
      }
      el0 = STAGED ? x0 : f.el[r0]; el1 = STAGED ? x1 : f.el[r1];
    } else {
#pragma unroll
      for (int hr = 0; hr < 2; ++hr) {
        const int tok = n * kC + r0 + 8 * hr;
        if (tok < T) {
          const int64_t at = o_base + (int64_t)tok * o_tok + 2 * t;
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            const float x = d[nt][2 * hr] + e[nt][2 * hr], y = d[nt][2 * hr + 1] + e[nt][2 * hr + 1];
            if (!in_bounds_run(p.status, at + 8 * nt, 2, p.n_v)) continue;
            if (p.out_dt == DR_BF16) *reinterpret_cast<uint32_t*>(reinterpret_cast<__nv_bfloat16*>(p.o) + at + 8 * nt) = mma::pack(x, y);
            else *reinterpret_cast<float2*>(reinterpret_cast<float*>(p.o) + at + 8 * nt) = make_float2(x, y);
          }
        }
      }
    }
  }
  if (state && p.hT) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      if (!in_bounds_run(p.status, s_at(r0, nt), 2, p.n_state) || !in_bounds_run(p.status, s_at(r1, nt), 2, p.n_state)) continue;
      *reinterpret_cast<float2*>(p.hT + s_at(r0, nt)) = make_float2(S[nt][0], S[nt][1]);
      *reinterpret_cast<float2*>(p.hT + s_at(r1, nt)) = make_float2(S[nt][2], S[nt][3]);
    }
  }
  if constexpr (STAGED) {
    if (tid == 0) sm100::report_wait(p.status, ctl.abort);
  }
}

// bytes per chunk: N, Y bf16; Z, A_qk U, e^{G_L} fp32
constexpr int64_t kTrN = 128 * 128 * 2, kTrY = 64 * 128 * 2, kTrZ = 128 * 128 * 4, kTrO = 64 * 128 * 4, kTrE = 512;
inline int64_t trans_workspace_bytes(int64_t units, int T) {
  return units * ((T + kC - 1) / kC) * (kTrN + kTrY + kTrZ + kTrO + kTrE);
}
inline cudaError_t launch_trans(const FwdParams& p, void* workspace, int sms, cudaStream_t stream) {
  thread_local int attr_dev = -1;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (attr_dev != dev) {
    e = cudaFuncSetAttribute(intra_trans_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, IT_TOTAL);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(trans_state_kernel<2, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, TrSmem<2>::kTotal);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(trans_state_kernel<4, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, TrSmem<4>::kTotal);
    if (e != cudaSuccess) return e;
    attr_dev = dev;
  }
  const int64_t units = (int64_t)p.map.B * p.map.H, nc = units * ((p.map.T + kC - 1) / kC);
  IntraTransParams P;
  uint8_t* w = reinterpret_cast<uint8_t*>(workspace);
  P.p = p;
  P.nf = reinterpret_cast<uint4*>(w); w += nc * kTrN;
  P.yf = reinterpret_cast<uint4*>(w); w += nc * kTrY;
  P.zf = reinterpret_cast<float4*>(w); w += nc * kTrZ;
  P.of = reinterpret_cast<float4*>(w); w += nc * kTrO;
  P.el = reinterpret_cast<float*>(w);
  P.chunks = nc;
  const SeqMap& m = p.map;
  if (!sm100::make_panel_map(&P.tq, p.q, m.B, m.Hq, m.T, m.bthd != 0) || !sm100::make_panel_map(&P.tk, p.k, m.B, m.Hq, m.T, m.bthd != 0) ||
      !sm100::make_panel_map(&P.tv, p.v, m.B, m.H, m.T, m.bthd != 0) ||
      (p.variant == DR_KDA && !sm100::make_output_map(&P.tg, const_cast<void*>(p.g), m, p.g_dt == DR_BF16 ? 2 : 4)))
    return cudaErrorInvalidValue;
  e = launch_pdl(intra_trans_kernel, dim3((unsigned)nc), dim3(kThreads), IT_TOTAL, stream, P);
  if (e != cudaSuccess) return e;
  // 16 columns per CTA while the slices fit one wave: the chain's length is what counts
  if (units <= 6) return launch_pdl(trans_state_kernel<2, false>, dim3((unsigned)(units * 8)), dim3(kTrThreads<false>), 0, stream, P);   // see the kernel
  if (units * 8 <= sms) return launch_pdl(trans_state_kernel<2, true>, dim3((unsigned)(units * 8)), dim3(kTrThreads<true>), TrSmem<2>::kTotal, stream, P);
  return launch_pdl(trans_state_kernel<4, true>, dim3((unsigned)(units * 4)), dim3(kTrThreads<true>), TrSmem<4>::kTotal, stream, P);
}

template <class IP, class SP>
inline cudaError_t launch_pair(IP& I, SP& S, const FwdParams& p, void* workspace, int64_t chunk_units, int64_t units, cudaStream_t stream,
                               cudaEvent_t after_intra = nullptr) {
  thread_local int attr_dev = -1, sms = 0;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (attr_dev != dev) {
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(intra_kernel<IP>, cudaFuncAttributeMaxDynamicSharedMemorySize, IS_TOTAL);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(state_kernel<SP>, cudaFuncAttributeMaxDynamicSharedMemorySize, ST_TOTAL);
    if (e != cudaSuccess) return e;
    attr_dev = dev;
  }
  I.p = p;
  S.p = p;
  S.ws = I.ws = reinterpret_cast<uint8_t*>(workspace);
  I.chunks = (int)chunk_units;
  I.use_tma = p.variant == DR_KDA && sm100::make_panel_map(&I.tq, p.q, p.map.B, p.map.Hq, p.map.T, p.map.bthd != 0) &&
              sm100::make_panel_map(&I.tk, p.k, p.map.B, p.map.Hq, p.map.T, p.map.bthd != 0) &&
              sm100::make_output_map(&I.tg, const_cast<void*>(p.g), p.map, p.g_dt == DR_BF16 ? 2 : 4);
  if (!sm100::make_panel_map(&S.tv, p.v, p.map.B, p.map.H, p.map.T, p.map.bthd != 0)) return cudaErrorInvalidValue;
  e = launch_pdl(intra_kernel<IP>, dim3((unsigned)std::min<int64_t>(chunk_units, 2 * sms)), dim3(kIntraThreads), IS_TOTAL, stream, I);
  if (e != cudaSuccess) return e;
  if (after_intra && (e = cudaEventRecord(after_intra, stream)) != cudaSuccess) return e;
  S.use_tma_out = p.o != nullptr && sm100::make_output_map(&S.to, p.o, p.map, p.out_dt == DR_BF16 ? 2 : 4);
  return launch_pdl(state_kernel<SP>, dim3((unsigned)units), dim3(kStateThreads), ST_TOTAL, stream, S);
}

inline cudaError_t launch_chunk(const FwdParams& p, void* workspace, cudaStream_t stream, int* launches, cudaEvent_t after_intra, WideMarks marks) {
  IntraParams I;
  StateParams S;
  I.marks = marks;
  const int64_t units = (int64_t)p.map.B * p.map.H;
  *launches = 2;
  return launch_pair(I, S, p, workspace, units * ((p.map.T + kC - 1) / kC), units, stream, after_intra);
}

// Every sequence of `seqs` in one pair of launches; the workspace holds seqs.chunks records per head.
inline cudaError_t launch_chunk_packed(const FwdParams& p, const SeqTable& seqs, void* workspace, cudaStream_t stream) {
  IntraPackedParams I;
  StatePackedParams S;
  I.seqs = S.seqs = seqs;
  I.marks = WideMarks{};
  return launch_pair(I, S, p, workspace, (int64_t)seqs.chunks * p.map.H, (int64_t)seqs.n * p.map.H, stream);
}

}  // namespace kda
}  // namespace dr
