// Backward of the chunkwise delta rule for bf16 inputs at K = V = 128, C = 64 (all three variants): the adjoint split
// into what is serial over the chunks and what is not.  Formulas and names: header of dr_bwd.cuh.
//
// With W = T diag(beta) K^ e^G, Y = Q^ e^G - A W and N = -W^T Kd (Kd = K^ e^{G_L - G}) the state gradient obeys
//     dS0 = e^{G_L} dS1 + N dS1 + Y^T dO
// one [128 x 128] product per chunk and nothing else on the chain.  Three kernels:
//
//   pre_kernel    one CTA per chunk, beside the forward (q, k, g, beta only): X, A, T, and N, Y as chain_kernel's tiles.  Per-channel decays:
//                 pre_sm100_kda_kernel (dr_bwd_pre_kda.cuh), persistent, on tcgen05, and pre_kernel for the chunks that it leaves.
//   chain_kernel  one CTA per (sequence, 64 value columns) walks the chunks backwards on tcgen05, dS in registers; stores dS1 of every
//                 chunk.  N and Y as two bf16 terms; per-channel decays: three.
//   the local pass, all chunks in parallel: everything else, from S0 (the forward's checkpoint), dS1 and the chunk's inputs; then the
//                 chain rule of the normalisation and the reverse cumulative sum of dG, so that dq, dk, dv, dbeta, dg
//                 leave in their final form (with grouped q/k heads dq^, dk^ leave as one fp32 copy per head for the
//                 finalize kernel).  Scalar decays: local_sm100_kernel (dr_bwd_local_sm100.cuh), persistent, on tcgen05.  Per-channel
//                 decays: local_sm100_kda_kernel (dr_bwd_local_kda.cuh), likewise, for chunks that decay by at most 2^40, and for the others
//                 local_kernel, looping over four value slices with the sums over v in registers.
//
// The one-CTA-per-sequence-slice adjoint it replaces here walked all of a chunk's work in sequence (B=2, T=4096, H=16:
// 1.26 ms; with per-channel decay 12 ms on the CUDA cores) and stored four fp32 copies of dq^, dk^.
//
// DeltaNet / Gated DeltaNet: products on tcgen05 with two bf16 terms per float32 operand (16 bits); in pre_kernel mma.sync bf16 for the exact
// ones of X and A and one tf32 product for W, Y and N.  KDA: three tf32 products per pair (x = hi + lo; see dr_tf32.cuh) on mma.sync, i.e.
// float32 precision, as the CUDA-core adjoint it replaces; on tcgen05 two bf16 terms, in the state pass three.  On mma.sync per-channel decays never
// appear as e^{-G}: inside a 16-row block the factors are referred to the row before the block, between blocks they are carried by
// the blocks' total decays, and a block whose decay range exceeds 2^64 is summed exactly.
#pragma once

#include "dr_common.cuh"
#include "dr_mma.cuh"
#include "dr_sm100_common.cuh"
#include "dr_tf32.cuh"

namespace dr {
namespace bwdc {

using sm100::LDT;
constexpr int kC = 64, kD = 128;
constexpr int kVS = 32;   // value columns per slice

struct Params {
  const void* q; const void* k; const void* v; const void* g; const float* beta; const void* d_o; const float* d_hT;
  void* dq; void* dk; void* dv; float* dbeta; float* dg; float* dh0;
  const float* ckpt;    // [units][N][128][128] state at the start of every chunk
  float4* nf;           // [units][N] kNTile bytes
  float4* yf;           // [units][N] kYTile bytes
  float* xat;           // [units][N][3][64][64] X, A, T; scalar decays: A and T as two bf16 terms, the tiles of local_sm100_kernel; KDA: see kXWide
  float* ds;            // [units][N][128][128] dS1
  float* el;            // [units][N][128] e^{G_L}
  float* norms;         // scalar decays: [units][N][2][64] norm factors of k and q
  float* part;          // grouped heads: dq^ [units][N*64][128], then dk^ (over nf)
  SeqMap map;
  int N, variant, g_dt, l2norm;
  int few;              // KDA: pre_kernel and local_kernel take every chunk, one per CTA (see kFewKda, make_params)
  float scale;
};

// float2 from shared memory
__device__ __forceinline__ float2 ld2(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float bf(const __nv_bfloat16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ float ex2(float x) { return tc::fast_exp2(x); }
constexpr float kLog2e = 1.4426950408889634f;

using mma::AFrag;
using mma::BFrag;
using mma::fma;
__device__ __forceinline__ void zero4(float (&d)[4]) { d[0] = d[1] = d[2] = d[3] = 0.f; }
// Operands of chain_kernel in memory: N [128][128] and Y^T [128][64] as two bf16 terms each, tiles of 8 x 8 core matrices.
constexpr int kNTile = 2 * 128 * 128 * 2, kYTile = 2 * 128 * 64 * 2, kYRbs = 8 * 128;
// an m16n8 accumulator (rows r, r + 8; two neighbouring columns) -> its two terms, `next` bytes to the rows 8 further on and `lo`
// bytes to the second term; a warp writes 128 contiguous bytes per store
__device__ __forceinline__ void store_terms(uint8_t* dst, int next, int lo, const float (&d)[4]) {
#pragma unroll
  for (int hr = 0; hr < 2; ++hr) {
    const uint32_t h = mma::pack(d[2 * hr], d[2 * hr + 1]);
    *reinterpret_cast<uint32_t*>(dst + hr * next) = h;
    *reinterpret_cast<uint32_t*>(dst + hr * next + lo) = mma::pack(d[2 * hr] - mma::lo_f(h), d[2 * hr + 1] - mma::hi_f(h));
  }
}

// two floats as two packed bf16 terms
__device__ __forceinline__ void split2(float x, float y, uint32_t& hi, uint32_t& lo) {
  hi = mma::pack(x, y);
  lo = mma::pack(x - mma::lo_f(hi), y - mma::hi_f(hi));
}
// four channels of the log decay in log2 units
__device__ __forceinline__ float4 load_g4(const void* g, int64_t at, int dt) {
  float4 x;
  if (dt == DR_BF16) {
    const uint2 u = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(g) + at);
    x = make_float4(mma::lo_f(u.x), mma::hi_f(u.x), mma::lo_f(u.y), mma::hi_f(u.y));
  } else {
    x = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(g) + at);
  }
  return make_float4(x.x * kLog2e, x.y * kLog2e, x.z * kLog2e, x.w * kLog2e);
}
// Per-channel decays: what is kept among X, A, T in places that neither form of X uses: the norm factors of k and q (four rows of 32; the pre-pass) and
// whether the chunk is pre_kernel's and local_kernel's (a channel decays by more than 2^40, or a decay is positive) or pre_sm100_kda_kernel's and
// local_sm100_kda_kernel's (the forward, see WideMarks).  local_kernel's chunks have X, A, T as rows, the others X by columns in fours, A and T - I as two bf16 terms in tiles.
constexpr float kWideKda = 40.f;   // log2 units
constexpr int kXNorms = 1056, kXNormRow = 256, kXWide = 2096;
// pre_kernel's and local_kernel's chunks in a list, entry i beside chunk i's mark, and in chunk 0's place its length and how many of them either kernel has
// taken; the forward's first kernel sets the three to zero, pre_sm100_kda_kernel fills the list.  CTAs take the entries one by one: dealt out
// beforehand, those whose SM the forward's state pass holds would do their share behind it (training step of 2048 such chunks 1711 us).
constexpr int kXList = kXWide + 1, kXCounts = kXWide + 2;

// The power of two that brings `top` to 2^40 .. 2^41 (none for zero and infinity; at most 2^126); its inverse
__device__ __forceinline__ float lift(uint32_t top) {
  const uint32_t e = top >> 23;
  return top == 0u || e == 255u ? 1.f : __uint_as_float(min(294u - e, 253u) << 23);
}
__device__ __forceinline__ float drop(uint32_t top) { return __uint_as_float((254u << 23) - __float_as_uint(lift(top))); }
// Per-channel decays: Y^T and the two halves of N's columns in float32, [128 rows][64 columns] each: eight columns of a row are a unit, eight rows'
// units of the same columns follow each other; the first four columns of all units, then the others.  An m16n8 accumulator (lane g, t) of column
// tile nt, rows r0 + g and eight further on.
constexpr int kHalf4 = 128 * 64 / 4;   // float4 of one such array
__device__ __forceinline__ void store_f32(float4* dst, int r0, int nt, int g, int t, const float (&d)[4]) {
#pragma unroll
  for (int hr = 0; hr < 2; ++hr)
    reinterpret_cast<float2*>(dst + (t >> 1) * (kHalf4 / 2) + ((r0 >> 3) + hr) * 64 + nt * 8 + g)[t & 1] = make_float2(d[2 * hr], d[2 * hr + 1]);
}
__device__ __forceinline__ void l2_panel(const void* tmap, int c0, int c1, int c2, int c3) {
  asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global [%0, {%1, %2, %3, %4}];" ::"l"(tmap), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
__device__ __forceinline__ void l2_bulk(const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}
// Those of the chunks blockIdx.x, + gridDim.x, .. that tcgen05 takes; warp-uniform, one read per 32 of them.
struct ChunkList {
  int base;
  uint32_t mask;
  __device__ __forceinline__ void start(const Params& p, int chunks, int lane) {
    base = blockIdx.x;
    fetch(p, chunks, lane);
  }
  __device__ __forceinline__ void fetch(const Params& p, int chunks, int lane) {
    const int64_t c = base + (int64_t)lane * gridDim.x;
    mask = __ballot_sync(0xffffffffu, c < chunks && __ldcg(p.xat + c * (3 * 64 * 64) + kXWide) == 0.f);
  }
  __device__ __forceinline__ int next(const Params& p, int chunks, int lane) {   // `chunks` behind the last
    while (mask == 0u) {
      if ((int64_t)base + 32 * gridDim.x >= chunks) return chunks;
      base += 32 * gridDim.x;
      fetch(p, chunks, lane);
    }
    const int i = __ffs(mask) - 1;
    mask &= mask - 1;
    return base + i * (int)gridDim.x;
  }
};
// The others: into the list (one warp per CTA) ..
__device__ __forceinline__ void list_wide(const Params& p, int chunks, int lane) {
  int* counts = reinterpret_cast<int*>(p.xat + kXCounts);
  for (int64_t base = blockIdx.x; base < chunks; base += 32 * (int64_t)gridDim.x) {
    const int64_t c = base + (int64_t)lane * gridDim.x;
    const bool wide = c < chunks && __ldcg(p.xat + c * (3 * 64 * 64) + kXWide) != 0.f;
    const uint32_t mask = __ballot_sync(0xffffffffu, wide);
    if (mask == 0u) continue;
    int at = 0;
    if (lane == 0) at = atomicAdd(counts, __popc(mask));
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(mask & ((1u << lane) - 1u));
    if (wide) reinterpret_cast<int*>(p.xat + (int64_t)at * (3 * 64 * 64))[kXList] = (int)c;
  }
}
// .. and from it (one thread per CTA): a number, and the chunk that has it, or `chunks`.  Kernel 0: pre_kernel, 1: local_kernel.  Without a list (p.few): one
// chunk per CTA.
__device__ __forceinline__ int take_number(const Params& p, int kernel, bool first) {
  int* counts = reinterpret_cast<int*>(p.xat + kXCounts);
  return p.few ? (first ? (int)blockIdx.x : 0x7fffffff) : __ldcg(counts) == 0 ? 0x7fffffff : atomicAdd(counts + 1 + kernel, 1);
}
__device__ __forceinline__ int numbered(const Params& p, int chunks, int i) {
  if (p.few) return min(i, chunks);
  return i < __ldcg(reinterpret_cast<const int*>(p.xat + kXCounts)) ? __ldcg(reinterpret_cast<const int*>(p.xat + (int64_t)i * (3 * 64 * 64)) + kXList) : chunks;
}
// Few chunks, in short sequences: a training step is bound by the host, and the two launches that look for wide chunks cost more than the kernels on
// tcgen05 give; every chunk is then treated as a wide one.  Whole step, so / as wide and narrow chunks: 20 chunks in 4 sequences 132 / 139 us, 40 in 4
// 134 / 140, 80 in 16 133 / 138; 64 in 4 152 / 139, 128 in 8 159 / 139.
constexpr int kFewKda = 80, kFewLength = 10;
// =====================================================================================================================
// pre_kernel
// =====================================================================================================================
constexpr int kPreThreads = 256;
constexpr int LDH = 136;   // row stride (bf16) of the raw k, q rows
constexpr int PR_K = 0, PR_Q = PR_K + 64 * LDH * 2, PR_X = PR_Q + 64 * LDH * 2, PR_A = PR_X + 64 * LDT * 4;
constexpr int PR_SC = PR_A + 64 * 72 * 4;     // beta, rk, rq, G, fw, fd (64 each)
constexpr int LDG = 136;   // row stride of G: pairs of eight rows are read without bank conflicts
constexpr int LDK = 130;   // row stride (16-byte entries) of the split Kd
constexpr int PR_G = PR_SC + 6 * 64 * 4;      // KDA: log2(e) G [64][136]; Kd as token pairs [32][130] (hi, hi, lo, lo) later over k, q, X, A
constexpr int PR_TAKEN = PR_G + 64 * LDG * 4;
template <bool KDA> constexpr int pre_smem() { return KDA ? PR_TAKEN + 16 : PR_G; }
static_assert(PR_SC >= 32 * LDK * 16 && 2 * (pre_smem<true>() + 1024) <= 233472, "two CTAs per SM");

template <bool KDA>
__global__ void __launch_bounds__(kPreThreads, 2) pre_kernel(const Params p, const int chunks) {
  pdl_entry();
  extern __shared__ __align__(16) uint8_t smem[];
  __nv_bfloat16* sK = reinterpret_cast<__nv_bfloat16*>(smem + PR_K);
  __nv_bfloat16* sQ = reinterpret_cast<__nv_bfloat16*>(smem + PR_Q);
  uint4* sKd = reinterpret_cast<uint4*>(smem + PR_K);
  float* sX = reinterpret_cast<float*>(smem + PR_X);
  float* sA = reinterpret_cast<float*>(smem + PR_A);
  float* sBeta = reinterpret_cast<float*>(smem + PR_SC);
  float *sRk = sBeta + 64, *sRq = sBeta + 128, *sGs = sBeta + 192, *sFw = sBeta + 256, *sFd = sBeta + 320;
  float* sG = reinterpret_cast<float*>(smem + PR_G);
  int* const taken = reinterpret_cast<int*>(smem + PR_TAKEN);   // KDA: [2], by turns
  if (KDA && threadIdx.x == 0) taken[0] = numbered(p, chunks, take_number(p, 0, true));
#pragma unroll 1
  for (int turn = 0; KDA || turn == 0; turn ^= 1) {
  int tid = threadIdx.x, c = blockIdx.x;
  if constexpr (KDA) {
    __syncthreads();   // the chunk before is done with shared memory
    c = taken[turn];
    if (c >= chunks) break;
    asm volatile("" : "+r"(tid));   // (see local_kernel)
    if (tid == 0) taken[turn ^ 1] = numbered(p, chunks, take_number(p, 0, false));
  }
  const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int64_t chunk = c;
  const int unit = c / p.N, n = c % p.N;
  const int b = unit / p.map.H, h = unit % p.map.H, t0 = n * kC, rows = min(kC, p.map.T - t0);
  const int64_t qk_base = p.map.base_qk(b, h, kD), qk_tok = p.map.tok_qk(kD);
  const int64_t gk_base = p.map.base(b, h, kD), gk_tok = p.map.tok(kD);
  const int64_t s_base = p.map.base(b, h, 1), s_tok = p.map.tok(1);
  // ---- raw rows, norm factors, decay --------------------------------------------------------------------------------
  {
    uint2 qr[8], kr[8];
    float4 gr[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int c = warp + 8 * i;
      qr[i] = kr[i] = make_uint2(0u, 0u);
      gr[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c < rows) {
        const int64_t at = qk_base + (t0 + c) * qk_tok + 4 * lane;
        qr[i] = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(p.q) + at);
        kr[i] = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(p.k) + at);
        if constexpr (KDA) gr[i] = load_g4(p.g, gk_base + (t0 + c) * gk_tok + 4 * lane, p.g_dt);
      }
    }
    float bt = 0.f, g_lo = 0.f, g_hi = 0.f;
    if (lane < 8 && warp + 8 * lane < rows) bt = p.beta[s_base + (t0 + warp + 8 * lane) * s_tok];
    if (!KDA && warp == 0 && p.variant == DR_GATED) {
      if (lane < rows) g_lo = ld_elem(p.g, s_base + (t0 + lane) * s_tok, p.g_dt);
      if (lane + 32 < rows) g_hi = ld_elem(p.g, s_base + (t0 + lane + 32) * s_tok, p.g_dt);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int c = warp + 8 * i;
      *reinterpret_cast<uint2*>(sQ + c * LDH + 4 * lane) = qr[i];
      *reinterpret_cast<uint2*>(sK + c * LDH + 4 * lane) = kr[i];
      if constexpr (KDA) *reinterpret_cast<float4*>(sG + c * LDG + 4 * lane) = gr[i];
    }
    // norm factors of the warp's 16 rows: the sums are scattered over the lanes as they are reduced, so that each lane takes one
    // square root and one quotient
    float ss[16];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float q0 = mma::lo_f(qr[i].x), q1 = mma::hi_f(qr[i].x), q2 = mma::lo_f(qr[i].y), q3 = mma::hi_f(qr[i].y);
      const float k0 = mma::lo_f(kr[i].x), k1 = mma::hi_f(kr[i].x), k2 = mma::lo_f(kr[i].y), k3 = mma::hi_f(kr[i].y);
      ss[i] = q0 * q0 + q1 * q1 + q2 * q2 + q3 * q3;
      ss[8 + i] = k0 * k0 + k1 * k1 + k2 * k2 + k3 * k3;
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
      (lane < 16 ? sRq : sRk)[warp + 8 * ((lane >> 1) & 7)] = p.l2norm ? top / (sqrtf(ss[0]) + 1e-6f) : top;
    }
    if (lane < 8) sBeta[warp + 8 * lane] = bt;
    if (!KDA && warp == 0) {
      mma::scan_scalars(g_lo, g_hi, lane);
      sGs[lane] = g_lo; sGs[lane + 32] = g_hi;
    }
  }
  __syncthreads();
  if constexpr (KDA) {
    mma::scan_channels<kPreThreads, kD, LDG>(sG, sX, tid);
    if (tid < 128) p.el[chunk * 128 + tid] = ex2(sG[63 * LDG + tid]);
    if (tid < 64) { sFw[tid] = sBeta[tid] * sRk[tid]; }
  } else {
    const float gl = sGs[63];
    if (tid < 128) p.el[chunk * 128 + tid] = expf(gl);
    if (tid < 64) {   // factors of row j of k in W and in Kd
      sFw[tid] = sBeta[tid] * sRk[tid] * expf(sGs[tid]);
      sFd[tid] = sRk[tid] * expf(fminf(gl - sGs[tid], 0.f));
    }
  }
  // ---- X = tril(K^K^^T.E, -1), A = tril(Q^K^^T.E): 20 tiles of 16 x 8 at or below the diagonal dealt to the warps ----------
  auto unsafe = [&](int blk) -> bool {   // KDA, warp-uniform: the decay inside the block exceeds 2^64 in some channel
    const float4 ga = *reinterpret_cast<const float4*>(sG + 16 * blk * LDG + 4 * lane);
    const float4 gb = *reinterpret_cast<const float4*>(sG + (16 * blk + 15) * LDG + 4 * lane);
    return __any_sync(0xffffffffu, !(fmaxf(fmaxf(ga.x - gb.x, ga.y - gb.y), fmaxf(ga.z - gb.z, ga.w - gb.w)) <= 64.f));
  };
  if constexpr (KDA) {
    // eight warp tasks (16-row block; 8-column tiles)  3;0-2  3;3-5  3;6-7  2;0-2  2;3-5  1;0-1  1;2-3  0;0-1: the decayed rows are formed
    // once for a task's tiles; the contraction runs over pairs of neighbouring channels
    const int mt = warp < 3 ? 3 : warp < 5 ? 2 : warp < 7 ? 1 : 0;
    const int nt0 = warp < 3 ? 3 * warp : warp < 5 ? 3 * (warp - 3) : warp < 7 ? 2 * (warp - 5) : 0;
    const int ntn = (warp == 2 || warp >= 5) ? 2 : 3;
    const bool skip = unsafe(mt);   // the diagonal block is done exactly below
    const int r0 = 16 * mt + g, r1 = r0 + 8, nrow = 16 * mt;
    float dk[3][4], dq[3][4];
#pragma unroll
    for (int x = 0; x < 3; ++x) { zero4(dk[x]); zero4(dq[x]); }
#pragma unroll 2
    for (int ks = 0; ks < 16; ++ks) {
      const int c = 8 * ks + 2 * t;
      const float2 gn = ld2(sG + nrow * LDG + c), ga = ld2(sG + r0 * LDG + c), gb = ld2(sG + r1 * LDG + c);
      const float e00 = ex2(ga.x - gn.x), e01 = ex2(ga.y - gn.y), e10 = ex2(gb.x - gn.x), e11 = ex2(gb.y - gn.y);
      const uint32_t k0 = *reinterpret_cast<const uint32_t*>(sK + r0 * LDH + c), k1 = *reinterpret_cast<const uint32_t*>(sK + r1 * LDH + c);
      const uint32_t q0 = *reinterpret_cast<const uint32_t*>(sQ + r0 * LDH + c), q1 = *reinterpret_cast<const uint32_t*>(sQ + r1 * LDH + c);
      AFrag<true> ak, aq;
      ak.set(mma::lo_f(k0) * e00, mma::lo_f(k1) * e10, mma::hi_f(k0) * e01, mma::hi_f(k1) * e11);
      aq.set(mma::lo_f(q0) * e00, mma::lo_f(q1) * e10, mma::hi_f(q0) * e01, mma::hi_f(q1) * e11);
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        if (x < ntn && !(skip && nt0 + x >= 2 * mt)) {
          const int j = 8 * (nt0 + x) + g;
          const float2 gj = ld2(sG + j * LDG + c);
          const uint32_t kj = *reinterpret_cast<const uint32_t*>(sK + j * LDH + c);
          BFrag<true> bk;
          bk.set(mma::lo_f(kj) * ex2(gn.x - gj.x), mma::hi_f(kj) * ex2(gn.y - gj.y));
          fma<true>(dk[x], ak, bk);
          fma<true>(dq[x], aq, bk);
        }
      }
    }
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      if (x < ntn && !(skip && nt0 + x >= 2 * mt)) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int i = 16 * mt + g + 8 * (e >> 1), j = 8 * (nt0 + x) + 2 * t + (e & 1);
          sX[i * LDT + j] = j < i ? dk[x][e] * sRk[j] * sRk[i] : 0.f;
          sA[i * 72 + j] = j <= i ? dq[x][e] * sRk[j] * sRq[i] : 0.f;
        }
      }
    }
  } else {
#pragma unroll 1
  for (int tile = warp; tile < 20; tile += kPreThreads / 32) {   // raw bf16 rows: exact products
    const int mt = tile < 2 ? 0 : tile < 6 ? 1 : tile < 12 ? 2 : 3, nt = tile - mt * (mt + 1);
    float dk[4], dq[4];
    zero4(dk); zero4(dq);
      const uint32_t aK = tc::smem_u32(sK), aQ = tc::smem_u32(sQ);
#pragma unroll
      for (int k2 = 0; k2 < 4; ++k2) {
        uint32_t a0[4], a1[4], q0[4], q1[4], bb[4];
        mma::ldsm4(bb, aK + 2u * ((8 * nt + (lane & 7)) * LDH + 32 * k2 + (lane >> 3) * 8));
        mma::ldsm4(a0, mma::frag_a(aK, LDH, 16 * mt, 32 * k2, lane));
        mma::ldsm4(a1, mma::frag_a(aK, LDH, 16 * mt, 32 * k2 + 16, lane));
        mma::ldsm4(q0, mma::frag_a(aQ, LDH, 16 * mt, 32 * k2, lane));
        mma::ldsm4(q1, mma::frag_a(aQ, LDH, 16 * mt, 32 * k2 + 16, lane));
        mma::bf16(dk, a0, bb[0], bb[1]);
        mma::bf16(dq, q0, bb[0], bb[1]);
        mma::bf16(dk, a1, bb[2], bb[3]);
        mma::bf16(dq, q1, bb[2], bb[3]);
      }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = 16 * mt + g + 8 * (e >> 1), j = 8 * nt + 2 * t + (e & 1);
      const float f = sRk[j] * __expf(fminf(sGs[i] - sGs[j], 0.f));
      sX[i * LDT + j] = j < i ? dk[e] * f * sRk[i] : 0.f;
      sA[i * 72 + j] = j <= i ? dq[e] * f * sRq[i] : 0.f;
    }
  }
  }
  if constexpr (KDA) {   // diagonal blocks with too wide a decay range: exactly, one entry per thread
    for (int blk = 0; blk < 4; ++blk) {
      if (!unsafe(blk)) continue;
      const int i = 16 * blk + (tid >> 4), j = 16 * blk + (tid & 15);
      float ak = 0.f, aq = 0.f;
      if (j <= i)
        for (int c = 0; c < kD; ++c) {
          const float w = bf(sK + j * LDH + c) * ex2(fminf(sG[i * LDG + c] - sG[j * LDG + c], 0.f));
          ak += bf(sK + i * LDH + c) * w;
          aq += bf(sQ + i * LDH + c) * w;
        }
      sX[i * LDT + j] = j < i ? ak * sRk[i] * sRk[j] : 0.f;
      sA[i * 72 + j] = j <= i ? aq * sRq[i] * sRk[j] : 0.f;
    }
  }
  __syncthreads();
  // ---- X, A -> global (16 x 16 blocks at or below the diagonal), then T in place of X ----------------------------------------
  float* xat = p.xat + chunk * (3 * 64 * 64);
  for (int i = tid; i < 64 * 16; i += kPreThreads) {
    const int r = i >> 4, c4 = (i & 15) * 4;
    if ((c4 >> 4) <= (r >> 4)) {
      // (scalar decays: columns in fours, so that a warp of the reader takes 32 rows of four at once)
      *reinterpret_cast<float4*>(xat + (KDA ? r * 64 + c4 : c4 * 64 + 4 * r)) = *reinterpret_cast<const float4*>(sX + r * LDT + c4);
      if constexpr (KDA) *reinterpret_cast<float4*>(xat + 4096 + r * 64 + c4) = *reinterpret_cast<const float4*>(sA + r * 72 + c4);
    }
  }
  // scalar decays: A, T as core matrices of 8 x 8, the blocks of eight rows next to each other; high terms, then low ones
  auto put_tile = [&](const float* src, int ld, float* dst) {
#pragma unroll
    for (int x = 0; x < 512 / kPreThreads; ++x) {
      const int i = tid + kPreThreads * x, r = 8 * ((i >> 3) & 7) + (i & 7), c = 8 * (i >> 6);
      if ((c >> 4) > (r >> 4)) continue;
      uint32_t h[4], l[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 y = ld2(src + r * ld + c + 2 * e);
        split2(c + 2 * e <= r ? y.x : 0.f, c + 2 * e + 1 <= r ? y.y : 0.f, h[e], l[e]);
      }
      reinterpret_cast<uint4*>(dst)[i] = make_uint4(h[0], h[1], h[2], h[3]);
      reinterpret_cast<uint4*>(dst)[512 + i] = make_uint4(l[0], l[1], l[2], l[3]);
    }
  };
  if constexpr (!KDA) {
    put_tile(sA, 72, xat + 4096);
    if (tid < 128) p.norms[chunk * 128 + tid] = (tid < 64 ? sRk : sRq - 64)[tid];
  }
  __syncthreads();
  sm100::block_inverse_64(sX, sBeta, sX, tid);   // ends with a barrier
  if constexpr (!KDA) put_tile(sX, LDT, xat + 8192);
  for (int i = tid; KDA && i < 64 * 16; i += kPreThreads) {
    const int r = i >> 4, c4 = (i & 15) * 4;
    if ((c4 >> 4) <= (r >> 4)) {
      float4 v = *reinterpret_cast<const float4*>(sX + r * LDT + c4);
      if (c4 + 0 > r) v.x = 0.f;
      if (c4 + 1 > r) v.y = 0.f;
      if (c4 + 2 > r) v.z = 0.f;
      if (c4 + 3 > r) v.w = 0.f;
      *reinterpret_cast<float4*>(xat + 8192 + r * 64 + c4) = v;
    }
  }
  // ---- W^T: rows = the warp's 16 channels, columns = tokens; W = T diag(beta) K^ e^G ----------------------------------------
  constexpr bool X3 = KDA;
  const int ch0 = 16 * warp + g, ch1 = ch0 + 8;
  float W[8][4];
#pragma unroll
  for (int nt = 0; nt < 8; ++nt) zero4(W[nt]);
#pragma unroll
  for (int ks = 0; ks < 8; ++ks) {
    const int j0 = 8 * ks + t, j1 = j0 + 4;
    float a0 = bf(sK + j0 * LDH + ch0), a1 = bf(sK + j0 * LDH + ch1), a2 = bf(sK + j1 * LDH + ch0), a3 = bf(sK + j1 * LDH + ch1);
    if constexpr (KDA) {
      a0 *= ex2(sG[j0 * LDG + ch0]); a1 *= ex2(sG[j0 * LDG + ch1]);
      a2 *= ex2(sG[j1 * LDG + ch0]); a3 *= ex2(sG[j1 * LDG + ch1]);
    }
    AFrag<X3> a;
    a.set(a0, a1, a2, a3);
    const float f0 = sFw[j0], f1 = sFw[j1];
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
      if (nt >= ks) {
        const int i = 8 * nt + g;
        BFrag<X3> bt;
        bt.set(j0 <= i ? sX[i * LDT + j0] * f0 : 0.f, j1 <= i ? sX[i * LDT + j1] * f1 : 0.f);
        fma<X3>(W[nt], a, bt);
      }
    }
  }
  // ---- Y^T = (Q^ e^G)^T - W^T A^T -> tiles (an accumulator is a fragment with its columns as k) ---------------------------------------
  {
    float Y[8][4];
#pragma unroll
    for (int nt = 0; nt < 8; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int ch = e < 2 ? ch0 : ch1, i = 8 * nt + 2 * t + (e & 1);
        Y[nt][e] = bf(sQ + i * LDH + ch) * sRq[i] * (KDA ? ex2(sG[i * LDG + ch]) : expf(sGs[i]));
      }
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      AFrag<X3> a;
      a.set(-W[ks][0], -W[ks][2], -W[ks][1], -W[ks][3]);
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) {
        if (nt >= ks) {
          const float2 y = ld2(sA + (8 * nt + g) * 72 + 8 * ks + 2 * t);
          BFrag<X3> ba;
          ba.set(y.x, y.y);
          fma<X3>(Y[nt], a, ba);
        }
      }
    }
    uint8_t* dst = reinterpret_cast<uint8_t*>(p.yf) + chunk * kYTile + 2 * warp * kYRbs + g * 16 + 4 * t;
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
      if constexpr (KDA) store_f32(p.yf + chunk * kHalf4, 16 * warp, nt, g, t, Y[nt]);
      else store_terms(dst + nt * 128, kYRbs, kYTile / 2, Y[nt]);
    }
  }
  // ---- N = -W^T Kd -> tiles -----------------------------------------------------------------------------------------------
  if constexpr (KDA) {
    // lane = channels lane, lane + 32, ..; warp = token pairs warp, warp + 8, ..; split into the two terms once
    uint4 kd[4][4];
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const int c = lane + 32 * x;
      const float gl = sG[63 * LDG + c];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = 2 * (warp + 8 * i);
        BFrag<true> f;
        f.set(bf(sK + r * LDH + c) * sRk[r] * ex2(gl - sG[r * LDG + c]), bf(sK + (r + 1) * LDH + c) * sRk[r + 1] * ex2(gl - sG[(r + 1) * LDG + c]));
        kd[i][x] = make_uint4(f.h[0], f.h[1], f.l[0], f.l[1]);
      }
    }
    __syncthreads();   // every read of k, q, X and A is done
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int x = 0; x < 4; ++x) sKd[(warp + 8 * i) * LDK + lane + 32 * x] = kd[i][x];
    __syncthreads();
  }
#pragma unroll 1
  for (int half = 0; half < 2; ++half) {
    float d[8][4];
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) zero4(d[nt]);
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      const int i0 = 8 * ks + 2 * t;
      const float f0 = KDA ? -1.f : -sFd[i0], f1 = KDA ? -1.f : -sFd[i0 + 1];
      AFrag<X3> a;
      a.set(W[ks][0] * f0, W[ks][2] * f0, W[ks][1] * f1, W[ks][3] * f1);
#pragma unroll
      for (int nt = 0; nt < 8; ++nt) {
        const int c = 64 * half + 8 * nt + g;
        BFrag<X3> bk;
        if constexpr (KDA) {
          const uint4 y = sKd[(4 * ks + t) * LDK + c];
          bk.h[0] = y.x; bk.h[1] = y.y; bk.l[0] = y.z; bk.l[1] = y.w;
        } else {
          bk.set(bf(sK + i0 * LDH + c), bf(sK + (i0 + 1) * LDH + c));
        }
        fma<X3>(d[nt], a, bk);
      }
    }
    uint8_t* dst = reinterpret_cast<uint8_t*>(p.nf) + chunk * kNTile + 2 * warp * sm100::RBS + 8 * half * 128 + g * 16 + 4 * t;
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
      if constexpr (KDA) store_f32(p.nf + (2 * chunk + half) * kHalf4, 16 * warp, nt, g, t, d[nt]);
      else store_terms(dst + nt * 128, sm100::RBS, kNTile / 2, d[nt]);
    }
  }
  }
}

// =====================================================================================================================
// chain_kernel: the state pass on tcgen05, one CTA per (sequence, 64 value columns)
//
// dS stays in registers (thread = channel row, 32 columns); its two bf16 terms are the B operand, N and Y^T arrive by bulk copies as
// the A operands, two terms each: three products N dS and two Y^T dO per 16 channels or tokens, 16 bits of every operand where
// one tf32 product had 11.  Y^T dO of a chunk is issued while the chunk before it is still on its way through the registers, into
// the other accumulator.  The chain per chunk: terms of dS -> 24 products -> multiply-add.
//
// What bounds it: B=2, T=4096, H=16 (64 CTAs): 105 us, 158 as mma.sync tf32 products over 128 CTAs (every warp read all of dS: shared
// memory 62 %); gradient of the initial state against float64 3.2e-4 -> 2.4e-4.  The products of a chunk take 1.2 K cycles, its 100 KB of
// operands 1.8 K at 55 bytes a clock.  Asking for the operands five chunks ahead in L2: 12 us slower.  Counters (16 sequences, 64
// chunks): 2.75 K cycles and 1.95 K warp instructions per chunk, tensor pipe 37 %, issue slots 18 %.
//
// Taken at every size.  The backward's kernels against those with the mma.sync pass, 16 sequences of one, two and three chunks: 35.2 ->
// 37.2 us, 37.5 -> 38.6, 39.4 -> 40.0, initial state's gradient included (asking for the tensor map earlier or leaving out N dS
// while dS is zero does not change that).  Forward and backward together, 1 to 256 sequences: 1 to 9 % faster at five chunks, 4 to
// 13 % at 16, 6 to 14 % at 64; from 48 sequences on ahead or level at every length.
// =====================================================================================================================
// Per-channel decays: the N of a strongly decaying chunk is as small as the decay, row by row, and what it adds to dS as large as the rest, so
// float32 operands are three bf16 terms each (24 bits of every entry, float32's exponents), six products per pair.  N and Y arrive in float32 by
// bulk copies; eight more warps turn them into terms in tensor memory, N in halves of 64 channels: the first as soon as the products with the chunk
// before's first half are done, so that it is ready when they all are.  Y^T d_o has accumulators of its own.  B=2, T=4096, H=16: 153 us under ncu, where
// two fp16 terms of operands scaled as a whole take 138 to 145 and lose N, and with it every gradient before such a chunk, from 0.35 nats a
// token in every channel on; with the terms in shared memory and N by loads into registers 310 us (no L1 to load through).
constexpr int kChThreads = 288, kChCols = 64;   // eight worker warps and one that issues
constexpr int kChSplit = 256;
template <bool KDA> constexpr int ch_threads() { return kChThreads + (KDA ? kChSplit : 0); }
// N hi twice, N lo, Y^T and d_o twice, the terms of dS, staging of its rows
constexpr int kNTerm = kNTile / 2, kSTerm = 128 * 128, kOTile = 64 * 128;
constexpr int CH_H = 0, CH_L = CH_H + 2 * kNTerm, CH_Y = CH_L + kNTerm, CH_O = CH_Y + 2 * kYTile, CH_S = CH_O + 2 * kOTile, CH_G = CH_S + 2 * kSTerm, CH_TOTAL = CH_G + 8 * 2048;
// per-channel decays: the terms of dS, d_o twice, staging, Y^T, three halves of N as they arrive
constexpr int kHalfTile = kHalf4 * 16, kHalfSlots = 3;
constexpr int CK_S = 0, CK_O = CK_S + 3 * kSTerm, CK_G = CK_O + 2 * kOTile, CK_Y = CK_G + 8 * 2048, CK_N = CK_Y + kHalfTile, CK_TOTAL = CK_N + kHalfSlots * kHalfTile;
static_assert(CH_O % 1024 == 0 && CH_S % 1024 == 0 && CK_O % 1024 == 0 && CH_TOTAL <= 232448 - 1024 && CK_TOTAL <= 232448 - 1024, "shared memory");
template <bool KDA> constexpr int ch_smem() { return KDA ? CK_TOTAL : CH_TOTAL; }
struct alignas(64) ChainParams {
  CUtensorMap to;   // panels of d_o (see sm100::make_panel_map)
  Params p;
  int32_t* status;
};

template <bool KDA>
__global__ void __launch_bounds__(ch_threads<KDA>(), 1) chain_kernel(const __grid_constant__ ChainParams P) {
  const Params& p = P.p;
  // a name of its own: declarations of one name in a namespace share the first one's alignment
  extern __shared__ __align__(1024) uint8_t chain_smem[];
  uint8_t* const smem = chain_smem;
  __shared__ __align__(8) struct {
    // (Y^T d_o of a chunk may be done before the slowest worker asks for the chunk before's, hence two barriers by turns; tests/test_chain_handover.py)
    // Per-channel decays: full_h: terms of N's halves, full_l: terms of Y, full_y[0]: Y has arrived, full_n: halves of N have, bar_e: products with N's first half
    uint64_t full_h[2], full_l, full_y[2], rdy, bar_y[2], bar_d, full_o[2], full_n[kHalfSlots], bar_e;
    uint32_t tmem_base;
    int abort;
  } ctl;
  // KDA: N dS behind the two accumulators of Y^T d_o, then the terms of N (64 columns each) and of Y
  constexpr uint32_t kTmem = KDA ? 512 : 128, kTmemN = 128, kTmemA = 192, kTmemY = kTmemA + 3 * 64;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int unit = blockIdx.x / (kD / kChCols), v0 = blockIdx.x % (kD / kChCols) * kChCols;
  const int b = unit / p.map.H, h = unit % p.map.H;
  if (warp == 0) {
    tc::tmem_alloc(tc::smem_u32(&ctl.tmem_base), kTmem);
    tc::tmem_relinquish();
  }
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(tc::smem_u32(&ctl.full_o[i]), 1);
      tc::mbar_init(tc::smem_u32(&ctl.full_h[i]), KDA ? kChSplit : 1);
      tc::mbar_init(tc::smem_u32(&ctl.full_y[i]), 1);
    }
    for (int i = 0; i < kHalfSlots; ++i) tc::mbar_init(tc::smem_u32(&ctl.full_n[i]), 1);
    tc::mbar_init(tc::smem_u32(&ctl.bar_e), 1);
    tc::mbar_init(tc::smem_u32(&ctl.full_l), KDA ? kChSplit : 1);
    tc::mbar_init(tc::smem_u32(&ctl.rdy), 256);
    tc::mbar_init(tc::smem_u32(&ctl.bar_y[0]), 1);
    tc::mbar_init(tc::smem_u32(&ctl.bar_y[1]), 1);
    tc::mbar_init(tc::smem_u32(&ctl.bar_d), 1);
    tc::fence_mbar_init();
    ctl.abort = 0;
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  pdl_entry();
  // local_kernel, behind the next kernel, takes its chunks from the first on, also in a second backward behind one forward
  if (KDA && blockIdx.x == 0 && tid == 0) reinterpret_cast<int*>(p.xat + kXCounts)[2] = 0;
  const uint32_t tbase = ctl.tmem_base, sbase = tc::smem_u32(smem);
  auto wait_bar = [&](uint64_t& bar, uint32_t parity) {
    const uint32_t at = tc::smem_u32(&bar);
    sm100::wait_inline(at, parity, &ctl.abort, at - tc::smem_u32(&ctl), min(warp >> 3, 1));
  };
  const int64_t chunk0 = (int64_t)unit * p.N;
  const int steps = p.dh0 ? p.N : p.N - 1;   // the product of the first chunk gives the initial state's gradient alone
  auto y_done = [&](int it) { wait_bar(ctl.bar_y[it & 1], (it >> 1) & 1); };
  constexpr uint32_t id = tc::idesc_bf16(128, 64, 0, 1);
  auto adv = [](uint64_t d, uint32_t bytes) { return d + (uint64_t)(bytes >> 4); };
  if (KDA && warp == 8) {
    if (tc::elect_one()) {
      auto load_o = [&](int it) {
        const uint32_t bar = tc::smem_u32(&ctl.full_o[it & 1]);
        tc::mbar_arrive_expect_tx(bar, kOTile);
        tc::tma_load_4d(sbase + CK_O + (it & 1) * kOTile, &P.to, v0, h, (p.N - 1 - it) * kC, b, bar);
      };
      auto load_y = [&](int it) {
        const uint32_t bar = tc::smem_u32(&ctl.full_y[0]);
        tc::mbar_arrive_expect_tx(bar, kHalfTile);
        tc::bulk_g2s(sbase + CK_Y, p.yf + (chunk0 + p.N - 1 - it) * kHalf4, kHalfTile, bar);
      };
      auto load_n = [&](int i) {   // half i & 1 of chunk i / 2
        const uint32_t bar = tc::smem_u32(&ctl.full_n[i % kHalfSlots]);
        tc::mbar_arrive_expect_tx(bar, kHalfTile);
        tc::bulk_g2s(sbase + CK_N + (i % kHalfSlots) * kHalfTile, p.nf + (2 * (chunk0 + p.N - 1 - (i >> 1)) + (i & 1)) * kHalf4, kHalfTile, bar);
      };
      if (steps > 0) { load_y(0); load_o(0); }
      for (int i = 0; i < kHalfSlots && i < 2 * steps; ++i) load_n(i);
      if (steps > 1) load_o(1);
      const uint64_t sd = tc::smem_desc_sw128(sbase + CK_S, kSTerm, 1024);
      const uint32_t acc_n = tbase + kTmemN;
      constexpr uint32_t left[6] = {0, 0, 0, 1, 1, 2}, right[6] = {0, 1, 2, 0, 1, 0};   // terms of N and of dS
#pragma unroll 1
      for (int it = 0; it < steps; ++it) {
        const uint32_t acc = tbase + (it & 1) * 64;   // (read for chunk it - 2 before its successor's dS was ready)
        const uint64_t od = tc::smem_desc_sw128(sbase + CK_O + (it & 1) * kOTile, kSTerm, 1024);
        wait_bar(ctl.full_o[it & 1], (it >> 1) & 1);
        wait_bar(ctl.full_l, it & 1);
        if (it + 1 < steps) load_y(it + 1);
        tc::tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
#pragma unroll
          for (int x = 0; x < 3; ++x) tc::mma_ts(acc, tbase + kTmemY + 32 * x + 8 * ks, adv(od, ks * 2048), id, ks + x > 0);
        tc::mma_commit(tc::smem_u32(&ctl.bar_y[it & 1]));
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          wait_bar(ctl.full_h[hf], it & 1);
          if (2 * it + hf + kHalfSlots < 2 * steps) load_n(2 * it + hf + kHalfSlots);
          if (hf == 0) wait_bar(ctl.rdy, it & 1);
          tc::tc_fence_after();
#pragma unroll
          for (int ks = 4 * hf; ks < 4 * hf + 4; ++ks)
#pragma unroll
            for (int x = 0; x < 6; ++x) tc::mma_ts(acc_n, tbase + kTmemA + 64 * left[x] + 8 * ks, adv(sd, right[x] * kSTerm + ks * 2048), id, ks + x > 0);
          tc::mma_commit(tc::smem_u32(hf ? &ctl.bar_d : &ctl.bar_e));
        }
        if (it + 2 < steps) {
          y_done(it);   // d_o has been read
          load_o(it + 2);
        }
      }
    }
    __syncwarp();
  } else if (warp == 8) {
    if (tc::elect_one()) {
      auto n_at = [&](int it) { return reinterpret_cast<const uint8_t*>(p.nf) + (chunk0 + p.N - 1 - it) * kNTile; };
      auto y_at = [&](int it) { return reinterpret_cast<const uint8_t*>(p.yf) + (chunk0 + p.N - 1 - it) * kYTile; };
      auto load_term = [&](uint64_t& full, uint32_t dst, const uint8_t* src) {
        const uint32_t bar = tc::smem_u32(&full);
        tc::mbar_arrive_expect_tx(bar, kNTerm);
        tc::bulk_g2s(dst, src, kNTerm, bar);
      };
      auto load_h = [&](int it) { load_term(ctl.full_h[it & 1], sbase + CH_H + (it & 1) * kNTerm, n_at(it)); };
      auto load_l = [&](int it) { load_term(ctl.full_l, sbase + CH_L, n_at(it) + kNTerm); };
      auto load_y = [&](int it) {
        const uint32_t bar = tc::smem_u32(&ctl.full_y[it & 1]);
        tc::mbar_arrive_expect_tx(bar, kYTile + kOTile);
        tc::tma_load_4d(sbase + CH_O + (it & 1) * kOTile, &P.to, v0, h, (p.N - 1 - it) * kC, b, bar);
        tc::bulk_g2s(sbase + CH_Y + (it & 1) * kYTile, y_at(it), kYTile, bar);
      };
      if (steps > 0) { load_y(0); load_h(0); load_l(0); }
      if (steps > 1) { load_y(1); load_h(1); }
      const uint64_t sd = tc::smem_desc_sw128(sbase + CH_S, 128 * 128, 1024), ld = tc::smem_desc(sbase + CH_L, 128, sm100::RBS);
#pragma unroll 1
      for (int it = 0; it < steps; ++it) {
        const uint32_t acc = tbase + (it & 1) * 64;   // (read for chunk it - 2 before its successor's dS was ready)
        const uint64_t yd = tc::smem_desc(sbase + CH_Y + (it & 1) * kYTile, 128, kYRbs);
        const uint64_t od = tc::smem_desc_sw128(sbase + CH_O + (it & 1) * kOTile, 128 * 128, 1024);
        const uint64_t hd = tc::smem_desc(sbase + CH_H + (it & 1) * kNTerm, 128, sm100::RBS);
        wait_bar(ctl.full_y[it & 1], (it >> 1) & 1);
        tc::tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          tc::mma_ss(acc, adv(yd, ks * 256), adv(od, ks * 2048), id, ks > 0);
          tc::mma_ss(acc, adv(yd, kYTile / 2 + ks * 256), adv(od, ks * 2048), id, 1);
        }
        tc::mma_commit(tc::smem_u32(&ctl.bar_y[it & 1]));
        wait_bar(ctl.full_h[it & 1], (it >> 1) & 1);
        wait_bar(ctl.rdy, it & 1);
        tc::tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
          tc::mma_ss(acc, adv(hd, ks * 256), adv(sd, ks * 2048), id, 1);
          tc::mma_ss(acc, adv(hd, ks * 256), adv(sd, kSTerm + ks * 2048), id, 1);
        }
        wait_bar(ctl.full_l, it & 1);
        tc::tc_fence_after();
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) tc::mma_ss(acc, adv(ld, ks * 256), adv(sd, ks * 2048), id, 1);
        tc::mma_commit(tc::smem_u32(&ctl.bar_d));
        y_done(it);   // Y^T and d_o have been read
        if (it + 2 < steps) load_y(it + 2);
        wait_bar(ctl.bar_d, it & 1);   // N has been read
        if (it + 1 < steps) load_l(it + 1);
        if (it + 2 < steps) load_h(it + 2);
      }
    }
    __syncwarp();
  } else if (KDA && warp > 8) {
    // thread = row; of 64 columns in shared memory half, as three terms to tensor memory
    const int row = 32 * (warp & 3) + lane, hc = (warp - 9) >> 2;
    const uint32_t at = (uint32_t)(32 * (warp & 3)) << 16;
    auto split = [&](int from, uint32_t to, uint32_t term, uint64_t& full) {
      const float4* src = reinterpret_cast<const float4*>(smem + from) + (row >> 3) * 64 + 4 * hc * 8 + (row & 7);
      uint32_t h[16], m[16], l[16];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 x = src[8 * i], y = src[kHalf4 / 2 + 8 * i];
        mma::split3_exact(x.x, x.y, h[4 * i], m[4 * i], l[4 * i]);
        mma::split3_exact(x.z, x.w, h[4 * i + 1], m[4 * i + 1], l[4 * i + 1]);
        mma::split3_exact(y.x, y.y, h[4 * i + 2], m[4 * i + 2], l[4 * i + 2]);
        mma::split3_exact(y.z, y.w, h[4 * i + 3], m[4 * i + 3], l[4 * i + 3]);
      }
      to += tbase + at + 16 * hc;
      tc::tmem_st16(to, h);
      tc::tmem_st16(to + term, m);
      tc::tmem_st16(to + 2 * term, l);
      tc::tc_wait_st();
      tc::tc_fence_before();
      sm100::mbar_arrive(tc::smem_u32(&full));
    };
#pragma unroll 1
    for (int it = 0; it < steps; ++it) {
      wait_bar(ctl.full_y[0], it & 1);
      if (it > 0) { y_done(it - 1); tc::tc_fence_after(); }
      split(CK_Y, kTmemY, 32, ctl.full_l);
#pragma unroll 1
      for (int hf = 0; hf < 2; ++hf) {
        const int i = 2 * it + hf;
        wait_bar(ctl.full_n[i % kHalfSlots], (i / kHalfSlots) & 1);
        if (it > 0) { wait_bar(hf ? ctl.bar_d : ctl.bar_e, (it - 1) & 1); tc::tc_fence_after(); }
        split(CK_N + (i % kHalfSlots) * kHalfTile, kTmemA + 32 * hf, 64, ctl.full_h[hf]);
      }
    }
  } else {
    const int row = 32 * (warp & 3) + lane, hc = warp >> 2;   // this thread's channel and half of the columns
    const uint32_t lane_addr = (uint32_t)(32 * (warp & 3)) << 16;
    const int64_t at = (int64_t)row * kD + v0 + 32 * hc;
    uint8_t* stage = smem + (KDA ? CK_G : CH_G) + warp * 2048;
    float S[32];
#pragma unroll
    for (int c = 0; c < 32; c += 2) {   // (d_hT and dh0 need not be aligned to more than eight bytes)
      const float2 x = p.d_hT ? ld2(p.d_hT + (int64_t)unit * kD * kD + at + c) : make_float2(0.f, 0.f);
      S[c] = x.x; S[c + 1] = x.y;
    }
#pragma unroll 1
    for (int it = 0; it < p.N; ++it) {
      const int64_t chunk = chunk0 + p.N - 1 - it;
      const float el = p.el[chunk * 128 + row];
      if (it < steps) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t hi[4], lo[4], last[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float x = S[8 * c + 2 * e], y = S[8 * c + 2 * e + 1];
            if constexpr (KDA) mma::split3_exact(x, y, hi[e], lo[e], last[e]); else split2(x, y, hi[e], lo[e]);
          }
          uint8_t* dst = smem + (KDA ? CK_S : CH_S) + row * 128 + (((4 * hc + c) ^ (row & 7)) << 4);
          *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
          *reinterpret_cast<uint4*>(dst + kSTerm) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
          if constexpr (KDA) *reinterpret_cast<uint4*>(dst + 2 * kSTerm) = make_uint4(last[0], last[1], last[2], last[3]);
        }
        tc::fence_async_smem();
        sm100::mbar_arrive(tc::smem_u32(&ctl.rdy));
      }
      // dS1 of this chunk -> memory, sixteen rows at a time through the warp's 2 KB: whole 128-byte lines (a thread's own row in 16-byte
      // pieces made the write the longest part of a chunk)
      float* ds = p.ds + chunk * (kD * kD) + (int64_t)(32 * (warp & 3)) * kD + v0 + 32 * hc;
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        const int r0 = lane & 15;
        if ((lane >> 4) == hf) {
#pragma unroll
          for (int q = 0; q < 8; ++q)
            *reinterpret_cast<float4*>(stage + r0 * 128 + ((q ^ (r0 & 7)) << 4)) = make_float4(S[4 * q], S[4 * q + 1], S[4 * q + 2], S[4 * q + 3]);
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int r = 4 * i + (lane >> 3), q = lane & 7;
          *reinterpret_cast<float4*>(ds + (int64_t)(16 * hf + r) * kD + 4 * q) = *reinterpret_cast<const float4*>(stage + r * 128 + ((q ^ (r & 7)) << 4));
        }
        __syncwarp();
      }
      if (it == steps) break;
      uint32_t d[32];
      if constexpr (KDA) {   // Y^T d_o is long done
        wait_bar(ctl.bar_y[it & 1], (it >> 1) & 1);
        tc::tc_fence_after();
        tc::tmem_ld32(tbase + lane_addr + (it & 1) * 64 + 32 * hc, d);
        tc::tc_wait_ld();
#pragma unroll
        for (int c = 0; c < 32; ++c) S[c] = S[c] * el + __uint_as_float(d[c]);
      }
      wait_bar(ctl.bar_d, it & 1);
      tc::tc_fence_after();
      tc::tmem_ld32(KDA ? tbase + lane_addr + kTmemN + 32 * hc : tbase + lane_addr + (it & 1) * 64 + 32 * hc, d);
      tc::tc_wait_ld();
#pragma unroll
      for (int c = 0; c < 32; ++c) S[c] = KDA ? S[c] + __uint_as_float(d[c]) : S[c] * el + __uint_as_float(d[c]);
      tc::tc_fence_before();
    }
    if (p.dh0) {
      float* out = p.dh0 + (int64_t)unit * kD * kD + at;
#pragma unroll
      for (int c = 0; c < 32; c += 2) *reinterpret_cast<float2*>(out + c) = make_float2(S[c], S[c + 1]);
    }
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    sm100::settle(ctl.abort);
    tc::tmem_dealloc(tbase, kTmem);
  }
  if (tid == 0) sm100::report_wait(P.status, ctl.abort);
}

// =====================================================================================================================
// local_kernel: sixteen warps; warp w works on token rows 16 (w >> 2) .. and on a quarter of the columns, w & 3
// =====================================================================================================================
constexpr int kLoThreads = 512;
constexpr int LDV = 40;    // row stride of the value-slice arrays
constexpr int LDA = 72;    // of A, dA, dX
// phase 1 (bytes): k^ e^G and k^ e^{G_L - G}, A, T, then V, dO, Vn, dR [64][40] and two buffers of S0, dS [128][40]
struct LoSmem {
  static constexpr int kK = 0, kKd = kK + 64 * 132 * 4;
  static constexpr int kA = kKd + 64 * 132 * 4, kT = kA + 64 * LDA * 4;
  static constexpr int kV = kT + 64 * LDT * 4, kSl = 64 * LDV * 4;   // V, dO, Vn, dR
  static constexpr int kSD = kV + 4 * kSl, kS1 = 128 * LDV * 4;        // [2][S0, dS]
  static constexpr int kSc = kSD + 4 * kS1;
  static constexpr int kTaken = kSc + (3 * 64 + 5 * 64 + 128 + 528) * 4;
  static constexpr int kTotal = kTaken + 16;
  // final phase: a map of its own from 0
  static constexpr int gQS = 0, gKS = 64 * 132 * 4, gKE = 2 * gKS, gG = 3 * gKS, gA = 4 * gKS, gX = gA + 64 * LDA * 4, gD = gX + 64 * LDA * 4;
  static constexpr int gSeg = gD + 4 * 128 * 4;   // [16][128] scan scratch
  static constexpr int kDot = gSeg + 16 * 128 * 4;   // final phase: q^ . dq^, k^ . dk^ per row, [2][4][64]
  static constexpr int gRaw = kDot + 2048;   // raw q and k rows, bf16 [2][64][136]
  static_assert(kTotal <= 232448 && gRaw + 2 * 64 * LDH * 2 <= kSc, "shared memory");
};

static __global__ void __launch_bounds__(kLoThreads, 1) local_kernel(const Params p, const int chunks) {
  using L = LoSmem;
  pdl_entry();
  extern __shared__ __align__(16) uint8_t smem[];
  auto F = [&](int off) { return reinterpret_cast<float*>(smem + off); };
  float *sK = F(L::kK), *sKd = F(L::kKd), *sA = F(L::kA), *sT = F(L::kT);
  float *sV = F(L::kV), *sdO = F(L::kV + L::kSl), *sVn = F(L::kV + 2 * L::kSl), *sdR = F(L::kV + 3 * L::kSl);
  float* sBeta = F(L::kSc);
  float *sRk = sBeta + 64, *sRq = sBeta + 128;
  // sums over a row's columns: one slot per quarter of the columns (sdB: and one for dR . V), added up by one thread at the
  // end -- no atomics, so that equal inputs give equal bits
  float *sdB = sBeta + 192, *sTS = sBeta + 512, *sU = sBeta + 640;   // dbeta [5][64]; <dS1, S0> per channel
  float *sEx = sU, *sUn = sU + 512;   // sums for dG_L [4][128], block flags
  float *sDq = F(L::kDot), *sDk = sDq + 256;
  int* const taken = reinterpret_cast<int*>(smem + L::kTaken);   // [2], by turns
  if (threadIdx.x == 0) taken[0] = numbered(p, chunks, take_number(p, 1, true));
#pragma unroll 1
  for (int turn = 0;; turn ^= 1) {
  __syncthreads();   // the chunk before is done with shared memory
  const int at_chunk = taken[turn];
  if (at_chunk >= chunks) break;
  int tid = threadIdx.x;
  asm volatile("" : "+r"(tid));   // (what follows from the thread's place is formed for each chunk: kept over the loop it costs the inner loops their registers)
  const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  int number = 0;   // (asked for early: the answer takes a while)
  if (tid == 0) number = take_number(p, 1, false);
  const int unit = at_chunk / p.N, n = at_chunk % p.N;
  const int b = unit / p.map.H, h = unit % p.map.H, t0 = n * kC, rows = min(kC, p.map.T - t0);
  const int64_t qk_base = p.map.base_qk(b, h, kD), qk_tok = p.map.tok_qk(kD);
  const int64_t gk_base = p.map.base(b, h, kD), gk_tok = p.map.tok(kD);
  const int64_t v_base = p.map.base(b, h, kD), v_tok = p.map.tok(kD);
  const int64_t s_base = p.map.base(b, h, 1), s_tok = p.map.tok(1);
  const int64_t chunk = (int64_t)unit * p.N + n;
  const float* xat = p.xat + chunk * (3 * 64 * 64);
  const __nv_bfloat16 *gq = reinterpret_cast<const __nv_bfloat16*>(p.q), *gk = reinterpret_cast<const __nv_bfloat16*>(p.k);
  const int m0 = 16 * (warp >> 2), wc = warp & 3;

  // S0, dS columns of one value slice -> buffer, 16 bytes per copy
  auto issue_slice = [&](int s) {
    float* dst = F(L::kSD + (s & 1) * 2 * L::kS1);
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int i = tid + kLoThreads * it, which = i >> 10, r = (i >> 3) & 127, c4 = (i & 7) * 4;
      const float* src = (which ? p.ds : p.ckpt) + chunk * (kD * kD) + r * kD + s * kVS + c4;
      tc::cp_async16(tc::smem_u32(dst + which * (128 * LDV) + r * LDV + c4), src, true);
    }
    tc::cp_async_commit();
  };
  // V, dO of one slice: thread = eight columns of one row of one of the two arrays
  const int vrow = (tid & 255) >> 2, vcol = (tid & 3) * 8;
  auto load_v = [&](int s) -> uint4 {
    if (vrow >= rows) return make_uint4(0u, 0u, 0u, 0u);
    const __nv_bfloat16* src = reinterpret_cast<const __nv_bfloat16*>(tid < 256 ? p.v : p.d_o);
    return *reinterpret_cast<const uint4*>(src + v_base + (int64_t)(t0 + vrow) * v_tok + s * kVS + vcol);
  };
  // ---- stage what all slices share ----------------------------------------------------------------------------------------------
  for (int i = tid; i < 2 * 64 * 16; i += kLoThreads) {
    const int m = i >> 10, r = (i >> 4) & 63, c4 = (i & 15) * 4;
    if ((c4 >> 4) <= (r >> 4))
      tc::cp_async16(tc::smem_u32((m ? sT + r * LDT : sA + r * LDA) + c4), xat + (1 + m) * 4096 + r * 64 + c4, true);
  }
  issue_slice(0);
  uint4 vr = load_v(0);
  {
    uint2 kr[4];
    float4 gr[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = warp + 16 * i;
      kr[i] = make_uint2(0u, 0u);
      gr[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c < rows) {
        kr[i] = *reinterpret_cast<const uint2*>(gk + qk_base + (t0 + c) * qk_tok + 4 * lane);
        gr[i] = load_g4(p.g, gk_base + (t0 + c) * gk_tok + 4 * lane, p.g_dt);
      }
    }
    if (tid < 64) {
      sBeta[tid] = tid < rows ? p.beta[s_base + (t0 + tid) * s_tok] : 0.f;
    }
    for (int i = tid; i < 320; i += kLoThreads) sdB[i] = 0.f;
    if (tid < 128) sTS[tid] = 0.f;
    float* sG = F(L::kSD + 2 * L::kS1);   // the second slice buffer, not yet in use (behind it: scan scratch)
#pragma unroll
    for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(sG + (warp + 16 * i) * 132 + 4 * lane) = gr[i];
    __syncthreads();
    mma::scan_channels<kLoThreads, kD>(sG, sVn, tid);   // scratch 8 KB
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = warp + 16 * i;
      const float k0 = mma::lo_f(kr[i].x), k1 = mma::hi_f(kr[i].x), k2 = mma::lo_f(kr[i].y), k3 = mma::hi_f(kr[i].y);
      const float nrm = p.l2norm ? sqrtf(warp_sum(k0 * k0 + k1 * k1 + k2 * k2 + k3 * k3)) : 0.f;
      const float m = p.l2norm ? 1.f / (nrm + 1e-6f) : 1.f;
      if (lane == 0) sRk[c] = m;
      const float4 gg = *reinterpret_cast<const float4*>(sG + c * 132 + 4 * lane), gl = *reinterpret_cast<const float4*>(sG + 63 * 132 + 4 * lane);
      *reinterpret_cast<float4*>(sK + c * 132 + 4 * lane) =
          make_float4(k0 * m * ex2(gg.x), k1 * m * ex2(gg.y), k2 * m * ex2(gg.z), k3 * m * ex2(gg.w));
      *reinterpret_cast<float4*>(sKd + c * 132 + 4 * lane) =
          make_float4(k0 * m * ex2(gl.x - gg.x), k1 * m * ex2(gl.y - gg.y), k2 * m * ex2(gl.z - gg.z), k3 * m * ex2(gl.w - gg.w));
    }
  }
  float dQ[4][4], dKr[4][4], dKc[4][4], da[2][4], dm[2][4];   // dQg, dKg (negated), dKt; dA, dR Vn^T
#pragma unroll
  for (int i = 0; i < 4; ++i) { zero4(dQ[i]); zero4(dKr[i]); zero4(dKc[i]); }
#pragma unroll
  for (int i = 0; i < 2; ++i) { zero4(da[i]); zero4(dm[i]); }

#pragma unroll 1
  for (int s = 0; s < kD / kVS; ++s) {
    const float *sS0 = F(L::kSD + (s & 1) * 2 * L::kS1), *sdS = sS0 + 128 * LDV;
    __syncthreads();   // the previous slice (s = 0: the scan scratch) is done with
    {
      const uint32_t w[4] = {vr.x, vr.y, vr.z, vr.w};
      float* dst = (tid < 256 ? sV : sdO) + vrow * LDV + vcol;
      *reinterpret_cast<float4*>(dst) = make_float4(mma::lo_f(w[0]), mma::hi_f(w[0]), mma::lo_f(w[1]), mma::hi_f(w[1]));
      *reinterpret_cast<float4*>(dst + 4) = make_float4(mma::lo_f(w[2]), mma::hi_f(w[2]), mma::lo_f(w[3]), mma::hi_f(w[3]));
    }
    tc::cp_async_wait_all();
    __syncthreads();
    if (s + 1 < kD / kVS) { issue_slice(s + 1); vr = load_v(s + 1); }
    // ---- R = beta V - beta (K^ e^G) S0,  dVn = A^T dO + Kd dS1 (eight columns per warp) ------------------------------------------
    const int n0 = 8 * wc;
    // different left operands, each split into two terms: half of the warps take R, half dVn, sixteen columns each, so that
    // a split serves two products (with both on every warp the splits were more than half of the instructions here)
    const bool second = warp >= 8;
    const int mr = 16 * ((warp & 7) >> 1), nc = 16 * (warp & 1);
    const uint32_t left = mma::lda_at(tc::smem_u32(second ? sKd : sK), 132, mr, lane);
    const float* right = second ? sdS : sS0;
    float d[2][4];
    zero4(d[0]); zero4(d[1]);
#pragma unroll 4
    for (int k0 = 0; k0 < kD; k0 += 8) {
      const int k = k0 + t;
      AFrag<true> a;
      mma::lda(a, left + 4u * k0);
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        BFrag<true> bs;
        bs.set(right[k * LDV + nc + 8 * nt + g], right[(k + 4) * LDV + nc + 8 * nt + g]);
        fma<true>(d[nt], a, bs);
      }
    }
    if (second) {
      for (int k0 = mr; k0 < kC; k0 += 8) {
        const int k = k0 + t;
        AFrag<true> a;
        a.set(sA[k * LDA + mr + g], sA[k * LDA + mr + g + 8], sA[(k + 4) * LDA + mr + g], sA[(k + 4) * LDA + mr + g + 8]);
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          BFrag<false> bo;   // bf16 values: one term
          bo.set(sdO[k * LDV + nc + 8 * nt + g], sdO[(k + 4) * LDV + nc + 8 * nt + g]);
          mma::fma_b1(d[nt], a, bo);
        }
      }
    }
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int hr = 0; hr < 2; ++hr) {
        const int c = mr + g + 8 * hr, at = c * LDV + nc + 8 * nt + 2 * t;
        if (second) {
          *reinterpret_cast<float2*>(sdR + at) = make_float2(d[nt][2 * hr], d[nt][2 * hr + 1]);
        } else {
          const float2 x = ld2(sV + at);
          const float bt = sBeta[c];
          *reinterpret_cast<float2*>(sVn + at) = make_float2(bt * (x.x - d[nt][2 * hr]), bt * (x.y - d[nt][2 * hr + 1]));
        }
      }
    __syncthreads();
    // ---- Vn = T R, dR = T^T dVn ------------------------------------------------------------------------------------------------------
    {
      const uint32_t aT = mma::lda_at(tc::smem_u32(sT), LDT, m0, lane);
      float vn[4], dr[4];
      zero4(vn); zero4(dr);
      for (int k0 = 0; k0 < m0 + 16; k0 += 8) {
        const int k = k0 + t;
        AFrag<true> a;
        mma::lda(a, aT + 4u * k0);
        BFrag<true> br;
        br.set(sVn[k * LDV + n0 + g], sVn[(k + 4) * LDV + n0 + g]);
        fma<true>(vn, a, br);
      }
      for (int k0 = m0; k0 < kC; k0 += 8) {
        const int k = k0 + t;
        AFrag<true> a;
        a.set(sT[k * LDT + m0 + g], sT[k * LDT + m0 + g + 8], sT[(k + 4) * LDT + m0 + g], sT[(k + 4) * LDT + m0 + g + 8]);
        BFrag<true> bd;
        bd.set(sdR[k * LDV + n0 + g], sdR[(k + 4) * LDV + n0 + g]);
        fma<true>(dr, a, bd);
      }
      __syncthreads();
#pragma unroll
      for (int hr = 0; hr < 2; ++hr) {
        const int at = (m0 + g + 8 * hr) * LDV + n0 + 2 * t;
        *reinterpret_cast<float2*>(sVn + at) = make_float2(vn[2 * hr], vn[2 * hr + 1]);
        *reinterpret_cast<float2*>(sdR + at) = make_float2(dr[2 * hr], dr[2 * hr + 1]);
      }
    }
    __syncthreads();
    // ---- dV = beta dR, dbeta += dR . V (half of the threads); <dS1, S0> per channel (the other half) -----------------------------------
    if (tid < 256) {
      float x[8], acc = 0.f;
      const float bt = sBeta[vrow];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        x[e] = sdR[vrow * LDV + vcol + e];
        acc += x[e] * sV[vrow * LDV + vcol + e];
        x[e] *= bt;
      }
      acc += __shfl_xor_sync(0xffffffffu, acc, 1);
      acc += __shfl_xor_sync(0xffffffffu, acc, 2);
      if ((tid & 3) == 0) sdB[256 + vrow] += acc;
      if (vrow < rows)
        *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.dv) + v_base + (int64_t)(t0 + vrow) * v_tok + s * kVS + vcol) =
            make_uint4(mma::pack(x[0], x[1]), mma::pack(x[2], x[3]), mma::pack(x[4], x[5]), mma::pack(x[6], x[7]));
    } else {
      const int u = tid - 256;
#pragma unroll
      for (int it = 0; it < 4; ++it) {   // eight lanes per channel row
        const int k = 32 * it + (u >> 3), c4 = (u & 7) * 4;
        const float4 x = *reinterpret_cast<const float4*>(sS0 + k * LDV + c4), y = *reinterpret_cast<const float4*>(sdS + k * LDV + c4);
        float acc = x.x * y.x + x.y * y.y + x.z * y.z + x.w * y.w;
        acc += __shfl_xor_sync(0xffffffffu, acc, 1);
        acc += __shfl_xor_sync(0xffffffffu, acc, 2);
        acc += __shfl_xor_sync(0xffffffffu, acc, 4);
        if ((u & 7) == 0) sTS[k] += acc;
      }
    }
    // ---- sums over v: dA += dO Vn^T, dM' += dR Vn^T; dQg += dO S0^T, dKg' += dR S0^T, dKt += Vn dS1^T (k taken in pairs) -----------------
#pragma unroll
    for (int k0 = 0; k0 < kVS; k0 += 8) {
      const int k = k0 + 2 * t;
      AFrag<false> ao;   // bf16 values: one term in either precision
      AFrag<true> ar, an;
      {
        const float2 x0 = ld2(sdO + (m0 + g) * LDV + k), x1 = ld2(sdO + (m0 + g + 8) * LDV + k);
        ao.set(x0.x, x1.x, x0.y, x1.y);
        const float2 y0 = ld2(sdR + (m0 + g) * LDV + k), y1 = ld2(sdR + (m0 + g + 8) * LDV + k);
        ar.set(y0.x, y1.x, y0.y, y1.y);
        const float2 z0 = ld2(sVn + (m0 + g) * LDV + k), z1 = ld2(sVn + (m0 + g + 8) * LDV + k);
        an.set(z0.x, z1.x, z0.y, z1.y);
      }
      if (16 * wc <= m0) {
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
          const float2 y = ld2(sVn + (16 * wc + 8 * nt + g) * LDV + k);
          BFrag<true> bv;
          bv.set(y.x, y.y);
          mma::fma_a1(da[nt], ao, bv);
          fma<true>(dm[nt], ar, bv);
        }
      }
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        const int ch = 32 * wc + 8 * nt + g;
        const float2 y = ld2(sS0 + ch * LDV + k), z = ld2(sdS + ch * LDV + k);
        BFrag<true> bs, bd;
        bs.set(y.x, y.y);
        bd.set(z.x, z.y);
        mma::fma_a1(dQ[nt], ao, bs);
        fma<true>(dKr[nt], ar, bs);
        fma<true>(dKc[nt], an, bd);
      }
    }
  }
  // ---- dA, dX with their decay factors; dbeta += dM . X -------------------------------------------------------------------------------------
  uint2 qr[4], kr[4];
  float4 gr[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {   // the chunk's q, k, g rows once more, in flight behind the next lines
    const int c = warp + 16 * i;
    qr[i] = kr[i] = make_uint2(0u, 0u);
    gr[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c < rows) {
      qr[i] = *reinterpret_cast<const uint2*>(gq + qk_base + (t0 + c) * qk_tok + 4 * lane);
      kr[i] = *reinterpret_cast<const uint2*>(gk + qk_base + (t0 + c) * qk_tok + 4 * lane);
      gr[i] = load_g4(p.g, gk_base + (t0 + c) * gk_tok + 4 * lane, p.g_dt);
    }
  }
  if (tid == 0) {
    const int next = numbered(p, chunks, number);
    taken[turn ^ 1] = next;
    if (next < chunks) {   // it begins with its states
      l2_bulk(p.ckpt + (int64_t)next * (kD * kD), kD * kD * 4);
      l2_bulk(p.ds + (int64_t)next * (kD * kD), kD * kD * 4);
    }
  }
  __syncthreads();   // phase 1 is over: its arrays may be written
  float *fA = F(L::gA), *fX = F(L::gX);
  {
    float dbacc[2] = {0.f, 0.f};
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int hr = 0; hr < 2; ++hr) {
        const int i = m0 + g + 8 * hr, j = 16 * wc + 8 * nt + 2 * t;
        float2 xx = make_float2(0.f, 0.f);
        if (16 * wc <= m0) xx = *reinterpret_cast<const float2*>(xat + i * 64 + j);   // zero at and above the diagonal
        float av[2], xv[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float ee = (j + e <= i) ? 1.f : 0.f;
          const float dmv = -dm[nt][2 * hr + e];
          dbacc[hr] += dmv * (e ? xx.y : xx.x);   // X carries its decay factor
          av[e] = da[nt][2 * hr + e] * ee;
          xv[e] = (j + e < i) ? sBeta[i] * dmv * ee : 0.f;
        }
        *reinterpret_cast<float2*>(fA + i * LDA + j) = make_float2(av[0], av[1]);
        *reinterpret_cast<float2*>(fX + i * LDA + j) = make_float2(xv[0], xv[1]);
      }
#pragma unroll
    for (int hr = 0; hr < 2; ++hr) {
      float x = dbacc[hr];
      x += __shfl_xor_sync(0xffffffffu, x, 1);
      x += __shfl_xor_sync(0xffffffffu, x, 2);
      if (t == 0) sdB[64 * wc + m0 + g + 8 * hr] += x;
    }
  }
  // ---- the decayed forms of q^ and k^ ---------------------------------------------------------------------------------------
  __nv_bfloat16* sRaw = reinterpret_cast<__nv_bfloat16*>(smem + L::gRaw);
  float* sDi = F(L::gSeg);   // 1 / total decay of each block (over the scan scratch)
  float *sQS = F(L::gQS), *sKS = F(L::gKS), *sKE = F(L::gKE), *sG = F(L::gG), *sD = F(L::gD);
#pragma unroll
  for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(sG + (warp + 16 * i) * 132 + 4 * lane) = gr[i];
  __syncthreads();
  mma::scan_channels<kLoThreads, kD>(sG, F(L::gSeg), tid);
  if (tid < 4) sUn[tid] = 0.f;
  __syncthreads();
  {   // total decay of each 16-row block; flag blocks whose range is too wide for the product form
    const int blk = tid >> 7, c = tid & 127;
    const float d = sG[(16 * blk + 15) * 132 + c] - (blk ? sG[(16 * blk - 1) * 132 + c] : 0.f);
    sD[blk * 128 + c] = ex2(d);
    sDi[blk * 128 + c] = 1.f / ex2(d);
    if (!(d >= -64.f)) sUn[blk] = 1.f;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int c = warp + 16 * i;
    const float q0 = mma::lo_f(qr[i].x), q1 = mma::hi_f(qr[i].x), q2 = mma::lo_f(qr[i].y), q3 = mma::hi_f(qr[i].y);
    const float nrm = p.l2norm ? sqrtf(warp_sum(q0 * q0 + q1 * q1 + q2 * q2 + q3 * q3)) : 0.f;
    const float m = p.l2norm ? p.scale / (nrm + 1e-6f) : p.scale;
    if (lane == 0) sRq[c] = m;
    *reinterpret_cast<uint2*>(sRaw + c * LDH + 4 * lane) = qr[i];
    *reinterpret_cast<uint2*>(sRaw + (64 + c) * LDH + 4 * lane) = kr[i];
    const int blk = c >> 4;
    const float4 gg = *reinterpret_cast<const float4*>(sG + c * 132 + 4 * lane);
    const float4 ge = *reinterpret_cast<const float4*>(sG + (16 * blk + 15) * 132 + 4 * lane);
    float4 gn = make_float4(0.f, 0.f, 0.f, 0.f);
    if (blk) gn = *reinterpret_cast<const float4*>(sG + (16 * blk - 1) * 132 + 4 * lane);
    const float mk = sRk[c];
    const float k0 = mma::lo_f(kr[i].x) * mk, k1 = mma::hi_f(kr[i].x) * mk, k2 = mma::lo_f(kr[i].y) * mk, k3 = mma::hi_f(kr[i].y) * mk;
    const float e0 = ex2(gg.x - gn.x), e1 = ex2(gg.y - gn.y), e2 = ex2(gg.z - gn.z), e3 = ex2(gg.w - gn.w);
    *reinterpret_cast<float4*>(sQS + c * 132 + 4 * lane) = make_float4(q0 * m * e0, q1 * m * e1, q2 * m * e2, q3 * m * e3);
    *reinterpret_cast<float4*>(sKS + c * 132 + 4 * lane) = make_float4(k0 * e0, k1 * e1, k2 * e2, k3 * e3);
    *reinterpret_cast<float4*>(sKE + c * 132 + 4 * lane) =
        make_float4(k0 * ex2(ge.x - gg.x), k1 * ex2(ge.y - gg.y), k2 * ex2(ge.z - gg.z), k3 * ex2(ge.w - gg.w));
  }
  __syncthreads();
  // ---- dQ^ = dQg e^G + (dA.E) K^ ; dK^ rows and columns (four channel tiles per warp: 32 wc ..) -------------------------------------------------
  float dbrow[2] = {0.f, 0.f};
  float Dg[4][4];   // dG of this lane's entries
  const int bi = warp >> 2;
  const bool exact = sUn[bi] != 0.f;
  // dbeta: -dKg . k^ e^G; dG_L: dKt . k^ e^{G_L - G}
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
    const int c = 32 * wc + 8 * nt + 2 * t;
    float2 en = make_float2(1.f, 1.f);   // decay before the block, and from its end to the chunk's
    if (bi) { const float2 x = ld2(sG + (16 * bi - 1) * 132 + c); en = make_float2(ex2(x.x), ex2(x.y)); }
    const float2 gl = ld2(sG + 63 * 132 + c), ge = ld2(sG + (16 * bi + 15) * 132 + c);
    const float2 ee = make_float2(ex2(gl.x - ge.x), ex2(gl.y - ge.y));
    float ex0 = 0.f, ex1 = 0.f;
#pragma unroll
    for (int hr = 0; hr < 2; ++hr) {
      const int i = m0 + g + 8 * hr;
      const float2 ks = ld2(sKS + i * 132 + c), ke = ld2(sKE + i * 132 + c);
      dbrow[hr] -= dKr[nt][2 * hr] * ks.x * en.x + dKr[nt][2 * hr + 1] * ks.y * en.y;
      ex0 += dKc[nt][2 * hr] * ke.x * ee.x;
      ex1 += dKc[nt][2 * hr + 1] * ke.y * ee.y;
      dKr[nt][2 * hr] *= -sBeta[i];
      dKr[nt][2 * hr + 1] *= -sBeta[i];
    }
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
      ex0 += __shfl_xor_sync(0xffffffffu, ex0, o);
      ex1 += __shfl_xor_sync(0xffffffffu, ex1, o);
    }
    if (g == 0) *reinterpret_cast<float2*>(sEx + 128 * bi + c) = make_float2(ex0, ex1);
  }
  auto carry = [&](float (&d)[4][4], int blk) {   // refer the sums to the end of block blk
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const float2 x = ld2(sD + blk * 128 + 32 * wc + 8 * nt + 2 * t);
      d[nt][0] *= x.x; d[nt][1] *= x.y; d[nt][2] *= x.x; d[nt][3] *= x.y;
    }
  };
  // rows: sums over the columns of earlier blocks, each block's decay carried on the way; then the diagonal block
#pragma unroll 1
  for (int bj = 0; bj <= bi; ++bj) {
    const bool diag = bj == bi;
    if (diag && exact) break;
    if (!diag) { carry(dQ, bj); carry(dKr, bj); }
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      const int k = 16 * bj + 8 * hf + 2 * t;
      AFrag<true> aa, ax;
      const float2 x0 = ld2(fA + (m0 + g) * LDA + k), x1 = ld2(fA + (m0 + g + 8) * LDA + k);
      aa.set(x0.x, x1.x, x0.y, x1.y);
      const float2 y0 = ld2(fX + (m0 + g) * LDA + k), y1 = ld2(fX + (m0 + g + 8) * LDA + k);
      ax.set(y0.x, y1.x, y0.y, y1.y);
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        const int c = 32 * wc + 8 * nt + g;
        float b0 = sKE[k * 132 + c], b1 = sKE[(k + 1) * 132 + c];
        if (diag) { const float iv = sDi[bi * 128 + c]; b0 *= iv; b1 *= iv; }
        BFrag<true> bk;
        bk.set(b0, b1);
        fma<true>(dQ[nt], aa, bk);
        fma<true>(dKr[nt], ax, bk);
      }
    }
  }
  // columns: the rows of later blocks, last first; then the diagonal block, referred to the block's start
#pragma unroll 1
  for (int bj = 3; bj >= bi; --bj) {
    const bool diag = bj == bi;
    if (diag && exact) break;
    carry(dKc, bj);
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      const int k = 16 * bj + 8 * hf + t;
      AFrag<true> aa, ax;
      aa.set(fA[k * LDA + m0 + g], fA[k * LDA + m0 + g + 8], fA[(k + 4) * LDA + m0 + g], fA[(k + 4) * LDA + m0 + g + 8]);
      ax.set(fX[k * LDA + m0 + g], fX[k * LDA + m0 + g + 8], fX[(k + 4) * LDA + m0 + g], fX[(k + 4) * LDA + m0 + g + 8]);
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        const int c = 32 * wc + 8 * nt + g;
        BFrag<true> bq, bk;
        bq.set(sQS[k * 132 + c], sQS[(k + 4) * 132 + c]);
        bk.set(sKS[k * 132 + c], sKS[(k + 4) * 132 + c]);
        fma<true>(dKc[nt], aa, bq);
        fma<true>(dKc[nt], ax, bk);
      }
    }
  }
  // the factors of the entries' own rows; dG
  float sq[2] = {0.f, 0.f}, sk[2] = {0.f, 0.f};
#pragma unroll
  for (int nt = 0; nt < 4; ++nt) {
    const int c = 32 * wc + 8 * nt + 2 * t;
    float2 gn = make_float2(0.f, 0.f);
    if (bi) gn = ld2(sG + (16 * bi - 1) * 132 + c);
    const float2 ge = ld2(sG + (16 * bi + 15) * 132 + c);
#pragma unroll
    for (int hr = 0; hr < 2; ++hr) {
      const int i = m0 + g + 8 * hr;
      const float2 gi = ld2(sG + i * 132 + c);
      const uint32_t uq = *reinterpret_cast<const uint32_t*>(sRaw + i * LDH + c), uk = *reinterpret_cast<const uint32_t*>(sRaw + (64 + i) * LDH + c);
      const float2 qh = make_float2(mma::lo_f(uq) * sRq[i], mma::hi_f(uq) * sRq[i]);
      const float2 kh = make_float2(mma::lo_f(uk) * sRk[i], mma::hi_f(uk) * sRk[i]);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int x = 2 * hr + e;
        const float Gi = e ? gi.y : gi.x, Gn = e ? gn.y : gn.x, Ge = e ? ge.y : ge.x;
        const float fr = ex2(Gi - Gn), fc = ex2((exact ? Ge : Gn) - Gi);
        float dq = dQ[nt][x] * fr, dkr = dKr[nt][x] * fr, dkc = dKc[nt][x] * fc;
        if (exact) {   // the diagonal block entry by entry
          for (int j = m0; j < m0 + 16; ++j) {
            const float Gj = sG[j * 132 + c + e];
            if (j >= rows) break;
            const int64_t at = qk_base + (t0 + j) * qk_tok + c + e;
            const float kj = bf(gk + at) * sRk[j], qj = bf(gq + at) * sRq[j];
            if (j <= i) {
              const float w = ex2(Gi - Gj) * kj;
              dq += fA[i * LDA + j] * w;
              dkr += fX[i * LDA + j] * w;
            }
            if (j >= i) {
              const float w = ex2(Gj - Gi);
              dkc += w * (fA[j * LDA + i] * qj + fX[j * LDA + i] * kj);
            }
          }
        }
        Dg[nt][x] = (e ? qh.y : qh.x) * dq + (e ? kh.y : kh.x) * (dkr - dkc);
        dQ[nt][x] = dq;
        dKr[nt][x] = dkr + dkc;
      }
      sq[hr] += qh.x * dQ[nt][2 * hr] + qh.y * dQ[nt][2 * hr + 1];
      sk[hr] += kh.x * dKr[nt][2 * hr] + kh.y * dKr[nt][2 * hr + 1];
    }
  }
#pragma unroll
  for (int hr = 0; hr < 2; ++hr) {
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      sq[hr] += __shfl_xor_sync(0xffffffffu, sq[hr], o);
      sk[hr] += __shfl_xor_sync(0xffffffffu, sk[hr], o);
    }
    if (t == 0) { sDq[64 * wc + m0 + g + 8 * hr] = sq[hr]; sDk[64 * wc + m0 + g + 8 * hr] = sk[hr]; }
  }
#pragma unroll
  for (int hr = 0; hr < 2; ++hr) {
    float db = dbrow[hr];
    db += __shfl_xor_sync(0xffffffffu, db, 1); db += __shfl_xor_sync(0xffffffffu, db, 2);
    if (t == 0) sdB[64 * wc + m0 + g + 8 * hr] += db;
  }
  __syncthreads();
  // ---- chain rule of the normalisation: y = s x / (|x| + eps), y^ = s x r:  dx = s r dy - y^ (y^ . dy) / (s |x|) ------------------------------------
  const bool grouped = p.map.Hq != p.map.H;
  __nv_bfloat16* oq = reinterpret_cast<__nv_bfloat16*>(smem + L::gKS);   // staging [64][136] bf16, twice
  __nv_bfloat16* ok = oq + 64 * 136;
  float* sDG = F(L::gQS);   // dG [64][132]
#pragma unroll
  for (int hr = 0; hr < 2; ++hr) {
    const int i = m0 + g + 8 * hr;
    const float mq = sRq[i], mk = sRk[i];
    float fq = 0.f, fk = 0.f;
    if (p.l2norm) {
      const float nq = p.scale / mq - 1e-6f, nk = 1.f / mk - 1e-6f;   // |q|, |k|
      fq = nq > 0.f ? ((sDq[i] + sDq[64 + i]) + (sDq[128 + i] + sDq[192 + i])) / (p.scale * nq) : 0.f;
      fk = nk > 0.f ? ((sDk[i] + sDk[64 + i]) + (sDk[128 + i] + sDk[192 + i])) / nk : 0.f;
    }
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const int c = 32 * wc + 8 * nt + 2 * t, e = 2 * hr;
      if (grouped) {
        const int64_t at = (chunk * kC + i) * kD + c;
        *reinterpret_cast<float2*>(p.part + at) = make_float2(dQ[nt][e], dQ[nt][e + 1]);
        *reinterpret_cast<float2*>(p.part + (int64_t)chunks * (kC * kD) + at) = make_float2(dKr[nt][e], dKr[nt][e + 1]);
      } else {
        float2 qh = make_float2(0.f, 0.f), kh = qh;
        const uint32_t uq = *reinterpret_cast<const uint32_t*>(sRaw + i * LDH + c), uk = *reinterpret_cast<const uint32_t*>(sRaw + (64 + i) * LDH + c);
        qh = make_float2(mma::lo_f(uq) * mq, mma::hi_f(uq) * mq);
        kh = make_float2(mma::lo_f(uk) * mk, mma::hi_f(uk) * mk);
        *reinterpret_cast<uint32_t*>(oq + i * 136 + c) = mma::pack(mq * dQ[nt][e] - qh.x * fq, mq * dQ[nt][e + 1] - qh.y * fq);
        *reinterpret_cast<uint32_t*>(ok + i * 136 + c) = mma::pack(mk * dKr[nt][e] - kh.x * fk, mk * dKr[nt][e + 1] - kh.y * fk);
      }
      *reinterpret_cast<float2*>(sDG + i * 132 + c) = make_float2(Dg[nt][e], Dg[nt][e + 1]);
    }
  }
  __syncthreads();
  if (!grouped) {
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int i = tid + kLoThreads * it, which = i >> 10, r = (i >> 4) & 63, c8 = (i & 15) * 8;
      if (r < rows)
        *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(which ? p.dk : p.dq) + qk_base + (t0 + r) * qk_tok + c8) =
            *reinterpret_cast<const uint4*>((which ? ok : oq) + r * 136 + c8);
    }
  }
  if (tid < rows) p.dbeta[s_base + (t0 + tid) * s_tok] = (sdB[tid] + sdB[64 + tid]) + (sdB[128 + tid] + sdB[192 + tid]) + sdB[256 + tid];
  // ---- dg: reverse cumulative sum of dG inside the chunk ---------------------------------------------------------------------------------------
  const int s = tid >> 7, c = tid & 127;   // 16-row segment, channel
  float acc = 0.f, loc[16];
  if (s == 3) acc = (sEx[c] + sEx[128 + c]) + (sEx[256 + c] + sEx[384 + c]) + sTS[c] * ex2(sG[63 * 132 + c]);
#pragma unroll
  for (int r = 15; r >= 0; --r) {
    acc += sDG[(16 * s + r) * 132 + c];
    loc[r] = acc;
  }
  sD[s * 128 + c] = acc;
  __syncthreads();
  float post = 0.f;
  for (int s2 = s + 1; s2 < 4; ++s2) post += sD[s2 * 128 + c];
#pragma unroll
  for (int r = 0; r < 16; ++r)
    if (16 * s + r < rows) p.dg[gk_base + (int64_t)(t0 + 16 * s + r) * gk_tok + c] = loc[r] + post;
  }
}

}  // namespace bwdc
}  // namespace dr

#include "dr_bwd_local_sm100.cuh"
#include "dr_bwd_local_kda.cuh"
#include "dr_bwd_pre_kda.cuh"

namespace dr {
namespace bwdc {
// =====================================================================================================================
// host side
// =====================================================================================================================
inline bool eligible(const DrDesc* d) {
  return d->K == kD && d->V == kD && d->chunk == kC && d->qkv_dtype == DR_BF16;
}
// floats per chunk: checkpoint, N (later the grouped heads' dq^, dk^), Y, X A T, dS1 (first the records of the two-kernel
// forward: 66048 bytes; scalar decays: and the norm factors), e^{G_L}
constexpr int64_t kCkpt = 16384, kNf = 16384, kYf = 8192, kXat = 3 * 4096, kDs = 16512, kEl = 128;
constexpr int64_t kFloats = kCkpt + kNf + kYf + kXat + kDs + kEl;
inline int64_t workspace_bytes(const DrDesc* d) {
  const int64_t N = (d->T + kC - 1) / kC;
  return (int64_t)d->B * d->H * N * kFloats * 4;
}
// Whether local_sm100_kda_kernel was given the registers that its split counts on (another compiler may give it others, and the split waits for good then).
inline bool split_fits(int regs) { return regs == kLkRegs; }
inline cudaError_t local_kernel_fits(bool* fits) {
  thread_local int attr_dev = -1;
  thread_local bool known = false;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess && attr_dev != dev) {
    cudaFuncAttributes at{};
    e = cudaFuncGetAttributes(&at, local_sm100_kda_kernel);
    if (e == cudaSuccess) { known = split_fits(at.numRegs); attr_dev = dev; }
  }
  *fits = known;
  return e;
}
inline bool tma_base(const void* g) { return (reinterpret_cast<uintptr_t>(g) & 15u) == 0; }
// Rows of per-channel decays where a tensor map does not take them (bf16 at eight bytes), and a local_sm100_kda_kernel that was not given its registers, leave
// every chunk to the kernels with 16-row blocks.  g: the decays that the pre-pass reads.
inline Params make_params(const DrDesc* d, void* workspace, const void* g) {
  Params p{};
  bool fits = true;
  if (d->variant == DR_KDA && local_kernel_fits(&fits) != cudaSuccess) fits = false;   // (the launches report what is wrong)
  p.N = (d->T + kC - 1) / kC;
  const int64_t nc = (int64_t)d->B * d->H * p.N;
  p.few = (nc <= kFewKda && p.N <= kFewLength) || (d->variant == DR_KDA && !(tma_base(g) && fits));
  float* f = reinterpret_cast<float*>(workspace);
  p.ckpt = f; f += nc * kCkpt;
  p.nf = reinterpret_cast<float4*>(f); p.part = f; f += nc * kNf;
  p.yf = reinterpret_cast<float4*>(f); f += nc * kYf;
  p.xat = f; f += nc * kXat;
  p.ds = f; p.norms = f + nc * kCkpt; f += nc * kDs;
  p.el = f;
  p.map.B = d->B; p.map.H = d->H; p.map.T = d->T; p.map.bthd = d->layout == DR_LAYOUT_BTHD;
  p.map.Hq = d->qk_heads > 0 ? d->qk_heads : d->H;
  p.variant = d->variant; p.g_dt = d->g_dtype; p.l2norm = d->use_qk_l2norm; p.scale = d->scale;
  return p;
}
template <bool KDA>
inline cudaError_t set_attributes(int* sms = nullptr) {
  thread_local int attr_dev = -1, count = 0;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess && attr_dev != dev) {
    e = cudaFuncSetAttribute(pre_kernel<KDA>, cudaFuncAttributeMaxDynamicSharedMemorySize, pre_smem<KDA>());
    if (e == cudaSuccess)
      e = KDA ? cudaFuncSetAttribute(local_sm100_kda_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LK_TOTAL)
              : cudaFuncSetAttribute(local_sm100_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LT_TOTAL);
    if (KDA && e == cudaSuccess) e = cudaFuncSetAttribute(local_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LoSmem::kTotal);
    if (KDA && e == cudaSuccess) e = cudaFuncSetAttribute(pre_sm100_kda_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, PK_TOTAL);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(chain_kernel<KDA>, cudaFuncAttributeMaxDynamicSharedMemorySize, ch_smem<KDA>());
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) attr_dev = dev;
  }
  if (sms) *sms = count;
  return e;
}
template <bool KDA>
inline cudaError_t launch_pre_t(const Params& p, int64_t units, int32_t* status, cudaStream_t stream, bool beside, int* launches) {
  int sms = 0;
  cudaError_t e = set_attributes<KDA>(&sms);
  if (e != cudaSuccess) return e;
  const int64_t chunks = units * p.N;
  if (KDA && !p.few) {
    PreParams pp;
    pp.p = p; pp.chunks = (int)chunks; pp.status = status; pp.n_tok = units * p.map.T;
    const SeqMap& m = p.map;
    if (!sm100::make_panel_map(&pp.tq, p.q, m.B, m.Hq, m.T, m.bthd != 0) || !sm100::make_panel_map(&pp.tk, p.k, m.B, m.Hq, m.T, m.bthd != 0) ||
        !sm100::make_output_map(&pp.tg, const_cast<void*>(p.g), m, p.g_dt == DR_BF16 ? 2 : 4))
      return cudaErrorInvalidValue;
    ++*launches;
    // Beside the forward's state pass, whose CTAs keep an SM each for 2.65 us a chunk (this kernel: 9 us), its own CTAs keep off those SMs while
    // there are few of them: those that wait for one would do their share of the chunks behind it.  32 sequences of 64 chunks: 160 us on
    // 116 SMs, by the same figures 170 + 125 on all of them; level at about 61 sequences.
    const int64_t free = beside && 5 * units <= 2 * sms ? sms - units : sms;
    e = launch_pdl(pre_sm100_kda_kernel, dim3((unsigned)(chunks < free ? chunks : free)), dim3(kLtThreads), PK_TOTAL, stream, pp);
    if (e != cudaSuccess) return e;
  }
  ++*launches;
  return launch_pdl(pre_kernel<KDA>, dim3((unsigned)(!KDA || p.few || chunks < 2 * sms ? chunks : 2 * sms)), dim3(kPreThreads), pre_smem<KDA>(), stream, p, (int)chunks);
}
inline cudaError_t launch_pre(const DrDesc* d, const void* q, const void* k, const void* g, const float* beta, void* workspace,
                              int32_t* status, cudaStream_t stream, bool beside, int* launches) {
  Params p = make_params(d, workspace, g);
  p.q = q; p.k = k; p.g = g; p.beta = beta;
  const int64_t units = (int64_t)d->B * d->H;
  return d->variant == DR_KDA ? launch_pre_t<true>(p, units, status, stream, beside, launches) : launch_pre_t<false>(p, units, status, stream, beside, launches);
}
template <bool KDA>
inline cudaError_t launch_adjoint_t(Params p, int64_t units, int32_t* status, cudaStream_t stream) {
  int sms = 0;
  cudaError_t e = set_attributes<KDA>(&sms);
  if (e != cudaSuccess) return e;
  const int64_t chunks = units * p.N;
  // the forward that this is the adjoint of had its decays where a tensor map takes them: so that its chunks are read as it left them, they move to Y's
  // place once that has been read (32 KB a chunk, 64 rows of 256 bytes)
  const void* const g_from = KDA && !p.few && !tma_base(p.g) ? p.g : nullptr;
  if (g_from) p.g = p.yf;
  const dim3 grid((unsigned)(chunks < sms ? chunks : sms));
  LocalParams lp;
  lp.p = p; lp.chunks = (int)chunks; lp.status = status;
  lp.n_tok = units * p.map.T; lp.n_part = 2 * chunks * (kC * kD);
  const SeqMap& m = p.map;
  auto panels = [&](CUtensorMap* t, const void* base, int heads) { return sm100::make_panel_map(t, base, m.B, heads, m.T, m.bthd != 0); };
  // (every map before the first launch: a call that fails leaves nothing half done)
  if (!panels(&lp.to, p.d_o, m.H) || !panels(&lp.tq, p.q, m.Hq) || !panels(&lp.tk, p.k, m.Hq) || !panels(&lp.tv, p.v, m.H) || !panels(&lp.tdq, p.dq, m.Hq) ||
      !panels(&lp.tdk, p.dk, m.Hq) || !panels(&lp.tdv, p.dv, m.H))
    return cudaErrorInvalidValue;
  if (KDA && !p.few && !sm100::make_output_map(&lp.tg, const_cast<void*>(p.g), m, p.g_dt == DR_BF16 ? 2 : 4)) return cudaErrorInvalidValue;
  ChainParams c;
  c.p = p;
  c.status = status;
  c.to = lp.to;
  e = launch_pdl(chain_kernel<KDA>, dim3((unsigned)(units * (kD / kChCols))), dim3(ch_threads<KDA>()), ch_smem<KDA>(), stream, c);
  if (g_from && e == cudaSuccess) e = cudaMemcpyAsync(p.yf, g_from, (size_t)units * m.T * kD * 2, cudaMemcpyDeviceToDevice, stream);
  if (e != cudaSuccess) return e;
  if constexpr (KDA) {
    if (p.few) return launch_pdl(local_kernel, dim3((unsigned)chunks), dim3(kLoThreads), LoSmem::kTotal, stream, p, (int)chunks);
    e = launch_pdl(local_sm100_kda_kernel, grid, dim3(kLkThreads), LK_TOTAL, stream, lp);
    if (e != cudaSuccess) return e;
    return launch_pdl(local_kernel, grid, dim3(kLoThreads), LoSmem::kTotal, stream, p, (int)chunks);
  } else {
    return launch_pdl(local_sm100_kernel, grid, dim3(kLtThreads), LT_TOTAL, stream, lp);
  }
}

}  // namespace bwdc
}  // namespace dr
