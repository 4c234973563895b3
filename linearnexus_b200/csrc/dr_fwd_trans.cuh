// Chunk forward in transition form (DeltaNet, Gated DeltaNet, KDA; K = V = D in {64, 128}): everything of a chunk that does
// not depend on the running state is computed chunk-parallel, including the chunk's whole effect on the state.
//
// With T = (I + diag(beta) X)^-1, W = T diag(beta) K^ e^G, U = T diag(beta) V, Kd = K^ e^{G_L - G}, A = tril(Q^K^^T.E):
//     S' = e^{G_L} S + N S + Z        N = -Kd^T W  [D x D],   Z = Kd^T U  [D x D]
//     O  = Y S + A U                  Y = Q^ e^G - A W
//   trans_pre_kernel    one CTA per chunk: N, Z, Y, A U, as mma.sync fragments in the order the lanes of the second kernel
//                       load them (16 bytes per lane)
//   trans_state_kernel  one CTA per (sequence, 8 NT value columns) walks the chunks: one [D x D] product per chunk on the
//                       chain, the output product beside it in warps of its own
//
// Decays are sums over a 16-row block up to a row, sums over its rest, and block totals, each summed by itself: a difference
// of long cumulative sums would lose what the recurrence keeps when a strong decay came earlier in the chunk.  Inside a block the
// scalar decays are differences all the same, so those sums are taken in 64 bits and kept as a float32 pair (eight tokens of -80, then
// eight of -0.02 a block: outputs off by 3.2e-5 with float32 sums, 6.5e-7 so); per-channel ones
// carry the rounding of their float32 sums along (one token of -40 a block: 5.3e-6 without, 6.4e-7 with).  Per-channel
// decays are folded into the rows once: q e^{prefix}, k e^{prefix}, k e^{suffix}; products between blocks carry the totals of
// the blocks in between.  A block whose decay exceeds 2^64 in some channel is summed entry by entry.
//
// It serves float32 storage (and bf16 at D = 64): three tf32 products per pair (dr_tf32.cuh), float32 precision throughout, the
// triangular inverse included.  The token recurrence it replaces there has one CTA per sequence and 64 value columns and a
// dependent chain of ~650 cycles per token: B=2, T=512, H=4, D=64 kept 8 SMs busy for 168 us.
#pragma once

#include "dr_common.cuh"
#include "dr_mma.cuh"
#include "dr_tcgen05.cuh"
#include "dr_tf32.cuh"

namespace dr {
namespace trans {

// operands in two tf32 terms: three products per pair, float32 precision
using AFrag = mma::AFrag<true>;
using BFrag = mma::BFrag<true>;
constexpr int kC = 64;
constexpr int LDX = 72;
constexpr float kLog2e = 1.4426950408889634f;
// A token's scalar log decay is cut off here: float32 has only zeros left for what crosses it, and -infinity (a hard reset) would
// leave infinity minus infinity between the tokens behind it.
constexpr float kDecayFloor = -200.f;

template <int D>
struct Sizes {
  static constexpr int NTHR = D == 128 ? 512 : 256, NW = NTHR / 32, CT = D / 16, LD = D + 4;
  static constexpr int kK = 0, kQ = kK + 64 * LD * 4, kV = kQ + 64 * LD * 4, kX = kV + 64 * LD * 4, kA = kX + 64 * LDX * 4;
  static constexpr int kSc = kA + 64 * LDX * 4;   // beta, prefix, suffix, e^G, e^{G_L - G}, norm factors of q and k, flags, rest of the prefix (64 each)
  static constexpr int kD = kSc + 9 * 64 * 4;     // KDA: per block and channel: its total decay, the decay before it, after it
  static constexpr int kE = kD + 3 * 4 * D * 4;   // KDA: k e^{suffix} [64][LD]
  static constexpr int smem(bool kda) { return kda ? kE + 64 * LD * 4 : kD; }
  // floats per chunk: N, Z, Y, A U, e^{G_L}
  static constexpr int64_t fN = D * D, fZ = D * D, fY = 64 * D, fO = 64 * D, fE = D, kFloats = fN + fZ + fY + fO + fE;
};

struct Params {
  FwdParams p;
  float4 *nf, *zf, *yf, *of;
  float* el;
  int N;
};

__device__ __forceinline__ void zero4(float (&d)[4]) { d[0] = d[1] = d[2] = d[3] = 0.f; }
__device__ __forceinline__ float2 ld2(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float ex2(float x) { return tc::fast_exp2(x); }
__device__ __forceinline__ float4 load4(const void* base, int64_t at, int dt) {
  if (dt == DR_BF16) {
    const uint2 u = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(base) + at);
    return make_float4(mma::lo_f(u.x), mma::hi_f(u.x), mma::lo_f(u.y), mma::hi_f(u.y));
  }
  return *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(base) + at);
}

// T = (I + diag(rs) A)^-1 in place for a strictly lower-triangular 64 x 64 A (row stride LDX): 8 x 8 diagonal blocks by
// substitution, then three merge levels T_10 = -T_11 (diag(rs) A_10) T_00.  Above the diagonal: scratch.
template <int NW>
__device__ __forceinline__ void inverse_64(float* sT, const float* rs, int tid) {
  const int warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  if (tid < 64) {
    const int o = (tid >> 3) * 8, c = tid & 7;
    float a[8][8], f[8], x[8];
#pragma unroll
    for (int i = 1; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < i; ++j) a[i][j] = sT[(o + i) * LDX + o + j];
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = rs[o + i];
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      float acc = 0.f;
#pragma unroll
      for (int j = 0; j < i; ++j) acc += a[i][j] * x[j];
      x[i] = ((i == c) ? 1.f : 0.f) - f[i] * acc;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) sT[(o + i) * LDX + o + c] = x[i];
  }
  __syncthreads();
#pragma unroll 1
  for (int bs = 8; bs < 64; bs *= 2) {
    const int mtn = bs >= 16 ? bs / 16 : 1, ntn = bs / 8, tpp = mtn * ntn, tiles = (32 / bs) * tpp;
#pragma unroll 1
    for (int step = 0; step < 2; ++step) {
#pragma unroll 1
      for (int tile = warp; tile < tiles; tile += NW) {
        const int pr = tile / tpp, mt = (tile % tpp) / ntn, nt = tile % ntn;
        const int r0 = 2 * bs * pr + bs, c0 = 2 * bs * pr, m0 = 16 * mt + g, m1 = m0 + 8, n = 8 * nt + g;
        float d[4];
        zero4(d);
#pragma unroll 1
        for (int k = t; k < bs; k += 8) {
          AFrag a;
          BFrag b;
          if (step == 0) {   // diag(rs) A_10 T_00 -> the mirrored block (rows c0 .., columns r0 ..)
            a.set(m0 < bs ? sT[(r0 + m0) * LDX + c0 + k] : 0.f, m1 < bs ? sT[(r0 + m1) * LDX + c0 + k] : 0.f,
                  m0 < bs ? sT[(r0 + m0) * LDX + c0 + k + 4] : 0.f, m1 < bs ? sT[(r0 + m1) * LDX + c0 + k + 4] : 0.f);
            b.set(n <= k ? sT[(c0 + k) * LDX + c0 + n] : 0.f, n <= k + 4 ? sT[(c0 + k + 4) * LDX + c0 + n] : 0.f);
          } else {           // -T_11 (...) -> T_10
            a.set(m0 < bs && k <= m0 ? sT[(r0 + m0) * LDX + r0 + k] : 0.f, m1 < bs && k <= m1 ? sT[(r0 + m1) * LDX + r0 + k] : 0.f,
                  m0 < bs && k + 4 <= m0 ? sT[(r0 + m0) * LDX + r0 + k + 4] : 0.f, m1 < bs && k + 4 <= m1 ? sT[(r0 + m1) * LDX + r0 + k + 4] : 0.f);
            b.set(sT[(c0 + k) * LDX + r0 + n], sT[(c0 + k + 4) * LDX + r0 + n]);
          }
          mma::fma<true>(d, a, b);
        }
#pragma unroll
        for (int hr = 0; hr < 2; ++hr) {
          const int m = m0 + 8 * hr;
          if (m < bs) {
            const float f = step == 0 ? rs[r0 + m] : -1.f;
            float* dst = step == 0 ? sT + (c0 + m) * LDX + r0 : sT + (r0 + m) * LDX + c0;
            *reinterpret_cast<float2*>(dst + 8 * nt + 2 * t) = make_float2(f * d[2 * hr], f * d[2 * hr + 1]);
          }
        }
      }
      __syncthreads();
    }
  }
}

template <int D, bool KDA>
__global__ void __launch_bounds__(Sizes<D>::NTHR, D == 64 ? 2 : 1) trans_pre_kernel(const __grid_constant__ Params P) {
  pdl_entry();
  using Z_ = Sizes<D>;
  constexpr int NTHR = Z_::NTHR, NW = Z_::NW, CT = Z_::CT, LD = Z_::LD;
  const FwdParams& p = P.p;
  extern __shared__ __align__(16) uint8_t smem[];
  auto F = [&](int off) { return reinterpret_cast<float*>(smem + off); };
  float *sK = F(Z_::kK), *sQ = F(Z_::kQ), *sV = F(Z_::kV), *sX = F(Z_::kX), *sA = F(Z_::kA), *sBeta = F(Z_::kSc);
  float *sPre = sBeta + 64, *sSuf = sBeta + 128, *sEG = sBeta + 192, *sWd = sBeta + 256, *sRq = sBeta + 320, *sRk = sBeta + 384, *sUn = sBeta + 448, *sPreLo = sBeta + 512;
  float *sD = F(Z_::kD), *sBef = sD + 4 * D, *sAft = sD + 8 * D, *sE = F(Z_::kE);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int unit = blockIdx.x / P.N, n = blockIdx.x % P.N;
  const int b = unit / p.map.H, h = unit % p.map.H, t0 = n * kC, rows = min(kC, p.map.T - t0);
  const int64_t qk_base = p.map.base_qk(b, h, D), qk_tok = p.map.tok_qk(D), vg_base = p.map.base(b, h, D), vg_tok = p.map.tok(D);
  const int64_t s_base = p.map.base(b, h, 1), s_tok = p.map.tok(1), chunk = (int64_t)unit * P.N + n;

  // index check of an entry of a scratch array that holds `per` floats a chunk
  auto scratch = [&](int64_t i, int width, int64_t per) { return in_bounds(p.status, i, (int64_t)p.map.B * p.map.H * P.N * (per / width)); };

  // ---- q^, k^ (normalised, scaled), v, decay, beta ---------------------------------------------------------------------------
  {
    constexpr int LPR = D / 4, RPP = NTHR / LPR, PASSES = 64 / RPP;   // lanes per row, rows per pass
    const int r0 = tid / LPR, c4 = 4 * (tid % LPR);
    float4 qv[PASSES], kv[PASSES], vv[PASSES], gv[KDA ? PASSES : 1];
#pragma unroll
    for (int i = 0; i < PASSES; ++i) {
      const int c = r0 + RPP * i;
      qv[i] = kv[i] = vv[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if constexpr (KDA) gv[i] = qv[i];
      const int64_t qk_at = qk_base + (t0 + c) * qk_tok + c4, vg_at = vg_base + (t0 + c) * vg_tok + c4;
      if (c < rows && in_bounds_run(p.status, qk_at, 4, p.n_qk) && in_bounds_run(p.status, vg_at, 4, p.n_v)) {
        qv[i] = load4(p.q, qk_at, p.qkv_dt);
        kv[i] = load4(p.k, qk_at, p.qkv_dt);
        vv[i] = load4(p.v, vg_at, p.qkv_dt);
        if constexpr (KDA) gv[i] = load4(p.g, vg_at, p.g_dt);   // (K = V: as many entries as v)
      }
    }
    auto token = [&](int r) { return r < rows && in_bounds(p.status, s_base + (t0 + r) * s_tok, p.n_tok); };
    if (tid < 64) sBeta[tid] = token(tid) ? p.beta[s_base + (t0 + tid) * s_tok] : 0.f;
    if (!KDA && warp == NW - 1) {
      float lo = 0.f, hi = 0.f;
      if (p.variant == DR_GATED) {
        if (token(lane)) lo = ld_elem(p.g, s_base + (t0 + lane) * s_tok, p.g_dt);
        if (token(lane + 32)) hi = ld_elem(p.g, s_base + (t0 + lane + 32) * s_tok, p.g_dt);
      }
      if (lo < kDecayFloor) lo = kDecayFloor;
      if (hi < kDecayFloor) hi = kDecayFloor;
      // sums inside the 16-row blocks (two blocks per 32 lanes), up to a row and over its rest
      double dlo = lo, dhi = hi;
      float slo = lo, shi = hi;
#pragma unroll
      for (int o = 1; o < 16; o <<= 1) {
        const double a = __shfl_up_sync(0xffffffffu, dlo, o), c = __shfl_up_sync(0xffffffffu, dhi, o);
        const float d = __shfl_down_sync(0xffffffffu, slo, o), e = __shfl_down_sync(0xffffffffu, shi, o);
        if ((lane & 15) >= o) { dlo += a; dhi += c; }
        if ((lane & 15) + o < 16) { slo += d; shi += e; }
      }
      const float plo = (float)dlo, phi = (float)dhi;
      sPreLo[lane] = (float)(dlo - plo); sPreLo[lane + 32] = (float)(dhi - phi);
      const float xlo = __shfl_down_sync(0xffffffffu, slo, 1), xhi = __shfl_down_sync(0xffffffffu, shi, 1);   // exclusive
      slo = (lane & 15) == 15 ? 0.f : xlo; shi = (lane & 15) == 15 ? 0.f : xhi;
      const float t0_ = __shfl_sync(0xffffffffu, plo, 15), t1_ = __shfl_sync(0xffffffffu, plo, 31), t2_ = __shfl_sync(0xffffffffu, phi, 15),
                  t3_ = __shfl_sync(0xffffffffu, phi, 31);
      if (lane == 0) { sUn[8] = t0_; sUn[9] = t1_; sUn[10] = t2_; sUn[11] = t3_; }   // block totals
      sPre[lane] = plo; sPre[lane + 32] = phi;
      sSuf[lane] = slo; sSuf[lane + 32] = shi;
      const bool up = lane >= 16;
      sEG[lane] = expf(plo + (up ? t0_ : 0.f)); sEG[lane + 32] = expf(phi + t0_ + t1_ + (up ? t2_ : 0.f));
      sWd[lane] = expf(slo + t2_ + t3_ + (up ? 0.f : t1_)); sWd[lane + 32] = expf(shi + (up ? 0.f : t3_));
      if (lane < 4) sUn[lane] = 0.f;
    }
#pragma unroll
    for (int i = 0; i < PASSES; ++i) {
      const int c = r0 + RPP * i;
      float mq = p.scale, mk = 1.f;
      if (p.l2norm) {
        float nq = qv[i].x * qv[i].x + qv[i].y * qv[i].y + qv[i].z * qv[i].z + qv[i].w * qv[i].w;
        float nk = kv[i].x * kv[i].x + kv[i].y * kv[i].y + kv[i].z * kv[i].z + kv[i].w * kv[i].w;
#pragma unroll
        for (int o = LPR / 2; o > 0; o >>= 1) {
          nq += __shfl_xor_sync(0xffffffffu, nq, o);
          nk += __shfl_xor_sync(0xffffffffu, nk, o);
        }
        mq = p.scale / (sqrtf(nq) + 1e-6f);
        mk = 1.f / (sqrtf(nk) + 1e-6f);
      }
      *reinterpret_cast<float4*>(sQ + c * LD + c4) = make_float4(qv[i].x * mq, qv[i].y * mq, qv[i].z * mq, qv[i].w * mq);
      *reinterpret_cast<float4*>(sK + c * LD + c4) = make_float4(kv[i].x * mk, kv[i].y * mk, kv[i].z * mk, kv[i].w * mk);
      *reinterpret_cast<float4*>(sV + c * LD + c4) = vv[i];
      if (c4 == 0) { sRq[c] = mq; sRk[c] = mk; }
      if constexpr (KDA)
        *reinterpret_cast<float4*>(sE + c * LD + c4) = make_float4(gv[i].x * kLog2e, gv[i].y * kLog2e, gv[i].z * kLog2e, gv[i].w * kLog2e);
    }
  }
  __syncthreads();
  if constexpr (KDA) {
    // thread = one channel of one block: its sixteen decays -> prefix and suffix sums -> the decayed rows in place
    static_assert(NTHR == 4 * D, "one thread per block and channel");
    const int blk = tid / D, c = tid % D;
    if (tid < 4) sUn[tid] = 0.f;
    float gr[16], suf = 0.f, rest = 0.f;
    auto add = [](float& sum, float& rest, float x) {   // sum + rest += x without a rounding of the sum
      const float s = sum + x, y = s - sum;
      rest += (sum - (s - y)) + (x - y);
      sum = s;
    };
    auto factor = [](float sum, float rest) {   // 2^(sum + rest)
      const float f = ex2(sum);
      return f > 0.f ? fmaf(f, rest * 0.69314718f, f) : f;
    };
#pragma unroll
    for (int r = 0; r < 16; ++r) gr[r] = sE[(16 * blk + r) * LD + c];
#pragma unroll
    for (int r = 15; r >= 0; --r) {
      sE[(16 * blk + r) * LD + c] = sK[(16 * blk + r) * LD + c] * factor(suf, rest);
      add(suf, rest, gr[r]);
    }
    sD[blk * D + c] = factor(suf, rest);
    float pre = 0.f;
    rest = 0.f;
#pragma unroll
    for (int r = 0; r < 16; ++r) {
      add(pre, rest, gr[r]);
      const float f = factor(pre, rest);
      sK[(16 * blk + r) * LD + c] *= f;
      sQ[(16 * blk + r) * LD + c] *= f;
    }
    __syncthreads();
    if (!(suf >= -64.f)) sUn[blk] = 1.f;
    float bef = 1.f, aft = 1.f;
    for (int x = 0; x < blk; ++x) bef *= sD[x * D + c];
    for (int x = blk + 1; x < 4; ++x) aft *= sD[x * D + c];
    sBef[blk * D + c] = bef;
    sAft[blk * D + c] = aft;
    __syncthreads();
    if (tid < D && scratch(chunk * D + tid, 1, Z_::fE)) P.el[chunk * D + tid] = sBef[3 * D + tid] * sD[3 * D + tid];
  } else if (tid < D && scratch(chunk * D + tid, 1, Z_::fE)) {
    P.el[chunk * D + tid] = sEG[63];
  }
  // ---- X = tril(K^K^^T.E, -1), A = tril(Q^K^^T.E) ----------------------------------------------------------------------------------
  auto unsafe = [&](int blk) -> bool { return KDA && sUn[blk] != 0.f; };   // the decay inside the block exceeds 2^64 in some channel
#pragma unroll 1
  for (int tile = warp; tile < 20; tile += NW) {
    const int mt = tile < 2 ? 0 : tile < 6 ? 1 : tile < 12 ? 2 : 3, nt = tile - mt * (mt + 1);
    if (KDA && nt >= 2 * mt && unsafe(mt)) continue;   // done exactly below
    const int r0 = 16 * mt + g, r1 = r0 + 8, j = 8 * nt + g;
    float dk[4], dq[4];
    zero4(dk); zero4(dq);
#pragma unroll 4
    for (int ks = 0; ks < D / 8; ++ks) {
      const int c0 = 8 * ks + t, c1 = c0 + 4;
      float f0 = 1.f, f1 = 1.f;
      const float* kj = sK;
      if constexpr (KDA) {   // k e^{suffix}, times the totals of the blocks in between; inside a block divided by its total
        kj = sE;
        const int bj = nt >> 1;
        if (bj == mt) { f0 = 1.f / sD[mt * D + c0]; f1 = 1.f / sD[mt * D + c1]; }
        for (int x = bj + 1; x < mt; ++x) { f0 *= sD[x * D + c0]; f1 *= sD[x * D + c1]; }
      }
      AFrag ak, aq;
      ak.set(sK[r0 * LD + c0], sK[r1 * LD + c0], sK[r0 * LD + c1], sK[r1 * LD + c1]);
      aq.set(sQ[r0 * LD + c0], sQ[r1 * LD + c0], sQ[r0 * LD + c1], sQ[r1 * LD + c1]);
      BFrag bk;
      bk.set(kj[j * LD + c0] * f0, kj[j * LD + c1] * f1);
      mma::fma<true>(dk, ak, bk);
      mma::fma<true>(dq, aq, bk);
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = 16 * mt + g + 8 * (e >> 1), jj = 8 * nt + 2 * t + (e & 1);
      float f = 1.f;
      if constexpr (!KDA) {
        const int bj = nt >> 1;
        float x = bj == mt ? (sPre[i] - sPre[jj]) + (sPreLo[i] - sPreLo[jj]) : sPre[i] + sSuf[jj];
        for (int y = bj + 1; y < mt; ++y) x += sUn[8 + y];
        f = expf(fminf(x, 0.f));
      }
      sX[i * LDX + jj] = jj < i ? dk[e] * f : 0.f;
      sA[i * LDX + jj] = jj <= i ? dq[e] * f : 0.f;
    }
  }
  if constexpr (KDA) {   // diagonal blocks with too wide a decay range: exactly, one entry per thread
    for (int blk = 0; blk < 4; ++blk) {
      if (!unsafe(blk) || tid >= 256) continue;
      const int i = 16 * blk + (tid >> 4), j = 16 * blk + (tid & 15);
      float ak = 0.f, aq = 0.f;
      auto qk = [&](const void* x, int r, int c) {
        const int64_t at = qk_base + (t0 + r) * qk_tok + c;
        return in_bounds(p.status, at, p.n_qk) ? ld_elem(x, at, p.qkv_dt) : 0.f;
      };
      if (j <= i && i < rows)
        for (int c = 0; c < D; ++c) {
          float x = 0.f;   // the decay of tokens j + 1 .. i, from the inputs
          for (int m = j + 1; m <= i; ++m) {
            const int64_t at = vg_base + (t0 + m) * vg_tok + c;
            if (in_bounds(p.status, at, p.n_gk)) x += ld_elem(p.g, at, p.g_dt);
          }
          const float w = qk(p.k, j, c) * sRk[j] * expf(x);
          ak += qk(p.k, i, c) * w;
          aq += qk(p.q, i, c) * w;
        }
      ak *= sRk[i];
      aq *= sRq[i];
      sX[i * LDX + j] = j < i ? ak : 0.f;
      sA[i * LDX + j] = j <= i ? aq : 0.f;
    }
  }
  __syncthreads();
  inverse_64<NW>(sX, sBeta, tid);   // ends with a barrier
  // ---- W^T and U^T of the warp's 16 channels / value columns (two warps share them): rows = columns of W / U, columns = tokens ---------
  const int own = warp % CT, part = warp / CT, ch0 = 16 * own + g, ch1 = ch0 + 8;
  float W[8][4], U[8][4];
#pragma unroll
  for (int nt = 0; nt < 8; ++nt) { zero4(W[nt]); zero4(U[nt]); }
#pragma unroll
  for (int ks = 0; ks < 8; ++ks) {
    const int j0 = 8 * ks + 2 * t, j1 = j0 + 1;
    const float b0 = sBeta[j0], b1 = sBeta[j1];
    float w00, w01, w10, w11;   // beta e^G at (token, channel) over what the rows already carry
    if constexpr (KDA) {
      const float f0 = sBef[(ks >> 1) * D + ch0], f1 = sBef[(ks >> 1) * D + ch1];
      w00 = b0 * f0; w01 = b0 * f1; w10 = b1 * f0; w11 = b1 * f1;
    } else {
      w00 = w01 = b0 * sEG[j0];
      w10 = w11 = b1 * sEG[j1];
    }
    AFrag aw, au;
    aw.set(sK[j0 * LD + ch0] * w00, sK[j0 * LD + ch1] * w01, sK[j1 * LD + ch0] * w10, sK[j1 * LD + ch1] * w11);
    au.set(sV[j0 * LD + ch0] * b0, sV[j0 * LD + ch1] * b0, sV[j1 * LD + ch0] * b1, sV[j1 * LD + ch1] * b1);
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
      if (nt >= ks) {
        const int i = 8 * nt + g;
        const float2 x = ld2(sX + i * LDX + j0);
        BFrag bt;
        bt.set(j0 <= i ? x.x : 0.f, j1 <= i ? x.y : 0.f);
        mma::fma<true>(W[nt], aw, bt);
        mma::fma<true>(U[nt], au, bt);
      }
    }
  }
  __syncthreads();
  // ---- K^ -> Kd = K^ e^{G_L - G} in place --------------------------------------------------------------------------------------------
  {
    constexpr int LPR = D / 4;
    for (int i = tid; i < 64 * LPR; i += NTHR) {
      const int c = i / LPR, c4 = 4 * (i % LPR);
      float4 x = *reinterpret_cast<const float4*>((KDA ? sE : sK) + c * LD + c4);
      if constexpr (KDA) {
        const float4 f = *reinterpret_cast<const float4*>(sAft + (c >> 4) * D + c4);
        x.x *= f.x; x.y *= f.y; x.z *= f.z; x.w *= f.w;
      } else {
        const float f = sWd[c];
        x.x *= f; x.y *= f; x.z *= f; x.w *= f;
      }
      *reinterpret_cast<float4*>(sK + c * LD + c4) = x;
    }
  }
  __syncthreads();
  // ---- [Kd^T; A] [W | U]: an accumulator of W^T or U^T is, register for register, the B operand of its columns ----------------------------
  auto products = [&](float (&w)[2][4], float (&u)[2][4], int ks, const AFrag& a) {
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      BFrag bw, bu;
      bw.set(W[ks][2 * hf], W[ks][2 * hf + 1]);
      bu.set(U[ks][2 * hf], U[ks][2 * hf + 1]);
      mma::fma<true>(w[hf], a, bw);
      mma::fma<true>(u[hf], a, bu);
    }
  };
#pragma unroll 1
  for (int mt = part * (CT / 2); mt < (part + 1) * (CT / 2); ++mt) {
    float w[2][4], u[2][4];
    zero4(w[0]); zero4(w[1]); zero4(u[0]); zero4(u[1]);
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      const float* k0 = sK + (8 * ks + 2 * t) * LD + 16 * mt + g;
      AFrag a;
      a.set(k0[0], k0[8], k0[LD], k0[LD + 8]);
      products(w, u, ks, a);
    }
    const int64_t at = ((chunk * CT + mt) * (2 * CT) + 2 * own) * 32 + lane;
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      if (!scratch(at + 32 * hf, 4, Z_::fN)) continue;
      P.nf[at + 32 * hf] = make_float4(-w[hf][0], -w[hf][2], -w[hf][1], -w[hf][3]);
      P.zf[at + 32 * hf] = make_float4(u[hf][0], u[hf][1], u[hf][2], u[hf][3]);
    }
  }
#pragma unroll 1
  for (int m = 0; m < 2; ++m) {
    const int mt = part ? 1 + m : 3 * m;   // token tiles 0, 3 and 1, 2: ten k-steps each
    float w[2][4], u[2][4];
    zero4(w[0]); zero4(w[1]); zero4(u[0]); zero4(u[1]);
#pragma unroll
    for (int ks = 0; ks < 8; ++ks) {
      if (ks <= 2 * mt + 1) {
        const float2 x0 = ld2(sA + (16 * mt + g) * LDX + 8 * ks + 2 * t), x1 = ld2(sA + (16 * mt + g + 8) * LDX + 8 * ks + 2 * t);
        AFrag a;
        a.set(x0.x, x1.x, x0.y, x1.y);
        products(w, u, ks, a);
      }
    }
    const int64_t at = ((chunk * 4 + mt) * (2 * CT) + 2 * own) * 32 + lane;
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      float y[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = 16 * mt + g + 8 * (e >> 1), c = 16 * own + 8 * hf + 2 * t + (e & 1);
        y[e] = sQ[i * LD + c] * (KDA ? sBef[mt * D + c] : sEG[i]) - w[hf][e];
      }
      if (!scratch(at + 32 * hf, 4, Z_::fY)) continue;
      P.yf[at + 32 * hf] = make_float4(y[0], y[2], y[1], y[3]);
      P.of[at + 32 * hf] = make_float4(u[hf][0], u[hf][1], u[hf][2], u[hf][3]);
    }
  }
}

// Warps 0 .. D/16 - 1: state rows 16 w ..; four more warps: output rows 16 (w - D/16) ...  NT: 8-column tiles per CTA.
template <int D, int NT>
__global__ void __launch_bounds__((D / 16 + 4) * 32, 1) trans_state_kernel(const __grid_constant__ Params P) {
  pdl_entry();
  constexpr int CT = D / 16, VS = 8 * NT, LDP = 2 * VS + 8;   // S in shared memory: row pairs interleaved [D / 2][VS][2]
  const FwdParams& p = P.p;
  __shared__ __align__(16) float sS[2][D / 2 * LDP];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  constexpr int SL = D / VS;
  const int unit = blockIdx.x / SL, v0 = (blockIdx.x % SL) * VS;
  const int b = unit / p.map.H, h = unit % p.map.H;
  const int64_t chunk0 = (int64_t)unit * P.N;
  const bool state = warp < CT;
  const int mt = state ? warp : warp - CT;
  const int r0 = 16 * mt + g, r1 = r0 + 8;
  const float4* fa = state ? P.nf : P.yf;   // A fragments [chunk][rows / 16][D / 8][32]
  const float4* fc = state ? P.zf : P.of;   // addends      [chunk][rows / 16][D / 8][32]
  const int tiles = state ? CT : 4;
  float4 a[D / 8], c[NT];
  float S[NT][4], el0 = 0.f, el1 = 0.f;
  // entry `i` of a scratch array; both halves of the warps read arrays of tiles * (D / 8) * 32 entries a chunk
  const int64_t entries = (int64_t)p.map.B * p.map.H * P.N * tiles * (D / 8) * 32;
  auto get = [&](const float4* f, int64_t i) { return in_bounds(p.status, i, entries) ? f[i] : make_float4(0.f, 0.f, 0.f, 0.f); };
  auto get_a = [&](int64_t ch, int ks) { return get(fa, ((ch * tiles + mt) * (D / 8) + ks) * 32 + lane); };
  auto get_c = [&](int64_t ch, int nt) { return get(fc, ((ch * tiles + mt) * (D / 8) + v0 / 8 + nt) * 32 + lane); };
  auto get_el = [&](int64_t ch, int r) { return in_bounds(p.status, ch * D + r, (int64_t)p.map.B * p.map.H * P.N * D) ? P.el[ch * D + r] : 0.f; };
  auto s_at = [&](int r, int nt) { return ((int64_t)unit * D + r) * D + v0 + 8 * nt + 2 * t; };
#pragma unroll
  for (int ks = 0; ks < D / 8; ++ks) a[ks] = get_a(chunk0, ks);
#pragma unroll
  for (int nt = 0; nt < NT; ++nt) c[nt] = get_c(chunk0, nt);
  if (state) {
    el0 = get_el(chunk0, r0); el1 = get_el(chunk0, r1);
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
  const int64_t o_base = p.map.base(b, h, D) + v0, o_tok = p.map.tok(D);
  for (int n = 0; n < P.N; ++n) {
    float* cS = sS[n & 1];
    if (state) {
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const int cc = 2 * (8 * nt + 2 * t);
        float* w0 = cS + (r0 >> 1) * LDP + cc + (r0 & 1);
        float* w1 = cS + (r1 >> 1) * LDP + cc + (r1 & 1);
        w0[0] = S[nt][0]; w0[2] = S[nt][1];
        w1[0] = S[nt][2]; w1[2] = S[nt][3];
      }
    }
    __syncthreads();
    float d[NT][4], e[NT][4];   // two accumulators: shorter chains
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      d[nt][0] = c[nt].x; d[nt][1] = c[nt].y; d[nt][2] = c[nt].z; d[nt][3] = c[nt].w;
      zero4(e[nt]);
    }
    const int64_t cn = chunk0 + (n + 1 < P.N ? n + 1 : n);   // the next chunk's operands replace this one's as they are used
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) c[nt] = get_c(cn, nt);
#pragma unroll
    for (int ks = 0; ks < D / 8; ++ks) {
      AFrag fr;
      fr.set(a[ks].x, a[ks].y, a[ks].z, a[ks].w);
      a[ks] = get_a(cn, ks);
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        const float2 y = ld2(cS + (4 * ks + t) * LDP + 2 * (8 * nt + g));
        BFrag bs;
        bs.set(y.x, y.y);
        if (ks & 1) mma::fma<true>(e[nt], fr, bs); else mma::fma<true>(d[nt], fr, bs);
      }
    }
    if (state) {
#pragma unroll
      for (int nt = 0; nt < NT; ++nt) {
        S[nt][0] = el0 * S[nt][0] + (d[nt][0] + e[nt][0]); S[nt][1] = el0 * S[nt][1] + (d[nt][1] + e[nt][1]);
        S[nt][2] = el1 * S[nt][2] + (d[nt][2] + e[nt][2]); S[nt][3] = el1 * S[nt][3] + (d[nt][3] + e[nt][3]);
      }
      el0 = get_el(cn, r0); el1 = get_el(cn, r1);
    } else {
#pragma unroll
      for (int hr = 0; hr < 2; ++hr) {
        const int tok = n * kC + r0 + 8 * hr;
        if (tok < p.map.T) {
          const int64_t at = o_base + (int64_t)tok * o_tok + 2 * t;
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            const float x = d[nt][2 * hr] + e[nt][2 * hr], y = d[nt][2 * hr + 1] + e[nt][2 * hr + 1];
            if (!in_bounds_run(p.status, at + 8 * nt, 2, p.n_v)) continue;
            if (p.out_dt == DR_BF16)
              *reinterpret_cast<uint32_t*>(reinterpret_cast<__nv_bfloat16*>(p.o) + at + 8 * nt) = mma::pack(x, y);
            else
              *reinterpret_cast<float2*>(reinterpret_cast<float*>(p.o) + at + 8 * nt) = make_float2(x, y);
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
}

inline int64_t workspace_bytes(int64_t units, int T, int D) {
  return units * ((T + kC - 1) / kC) * 4 * (D == 128 ? Sizes<128>::kFloats : Sizes<64>::kFloats);
}

template <int D, bool KDA>
inline cudaError_t launch_t(const FwdParams& p, void* workspace, int sms, cudaStream_t stream) {
  using Z = Sizes<D>;
  thread_local int attr_dev = -1;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (attr_dev != dev) {
    e = cudaFuncSetAttribute(trans_pre_kernel<D, KDA>, cudaFuncAttributeMaxDynamicSharedMemorySize, Z::smem(KDA));
    if (e != cudaSuccess) return e;
    attr_dev = dev;
  }
  Params P;
  P.p = p;
  P.N = (p.map.T + kC - 1) / kC;
  const int64_t units = (int64_t)p.map.B * p.map.H, nc = units * P.N;
  float* f = reinterpret_cast<float*>(workspace);
  P.nf = reinterpret_cast<float4*>(f); f += nc * Z::fN;
  P.zf = reinterpret_cast<float4*>(f); f += nc * Z::fZ;
  P.yf = reinterpret_cast<float4*>(f); f += nc * Z::fY;
  P.of = reinterpret_cast<float4*>(f); f += nc * Z::fO;
  P.el = f;
  e = launch_pdl(trans_pre_kernel<D, KDA>, dim3((unsigned)nc), dim3(Z::NTHR), Z::smem(KDA), stream, P);
  if (e != cudaSuccess) return e;
  // narrow slices while they fit one wave: the chain's length is what counts, and every slice adds readers of N and Y
  if (units * (D / 16) <= sms)
    return launch_pdl(trans_state_kernel<D, 2>, dim3((unsigned)(units * (D / 16))), dim3((D / 16 + 4) * 32), 0, stream, P);
  return launch_pdl(trans_state_kernel<D, 4>, dim3((unsigned)(units * (D / 32))), dim3((D / 16 + 4) * 32), 0, stream, P);
}

template <int D>
inline cudaError_t launch_d(const FwdParams& p, void* workspace, int sms, cudaStream_t stream) {
  return p.variant == DR_KDA ? launch_t<D, true>(p, workspace, sms, stream) : launch_t<D, false>(p, workspace, sms, stream);
}

}  // namespace trans
}  // namespace dr
