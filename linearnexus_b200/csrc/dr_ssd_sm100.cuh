// Mamba-2 SSD scan in chunk form on tcgen05, bf16 storage, float32 operands of the products as three bf16 terms (24 bits), decay
// factors to float32 precision (measured in the tests: test_ssd_decay_weights_inside_a_chunk).  Formulas: header of dr_ssd_chunk.cuh,
// with chunks of 128 tokens; per chunk, with S^T [N][P] the state at its start,
//     G  = C B^T                                      128 x 128 x N   both from shared memory
//     P  = tril(G e^{G_i - G_j} dt_j), three bf16 terms over G in tensor memory (the third beside it)
//     Y2 = P x                                        128 x 64 x 128  A from tensor memory, three terms
//     Y1 = C S^T                                      128 x 64 x N    S^T as three bf16 tiles, [hi | mid] as one N = 128 product
//     D  = B^T xs,  xs = dt e^{G_L - G} x             N x 64 x 128    xs as three bf16 tiles, likewise
//     y  = e^{G_i} Y1 + Y2 + D x;  S^T <- e^{G_L} S^T + D
// The state stays in the registers of the group that owns it (thread = state column n, 64 values) and only its terms go through
// shared memory, so no product waits for another chunk's product: the chain is one multiply-add per entry and the split, and the
// step follows the sum of the tensor work (N = 128: 48 products of N = 64 at 49 cycles or 33 and 24 of N = 128 at 65, 3.1 K cycles), the
// waits between them, or the longest group, whichever is longer.
//
// 20 warps, one CTA per (batch, head, 64 value columns):
//   0-7    G -> P; warp = rows of a quarter (warp & 3) and half of the columns (warp >> 2)
//   8-11   the state: D -> S, S -> its three terms
//   12-15  x -> xs (thread = token), outputs (thread = token)
//   16     issues every product (one elected thread)
//   17     copies B, C, x (one thread, TMA, 128-byte swizzle; tokens past the end arrive as zeros)
//   18, 19 dt -> scalars of a chunk
// B, C, the terms of S and of xs have one tile each, x three (it is read again for the outputs, whose rows are staged over it),
// the scalars three stages.  A product that accumulates onto one of another shape waits for it: only products of equal shape are ordered.
//
// What bounds it: B=8, T=4096, H=16, N=128: 133 to 137 us on different boxes, 318 in the mma.sync form (tensor pipe 41 % of 1024
// multiply-adds per clock and SM; tcgen05 takes 4096).  A chunk takes 7.1 K cycles: tensor pipe 40 %, issue slots 53 %, 15.0 K warp
// instructions; per instruction issued a warp waits 4.0 cycles on hand-overs and tensor memory and 0.8 on the instruction fetch, so
// the loops are kept rolled (75 KB of code; 150 KB: 215 us, 100 KB: 162).  Twenty-four warps with the outputs on their own
// (setmaxnreg for the state's group): 137, 133 without; xs by the warps with the least of P: 136; the issue loops unrolled by four:
// 142.  Segments over a cluster for few sequences, decay sums in 64 bits and their cut-off: as there.
//
// Infinities and NaN in x: P is 0 above the diagonal, but 0 x inf is NaN, and a whole chunk is one product.  Such an entry is
// taken out of the tile of Y2 (it stays in xs, so the state gets it) and the outputs of its column from its token on become NaN.
#pragma once

#include <cooperative_groups.h>

#include <type_traits>

#include "dr_linrec.cuh"
#include "dr_mma.cuh"
#include "dr_sm100_common.cuh"
#include "dr_tcgen05.cuh"

namespace dr {
namespace ssdu {

constexpr int kC = 128, kP = 64, kThreads = 20 * 32;
constexpr float kDecayFloor = -200.f;   // as in the mma.sync form
constexpr int kPanel = 128 * 128;       // 128 rows of 64 bf16, 128-byte swizzle
constexpr int kXs = 3;                  // x tiles, and scalars of a chunk, in flight
// per chunk and token j: G as a float32 pair (log2 units), dt, e^G, dt e^{G_L - G}; dt e^{G_r - G_j} for r = 32, 64, 96 (j < r)
constexpr int kScalars = 8, SC_G = 0, SC_R = kC, SC_DT = 2 * kC, SC_EG = 3 * kC, SC_W = 4 * kC, SC_H = 5 * kC;

constexpr int kBadRow = kP + 4;         // per column, then one word for the whole chunk

// tensor-memory columns
constexpr uint32_t TM_G = 0;      // G, then P: per 16 tokens j the hi and mid terms (8 + 8 columns)   128
constexpr uint32_t TM_PL = 128;   // lo terms of P                                                     64
constexpr uint32_t TM_Y2 = 192;   // P x                                                               64
constexpr uint32_t TM_Y1 = 256;   // C [hi + lo | mid] of S^T                                         128
constexpr uint32_t TM_D = 384;    // B^T [hi + lo | mid] of xs                                        128

template <int N>
struct Smem {
  static constexpr int kB = 0;                          // two panels (N = 64: the second is zero)
  static constexpr int kCt = kB + 2 * kPanel;
  static constexpr int kX = kCt + (N / 64) * kPanel;
  static constexpr int kXt = kX + kXs * kPanel;         // terms of xs
  static constexpr int kSt = kXt + 3 * kPanel;          // terms of S^T; a segment's end state [64][128] fp32 between the passes
  static constexpr int kSc = kSt + 3 * kPanel;          // kXs stages of kScalars arrays
  static constexpr int kBad = kSc + kXs * kScalars * kC * 4;     // kXs stages of kBadRow words, see bad_of
  static constexpr int kTotal = kBad + kXs * kBadRow * 4;
};

// 2^{(a + b) - (c + d)} of two float32 pairs, to about one unit in the last place: the difference is taken whole (what a - c loses joins
// the rests), and e^{f ln 2}, |f| <= 1/2, is its Taylor series to f^7 (the next term is below 6e-9).  Underflows gradually, as exp2f does.
__device__ __forceinline__ float exp2_diff(float a, float b, float c, float d) {
  const float s = a - c, t = s - a;
  const float rest = ((a - (s - t)) - (c + t)) + (b - d);   // (two-sum)
  const float x = fminf(fmaxf(s, -252.f), 254.f), n = rintf(x), f = (x - n) + rest;
  float p = 1.5252734e-5f;   // (ln 2)^k / k!
  p = fmaf(p, f, 1.5403530e-4f);
  p = fmaf(p, f, 1.3333558e-3f);
  p = fmaf(p, f, 9.6181291e-3f);
  p = fmaf(p, f, 5.5504109e-2f);
  p = fmaf(p, f, 2.4022651e-1f);
  p = fmaf(p, f, 6.9314718e-1f);
  p = fmaf(p, f, 1.f);
  const int e = (int)n, half = e / 2;
  return p * __int_as_float((127 + half) << 23) * __int_as_float((127 + e - half) << 23);
}

struct Ctl {
  uint64_t fullB, fullC, fullX[kXs], scal[kXs], xs, d_read[kXs], x_free[kXs], s_rdy, y_read, p_rdy[4];
  uint64_t barDa, barD, barG, barY1a, barY1, barY;
  uint32_t tmem_base;
  int abort;
  float seg_decay;
};

// byte offset of 16-byte piece c of row r of a panel
__device__ __forceinline__ uint32_t piece_at(int r, int c) { return (uint32_t)(r * 128 + ((c ^ (r & 7)) << 4)); }
__device__ __forceinline__ void cluster_barrier() {   // whole warps
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

struct alignas(64) Params {
  CUtensorMap tb, tc, tx;   // {columns, heads or groups, T, B} of B, C and x; a box is 64 columns of 128 tokens
  LinRecParams p;
  int nseg;
};

template <int N>
__global__ void __launch_bounds__(kThreads, 1) ssd_sm100_kernel(const __grid_constant__ Params P) {
  const LinRecParams& p = P.p;
  const int nseg = P.nseg;
  using L = Smem<N>;
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ __align__(16) Ctl ctl;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31, wq = warp & 3;
  const int lt = 32 * wq + lane;   // tensor-memory lane of the thread (warps 0-15)
  const int seg = blockIdx.x % nseg;
  const int slices = p.V / kP, unit = blockIdx.x / nseg / slices, slice = blockIdx.x / nseg % slices;
  const int b = unit / p.H, h = unit % p.H, T = p.T;
  const int nchunks = (T + kC - 1) / kC, per = (nchunks + nseg - 1) / nseg;
  const int c_lo = min(seg * per, nchunks), c_hi = min(c_lo + per, nchunks);
  // the CTA's steps: its chunks for their effect on the state alone (all but the last segment), then in full
  const int n1 = seg + 1 < nseg ? c_hi - c_lo : 0, steps = n1 + c_hi - c_lo;
  auto chunk_of = [&](int it) { return c_lo + (it < n1 ? it : it - n1); };

  if (warp == 0) {
    tc::tmem_alloc(tc::smem_u32(&ctl.tmem_base), 512);
    tc::tmem_relinquish();
  }
  if (tid == 0) {
    auto init = [&](uint64_t& bar, uint32_t count) { tc::mbar_init(tc::smem_u32(&bar), count); };
    init(ctl.fullB, 1); init(ctl.fullC, 1);
    for (int i = 0; i < kXs; ++i) { init(ctl.fullX[i], 1); init(ctl.x_free[i], 128); init(ctl.scal[i], 1); init(ctl.d_read[i], 128); }
    for (int i = 0; i < 4; ++i) init(ctl.p_rdy[i], 128);
    init(ctl.y_read, 128);
    init(ctl.xs, 128); init(ctl.s_rdy, 128);
    init(ctl.barDa, 1); init(ctl.barD, 1); init(ctl.barG, 1); init(ctl.barY1a, 1); init(ctl.barY1, 1); init(ctl.barY, 1);
    tc::fence_mbar_init();
    ctl.abort = 0;
  }
  if (tid < kXs * kBadRow) reinterpret_cast<uint32_t*>(smem + L::kBad)[tid] = 0u;
  if (N == 64)
    for (int i = tid; i < kPanel / 16; i += kThreads) *reinterpret_cast<uint4*>(smem + L::kB + kPanel + 16 * i) = make_uint4(0u, 0u, 0u, 0u);
  tc::fence_async_smem();
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  pdl_entry();
  const uint32_t tbase = ctl.tmem_base, lane_addr = (uint32_t)(wq * 32) << 16, sbase = tc::smem_u32(smem);
  auto wait_bar = [&](uint64_t& bar, uint32_t parity) {
    const uint32_t at = tc::smem_u32(&bar);
    sm100::wait_inline(at, parity, &ctl.abort, at - tc::smem_u32(&ctl), warp < 8 ? 0 : warp < 12 ? 1 : warp < 16 ? 2 : 3);
  };
  auto arrive = [&](uint64_t& bar) { sm100::mbar_arrive(tc::smem_u32(&bar)); };
  auto scalars = [&](int it) { return reinterpret_cast<float*>(smem + L::kSc) + (it % kXs) * kScalars * kC; };
  // between the two passes of a segmented run: the segments' ends are out, then every segment has read them
  auto boundary = [&]() {
    if (nseg > 1) { cluster_barrier(); cluster_barrier(); }
  };

  if (warp < 8) {
    // =========================== G -> P ==========================================================================
    const int jh = warp >> 2;
    boundary();
#pragma unroll 1
    for (int it = n1; it < steps; ++it) {
      const int m = it - n1;
      const float* sc = scalars(it);
      wait_bar(ctl.scal[it % kXs], (it / kXs) & 1);
      const float Gi = sc[SC_G + lt], ri = sc[SC_R + lt];
      // Left of the warp's 32 x 32 diagonal block the decay is a product of two: to its first row r, and from there.  Both factors are
      // exact to about one unit in the last place, since the rounding of a long difference would cost more than the product does:
      // rms error of a weight between the halves of a chunk 4.0e-8 (decays of 2^-0.2 a token) and 4.1e-8 (2^-1); as one exponential
      // of the rounded difference 1.8e-7 and 9.8e-7, as the mma.sync form has it across its chunks 9e-8 and 3.9e-7.
      const float fi = exp2_diff(Gi, ri, sc[SC_G + 32 * wq], sc[SC_R + 32 * wq]);
      const float* sH = sc + SC_H + (wq - 1) * kC;
      wait_bar(ctl.barG, m & 1);
      tc::tc_fence_after();
#pragma unroll 1
      for (int kb = 0; kb < 4; ++kb) {
        const int j0 = 64 * jh + 16 * kb;
        uint32_t hm[16], lo[8];
        if (j0 < 32 * wq + 32) {
          uint32_t r[16];
          tc::tmem_ld16(tbase + TM_G + lane_addr + j0, r);
          float x[16];
          if (j0 < 32 * wq) {
            float f[16];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const float4 H = *reinterpret_cast<const float4*>(sH + j0 + 4 * q);
              f[4 * q] = fi * H.x; f[4 * q + 1] = fi * H.y; f[4 * q + 2] = fi * H.z; f[4 * q + 3] = fi * H.w;
            }
            tc::tc_wait_ld();
#pragma unroll
            for (int e = 0; e < 16; ++e) x[e] = __uint_as_float(r[e]) * f[e];
          } else {
            float f[16];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const float4 G = *reinterpret_cast<const float4*>(sc + SC_G + j0 + 4 * q), r2 = *reinterpret_cast<const float4*>(sc + SC_R + j0 + 4 * q);
              f[4 * q] = (Gi - G.x) + (ri - r2.x); f[4 * q + 1] = (Gi - G.y) + (ri - r2.y);
              f[4 * q + 2] = (Gi - G.z) + (ri - r2.z); f[4 * q + 3] = (Gi - G.w) + (ri - r2.w);
            }
            // the fast form drops what lies below the normal range; the sums run one way, so the first column has the smallest
            if (__any_sync(0xffffffffu, f[0] < -125.f)) {
#pragma unroll
              for (int e = 0; e < 16; ++e) f[e] = exp2f(f[e]);
            } else {
#pragma unroll
              for (int e = 0; e < 16; ++e) f[e] = tc::fast_exp2(f[e]);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const float4 d = *reinterpret_cast<const float4*>(sc + SC_DT + j0 + 4 * q);
              f[4 * q] *= d.x; f[4 * q + 1] *= d.y; f[4 * q + 2] *= d.z; f[4 * q + 3] *= d.w;
            }
            tc::tc_wait_ld();
#pragma unroll
            for (int e = 0; e < 16; ++e) x[e] = e <= lt - j0 ? __uint_as_float(r[e]) * f[e] : 0.f;
          }
#pragma unroll
          for (int e = 0; e < 8; ++e) mma::split3_exact(x[2 * e], x[2 * e + 1], hm[e], hm[8 + e], lo[e]);
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) hm[e] = hm[8 + e] = lo[e] = 0u;
        }
        tc::tmem_st16(tbase + TM_G + lane_addr + j0, hm);
        tc::tmem_st8(tbase + TM_PL + lane_addr + j0 / 2, lo);
        if (kb & 1) {   // 32 tokens: their product need not wait for the rest
          tc::tc_wait_st();
          tc::tc_fence_before();
          arrive(ctl.p_rdy[2 * jh + (kb >> 1)]);
        }
      }
    }
  } else if (warp < 12) {
    // =========================== the state: thread = state column lt ============================================
    const bool live = lt < N;
    const int64_t s_unit = ((int64_t)unit * p.V + slice * kP) * N + lt;
    float S[kP];
#pragma unroll
    for (int q = 0; q < kP; ++q) S[q] = 0.f;
    float dec_all = 1.f;
    auto update = [&](int it) {
      wait_bar(ctl.barD, it & 1);
      tc::tc_fence_after();
      const float dec = scalars(it)[SC_EG + kC - 1];
      dec_all *= dec;
#pragma unroll
      for (int q = 0; q < kP; q += 8) {
        uint32_t x[8], y[8];
        tc::tmem_ld8(tbase + TM_D + lane_addr + q, x);
        tc::tmem_ld8(tbase + TM_D + 64 + lane_addr + q, y);
        tc::tc_wait_ld();
#pragma unroll
        for (int e = 0; e < 8; ++e) S[q + e] = S[q + e] * dec + (__uint_as_float(x[e]) + __uint_as_float(y[e]));
      }
      tc::tc_fence_before();
      arrive(ctl.d_read[it % kXs]);
    };
    auto publish = [&](int m) {   // the terms of the state at the start of full step m
      if (m >= 1) wait_bar(ctl.barY1, (m - 1) & 1);
      if (live) {
        uint8_t* dst = smem + L::kSt;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          uint4 w1, w2, w3;
          uint32_t *a = reinterpret_cast<uint32_t*>(&w1), *bb = reinterpret_cast<uint32_t*>(&w2), *cc = reinterpret_cast<uint32_t*>(&w3);
#pragma unroll
          for (int e = 0; e < 4; ++e) mma::split3(S[8 * c + 2 * e], S[8 * c + 2 * e + 1], a[e], bb[e], cc[e]);
          const uint32_t at = piece_at(lt, c);
          *reinterpret_cast<uint4*>(dst + at) = w1;
          *reinterpret_cast<uint4*>(dst + kPanel + at) = w2;
          *reinterpret_cast<uint4*>(dst + 2 * kPanel + at) = w3;
        }
      }
      tc::fence_async_smem();
      arrive(ctl.s_rdy);
    };
    // The state at the CTA's first step; between the passes the segment's own effect goes out first, and the start of the second
    // pass is the earlier segments' ends, decayed.
    auto start = [&](bool exchange) {
      namespace cg = cooperative_groups;
      cg::cluster_group cluster = cg::this_cluster();
      float* own = reinterpret_cast<float*>(smem + L::kSt) + lt;
      if (exchange) {
#pragma unroll
        for (int q = 0; q < kP; ++q) own[q * kC] = S[q];
        if (lt == 0) ctl.seg_decay = dec_all;
        cluster_barrier();
      }
      const bool from_h0 = seg == 0 && p.h0 && live;
#pragma unroll
      for (int q = 0; q < kP; ++q) S[q] = from_h0 && in_bounds(p.status, s_unit + q * N, p.n_state) ? p.h0[s_unit + q * N] : 0.f;
      if (exchange) {
#pragma unroll 1
        for (int s = 0; s < seg; ++s) {
          const float* other = cluster.map_shared_rank(own, s);
          const float d = *cluster.map_shared_rank(&ctl.seg_decay, s);
#pragma unroll
          for (int q = 0; q < kP; ++q) S[q] = S[q] * d + other[q * kC];
        }
        cluster_barrier();   // the others have read this CTA's copy (and p.hT may alias p.h0)
      }
    };
#pragma unroll 1
    for (int it = 0;; ++it) {
      if (it == 0 || it == n1) start(it == n1 && nseg > 1);
      if (it == steps) break;
      if (it >= n1) publish(it - n1);
      update(it);
    }
    if (p.hT && seg == nseg - 1 && live) {
#pragma unroll
      for (int q = 0; q < kP; ++q)
        if (in_bounds(p.status, s_unit + q * N, p.n_state)) p.hT[s_unit + q * N] = S[q];
    }
  } else if (warp < 16) {
    // =========================== xs and the outputs: thread = token lt ===========================================
    const int64_t y_at = b * p.o_sb + h * p.o_sh + slice * kP;
    __nv_bfloat16* gy = reinterpret_cast<__nv_bfloat16*>(p.o) + y_at;
    const float D_h = p.D[h];
    auto x_tile = [&](int it) { return smem + L::kX + (it % kXs) * kPanel; };
    // Which columns of step `it` have a non-finite x, and from which token on: per column the largest bad_key of such a token (a word of
    // an earlier step is smaller than every key of this one, so nothing is reset), then one word for the whole chunk.  A stage is
    // written again three steps on, once the tile is: every thread has read it by then (x_free).
    auto bad_of = [&](int it) { return reinterpret_cast<uint32_t*>(smem + L::kBad) + (it % kXs) * kBadRow; };
    auto bad_key = [&](int it, int token) { return (uint32_t)(it + 1) * kC + (kC - 1 - token); };
    auto make_xs = [&](int it) {
      if (it == n1) boundary();
      wait_bar(ctl.scal[it % kXs], (it / kXs) & 1);
      wait_bar(ctl.fullX[it % kXs], (it / kXs) & 1);
      if (it >= 1) wait_bar(ctl.barD, (it - 1) & 1);
      const float w = scalars(it)[SC_W + lt];
      uint8_t *tile = x_tile(it), *dst = smem + L::kXt;
      __nv_bfloat162 inf = __floats2bfloat162_rn(0.f, 0.f);   // 0 x every entry: NaN if one is not finite
#pragma unroll 1
      for (int c = 0; c < 8; ++c) {
        const uint32_t at = piece_at(lt, c);
        const uint4 u = *reinterpret_cast<const uint4*>(tile + at);
        const uint32_t v[4] = {u.x, u.y, u.z, u.w};
        uint4 w1, w2, w3;
        uint32_t *a = reinterpret_cast<uint32_t*>(&w1), *bb = reinterpret_cast<uint32_t*>(&w2), *cc = reinterpret_cast<uint32_t*>(&w3);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          inf = __hfma2(*reinterpret_cast<const __nv_bfloat162*>(&v[e]), __floats2bfloat162_rn(0.f, 0.f), inf);
          mma::split3(mma::lo_f(v[e]) * w, mma::hi_f(v[e]) * w, a[e], bb[e], cc[e]);
        }
        *reinterpret_cast<uint4*>(dst + at) = w1;
        *reinterpret_cast<uint4*>(dst + kPanel + at) = w2;
        *reinterpret_cast<uint4*>(dst + 2 * kPanel + at) = w3;
      }
      if ((__hisnan(inf.x) || __hisnan(inf.y)) && it >= n1) {
#pragma unroll 1
        for (int q = 0; q < kP; ++q) {
          uint16_t* x = reinterpret_cast<uint16_t*>(tile + piece_at(lt, q >> 3)) + (q & 7);
          if ((*x & 0x7f80) == 0x7f80) {
            *x = 0;
            atomicMax(bad_of(it) + q, bad_key(it, lt));
          }
        }
        bad_of(it)[kP] = bad_key(it, kC - 1);
      }
      tc::fence_async_smem();
      arrive(ctl.xs);
      if (it < n1) arrive(ctl.x_free[it % kXs]);
    };
    auto outputs = [&](int it) {
      wait_bar(ctl.barY, (it - n1) & 1);
      tc::tc_fence_after();
      const float eg = scalars(it)[SC_EG + lt];
      uint8_t* tile = x_tile(it);
      const uint32_t* bad_at = bad_of(it);
      const bool bad = bad_at[kP] == bad_key(it, kC - 1);
#pragma unroll 1
      for (int c0 = 0; c0 < kP; c0 += 16) {
        uint32_t y1[16], y1b[16], y2[16];
        tc::tmem_ld16(tbase + TM_Y1 + lane_addr + c0, y1);
        tc::tmem_ld16(tbase + TM_Y1 + 64 + lane_addr + c0, y1b);
        tc::tmem_ld16(tbase + TM_Y2 + lane_addr + c0, y2);
        tc::tc_wait_ld();
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const uint32_t at = piece_at(lt, (c0 >> 3) + c);
          uint4 u = *reinterpret_cast<const uint4*>(tile + at);
          uint32_t* v = reinterpret_cast<uint32_t*>(&u);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int q = 8 * c + 2 * e;
            auto out = [&](int i, float x) {
              return eg * (__uint_as_float(y1[i]) + __uint_as_float(y1b[i])) + __uint_as_float(y2[i]) + D_h * x;
            };
            v[e] = mma::pack(out(q, mma::lo_f(v[e])), out(q + 1, mma::hi_f(v[e])));
          }
          if (bad) {
#pragma unroll
            for (int e = 0; e < 8; ++e)
              if (bad_at[c0 + 8 * c + e] >= bad_key(it, lt)) v[e >> 1] |= 0x7fffu << (16 * (e & 1));
          }
          *reinterpret_cast<uint4*>(tile + at) = u;
        }
      }
      tc::tc_fence_before();
      arrive(ctl.y_read);
      __syncwarp();
      const int t0 = chunk_of(it) * kC + 32 * wq + (lane >> 3);   // the warp's own 32 rows leave as whole rows
      int64_t at = (int64_t)t0 * p.o_st + 8 * (lane & 7);
#pragma unroll 2
      for (int r = 0; r < 8; ++r) {
        if (t0 + 4 * r < T && in_bounds_run(p.status, y_at + at, 8, p.n_o))
          *reinterpret_cast<uint4*>(gy + at) = *reinterpret_cast<const uint4*>(tile + piece_at(32 * wq + 4 * r + (lane >> 3), lane & 7));
        at += 4 * p.o_st;
      }
      tc::fence_async_smem();
      arrive(ctl.x_free[it % kXs]);
    };
#pragma unroll 1
    for (int it = 0; it <= steps; ++it) {   // the outputs one step behind
      if (it < steps) make_xs(it);
      if (it > n1) outputs(it - 1);
    }
    if (n1 == steps) boundary();   // no step of the second pass
  } else if (warp == 16) {
    // =========================== issue ==============================================================================
    constexpr uint32_t idG = tc::idesc_bf16(128, 128, 0, 0), idD = tc::idesc_bf16(128, 128, 1, 1), idDl = tc::idesc_bf16(128, 64, 1, 1);
    constexpr uint32_t idY = tc::idesc_bf16(128, 128, 0, 1), idYl = tc::idesc_bf16(128, 64, 0, 1);
    auto adv = [](uint64_t d, uint32_t bytes) { return d + (uint64_t)(bytes >> 4); };
    // rows along M or N, 16 columns per step of the contraction
    const uint64_t bK = tc::smem_desc_sw128(sbase + L::kB, 16, 1024), cK = tc::smem_desc_sw128(sbase + L::kCt, 16, 1024);
    // rows along the contraction, 16 per step
    const uint64_t bM = tc::smem_desc_sw128(sbase + L::kB, kPanel, 1024), xt = tc::smem_desc_sw128(sbase + L::kXt, kPanel, 1024);
    const uint64_t st = tc::smem_desc_sw128(sbase + L::kSt, kPanel, 1024);
    auto issue = [&](bool full, int it) {
      const int m = it - n1;
      wait_bar(ctl.fullB, it & 1);
      // D first if its operands are there: it fills the wait for P of the chunk before
      const bool early = !full || tc::mbar_test(tc::smem_u32(&ctl.xs), it & 1);
#pragma unroll 1
      for (int k = 0; k < 2; ++k) {
        if ((k == 0) == early) {
          wait_bar(ctl.xs, it & 1);
          if (it >= 1) wait_bar(ctl.d_read[(it - 1) % kXs], ((it - 1) / kXs) & 1);
          tc::tc_fence_after();
#pragma unroll 1
          for (int ks = 0; ks < 8; ++ks) tc::mma_ss(tbase + TM_D, adv(bM, ks * 2048), adv(xt, ks * 2048), idD, ks > 0);
          tc::mma_commit(tc::smem_u32(&ctl.barDa));
        } else if (full) {
          wait_bar(ctl.fullC, m & 1);
          if (m >= 1) wait_bar(ctl.barY, (m - 1) & 1);   // P of the chunk before has been read
          tc::tc_fence_after();
#pragma unroll 1
          for (int ks = 0; ks < N / 16; ++ks) {
            const uint32_t o = (ks >> 2) * kPanel + (ks & 3) * 32;
            tc::mma_ss(tbase + TM_G, adv(cK, o), adv(bK, o), idG, ks > 0);
          }
          tc::mma_commit(tc::smem_u32(&ctl.barG));
        }
      }
      wait_bar(ctl.barDa, it & 1);
      tc::tc_fence_after();
#pragma unroll 1
      for (int ks = 0; ks < 8; ++ks) tc::mma_ss(tbase + TM_D, adv(bM, ks * 2048), adv(xt, 2 * kPanel + ks * 2048), idDl, 1);
      tc::mma_commit(tc::smem_u32(&ctl.barD));
      if (full) {
        wait_bar(ctl.s_rdy, m & 1);
        if (m >= 1) wait_bar(ctl.y_read, (m - 1) & 1);   // Y1, Y2 of the chunk before have been read
        tc::tc_fence_after();
#pragma unroll 1
        for (int ks = 0; ks < N / 16; ++ks)
          tc::mma_ss(tbase + TM_Y1, adv(cK, (ks >> 2) * kPanel + (ks & 3) * 32), adv(st, ks * 2048), idY, ks > 0);
        tc::mma_commit(tc::smem_u32(&ctl.barY1a));
        wait_bar(ctl.barY1a, m & 1);
        tc::tc_fence_after();
#pragma unroll 1
        for (int ks = 0; ks < N / 16; ++ks)
          tc::mma_ss(tbase + TM_Y1, adv(cK, (ks >> 2) * kPanel + (ks & 3) * 32), adv(st, 2 * kPanel + ks * 2048), idYl, 1);
        tc::mma_commit(tc::smem_u32(&ctl.barY1));
        const uint64_t xd = tc::smem_desc_sw128(sbase + L::kX + (it % kXs) * kPanel, kPanel, 1024);
#pragma unroll 1
        for (int x = 0; x < 4; ++x) {   // in the order in which the two halves come
          const int part = 2 * (x & 1) + (x >> 1);
          wait_bar(ctl.p_rdy[part], m & 1);
          tc::tc_fence_after();
#pragma unroll 1
          for (int k = 0; k < 2; ++k) {
            const int ks = 2 * part + k;
            tc::mma_ts(tbase + TM_Y2, tbase + TM_G + 16 * ks, adv(xd, ks * 2048), idYl, x + k > 0);
            tc::mma_ts(tbase + TM_Y2, tbase + TM_G + 16 * ks + 8, adv(xd, ks * 2048), idYl, 1);
            tc::mma_ts(tbase + TM_Y2, tbase + TM_PL + 8 * ks, adv(xd, ks * 2048), idYl, 1);
          }
        }
        tc::mma_commit(tc::smem_u32(&ctl.barY));
      }
    };
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
      if (tc::elect_one())
#pragma unroll 1
        for (int it = pass ? n1 : 0; it < (pass ? steps : n1); ++it) issue(pass != 0, it);
      __syncwarp();
      if (pass == 0) boundary();
    }
  } else if (warp == 17) {
    // =========================== copies (one thread) ================================================================
    const int hx = h / p.v.hdiv, hb = h / p.k.hdiv, hc = h / p.q.hdiv;
    auto panels = [&](uint64_t& bar, const CUtensorMap* map, uint32_t dst, int n, int col, int head, int it) {
      const uint32_t at = tc::smem_u32(&bar);
      tc::mbar_arrive_expect_tx(at, n * kPanel);
      for (int i = 0; i < n; ++i) tc::tma_load_4d(dst + i * kPanel, map, col + 64 * i, head, chunk_of(it) * kC, b, at);
    };
    auto load_x = [&](int it) { panels(ctl.fullX[it % kXs], &P.tx, sbase + L::kX + (it % kXs) * kPanel, 1, slice * kP, hx, it); };
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
      if (tc::elect_one()) {
#pragma unroll 1
        for (int it = pass ? n1 : 0; it < (pass ? steps : n1); ++it) {
          if (it == 0) load_x(0);
          else wait_bar(ctl.barD, (it - 1) & 1);   // B has been read
          panels(ctl.fullB, &P.tb, sbase + L::kB, N / 64, 0, hb, it);
          if (it + 1 < steps) {
            if (it >= 2) wait_bar(ctl.x_free[(it + 1) % kXs], ((it - 2) / kXs) & 1);
            load_x(it + 1);
          }
          if (pass) {
            if (it > n1) wait_bar(ctl.barY1, (it - n1 - 1) & 1);   // C has been read
            panels(ctl.fullC, &P.tc, sbase + L::kCt, N / 64, 0, hc, it);
          }
        }
      }
      __syncwarp();
      if (pass == 0) boundary();
    }
  } else {
    // =========================== scalars (warps 18, 19 in turn); lane = a token of each 32 ==========================
    const int64_t dt_at = p.dt.at(b, h, 0);
    const float* gdt = reinterpret_cast<const float*>(p.dt.p) + dt_at;
    const float A_h = p.A[h], bias = p.dt_bias ? p.dt_bias[h] : 0.f;
    constexpr float kLn2 = 0.69314718f;
    bool met = false;
#pragma unroll 1
    for (int it = warp - 18; it < steps; it += 2) {
      if (it >= n1 && !met) { boundary(); met = true; }
      if (it >= kXs) {   // the stage's chunk has been used
        wait_bar(ctl.x_free[it % kXs], (it / kXs - 1) & 1);
        wait_bar(ctl.d_read[it % kXs], (it / kXs - 1) & 1);
      }
      float* sc = scalars(it);
      const int t0 = chunk_of(it) * kC + lane;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int64_t at = (int64_t)(t0 + 32 * r) * p.dt.st;
        sc[SC_DT + 32 * r + lane] = t0 + 32 * r < T && in_bounds(p.status, dt_at + at, p.dt.n) ? gdt[at] : 0.f;
      }
#pragma unroll 1
      for (int r = 0; r < 4; ++r)
        sc[SC_DT + 32 * r + lane] = t0 + 32 * r < T ? fminf(fmaxf(softplus_f(sc[SC_DT + 32 * r + lane] + bias), p.dt_lo), p.dt_hi) : 0.f;
      double a[4];   // in log2 units
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float l = A_h * sc[SC_DT + 32 * r + lane];
        a[r] = (double)(l < kDecayFloor ? kDecayFloor : l) * 1.4426950408889634;
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const double x = __shfl_up_sync(0xffffffffu, a[r], o);
          if (lane >= o) a[r] += x;
        }
      }
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        if (r) a[r] += __shfl_sync(0xffffffffu, a[r - 1], 31);
        const float hi = (float)a[r];
        sc[SC_G + 32 * r + lane] = hi;
        sc[SC_R + 32 * r + lane] = (float)(a[r] - hi);
      }
      __syncwarp();
      const float GL = sc[SC_G + kC - 1], RL = sc[SC_R + kC - 1];
#pragma unroll 1
      for (int r = 0; r < 4; ++r) {
        const int j = 32 * r + lane;
        const float G = sc[SC_G + j], R = sc[SC_R + j], d = sc[SC_DT + j];
        const float x = GL - G;   // the sums of a head run one way: what is lost here is (GL - x) - G
        sc[SC_EG + j] = exp2f(G) * (1.f + kLn2 * R);
        sc[SC_W + j] = d * exp2f(x) * (1.f + kLn2 * (((GL - x) - G) + (RL - R)));
#pragma unroll 1
        for (int q = it < n1 ? 4 : r + 1; q < 4; ++q)   // (P alone needs them)
          sc[SC_H + (q - 1) * kC + j] = d * exp2_diff(sc[SC_G + 32 * q], sc[SC_R + 32 * q], G, R);
      }
      __syncwarp();
      if (lane == 0) arrive(ctl.scal[it % kXs]);
    }
    if (!met) boundary();
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    sm100::settle(ctl.abort);
    tc::tmem_dealloc(tbase, 512);
  }
  if (tid == 0) sm100::report_wait(p.status, ctl.abort);
}

// Rows of 64 columns of 128 tokens of a [B][T][heads][cols] array (any strides), 128-byte swizzle; tokens past T arrive as zeros.
// Encoded anew for each call, 0.05 us each on the host (measured), less than looking one up by its strides would save.  What
// ssd::eligible takes can be encoded: base and strides are multiples of 16 bytes, and the strides of an array in memory stay below 2^40.
inline bool make_map(CUtensorMap* m, const LrVec& v, int cols, int B, int heads, int T) {
  sm100::EncodeTiledFn encode = sm100::encode_tiled_fn();
  if (!encode) return false;
  const cuuint64_t dims[4] = {(cuuint64_t)cols, (cuuint64_t)heads, (cuuint64_t)T, (cuuint64_t)B};
  const cuuint64_t strides[3] = {(cuuint64_t)v.sh * 2, (cuuint64_t)v.st * 2, (cuuint64_t)v.sb * 2};
  const cuuint32_t box[4] = {64, 1, kC, 1}, es[4] = {1, 1, 1, 1};
  return encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(v.p), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// How many clusters of 2, 4 and 8 CTAs run at once (B200: 74, 33, 15, as the SMs of a GPC divide), once per host thread and device.
struct ClusterFit { int dev = -1, n[4] = {0, 0, 0, 0}; };
template <int N>
inline cudaError_t cluster_fit(const ClusterFit** out) {
  thread_local ClusterFit fit;
  *out = &fit;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || fit.dev == dev) return e;
  e = cudaFuncSetAttribute(ssd_sm100_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, Smem<N>::kTotal);
  for (int i = 1; i < 4 && e == cudaSuccess; ++i) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(1u << i);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = Smem<N>::kTotal;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1u << i;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaOccupancyMaxActiveClusters(&fit.n[i], ssd_sm100_kernel<N>, &cfg);
  }
  if (e == cudaSuccess) fit.dev = dev;
  return e;
}

template <int N>
inline cudaError_t launch_n(const LinRecParams& p, cudaStream_t stream) {
  auto kern = ssd_sm100_kernel<N>;
  const ClusterFit* fit;
  const cudaError_t e = cluster_fit<N>(&fit);
  if (e != cudaSuccess) return e;
  const int64_t ctas = (int64_t)p.B * p.H * (p.V / kP);
  const int nchunks = (p.T + kC - 1) / kC;
  // Segments: a step of the first pass costs half of a full one, and every segment reads all earlier ends; clusters that do not all run
  // at once cost a second wave (N = 128, T=400 in fours: 33 CTAs 20.8 us, 34 of them 37.8; 20.8 whole).  Us at N = 128, chunks:
  //   8 CTAs    4: 19.8 whole, 19.1 in fours, 31.5 in eights   5: 23.3, 24.4, 31.6   7: 30.6, 24.5, 31.8   8: 34.1, 24.6, 31.9
  //             16: 62.3, 35.7, 37.1   20: 41.6 in fours, 42.7 in eights   22: 47.2, 42.9   32: 57.8, 48.2   (6, 28 CTAs: 28.2, 26.2)
  //   74 CTAs   4: 20.6 whole, 22.7 in pairs   7: 31.5, 34.3   8: 35.0, 34.3   9: 38.6, 40.3   12: 49.2, 46.2   16: 63.5, 58.0
  // N = 64 is up to 8 % below, with the same crossings (four chunks whole: 18.0, in fours 18.5).
  int nseg = 1;
  if (nchunks > 20 && ctas <= fit->n[3]) nseg = 8;
  else if ((nchunks == 4 || nchunks > 5) && ctas <= fit->n[2]) nseg = 4;
  else if (nchunks >= 8 && ctas <= fit->n[1]) nseg = 2;
  Params P;
  P.p = p;
  P.nseg = nseg;
  if (!make_map(&P.tb, p.k, N, p.B, p.H / p.k.hdiv, p.T) || !make_map(&P.tc, p.q, N, p.B, p.H / p.q.hdiv, p.T) ||
      !make_map(&P.tx, p.v, p.V, p.B, p.H / p.v.hdiv, p.T))
    return cudaErrorInvalidValue;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(ctas * nseg));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = Smem<N>::kTotal;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = nseg;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;   // see pdl_entry
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, kern, P);
}

// What ssd::eligible takes, but for
//  * a single 64-token chunk (8 heads, T=64: 9.6 us here, 8.5 there; 256 heads 20.7 / 16.3);
//  * half-size states in few sequences where the other form's segments, of half the chunk and less fixed cost, come out ahead while
//    they all run at once: four of them for 513 to 768 tokens (N = 64, 28 CTAs, T = 513 / 640 / 768: 22.5 / 22.8 / 25.2 here, 21.9 /
//    22.0 / 22.2 there; T = 800, 16 CTAs: 23.8 / 26.5), eight for 961 to 2560 (8 CTAs, T = 960 / 961 / 1300 / 2048 / 2560 / 2816: 23.5 /
//    23.5 / 28.7 / 34.0 / 39.3 / 41.2 here, 26.4 / 21.6 / 26.3 / 32.0 / 37.1 / 41.8 there; 16 CTAs, T = 1024: 23.9 / 38.1).
inline bool ahead(const LinRecParams& p) {
  if (p.T <= 64 || !sm100::encode_tiled_fn()) return false;
  const bool four = p.T > 512 && p.T <= 768, eight = p.T > 960 && p.T <= 2560;
  if (p.K != 64 || !(four || eight)) return true;
  const ClusterFit* fit;
  return cluster_fit<64>(&fit) != cudaSuccess || (int64_t)p.B * p.H * (p.V / kP) > fit->n[four ? 2 : 3];
}

inline cudaError_t launch(const LinRecParams& p, cudaStream_t stream) {
  return p.K == 64 ? launch_n<64>(p, stream) : launch_n<128>(p, stream);
}

}  // namespace ssdu
}  // namespace dr
