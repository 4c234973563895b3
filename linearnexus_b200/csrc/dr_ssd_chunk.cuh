// Mamba-2 SSD scan in chunk form on the warp-level tensor cores, bf16 storage, float32-exact products.  One chunk, and few
// sequences of medium length with half-size states; the rest runs on tcgen05 (dr_ssd_sm100.cuh, ssdu::ahead).
//
// With a_t = A dt_t, G the running sum of a over a 64-token chunk and S [P][N] the state at its start:
//     P_ij = (C_i . B_j) e^{G_i - G_j} dt_j   (j <= i)
//     y_i  = e^{G_i} S C_i + sum_j P_ij x_j + D x_i
//     S'   = e^{G_L} S + sum_j (dt_j e^{G_L - G_j} x_j) B_j^T
// B, C and x are bf16 as stored and enter the products exactly; the float32 operand of each product (P, S, the scaled x)
// is split into three bf16 terms (dr_mma.cuh), so the results carry float32 precision as those of the token
// recurrence do.  C B^T is one bf16 product.
//
// The recurrence multiplies decays up token by token; here they are differences of running sums, and after a strong decay (the
// selective reset: A dt of -80 a token) a float32 sum has lost the small decays of the tokens behind it.  So G is summed in
// 64 bits and kept as a float32 pair, and a difference is formed part by part: its error is that of the difference itself.  Reset of
// 32 tokens at A dt = -80, then 0.32 a token: the state is off by 2.6e-7 of its largest entry (T = 64; 1.2e-7 at T = 1100), 8.3e-5
// with float32 sums; the token recurrence by 9e-8.  B=8, T=4096, H=16, N=128:
// 319 us (334 with the scan behind the state update on a warp with three tiles of P; float32 sums there: 322).
//
// One CTA of eight warps per (batch, head, 64 value rows).  Warp w keeps S rows 16 (w & 3).. and state columns of half
// w >> 2 in accumulator registers for the whole sequence: an m16n8 accumulator of S is, register for register, the B
// operand S^T of the output product, so the state never passes through memory.  Each warp adds its half of the
// contraction to a 64 x 16 block of y; the two halves meet through shared memory.
//
// Few sequences (B H P / 64 below the SM count) leave SMs idle, so the sequence is cut into the CTAs of a cluster: every
// CTA but the last first runs the state update alone over its segment, the segments' states are combined through
// distributed shared memory (S is linear in its start: S_end = decay S_start + S_local), then each runs its segment in
// full from its true start.  That costs 1.4x the work and divides the chain by the cluster size.
//
// Infinities and NaN in x: P is 0 above the diagonal, but 0 x inf is NaN, and sixteen tokens enter one product.  Such an entry is taken
// out of the operand of P x (the state gets it), and the outputs of its column from its token on become NaN.
//
// What bounds it: 1940 mma per chunk and head (N = 128) of 8 cycles each per scheduler, 3.9 K cycles; the token
// recurrence needs 3 K V FMAs per token = 64 x 192 cycles and ran at 64 x 900.
#pragma once

#include <cooperative_groups.h>

#include "dr_linrec.cuh"
#include "dr_mma.cuh"
#include "dr_tcgen05.cuh"

namespace dr {
namespace ssd {

constexpr int kC = 64, kP = 64, kThreads = 256;
constexpr int LDX = kP + 8;    // row stride of the x, P and y tiles (bf16)
constexpr int kScanWarp = 5;       // takes dt to the scalars; one of the warps with two tiles of P (0-3 have three)
constexpr int kScalars = 5 * kC;   // per-token scalars of a stage
// A token's log decay is cut off here: what crosses the token is 0 in float32 either way (the decays of a head have one sign),
// and the sums stay finite and within the pair's 48 bits.
constexpr float kDecayFloor = -200.f;

template <int N>
struct Smem {
  static constexpr int LDN = N + 8;
  static constexpr int kB = 0;                              // two stages of: B [64][LDN], C [64][LDN], x [64][LDX] bf16
  static constexpr int kTileN = kC * LDN * 2, kTileX = kC * LDX * 2;
  static constexpr int kStage = 2 * kTileN + kTileX;
  static constexpr int kPm = kB + 2 * kStage;               // P, three bf16 terms [3][64][LDX]
  static constexpr int kY = kPm + 3 * kTileX;               // partial y fp32 [64][68]; then the bf16 rows [64][LDX]
  static constexpr int kSt = kY + kC * 68 * 4;              // this segment's end state fp32 [64][N] (clusters)
  static constexpr int kSc = kSt + kP * N * 4;              // per stage: G[64], e^G[64], dt[64], dt e^{G_L - G}[64], rest of G[64]
  static constexpr int kDec = kSc + 2 * kScalars * 4;       // this segment's decay
  static constexpr int kBad = kDec + 16;                     // see bad_key; one word per value column, one for the whole chunk
  static constexpr int kTotal = kBad + (kP + 4) * 4;
};

template <int N>
__global__ void __launch_bounds__(kThreads, 1) ssd_chunk_kernel(const LinRecParams p, const int nseg) {
  pdl_entry();
  using L = Smem<N>;
  constexpr int LDN = L::LDN, NT = N / 16, KS = N / 32;   // state tiles (8 columns) per warp, 16-column k-steps per warp
  extern __shared__ __align__(16) uint8_t smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int pw = warp & 3, nh = warp >> 2;   // 16 value rows, half of the state columns
  const int p0 = 16 * pw, n0 = nh * (N / 2);
  const int seg = blockIdx.x % nseg;
  const int slices = p.V / kP, unit = blockIdx.x / nseg / slices, slice = blockIdx.x / nseg % slices;
  const int b = unit / p.H, h = unit % p.H, T = p.T;
  const int nchunks = (T + kC - 1) / kC, per = (nchunks + nseg - 1) / nseg;
  const int c_lo = min(seg * per, nchunks), c_hi = min(c_lo + per, nchunks);
  const int64_t c_at = p.q.at(b, h, 0), b_at = p.k.at(b, h, 0), x_at = p.v.at(b, h, 0) + slice * kP, dt_at = p.dt.at(b, h, 0);
  const int64_t y_at = b * p.o_sb + h * p.o_sh + slice * kP;
  const __nv_bfloat16* gC = reinterpret_cast<const __nv_bfloat16*>(p.q.p) + c_at;
  const __nv_bfloat16* gB = reinterpret_cast<const __nv_bfloat16*>(p.k.p) + b_at;
  const __nv_bfloat16* gx = reinterpret_cast<const __nv_bfloat16*>(p.v.p) + x_at;
  __nv_bfloat16* gy = reinterpret_cast<__nv_bfloat16*>(p.o) + y_at;
  const float* gdt = reinterpret_cast<const float*>(p.dt.p) + dt_at;
  const float A_h = p.A[h], D_h = p.D[h], bias_h = p.dt_bias ? p.dt_bias[h] : 0.f;
  const uint32_t sbase = tc::smem_u32(smem);

  // state tile nt: rows p0 + g, p0 + g + 8, columns n0 + 8 nt + 2t, + 1; stored [P][N] per unit
  float S[NT][4];
  const int64_t s_unit = ((int64_t)unit * p.V + slice * kP + p0 + g) * N + n0 + 2 * t;
  auto zero_state = [&]() {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) S[nt][0] = S[nt][1] = S[nt][2] = S[nt][3] = 0.f;
  };
  zero_state();
  auto load_h0 = [&]() {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      if (!in_bounds_run(p.status, s_unit + 8 * nt, 2, p.n_state) || !in_bounds_run(p.status, s_unit + 8 * N + 8 * nt, 2, p.n_state)) continue;
      const float2 lo = *reinterpret_cast<const float2*>(p.h0 + s_unit + 8 * nt);
      const float2 hi = *reinterpret_cast<const float2*>(p.h0 + s_unit + 8 * N + 8 * nt);
      S[nt][0] = lo.x; S[nt][1] = lo.y; S[nt][2] = hi.x; S[nt][3] = hi.y;
    }
  };
  if (p.h0 && seg == 0) load_h0();

  auto tile_B = [&](int st) { return sbase + L::kB + st * L::kStage; };
  auto tile_C = [&](int st) { return sbase + L::kB + st * L::kStage + L::kTileN; };
  auto tile_X = [&](int st) { return sbase + L::kB + st * L::kStage + 2 * L::kTileN; };
  auto scalars = [&](int st) { return reinterpret_cast<float*>(smem + L::kSc) + st * kScalars; };
  // rows of chunk c -> stage st by 16-byte asynchronous copies; rows past the end become zeros
  auto issue = [&](int c, int st, bool full) {
    const int t0 = c * kC, rows = min(kC, T - t0);
#pragma unroll
    for (int i = tid; i < kC * (N / 8); i += kThreads) {
      const int r = i / (N / 8), q = (i % (N / 8)) * 8;
      const int64_t row = t0 + (r < rows ? r : 0);
      tc::cp_async16(tile_B(st) + 2u * (r * LDN + q), gB + row * p.k.st + q,
                     r < rows && in_bounds_run(p.status, b_at + row * p.k.st + q, 8, p.k.n));
      if (full) tc::cp_async16(tile_C(st) + 2u * (r * LDN + q), gC + row * p.q.st + q,
                               r < rows && in_bounds_run(p.status, c_at + row * p.q.st + q, 8, p.q.n));
    }
#pragma unroll
    for (int i = tid; i < kC * (kP / 8); i += kThreads) {
      const int r = i / (kP / 8), q = (i % (kP / 8)) * 8;
      const int64_t at = (int64_t)(t0 + (r < rows ? r : 0)) * p.v.st + q;
      tc::cp_async16(tile_X(st) + 2u * (r * LDX + q), gx + at, r < rows && in_bounds_run(p.status, x_at + at, 8, p.v.n));
    }
    tc::cp_async_commit();
  };
  // dt of the next chunk (one warp, two tokens per lane), then its scan: G, e^G, dt, dt e^{G_L - G}
  float dt_lo = 0.f, dt_hi = 0.f;
  auto fetch_dt = [&](int c) {
    if (warp == kScanWarp) {
      const int t0 = c * kC + lane;
      const int64_t at = (int64_t)t0 * p.dt.st, at32 = (int64_t)(t0 + 32) * p.dt.st;
      dt_lo = t0 < T && in_bounds(p.status, dt_at + at, p.dt.n) ? gdt[at] : 0.f;
      dt_hi = t0 + 32 < T && in_bounds(p.status, dt_at + at32, p.dt.n) ? gdt[at32] : 0.f;
    }
  };
  auto scan_dt = [&](int c, int st) {
    if (warp == kScanWarp) {
      const int t0 = c * kC + lane;
      float* sc = scalars(st);
      const float d0 = t0 < T ? fminf(fmaxf(softplus_f(dt_lo + bias_h), p.dt_lo), p.dt_hi) : 0.f;
      const float d1 = t0 + 32 < T ? fminf(fmaxf(softplus_f(dt_hi + bias_h), p.dt_lo), p.dt_hi) : 0.f;
      auto log_decay = [&](float d) -> double {
        const float a = A_h * d;
        return a < kDecayFloor ? kDecayFloor : a;
      };
      double a0 = log_decay(d0), a1 = log_decay(d1);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double x = __shfl_up_sync(0xffffffffu, a0, o), y = __shfl_up_sync(0xffffffffu, a1, o);
        if (lane >= o) { a0 += x; a1 += y; }
      }
      a1 += __shfl_sync(0xffffffffu, a0, 31);
      const double last = __shfl_sync(0xffffffffu, a1, 31);
      const float g0 = (float)a0, g1 = (float)a1;
      sc[lane] = g0; sc[32 + lane] = g1;
      sc[64 + lane] = expf(g0); sc[96 + lane] = expf(g1);
      sc[128 + lane] = d0; sc[160 + lane] = d1;
      sc[192 + lane] = d0 * expf((float)(last - a0)); sc[224 + lane] = d1 * expf((float)(last - a1));
      sc[256 + lane] = (float)(a0 - g0); sc[288 + lane] = (float)(a1 - g1);
    }
  };

  // S' = e^{G_L} S + (scaled x)^T B
  auto state_update = [&](int st) {
    const float* sc = scalars(st);
    const float dec = sc[64 + 63];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) { S[nt][0] *= dec; S[nt][1] *= dec; S[nt][2] *= dec; S[nt][3] *= dec; }
#pragma unroll
    for (int kt = 0; kt < 4; ++kt) {
      uint32_t xr[4], a1[4], a2[4], a3[4];
      mma::ldsm4t(xr, mma::frag_at(tile_X(st), LDX, 16 * kt, p0, lane));
      const float2 s0 = *reinterpret_cast<const float2*>(sc + 192 + 16 * kt + 2 * t);
      const float2 s1 = *reinterpret_cast<const float2*>(sc + 192 + 16 * kt + 8 + 2 * t);
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const float2 s = r < 2 ? s0 : s1;
        mma::split3(mma::lo_f(xr[r]) * s.x, mma::hi_f(xr[r]) * s.y, a1[r], a2[r], a3[r]);
      }
#pragma unroll
      for (int n2 = 0; n2 < NT / 2; ++n2) {
        uint32_t br[4];
        mma::ldsm4t(br, mma::frag_bt(tile_B(st), LDN, 16 * kt, n0 + 16 * n2, lane));
        mma::bf16(S[2 * n2], a1, br[0], br[1]);
        mma::bf16(S[2 * n2 + 1], a1, br[2], br[3]);
        mma::bf16(S[2 * n2], a2, br[0], br[1]);
        mma::bf16(S[2 * n2 + 1], a2, br[2], br[3]);
        mma::bf16(S[2 * n2], a3, br[0], br[1]);
        mma::bf16(S[2 * n2 + 1], a3, br[2], br[3]);
      }
    }
  };

  if (nseg > 1) {
    // ---- the segment's own contribution to the state, and its decay ------------------------------------------------
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    float* seg_decay = reinterpret_cast<float*>(smem + L::kDec);
    float dec = 1.f;
    if (seg + 1 < nseg && c_lo < c_hi) {
      issue(c_lo, 0, false);
      fetch_dt(c_lo);
      scan_dt(c_lo, 0);
      for (int c = c_lo; c < c_hi; ++c) {
        const int st = (c - c_lo) & 1;
        tc::cp_async_wait_all();
        __syncthreads();
        if (c + 1 < c_hi) { issue(c + 1, st ^ 1, false); fetch_dt(c + 1); }
        state_update(st);
        dec *= scalars(st)[64 + 63];
        if (c + 1 < c_hi) scan_dt(c + 1, st ^ 1);
      }
    }
    float* own = reinterpret_cast<float*>(smem + L::kSt);
    const int at = (p0 + g) * N + n0 + 2 * t;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      *reinterpret_cast<float2*>(own + at + 8 * nt) = make_float2(S[nt][0], S[nt][1]);
      *reinterpret_cast<float2*>(own + at + 8 * N + 8 * nt) = make_float2(S[nt][2], S[nt][3]);
    }
    if (tid == 0) *seg_decay = dec;
    cluster.sync();
    // ---- this segment's start: the earlier segments' ends, decayed ----------------------------------------------------
    if (seg > 0) {
      zero_state();
      for (int s = 0; s < seg; ++s) {
        const float* other = cluster.map_shared_rank(own, s);
        const float d = *cluster.map_shared_rank(seg_decay, s);
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) {
          const float2 lo = *reinterpret_cast<const float2*>(other + at + 8 * nt);
          const float2 hi = *reinterpret_cast<const float2*>(other + at + 8 * N + 8 * nt);
          S[nt][0] = S[nt][0] * d + lo.x; S[nt][1] = S[nt][1] * d + lo.y;
          S[nt][2] = S[nt][2] * d + hi.x; S[nt][3] = S[nt][3] * d + hi.y;
        }
      }
    } else {
      zero_state();
      if (p.h0) load_h0();
    }
    cluster.sync();   // the others have read this CTA's copy (and p.hT may alias p.h0)
  }

  // Non-finite x of a chunk: per column the largest bad_key of such a token.  A word of an earlier chunk is smaller than every key of
  // this one; words are written behind the barrier at "P is complete" and read behind the next.
  uint32_t* sBad = reinterpret_cast<uint32_t*>(smem + L::kBad);
  auto bad_key = [&](int c, int token) { return (uint32_t)(c + 1) * kC + (kC - 1 - token); };
  if (tid <= kP) sBad[tid] = 0u;   // (the first barrier of the loop lies before the first use)

  const uint32_t sPm = sbase + L::kPm;
  float* sY = reinterpret_cast<float*>(smem + L::kY);
  __nv_bfloat16* sYo = reinterpret_cast<__nv_bfloat16*>(smem + L::kPm);   // output rows: the P tiles are dead by then
  if (c_lo < c_hi) {
    issue(c_lo, 0, true);
    fetch_dt(c_lo);
    scan_dt(c_lo, 0);
  }
  for (int c = c_lo; c < c_hi; ++c) {
    const int st = (c - c_lo) & 1, t0 = c * kC;
    const float* sc = scalars(st);
    tc::cp_async_wait_all();
    __syncthreads();
    if (c + 1 < c_hi) { issue(c + 1, st ^ 1, true); fetch_dt(c + 1); }
    // ---- P = tril(C B^T e^{G_i - G_j} dt_j), 20 tiles of 16 x 8 at or below the diagonal dealt to the warps ---------
#pragma unroll 1
    for (int tile = warp; tile < 20; tile += 8) {
      const int mt = tile < 2 ? 0 : tile < 6 ? 1 : tile < 12 ? 2 : 3;
      const int nt = tile - mt * (mt + 1);
      float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int k2 = 0; k2 < N / 32; ++k2) {   // two k-steps: one ldmatrix for both B fragments
        uint32_t a0[4], a1[4], bb[4];
        mma::ldsm4(a0, mma::frag_a(tile_C(st), LDN, 16 * mt, 32 * k2, lane));
        mma::ldsm4(a1, mma::frag_a(tile_C(st), LDN, 16 * mt, 32 * k2 + 16, lane));
        mma::ldsm4(bb, tile_B(st) + 2u * ((8 * nt + (lane & 7)) * LDN + 32 * k2 + (lane >> 3) * 8));
        mma::bf16(d, a0, bb[0], bb[1]);
        mma::bf16(d, a1, bb[2], bb[3]);
      }
      const int j = 8 * nt + 2 * t;
      const float2 Gj = *reinterpret_cast<const float2*>(sc + j), dj = *reinterpret_cast<const float2*>(sc + 128 + j);
      const float2 rj = *reinterpret_cast<const float2*>(sc + 256 + j);
#pragma unroll
      for (int hr = 0; hr < 2; ++hr) {
        const int i = 16 * mt + g + 8 * hr;
        const float Gi = sc[i], ri = sc[256 + i];
        const float x = j <= i ? d[2 * hr] * (expf((Gi - Gj.x) + (ri - rj.x)) * dj.x) : 0.f;
        const float y = j + 1 <= i ? d[2 * hr + 1] * (expf((Gi - Gj.y) + (ri - rj.y)) * dj.y) : 0.f;
        uint32_t w1, w2, w3;
        mma::split3(x, y, w1, w2, w3);
        uint8_t* dst = smem + L::kPm + 2 * (i * LDX + j);
        *reinterpret_cast<uint32_t*>(dst) = w1;
        *reinterpret_cast<uint32_t*>(dst + L::kTileX) = w2;
        *reinterpret_cast<uint32_t*>(dst + 2 * L::kTileX) = w3;
      }
    }
    // ---- y: e^{G_i} S C_i over this warp's state columns -----------------------------------------------------------
    float y[4][2][4];
#pragma unroll
    for (int mt = 0; mt < 4; ++mt)
#pragma unroll
      for (int n2 = 0; n2 < 2; ++n2) y[mt][n2][0] = y[mt][n2][1] = y[mt][n2][2] = y[mt][n2][3] = 0.f;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      uint32_t b1[2][2], b2[2][2], b3[2][2];   // [value rows g / g + 8][k half]
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int kh = 0; kh < 2; ++kh)
          mma::split3(S[2 * ks + kh][2 * r], S[2 * ks + kh][2 * r + 1], b1[r][kh], b2[r][kh], b3[r][kh]);
#pragma unroll
      for (int mt = 0; mt < 4; ++mt) {
        uint32_t a[4];
        mma::ldsm4(a, mma::frag_a(tile_C(st), LDN, 16 * mt, n0 + 16 * ks, lane));
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          mma::bf16(y[mt][r], a, b1[r][0], b1[r][1]);
          mma::bf16(y[mt][r], a, b2[r][0], b2[r][1]);
          mma::bf16(y[mt][r], a, b3[r][0], b3[r][1]);
        }
      }
    }
#pragma unroll
    for (int mt = 0; mt < 4; ++mt) {
      const float e0 = sc[64 + 16 * mt + g], e1 = sc[64 + 16 * mt + g + 8];
#pragma unroll
      for (int r = 0; r < 2; ++r) { y[mt][r][0] *= e0; y[mt][r][1] *= e0; y[mt][r][2] *= e1; y[mt][r][3] *= e1; }
    }
    if (c + 1 < c_hi) scan_dt(c + 1, st ^ 1);   // (the last reader of that stage's scalars was the previous chunk's state update)
    __syncthreads();   // P is complete
    // ---- + P x: the 16-token blocks 0 and 3 by one half of the warps, 1 and 2 by the other (five products each) --------
#pragma unroll
    for (int kk = 0; kk < 2; ++kk) {
      const int kt = nh ? 1 + kk : 3 * kk;
      uint32_t xb[4];
      mma::ldsm4t(xb, mma::frag_bt(tile_X(st), LDX, 16 * kt, p0, lane));
      __nv_bfloat162 inf = __floats2bfloat162_rn(0.f, 0.f);   // 0 x every entry: NaN if one is not finite
#pragma unroll
      for (int r = 0; r < 4; ++r) inf = __hfma2(*reinterpret_cast<const __nv_bfloat162*>(&xb[r]), __floats2bfloat162_rn(0.f, 0.f), inf);
      if (__hisnan(inf.x) || __hisnan(inf.y)) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {   // entry: token 16 kt + 2t + (e & 1) + 8 (e >> 1 & 1), column p0 + g + 8 (e >> 2)
          const uint32_t half = (e & 1) ? 0xffff0000u : 0xffffu, exp = half & 0x7f807f80u;
          if ((xb[e >> 1] & exp) == exp) {
            xb[e >> 1] &= ~half;
            atomicMax(sBad + p0 + g + 8 * (e >> 2), bad_key(c, 16 * kt + 2 * t + (e & 1) + 8 * ((e >> 1) & 1)));
          }
        }
        sBad[kP] = bad_key(c, kC - 1);
      }
      __syncwarp();
#pragma unroll
      for (int mt = 0; mt < 4; ++mt) {
        if (mt >= kt) {
#pragma unroll
          for (int s = 0; s < 3; ++s) {
            uint32_t a[4];
            mma::ldsm4(a, mma::frag_a(sPm + s * L::kTileX, LDX, 16 * mt, 16 * kt, lane));
            mma::bf16(y[mt][0], a, xb[0], xb[1]);
            mma::bf16(y[mt][1], a, xb[2], xb[3]);
          }
        }
      }
    }
    // ---- the halves meet: this warp finishes 32 of the 64 tokens ----------------------------------------------------
#pragma unroll
    for (int m = 0; m < 2; ++m) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int mt = nh ? m : 2 + m;   // the other half's tokens
        float* dst = sY + (16 * mt + g) * 68 + p0 + 8 * r + 2 * t;
        const float (&v)[4] = nh ? y[m][r] : y[2 + m][r];
        *reinterpret_cast<float2*>(dst) = make_float2(v[0], v[1]);
        *reinterpret_cast<float2*>(dst + 8 * 68) = make_float2(v[2], v[3]);
      }
    }
    __syncthreads();   // partials written; every warp is done with P
    const bool bad = sBad[kP] == bad_key(c, kC - 1);
#pragma unroll
    for (int m = 0; m < 2; ++m) {
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int mt = nh ? 2 + m : m;
        const float (&v)[4] = nh ? y[2 + m][r] : y[m][r];
#pragma unroll
        for (int hr = 0; hr < 2; ++hr) {
          const int i = 16 * mt + g + 8 * hr, cc = p0 + 8 * r + 2 * t;
          const float2 o = *reinterpret_cast<const float2*>(sY + i * 68 + cc);
          const uint32_t xx = *reinterpret_cast<const uint32_t*>(smem + L::kB + st * L::kStage + 2 * L::kTileN + 2 * (i * LDX + cc));
          uint32_t out = mma::pack(v[2 * hr] + o.x + D_h * mma::lo_f(xx), v[2 * hr + 1] + o.y + D_h * mma::hi_f(xx));
          if (bad) out |= (sBad[cc] >= bad_key(c, i) ? 0x7fffu : 0u) | (sBad[cc + 1] >= bad_key(c, i) ? 0x7fff0000u : 0u);
          *reinterpret_cast<uint32_t*>(sYo + i * LDX + cc) = out;
        }
      }
    }
    state_update(st);
    __syncthreads();   // the output rows are complete
#pragma unroll
    for (int i = tid; i < kC * (kP / 8); i += kThreads) {
      const int r = i / (kP / 8), q = (i % (kP / 8)) * 8;
      if (t0 + r < T && in_bounds_run(p.status, y_at + (int64_t)(t0 + r) * p.o_st + q, 8, p.n_o))
        *reinterpret_cast<uint4*>(gy + (int64_t)(t0 + r) * p.o_st + q) = *reinterpret_cast<const uint4*>(sYo + r * LDX + q);
    }
  }
  if (p.hT && seg == nseg - 1) {
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      if (!in_bounds_run(p.status, s_unit + 8 * nt, 2, p.n_state) || !in_bounds_run(p.status, s_unit + 8 * N + 8 * nt, 2, p.n_state)) continue;
      *reinterpret_cast<float2*>(p.hT + s_unit + 8 * nt) = make_float2(S[nt][0], S[nt][1]);
      *reinterpret_cast<float2*>(p.hT + s_unit + 8 * N + 8 * nt) = make_float2(S[nt][2], S[nt][3]);
    }
  }
}

// bf16 rows that 16-byte copies can read, whole 64-row value slices, a state that fits the warps' registers; and at
// least half a chunk of tokens (a decode step is a handful of FMAs per state entry).
inline bool eligible(const LinRecParams& p) {
  auto ok = [](const LrVec& v) { return (reinterpret_cast<uintptr_t>(v.p) & 15) == 0 && v.sb % 8 == 0 && v.sh % 8 == 0 && v.st % 8 == 0; };
  return (p.K == 64 || p.K == 128) && p.V % kP == 0 && p.T >= 32 && ok(p.q) && ok(p.k) && ok(p.v) &&
         (reinterpret_cast<uintptr_t>(p.o) & 15) == 0 && p.o_sb % 8 == 0 && p.o_sh % 8 == 0 && p.o_st % 8 == 0 &&
         (!p.h0 || (reinterpret_cast<uintptr_t>(p.h0) & 15) == 0) && (!p.hT || (reinterpret_cast<uintptr_t>(p.hT) & 15) == 0);
}

template <int N>
inline cudaError_t launch_n(const LinRecParams& p, int sms, cudaStream_t stream) {
  auto kern = ssd_chunk_kernel<N>;
  thread_local int attr_dev = -1;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (attr_dev != dev) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Smem<N>::kTotal);
    if (e != cudaSuccess) return e;
    attr_dev = dev;
  }
  const int64_t ctas = (int64_t)p.B * p.H * (p.V / kP);
  const int nchunks = (p.T + kC - 1) / kC;
  // segments: as many as fit one wave (a segmented run costs 1.4x the work), two chunks each at least
  int nseg = 1;
  while (nseg < 8 && ctas * nseg * 2 <= sms && nchunks >= 4 * nseg) nseg *= 2;
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
  return cudaLaunchKernelEx(&cfg, kern, p, nseg);
}

inline cudaError_t launch(const LinRecParams& p, int sms, cudaStream_t stream) {
  return p.K == 64 ? launch_n<64>(p, sms, stream) : launch_n<128>(p, sms, stream);
}

}  // namespace ssd
}  // namespace dr
