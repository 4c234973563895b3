// The chunk-parallel part of the backward for scalar decays (DeltaNet, Gated DeltaNet) on tcgen05: every gradient of a chunk from its
// state S0, the state gradient dS1 behind it and its inputs.  Formulas and names: header of dr_bwd.cuh; the kernels around it:
// dr_bwd_chunk.cuh.
//
// All products have M = 128 (value or key channels, or [dO; dR] rows) and tokens as N, so that a thread of an epilogue owns one
// channel and sixteen tokens.  float32 operands are two bf16 terms each (16 bits); K, Q, dO are bf16 and exact:
//   1  KS^T = S0^T K^T,  KD^T = dS1^T K^T,  AO^T = dO^T A,  dQ1^T = S0 dO^T
//   2  Vn^T = R^T T^T,   dR^T = dVn^T T         R = beta (V - e^G rk KS),  dVn = e^{G_L - G} rk KD + AO   (terms in tensor memory)
//   3  [dA; dM] = [dO; dR] Vn^T,  dKr1^T = S0 dR^T,  dKc1^T = dS1 Vn^T
//   4  dQ2^T = K^T P^T,  dKr2^T = K^T Px^T,  dKc2^T = Q^T P + K^T Px      P = rq rk dA.E, Px = rk rk dX.E, so that K, Q stay as they are
// Triangular operands are taken by 16-token blocks, N = the columns that a block reaches.
//
// One persistent CTA per SM: sixteen warps that split and finish, one that issues.  The states, 128 KB of the 220 KB a chunk reads, arrive
// by bulk copies during the end of the chunk before, as soon as its last product with them is done, and are split where they lie; the
// other operands follow at its end (asked for in L2 a chunk ahead).  Outputs leave by TMA from tiles that are no longer needed.  Only
// three sums over the channels of a token are formed: k^ . (dX.E) K^ is the sum of dX . X, which the rows of dX have at hand.
//
// What bounds it: B=2, T=4096, H=16 (2048 chunks, 14 per CTA): 25 K cycles per chunk, 59 K as tf32 products on mma.sync with one CTA per chunk
// (450 us -> 200, the training step 779 -> 548).  Of them 6 K are waits for products and copies, the rest the element-wise work between the
// products, 2.4 K instructions per warp at four warps per scheduler (issue slots 35 %); the products take 6.5 K, 1.2 K before and
// after hidden behind it, the memory's share is 11.7 K at the copy rate.  Without the bulk copies a chunk ahead, with the operands by
// 2-byte loads: 51 K.  Two terms have 16 bits where one tf32 product had 11: errors of dbeta, dg against float64 at one chunk
// 1.1e-3, 1.2e-3 -> 5.5e-5, 4.0e-5 (over many chunks the forward's checkpoints decide), of dq, dk 2.2e-3 -> 1.7e-3 (bf16 rounding).
#pragma once

namespace dr {
namespace bwdc {

constexpr int kLtThreads = 544, kLtWorkers = 512;
constexpr int kTile = 64 * 128 * 2;   // 64 tokens x 128 channels, bf16
// S0 and dS1 (fp32 rows as they arrive, then per 8 channels the core matrices of the high and of the low terms); K (128-byte swizzle);
// dO^T, dR^T hi, lo (before: dO and V as they arrive); A hi, lo, T hi, lo, then Vn^T hi, lo
constexpr int LT_S = 0, LT_D = LT_S + 65536, LT_K = LT_D + 65536, LT_O = LT_K + kTile, LT_N = LT_O + 3 * kTile, LT_CTL = LT_N + 32768;
// once the products with dR and Vn are done: P hi, lo, Px hi, lo, Q over dO, dR, later dq, dk; dv and sums over Vn
constexpr int LT_P = LT_O, LT_Q = LT_O + 2 * kTile, LT_SUM = LT_N + kTile;
struct LtSums {
  float row[3][4][64];            // per quarter of the channels: q^ . dq^, k^ . dkc, beta's part of k^ . dkr
  float x[4][64], v[4][64];       // dM . X per quarter of the columns, dR . V per quarter of the channels
  float f[16][32];                // per warp: the chain rule's factors of its tokens, q and k
  float ex[16], ts[16];
};
static_assert(sizeof(LtSums) <= kTile, "behind dv");
struct LtCtl {
  uint64_t bar[6], full_s, full_d, full_i, full_q;
  float beta[64], rk[64], rq[64], ik[64], cq[64], ck[64], G[64], eg[64], wd[64];   // norm factors, 1 / rk, r / (s |x|); G, e^G, e^{G_L - G}
  uint32_t tmem_base;
  int abort;
};
constexpr int LT_TOTAL = LT_CTL + sizeof(LtCtl);
static_assert(LT_TOTAL <= 232448, "shared memory");
struct alignas(64) LocalParams {
  CUtensorMap tq, tk, tv, to, tdq, tdk, tdv;   // panels of 64 columns (see sm100::make_panel_map)
  CUtensorMap tg;   // per-channel decays: boxes of 64 rows
  Params p;
  int chunks;
  int32_t* status;
  int64_t n_tok, n_part;   // entries of the arrays with one number per token, of dq^ and dk^ per head (index checks of the debug build)
};
static __global__ void __launch_bounds__(kLtThreads, 1) local_sm100_kernel(const __grid_constant__ LocalParams P) {
  const Params& p = P.p;
  extern __shared__ __align__(1024) uint8_t lt_smem[];
  uint8_t* const smem = lt_smem;
  LtCtl& ctl = *reinterpret_cast<LtCtl*>(smem + LT_CTL);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  if (warp == 16) {
    tc::tmem_alloc(tc::smem_u32(&ctl.tmem_base), 512);
    tc::tmem_relinquish();
  }
  if (tid == 0) {
    for (int i = 0; i < 6; ++i) tc::mbar_init(tc::smem_u32(&ctl.bar[i]), 1);
    tc::mbar_init(tc::smem_u32(&ctl.full_s), 1);
    tc::mbar_init(tc::smem_u32(&ctl.full_d), 1);
    tc::mbar_init(tc::smem_u32(&ctl.full_i), 1);
    tc::mbar_init(tc::smem_u32(&ctl.full_q), 1);
    tc::fence_mbar_init();
    ctl.abort = 0;
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  pdl_entry();
  const uint32_t tb = ctl.tmem_base, sb = tc::smem_u32(smem);
  auto wait_at = [&](uint64_t& bar, uint32_t parity) {
    const uint32_t at = tc::smem_u32(&bar);
    sm100::wait_inline(at, parity, &ctl.abort, at - tc::smem_u32(&ctl), warp == 16);
  };
  auto wait_bar = [&](int i, uint32_t parity) { wait_at(ctl.bar[i], parity); };
  LtSums& sum = *reinterpret_cast<LtSums*>(smem + LT_SUM);
  auto total = [](const float (&a)[4][64], int i) { return (a[0][i] + a[1][i]) + (a[2][i] + a[3][i]); };
  // tensor memory: columns of the accumulators and of the two terms of R^T, dVn^T
  constexpr uint32_t tKS = 0, tKD = 64, tAO = 128, tQ1 = 192, tR = 256, tV = 320, tVn = 384, tdR = 448;
  constexpr uint32_t tKr1 = 0, tKc1 = 64, tA = 128, tM = 256, tQ2 = 128, tKr2 = 256, tKc2 = 320;

  if (warp == 16) {
    auto adv = [](uint64_t d, uint32_t bytes) { return d + (uint64_t)(bytes >> 4); };
    auto commit = [&](int i) { tc::mma_commit(tc::smem_u32(&ctl.bar[i])); };
    auto in = [&](int64_t i) { return in_bounds(P.status, i, P.n_tok); };
    struct At { int b, h, hq, t0; };
    auto place = [&](int c) {
      const int unit = c / p.N, b = unit / p.map.H, h = unit % p.map.H;
      return At{b, h, p.map.hq(h), (c % p.N) * kC};
    };
    auto load_panels = [&](const CUtensorMap& m, uint32_t dst, int h, const At& x, uint64_t& bar) {
      tc::tma_load_4d(sb + dst, &m, 0, h, x.t0, x.b, tc::smem_u32(&bar));
      tc::tma_load_4d(sb + dst + 8192, &m, 64, h, x.t0, x.b, tc::smem_u32(&bar));
    };
    auto load_state = [&](uint64_t& bar, uint32_t dst, const float* src) {
      tc::mbar_arrive_expect_tx(tc::smem_u32(&bar), 65536);
      tc::bulk_g2s(sb + dst, src, 65536, tc::smem_u32(&bar));
    };
    // K, V, the tiles of A and T; then dO
    auto load_inputs = [&](int c) {
      const At x = place(c);
      tc::mbar_arrive_expect_tx(tc::smem_u32(&ctl.full_i), 3 * kTile + 32768);
      load_panels(P.tk, LT_K, x.hq, x, ctl.full_i);
      load_panels(P.tv, LT_O + 2 * kTile, x.h, x, ctl.full_i);
      tc::bulk_g2s(sb + LT_N, p.xat + (int64_t)c * (3 * 64 * 64) + 4096, 32768, tc::smem_u32(&ctl.full_i));
    };
    auto load_do = [&](int c) {
      const At x = place(c);
      load_panels(P.to, LT_O + kTile, x.h, x, ctl.full_i);
    };
    // the token vectors of a chunk, lane = token and token + 32
    float g_lo = 0.f, g_hi = 0.f, b0 = 0.f, b1 = 0.f, k0 = 0.f, k1 = 0.f, q0 = 0.f, q1 = 0.f;
    auto load_vectors = [&](int c) {
      const At x = place(c);
      const int rows = min(kC, p.map.T - x.t0);
      const int64_t at = p.map.base(x.b, x.h, 1) + (int64_t)x.t0 * p.map.tok(1), tok = p.map.tok(1);
      g_lo = g_hi = b0 = b1 = 0.f;
      if (p.variant == DR_GATED) {
        if (lane < rows && in(at + lane * tok)) g_lo = ld_elem(p.g, at + lane * tok, p.g_dt);
        if (lane + 32 < rows && in(at + (lane + 32) * tok)) g_hi = ld_elem(p.g, at + (lane + 32) * tok, p.g_dt);
      }
      if (lane < rows && in(at + lane * tok)) b0 = p.beta[at + lane * tok];
      if (lane + 32 < rows && in(at + (lane + 32) * tok)) b1 = p.beta[at + (lane + 32) * tok];
      const float* nrm = p.norms + (int64_t)c * 128;
      k0 = nrm[lane]; k1 = nrm[lane + 32]; q0 = nrm[lane + 64]; q1 = nrm[lane + 96];
    };
    const int first = blockIdx.x;
    if (tc::elect_one()) {
      load_state(ctl.full_s, LT_S, p.ckpt + (int64_t)first * (kD * kD));
      load_inputs(first);
      load_do(first);
      load_state(ctl.full_d, LT_D, p.ds + (int64_t)first * (kD * kD));
    }
    __syncwarp();
    load_vectors(first);
    uint32_t ph = 0;
#pragma unroll 1
    for (int c = first; c < P.chunks; c += gridDim.x, ph ^= 1) {
      const int next = c + gridDim.x;
      {
        mma::scan_scalars(g_lo, g_hi, lane);
        const float gl = __shfl_sync(0xffffffffu, g_hi, 31);
        ctl.beta[lane] = b0; ctl.beta[lane + 32] = b1;
        ctl.rk[lane] = k0; ctl.rk[lane + 32] = k1;
        ctl.rq[lane] = q0; ctl.rq[lane + 32] = q1;
        ctl.ik[lane] = k0 != 0.f ? 1.f / k0 : 0.f; ctl.ik[lane + 32] = k1 != 0.f ? 1.f / k1 : 0.f;   // (a factor of zero: no row)
        // chain rule of the normalisation: y = s x / (|x| + eps), y^ = s x r:  dx = s r dy - y^ (y^ . dy) / (s |x|)
        auto chain = [&](float r, float top) {
          const float nrm = top / r - 1e-6f;   // |x|
          return p.l2norm && nrm > 0.f ? r / (top * nrm) : 0.f;
        };
        ctl.ck[lane] = chain(k0, 1.f); ctl.ck[lane + 32] = chain(k1, 1.f);
        ctl.cq[lane] = chain(q0, p.scale); ctl.cq[lane + 32] = chain(q1, p.scale);
        ctl.G[lane] = g_lo; ctl.G[lane + 32] = g_hi;
        ctl.eg[lane] = expf(g_lo); ctl.eg[lane + 32] = expf(g_hi);
        ctl.wd[lane] = expf(fminf(gl - g_lo, 0.f)); ctl.wd[lane + 32] = expf(fminf(gl - g_hi, 0.f));
      }
      asm volatile("bar.sync 7, 544;" ::: "memory");
      tc::tc_fence_after();
      if (tc::elect_one()) {
        const uint64_t kd = tc::smem_desc_sw128(sb + LT_K, 128, 1024), sT = tc::smem_desc(sb + LT_S, 4096, 128);
        wait_at(ctl.full_i, ph);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
#pragma unroll
          for (int x = 0; x < 2; ++x) tc::mma_ss(tb + tKS, adv(sT, x * 2048 + ks * 8192), adv(kd, (ks >> 2) * 8192 + (ks & 3) * 32), tc::idesc_bf16(128, 64, 1, 0), ks + x > 0);
      }
      __syncwarp();
      asm volatile("bar.sync 2, 544;" ::: "memory");
      tc::tc_fence_after();
      if (tc::elect_one()) {
        const uint64_t kd = tc::smem_desc_sw128(sb + LT_K, 128, 1024), od = tc::smem_desc(sb + LT_O, 128, 2048);
        const uint64_t odT = tc::smem_desc(sb + LT_O, 2048, 128), ad = tc::smem_desc(sb + LT_N, 128, 1024);
        const uint64_t dT = tc::smem_desc(sb + LT_D, 4096, 128), sd = tc::smem_desc(sb + LT_S, 128, 4096);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
#pragma unroll
          for (int x = 0; x < 2; ++x) tc::mma_ss(tb + tKD, adv(dT, x * 2048 + ks * 8192), adv(kd, (ks >> 2) * 8192 + (ks & 3) * 32), tc::idesc_bf16(128, 64, 1, 0), ks + x > 0);
#pragma unroll
        for (int ks = 3; ks >= 0; --ks)
#pragma unroll
          for (int x = 0; x < 2; ++x) tc::mma_ss(tb + tAO, adv(odT, ks * 4096), adv(ad, x * 8192 + ks * 256), tc::idesc_bf16(128, 16 * (ks + 1), 0, 1), ks < 3 || x > 0);
        commit(0);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
#pragma unroll
          for (int x = 0; x < 2; ++x) tc::mma_ss(tb + tQ1, adv(sd, x * 2048 + ks * 256), adv(od, ks * 256), tc::idesc_bf16(128, 64, 0, 1), ks + x > 0);
        if (next < P.chunks) {   // what the next chunk reads late, and Q of this one
          const At x = place(next);
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            l2_panel(&P.tq, 64 * e, x.hq, x.t0, x.b);
            l2_panel(&P.tk, 64 * e, x.hq, x.t0, x.b);
            l2_panel(&P.tv, 64 * e, x.h, x.t0, x.b);
            l2_panel(&P.to, 64 * e, x.h, x.t0, x.b);
          }
          l2_bulk(p.xat + (int64_t)next * (3 * 64 * 64), 3 * 16384);
        }
      }
      __syncwarp();
      if (next < P.chunks) load_vectors(next);
      asm volatile("bar.sync 3, 544;" ::: "memory");
      tc::tc_fence_after();
      if (tc::elect_one()) {
        const uint64_t tk = tc::smem_desc(sb + LT_N + 16384, 1024, 128), tm = tc::smem_desc(sb + LT_N + 16384, 128, 1024);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          const uint32_t id = tc::idesc_bf16(128, 64 - 16 * ks, 0, 0);
          tc::mma_ts(tb + tVn + 16 * ks, tb + tR + 8 * ks, adv(tk, ks * 2304), id, ks > 0);
          tc::mma_ts(tb + tVn + 16 * ks, tb + tR + 32 + 8 * ks, adv(tk, ks * 2304), id, 1);
          tc::mma_ts(tb + tVn + 16 * ks, tb + tR + 8 * ks, adv(tk, 8192 + ks * 2304), id, 1);
        }
#pragma unroll
        for (int ks = 3; ks >= 0; --ks) {
          const uint32_t id = tc::idesc_bf16(128, 16 * (ks + 1), 0, 1);
          tc::mma_ts(tb + tdR, tb + tV + 8 * ks, adv(tm, ks * 256), id, ks < 3);
          tc::mma_ts(tb + tdR, tb + tV + 32 + 8 * ks, adv(tm, ks * 256), id, 1);
          tc::mma_ts(tb + tdR, tb + tV + 8 * ks, adv(tm, 8192 + ks * 256), id, 1);
        }
        commit(1);
      }
      __syncwarp();
      asm volatile("bar.sync 4, 544;" ::: "memory");
      tc::tc_fence_after();
      if (tc::elect_one()) {
        const uint64_t od = tc::smem_desc(sb + LT_O, 128, 2048), nd = tc::smem_desc(sb + LT_N, 128, 2048);
        const uint64_t sd = tc::smem_desc(sb + LT_S, 128, 4096), dd = tc::smem_desc(sb + LT_D, 128, 4096);
        constexpr uint32_t id = tc::idesc_bf16(128, 64, 1, 1), ik = tc::idesc_bf16(128, 64, 0, 1);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
          tc::mma_ss(tb + tA, adv(od, ks * 256), adv(nd, ks * 256), id, ks > 0);
          tc::mma_ss(tb + tA, adv(od, ks * 256), adv(nd, 16384 + ks * 256), id, 1);
          tc::mma_ss(tb + tM, adv(od, 16384 + ks * 256), adv(nd, ks * 256), id, ks > 0);   // rows 64 ..: the low term of dR
        }
        commit(2);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
          tc::mma_ss(tb + tKr1, adv(sd, ks * 256), adv(od, 16384 + ks * 256), ik, ks > 0);
          tc::mma_ss(tb + tKr1, adv(sd, 2048 + ks * 256), adv(od, 16384 + ks * 256), ik, 1);
          tc::mma_ss(tb + tKr1, adv(sd, ks * 256), adv(od, 32768 + ks * 256), ik, 1);
        }
        commit(3);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
          tc::mma_ss(tb + tKc1, adv(dd, ks * 256), adv(nd, ks * 256), ik, ks > 0);
          tc::mma_ss(tb + tKc1, adv(dd, 2048 + ks * 256), adv(nd, ks * 256), ik, 1);
          tc::mma_ss(tb + tKc1, adv(dd, ks * 256), adv(nd, 16384 + ks * 256), ik, 1);
        }
        commit(4);
        wait_bar(3, ph);   // S0, dO, dR have been read
        const At x = place(c);
        tc::mbar_arrive_expect_tx(tc::smem_u32(&ctl.full_q), kTile);
        load_panels(P.tq, LT_Q, x.hq, x, ctl.full_q);
        if (next < P.chunks) load_state(ctl.full_s, LT_S, p.ckpt + (int64_t)next * (kD * kD));
        wait_bar(4, ph);   // dS1, Vn
        if (next < P.chunks) load_state(ctl.full_d, LT_D, p.ds + (int64_t)next * (kD * kD));
      }
      __syncwarp();
      asm volatile("bar.sync 5, 544;" ::: "memory");
      tc::tc_fence_after();
      if (tc::elect_one()) {
        const uint64_t kT = tc::smem_desc_sw128(sb + LT_K, 8192, 1024), qT = tc::smem_desc_sw128(sb + LT_Q, 8192, 1024);
        const uint64_t pk = tc::smem_desc(sb + LT_P, 1024, 128), pm = tc::smem_desc(sb + LT_P, 128, 1024);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          const uint32_t id = tc::idesc_bf16(128, 64 - 16 * ks, 1, 0);
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            tc::mma_ss(tb + tQ2 + 16 * ks, adv(kT, ks * 2048), adv(pk, x * 8192 + ks * 2304), id, ks + x > 0);
            tc::mma_ss(tb + tKr2 + 16 * ks, adv(kT, ks * 2048), adv(pk, 16384 + x * 8192 + ks * 2304), id, ks + x > 0);
          }
        }
        wait_at(ctl.full_q, ph);
        tc::tc_fence_after();
#pragma unroll
        for (int ks = 3; ks >= 0; --ks) {
          const uint32_t id = tc::idesc_bf16(128, 16 * (ks + 1), 1, 1);
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            tc::mma_ss(tb + tKc2, adv(qT, ks * 2048), adv(pm, x * 8192 + ks * 256), id, ks < 3 || x > 0);
            tc::mma_ss(tb + tKc2, adv(kT, ks * 2048), adv(pm, 16384 + x * 8192 + ks * 256), id, 1);
          }
        }
        commit(5);
      }
      __syncwarp();
      asm volatile("bar.sync 6, 544;" ::: "memory");
      {   // dbeta; dg = reverse cumulative sum of dG inside the chunk.  k^ . dkr = beta (beta's part + dM . X), since k^ . (dX.E) K^ = sum of dX . X
        const At x = place(c);
        const int rows = min(kC, p.map.T - x.t0);
        const int64_t at = p.map.base(x.b, x.h, 1) + (int64_t)x.t0 * p.map.tok(1), tok = p.map.tok(1);
        float lo = total(sum.x, lane) - total(sum.row[2], lane), hi = total(sum.x, lane + 32) - total(sum.row[2], lane + 32);
        const bool in0 = lane < rows && in(at + lane * tok), in1 = lane + 32 < rows && in(at + (lane + 32) * tok);
        if (in0) p.dbeta[at + lane * tok] = lo + total(sum.v, lane);
        if (in1) p.dbeta[at + (lane + 32) * tok] = hi + total(sum.v, lane + 32);
        if (p.variant == DR_GATED) {
          const float gs = warp_sum(lane < 16 ? sum.ts[lane] : 0.f) * expf(ctl.G[63]) + warp_sum(lane < 16 ? sum.ex[lane] : 0.f);
          lo = total(sum.row[0], lane) - total(sum.row[1], lane) + ctl.beta[lane] * lo;
          hi = total(sum.row[0], lane + 32) - total(sum.row[1], lane + 32) + ctl.beta[lane + 32] * hi + (lane == 31 ? gs : 0.f);
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const float y = __shfl_down_sync(0xffffffffu, lo, o), z = __shfl_down_sync(0xffffffffu, hi, o);
            if (lane + o < 32) { lo += y; hi += z; }
          }
          lo += __shfl_sync(0xffffffffu, hi, 0);
          if (in0) p.dg[at + lane * tok] = lo;
          if (in1) p.dg[at + (lane + 32) * tok] = hi;
        }
      }
      asm volatile("bar.sync 1, 544;" ::: "memory");   // dq, dk are staged; everything but the next states is free
      if (tc::elect_one()) {
        if (p.map.Hq == p.map.H) {
          const At x = place(c);
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            tc::tma_store_4d(&P.tdq, sb + LT_P + 8192 * e, 64 * e, x.h, x.t0, x.b);
            tc::tma_store_4d(&P.tdk, sb + LT_P + kTile + 8192 * e, 64 * e, x.h, x.t0, x.b);
          }
          tc::bulk_commit();
        }
        if (next < P.chunks) {
          load_inputs(next);
          tc::bulk_wait_read_all();
          load_do(next);
        } else {
          tc::bulk_wait_all();
        }
      }
      __syncwarp();
    }
  } else {
    const int qd = warp & 3, cg = warp >> 2, row = 32 * qd + lane;   // this thread's channel (or row of [dO; dR]) and sixteen tokens from 16 cg
    const uint32_t ta = tb + ((uint32_t)(32 * qd) << 16) + 16 * cg;
    const int own = (row >> 3) * 128 + (row & 7) * 16;               // this channel's row in the [8 tokens][8 channels] tiles
    // its entry of token 16 cg in the swizzled panels; token 16 cg + e: ^ (e & 7) << 4, + 128 e
    const uint32_t el = (row >> 6) * 8192 + 16 * cg * 128 + ((row >> 3) & 7) * 16 + (row & 7) * 2;
    auto entry = [&](int base, int e) { return reinterpret_cast<__nv_bfloat16*>(smem + base + (el ^ ((e & 7) << 4)) + 128 * e); };
    auto four = [&](const float (&a)[64], int e) { return *reinterpret_cast<const float4*>(a + 16 * cg + e); };
    auto hand_over = [](int id) {
      tc::fence_async_smem();
      tc::tc_fence_before();
      asm volatile("bar.arrive %0, 544;" ::"r"(id) : "memory");
    };
    // sums of sixteen values over the lanes: lane l ends up with value l >> 1
    auto reduce16 = [&](float (&w)[16]) -> float {
#pragma unroll
      for (int o = 16, m = 8; o > 1; o >>= 1, m >>= 1)
#pragma unroll
        for (int i = 0; i < m; ++i) {
          const bool up = lane & o;
          const float send = up ? w[i] : w[i + m], keep = up ? w[i + m] : w[i];
          w[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
      return w[0] + __shfl_xor_sync(0xffffffffu, w[0], 1);
    };
    uint32_t ph = 0;
#pragma unroll 1
    for (int c = blockIdx.x; c < P.chunks; c += gridDim.x, ph ^= 1) {
      const int unit = c / p.N, b = unit / p.map.H, h = unit % p.map.H, t0 = (c % p.N) * kC;
      const float* xat = p.xat + (int64_t)c * (3 * 64 * 64);
      // ---- S0, dS1: each warp splits its eight rows in place; <dS1, S0> on the way.  A lane's pieces of eight columns are skewed by the
      // row, and rows 4 .. 7 read the halves of a piece in the other order: no bank conflicts on either side --------------------------------
      float ts = 0.f;
      {
        const int r = lane & 7, turn = r >> 2;
        float4 s[8], d[8];
        auto load = [&](int base, float4 (&x)[8]) {
#pragma unroll
          for (int it = 0; it < 4; ++it) {
            const uint8_t* src = smem + base + warp * 4096 + r * 512 + ((4 * it + (lane >> 3) + r) & 15) * 32;
            x[2 * it] = *reinterpret_cast<const float4*>(src + 16 * turn);
            x[2 * it + 1] = *reinterpret_cast<const float4*>(src + 16 - 16 * turn);
          }
          __syncwarp();
        };
        auto store = [&](int base, const float4 (&x)[8]) {
#pragma unroll
          for (int it = 0; it < 4; ++it) {
            uint32_t h[4], l[4];
            split2(x[2 * it].x, x[2 * it].y, h[0], l[0]);
            split2(x[2 * it].z, x[2 * it].w, h[1], l[1]);
            split2(x[2 * it + 1].x, x[2 * it + 1].y, h[2], l[2]);
            split2(x[2 * it + 1].z, x[2 * it + 1].w, h[3], l[3]);
            uint8_t* dst = smem + base + warp * 4096 + ((4 * it + (lane >> 3) + r) & 15) * 128 + r * 16;
            *reinterpret_cast<uint4*>(dst) = turn ? make_uint4(h[2], h[3], h[0], h[1]) : make_uint4(h[0], h[1], h[2], h[3]);
            *reinterpret_cast<uint4*>(dst + 2048) = turn ? make_uint4(l[2], l[3], l[0], l[1]) : make_uint4(l[0], l[1], l[2], l[3]);
          }
        };
        wait_at(ctl.full_s, ph);
        load(LT_S, s);
        store(LT_S, s);
        hand_over(7);
        wait_at(ctl.full_d, ph);
        load(LT_D, d);
        store(LT_D, d);
#pragma unroll
        for (int i = 0; i < 8; ++i) ts += (s[i].x * d[i].x + s[i].y * d[i].y) + (s[i].z * d[i].z + s[i].w * d[i].w);
      }
      // ---- dO^T (warp = eight channels), V -> registers ------------------------------------------------------------------------------------
      uint32_t vp[8];
      wait_at(ctl.full_i, ph);
      {
        const uint32_t src = sb + LT_O + kTile + (warp >> 3) * 8192 + (lane & 7) * 128 + (((warp & 7) ^ (lane & 7)) << 4);
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          uint32_t r[4];
          mma::ldsm4t(r, src + (4 * x + (lane >> 3)) * 1024);
#pragma unroll
          for (int m = 0; m < 4; ++m) *reinterpret_cast<uint32_t*>(smem + LT_O + (4 * x + m) * 2048 + warp * 128 + lane * 4) = r[m];
        }
#pragma unroll
        for (int e = 0; e < 8; ++e)
          vp[e] = (uint32_t)__bfloat16_as_ushort(*entry(LT_O + 2 * kTile, 2 * e)) | ((uint32_t)__bfloat16_as_ushort(*entry(LT_O + 2 * kTile, 2 * e + 1)) << 16);
      }
      tc::fence_async_smem();
      tc::tc_fence_before();
      asm volatile("bar.sync 2, 544;" ::: "memory");
      // ---- R and dVn, as two terms in tensor memory ----------------------------------------------------------------------------------
      wait_bar(0, ph);
      tc::tc_fence_after();
      {
        uint32_t ks[16], kd[16], ao[16];
        tc::tmem_ld16(ta + tKS, ks);
        tc::tmem_ld16(ta + tKD, kd);
        tc::tmem_ld16(ta + tAO, ao);
        tc::tc_wait_ld();
        uint32_t rh[8], rl[8], dh[8], dl[8];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float4 bt4 = four(ctl.beta, 4 * e), rk4 = four(ctl.rk, 4 * e), eg4 = four(ctl.eg, 4 * e), wd4 = four(ctl.wd, 4 * e);
          const float bt[4] = {bt4.x, bt4.y, bt4.z, bt4.w}, rk[4] = {rk4.x, rk4.y, rk4.z, rk4.w};
          const float eg[4] = {eg4.x, eg4.y, eg4.z, eg4.w}, wd[4] = {wd4.x, wd4.y, wd4.z, wd4.w};
          float r[4], d[4];
#pragma unroll
          for (int f = 0; f < 4; ++f) {
            const uint32_t v = vp[2 * e + (f >> 1)];
            r[f] = bt[f] * ((f & 1 ? mma::hi_f(v) : mma::lo_f(v)) - eg[f] * (rk[f] * __uint_as_float(ks[4 * e + f])));
            d[f] = wd[f] * (rk[f] * __uint_as_float(kd[4 * e + f])) + __uint_as_float(ao[4 * e + f]);
          }
#pragma unroll
          for (int f = 0; f < 2; ++f) {
            split2(r[2 * f], r[2 * f + 1], rh[2 * e + f], rl[2 * e + f]);
            split2(d[2 * f], d[2 * f + 1], dh[2 * e + f], dl[2 * e + f]);
          }
        }
        const uint32_t tt = ta - 8 * cg;   // eight columns for sixteen tokens
        tc::tmem_st8(tt + tR, rh);
        tc::tmem_st8(tt + tR + 32, rl);
        tc::tmem_st8(tt + tV, dh);
        tc::tmem_st8(tt + tV + 32, dl);
        tc::tc_wait_st();
      }
      hand_over(3);
      // ---- Vn, dR -> tiles -----------------------------------------------------------------------------------------
      wait_bar(1, ph);
      tc::tc_fence_after();
      {
        uint32_t vn[16], dr[16];
        tc::tmem_ld16(ta + tVn, vn);
        tc::tmem_ld16(ta + tdR, dr);
        tc::tc_wait_ld();
        auto put = [&](const uint32_t (&y)[16], int base) {
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            uint32_t hi[4], lo[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) split2(__uint_as_float(y[8 * x + 2 * e]), __uint_as_float(y[8 * x + 2 * e + 1]), hi[e], lo[e]);
            uint8_t* dst = smem + base + (2 * cg + x) * 2048 + own;
            *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
            *reinterpret_cast<uint4*>(dst + kTile) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
          }
        };
        put(vn, LT_N);
        put(dr, LT_O + kTile);
        hand_over(4);
      }
      // ---- P = rq rk dA.E (rows 0 .. 63 of the product), Px = rk rk dX.E and dM . X (rows 64 ..) ------------------------------------------
      float xs = 0.f;
      const bool second = row >= 64;
      {
        const int i = row & 63;
        float x[16], f[16];
        if (second && cg <= (i >> 4)) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float4 y = __ldcs(reinterpret_cast<const float4*>(xat) + (4 * cg + e) * 64 + i);
            x[4 * e] = y.x; x[4 * e + 1] = y.y; x[4 * e + 2] = y.z; x[4 * e + 3] = y.w;
          }
        } else {
#pragma unroll
          for (int e = 0; e < 16; ++e) x[e] = 0.f;
        }
        const float gi = ctl.G[i], top = second ? -ctl.beta[i] * ctl.rk[i] : ctl.rq[i];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float4 g4 = four(ctl.G, 4 * e), k4 = four(ctl.rk, 4 * e);
          f[4 * e] = top * k4.x * __expf(fminf(gi - g4.x, 0.f)); f[4 * e + 1] = top * k4.y * __expf(fminf(gi - g4.y, 0.f));
          f[4 * e + 2] = top * k4.z * __expf(fminf(gi - g4.z, 0.f)); f[4 * e + 3] = top * k4.w * __expf(fminf(gi - g4.w, 0.f));
        }
        wait_bar(2, ph);
        tc::tc_fence_after();
        uint32_t a[16];
        tc::tmem_ld16(ta + tA, a);
        if (second) {
          uint32_t a2[16];
          tc::tmem_ld16(ta + tM, a2);
          tc::tc_wait_ld();
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            const float dm = __uint_as_float(a[e]) + __uint_as_float(a2[e]);   // negated
            xs -= dm * x[e];   // X carries its decay factor
            a[e] = __float_as_uint(dm);
          }
        } else {
          tc::tc_wait_ld();
        }
        const int last = (second ? i - 1 : i) - 16 * cg;   // dX is strictly below the diagonal
#pragma unroll
        for (int e = 0; e < 16; ++e) x[e] = e <= last ? __uint_as_float(a[e]) * f[e] : 0.f;
        wait_bar(3, ph);   // dO and dR have been read
        uint8_t* dst = smem + LT_P + (second ? 16384 : 0) + 2 * cg * 1024 + (i >> 3) * 128 + (i & 7) * 16;
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          uint32_t hi[4], lo[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) split2(x[8 * hf + 2 * e], x[8 * hf + 2 * e + 1], hi[e], lo[e]);
          *reinterpret_cast<uint4*>(dst + hf * 1024) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
          *reinterpret_cast<uint4*>(dst + 8192 + hf * 1024) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        }
        hand_over(5);
      }
      // ---- dV = beta dR; dR . V (while the last products run) --------------------------------------------------------------------------------
      {
        uint32_t dr[16];
        tc::tmem_ld16(ta + tdR, dr);
        tc::tc_wait_ld();
        wait_bar(4, ph);   // Vn has been read
        float w[16];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float4 bt4 = four(ctl.beta, 4 * e);
          const float bt[4] = {bt4.x, bt4.y, bt4.z, bt4.w};
#pragma unroll
          for (int f = 0; f < 4; ++f) {
            const float x = __uint_as_float(dr[4 * e + f]);
            const uint32_t v = vp[2 * e + (f >> 1)];
            w[4 * e + f] = x * (f & 1 ? mma::hi_f(v) : mma::lo_f(v));
            *entry(LT_N, 4 * e + f) = __float2bfloat16_rn(bt[f] * x);
          }
        }
        const float vs = reduce16(w);
        ts = warp_sum(ts);
        if (second) sum.x[cg][row & 63] = xs;
        if (!(lane & 1)) sum.v[qd][16 * cg + (lane >> 1)] = vs;
        if (lane == 0) sum.ts[warp] = ts;
      }
      // ---- dq^, dk^ and their sums over the channels ----------------------------------------------------------------------------------------
      wait_at(ctl.full_q, ph);
      wait_bar(5, ph);
      tc::tc_fence_after();
      float dq[16], dk[16];
      {
        uint32_t q1[16], q2[16];
        tc::tmem_ld16(ta + tQ1, q1);
        tc::tmem_ld16(ta + tQ2, q2);
        tc::tc_wait_ld();
        float w[16];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float4 eg4 = four(ctl.eg, 4 * e), rq4 = four(ctl.rq, 4 * e);
          const float eg[4] = {eg4.x, eg4.y, eg4.z, eg4.w}, rq[4] = {rq4.x, rq4.y, rq4.z, rq4.w};
#pragma unroll
          for (int f = 0; f < 4; ++f) {
            const int j = 4 * e + f;
            // rq dq^: dq^ itself is not needed
            dq[j] = rq[f] * eg[f] * __uint_as_float(q1[j]) + __uint_as_float(q2[j]);
            w[j] = dq[j] * bf(entry(LT_Q, j));
          }
        }
        const float x = reduce16(w);
        if (!(lane & 1)) sum.row[0][qd][16 * cg + (lane >> 1)] = x;
      }
      float extra = 0.f;
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t r1[8], r2[8], c1[8], c2[8];
        tc::tmem_ld8(ta + tKr1 + 8 * hf, r1);
        tc::tmem_ld8(ta + tKr2 + 8 * hf, r2);
        tc::tmem_ld8(ta + tKc1 + 8 * hf, c1);
        tc::tmem_ld8(ta + tKc2 + 8 * hf, c2);
        tc::tc_wait_ld();
        float w[16];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float4 eg4 = four(ctl.eg, 8 * hf + 4 * e), wd4 = four(ctl.wd, 8 * hf + 4 * e), rk4 = four(ctl.rk, 8 * hf + 4 * e);
          const float4 ik4 = four(ctl.ik, 8 * hf + 4 * e), bt4 = four(ctl.beta, 8 * hf + 4 * e);
          const float eg[4] = {eg4.x, eg4.y, eg4.z, eg4.w}, wd[4] = {wd4.x, wd4.y, wd4.z, wd4.w}, rk[4] = {rk4.x, rk4.y, rk4.z, rk4.w};
          const float ik[4] = {ik4.x, ik4.y, ik4.z, ik4.w}, bt[4] = {bt4.x, bt4.y, bt4.z, bt4.w};
#pragma unroll
          for (int f = 0; f < 4; ++f) {
            const int j = 4 * e + f;
            const float kh = rk[f] * bf(entry(LT_K, 8 * hf + j));
            const float g1 = eg[f] * __uint_as_float(r1[j]), g3 = wd[f] * __uint_as_float(c1[j]);
            const float kc = ik[f] * __uint_as_float(c2[j]) + g3;
            extra += g3 * kh;
            w[j] = kc * kh;
            w[8 + j] = g1 * kh;
            dk[8 * hf + j] = (ik[f] * __uint_as_float(r2[j]) - bt[f] * g1) + kc;
          }
        }
        const float x = reduce16(w);
        if (!(lane & 1)) sum.row[1 + (lane >> 4)][qd][16 * cg + 8 * hf + ((lane >> 1) & 7)] = x;
      }
      extra = warp_sum(extra);
      if (lane == 0) sum.ex[warp] = extra;
      tc::fence_async_smem();
      tc::tc_fence_before();
      asm volatile("bar.sync 6, 544;" ::: "memory");   // the sums of all warps
      // ---- the chain rule's factors, dq, dk ---------------------------------------------------------------------------------------------------
      {   // each warp for its own sixteen tokens: q in the lower lanes, k in the upper ones
        const int i = 16 * cg + (lane & 15);
        float f;
        if (lane < 16)
          f = ctl.cq[i] * total(sum.row[0], i);
        else
          f = ctl.ck[i] * (total(sum.row[1], i) + ctl.beta[i] * (total(sum.x, i) - total(sum.row[2], i)));
        sum.f[warp][lane] = f;
        __syncwarp();
      }
      if (tid == 256) {
#pragma unroll
        for (int e = 0; e < 2; ++e) tc::tma_store_4d(&P.tdv, sb + LT_N + 8192 * e, 64 * e, h, t0, b);
        tc::bulk_commit();
      }
      if (p.map.Hq != p.map.H) {   // grouped heads: dq^, dk^ per head for the finalize kernel
        const int64_t at = ((int64_t)c * kC + 16 * cg) * kD + row, half = (int64_t)P.chunks * (kC * kD);
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const float rq = ctl.rq[16 * cg + e];
          if (in_bounds(P.status, at + e * kD, half) && in_bounds(P.status, half + at + e * kD, P.n_part)) {
            p.part[at + e * kD] = rq != 0.f ? dq[e] / rq : 0.f;
            p.part[half + at + e * kD] = dk[e];
          }
        }
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float4 fq4 = *reinterpret_cast<const float4*>(sum.f[warp] + 4 * e), fk4 = *reinterpret_cast<const float4*>(sum.f[warp] + 16 + 4 * e), rk4 = four(ctl.rk, 4 * e);
          const float fq[4] = {fq4.x, fq4.y, fq4.z, fq4.w}, fk[4] = {fk4.x, fk4.y, fk4.z, fk4.w};
          const float rk[4] = {rk4.x, rk4.y, rk4.z, rk4.w};
#pragma unroll
          for (int f = 0; f < 4; ++f) {
            const int j = 4 * e + f;
            *entry(LT_P, j) = __float2bfloat16_rn(dq[j] - fq[f] * bf(entry(LT_Q, j)));
            *entry(LT_P + kTile, j) = __float2bfloat16_rn(rk[f] * dk[j] - fk[f] * bf(entry(LT_K, j)));
          }
        }
      }
      if (tid == 256) tc::bulk_wait_read_all();
      tc::fence_async_smem();
      asm volatile("bar.sync 1, 544;" ::: "memory");
    }
    if (tid == 256) tc::bulk_wait_all();
  }
  tc::tc_fence_before();
  __syncthreads();
  if (warp == 16) {
    sm100::settle(ctl.abort);
    tc::tmem_dealloc(tb, 512);
  }
  if (tid == 0) sm100::report_wait(P.status, ctl.abort);
}

}  // namespace bwdc
}  // namespace dr
