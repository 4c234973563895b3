// The chunk-parallel part of the backward for per-channel decays (KDA) on tcgen05: every gradient of a chunk from its state S0, the state
// gradient dS1 behind it and its inputs.  Formulas and names: header of dr_bwd.cuh; the kernels around it: dr_bwd_chunk.cuh; the form for
// scalar decays, whose layout of work this one has: dr_bwd_local_sm100.cuh.
//
// float32 operands are two bf16 terms, three products per pair: 17 bits of every entry, whatever lies beside it, with float32's exponents.  (Two fp16
// terms of a power of two times the tile have 22 bits of its largest entries, none of those below 2^-39 of them; three bf16 terms
// do not fit: the states alone would take 192 KB.)  dO is a bf16 value: one term.
//
// Decays: with Kg = k^ e^G, Qg = q^ e^G, Kd = k^ e^{G_L - G}, all at most the rows themselves,
//   1  KS^T = S0^T Kg^T,  KD^T = dS1^T Kd^T,  AO^T = dO^T A,  dQ1^T = S0 dO^T
//   2  Vn^T = R^T T^T,   dR^T = dVn^T T         R = beta (V - KS),  dVn = KD + AO   (terms in tensor memory)
//   3  [dA; dM] = [dO; dR] Vn^T,  dKr1^T = S0 dR^T,  dKc1^T = dS1 Vn^T
//   4  dQ2^T = Kd^T P^T,  dKr2^T = Kd^T Px^T,  dKc2^T = Qg^T P,  dKc3^T = Kg^T Px       P = dA, Px = dX below the diagonal
//   dq^ = e^G (dQ1 + e^{-G_L} dQ2) + diag(dA) k^,  dk^ = e^G (-beta dKr1 + e^{-G_L} dKr2) + e^{G_L - G} dKc1 + e^{-G} (dKc2 + dKc3) + diag(dA) q^
// What the diagonals contribute is added in float32: T's (R and dVn lie in the accumulators that T - I adds to) and dA's, whose parts of q^ dq^
// and k^ dk^ are equal and stay out of dG -- behind strong decays they are most of both.
// The factors of a term multiply to decays of at most 1, so what each of them may reach is a matter of exponents alone.  P and Px, whose products
// are the ones with a factor of more than 1 behind them, come with a power of two that brings their largest entries to 2^40, so that gradients as small as
// float32 has them pass.  A chunk may decay by 2^40 in any channel (kWideKda).  The forward marks those that
// decay by more, and local_kernel, which refers the decays to 16-row blocks, takes them.
//
// A thread of an epilogue owns one channel and sixteen tokens, and so does the one that forms Kg, Kd and Qg: G stays in its registers.  The
// three are formed twice, before the products of 1 and of 4: beside the states (128 KB) there is no room to keep them.
//
// What bounds it: B=2, T=4096, H=16 (2048 chunks, 14 per CTA): 319 us, 46 K cycles per chunk, where local_kernel takes 884 us (three tf32 products on
// mma.sync, 119 K).  Issue slots 34 %, tensor pipe 16 %: the element-wise work between the products, 4 K instructions per warp.  Almost nothing is left for an L1, so what is not in
// shared memory costs an L2 access: with g, q, X, A and T by loads of the warps 71 K cycles, with everything the compiler would keep over the
// chunk loop in spilled registers 57 K; hence the opaque thread index, and G parked in tensor memory.
// Errors against float64 at one chunk (2-norm, 82 sequences; in brackets pre_kernel and local_kernel): dbeta 4.9e-5 (4.9e-5), dg 4.6e-5 (4.6e-5), dh0
// 1.5e-5 (1.5e-5): T's tf32 merges decide; dq, dk, dv 1.7e-3 (bf16 rounding).  Where T is near I (beta a twentieth) 5.2e-6 (2.7e-6), 4.7e-6 (2.0e-6),
// 2.2e-6 (1.3e-6).
#pragma once

namespace dr {
namespace bwdc {

// S0, dS1 (as in local_sm100_kernel); Kg hi, lo, later Vn, later Kg again (before: K and V as they arrive); dO^T (before: dO as it arrives); Kd hi,
// lo, later dR (before: the log decay); A, later T, later X.  In the end q over part of S0, P hi, lo over dO^T, Px over dR hi, Kd over dR lo and X, Qg
// over half of dS1; then dq, dk, dv over dO^T and dR, the sums over Kd lo.
constexpr int LK_S = 0, LK_D = LK_S + 65536, LK_N = LK_D + 65536, LK_O = LK_N + 2 * kTile, LK_R = LK_O + kTile, LK_T = LK_R + 2 * kTile, LK_CTL = LK_T + kTile;
constexpr int LK_P = LK_O, LK_KD = LK_R + kTile, LK_QG = LK_D;
struct LkSums {
  float row[3][4][64];            // per quarter of the channels: q^ . dq^, k^ . dk^, beta's part of k^ . dkr
  float x[4][64], v[4][64];       // dM . X per quarter of the columns, dR . V per quarter of the channels
  float f[16][32];                // per warp: the chain rule's factors of its tokens, q and k
  float g[4][128], ex[4][128];    // dG and dKt . Kt, sums over sixteen tokens
  float ts[128];                  // <dS1, S0> per channel
};
static_assert(sizeof(LkSums) <= kTile, "over T");
struct LkCtl {
  uint64_t bar[6], full_s, full_d, full_i, full_kv, full_t, full_x, full_q;
  uint32_t top[2][2];             // largest entries (bits) of P and Px, by turns
  alignas(16) float beta[64];     // (read four at a time)
  float rk[64], rq[64];
  float g[4][128];                // decay of sixteen tokens, later the diagonal of dA
  uint32_t tmem_base;
  int abort;
};
constexpr int LK_TOTAL = LK_CTL + sizeof(LkCtl);
static_assert(LK_TOTAL <= 232448 && LK_CTL % 16 == 0 && offsetof(LkCtl, beta) % 16 == 0 && offsetof(LkSums, f) % 16 == 0, "shared memory");
// Registers: 640 threads of 96 (the fifth warp group is the issuing warp and three that leave); the workers take 104, the issuing group keeps 64, which
// adds up to what the block was launched with (make_params sees to it that it was 96).  With 544 threads and 96 each 1.4 % slower, spills 308 bytes against 136.
constexpr int kLkThreads = 640, kLkRegs = 96, kLkWorkerRegs = 104, kLkIssueRegs = 64;
static_assert(512 * kLkWorkerRegs + 128 * kLkIssueRegs <= kLkThreads * kLkRegs, "the split waits for good otherwise");
static __global__ void __launch_bounds__(kLkThreads, 1) local_sm100_kda_kernel(const __grid_constant__ LocalParams P) {
  const Params& p = P.p;
  extern __shared__ __align__(1024) uint8_t lk_smem[];
  uint8_t* const smem = lk_smem;
  LkCtl& ctl = *reinterpret_cast<LkCtl*>(smem + LK_CTL);
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
    tc::mbar_init(tc::smem_u32(&ctl.full_kv), 1);
    tc::mbar_init(tc::smem_u32(&ctl.full_t), 1);
    tc::mbar_init(tc::smem_u32(&ctl.full_x), 1);
    tc::mbar_init(tc::smem_u32(&ctl.full_q), 1);
    tc::fence_mbar_init();
    ctl.abort = 0;
    ctl.top[0][0] = ctl.top[0][1] = 0u;
  }
  tc::tc_fence_before();
  __syncthreads();
  tc::tc_fence_after();
  pdl_entry();
  uint32_t tb = ctl.tmem_base, sb = tc::smem_u32(smem);
  auto wait_at = [&](uint64_t& bar, uint32_t parity) {
    const uint32_t at = tc::smem_u32(&bar);
    sm100::wait_inline(at, parity, &ctl.abort, at - tc::smem_u32(&ctl), warp == 16);
  };
  auto wait_bar = [&](int i, uint32_t parity) { wait_at(ctl.bar[i], parity); };
  LkSums& sum = *reinterpret_cast<LkSums*>(smem + LK_T);
  float(&dA)[64] = *reinterpret_cast<float(*)[64]>(ctl.g[0]);
  auto total = [](const float (&a)[4][64], int i) { return (a[0][i] + a[1][i]) + (a[2][i] + a[3][i]); };
  // tensor memory: columns of the accumulators and of the two terms of R^T, dVn^T
  constexpr uint32_t tKS = 0, tKD = 64, tAO = 128, tQ1 = 192, tR = 256, tV = 320, tVn = 384, tdR = 448;
  constexpr uint32_t tKr1 = 0, tKc1 = 64, tA = 128, tM = 256, tQ2 = 128, tKr2 = 256, tKc2 = 320, tKc3 = 384;
  ChunkList list;
  list.start(p, P.chunks, lane);

  if (warp >= 16) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kLkIssueRegs));
    if (warp == 16) {
    // (only the low word changes: the address field does not carry into the other)
    auto adv = [](uint64_t d, uint32_t bytes) { return (d & 0xffffffff00000000ull) | ((uint32_t)d + (bytes >> 4)); };
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
    auto load_part = [&](uint64_t& bar, uint32_t dst, const float* src, uint32_t bytes) { tc::bulk_g2s(sb + dst, src, bytes, tc::smem_u32(&bar)); };
    auto expect = [&](uint64_t& bar, uint32_t bytes) { tc::mbar_arrive_expect_tx(tc::smem_u32(&bar), bytes); };
    auto state = [&](const float* base, int c) { return base + (int64_t)c * (kD * kD); };
    auto tile = [&](int c, int i) { return p.xat + ((int64_t)c * 3 + i) * (64 * 64); };
    // the states arrive in two parts: q lies where the first quarter of S0 goes, Qg where the first half of dS1 does
    auto load_s_upper = [&](int c) { expect(ctl.full_s, 65536); load_part(ctl.full_s, LK_S + kTile, state(p.ckpt, c) + kTile / 4, 65536 - kTile); };
    auto load_s_lower = [&](int c) { load_part(ctl.full_s, LK_S, state(p.ckpt, c), kTile); };
    auto load_d_upper = [&](int c) { expect(ctl.full_d, 65536); load_part(ctl.full_d, LK_D + 32768, state(p.ds, c) + 8192, 32768); };
    auto load_d_lower = [&](int c) { load_part(ctl.full_d, LK_D, state(p.ds, c), 32768); };
    auto load_kv = [&](int c) {
      const At x = place(c);
      expect(ctl.full_kv, 2 * kTile);
      load_panels(P.tk, LK_N, x.hq, x, ctl.full_kv);
      load_panels(P.tv, LK_N + kTile, x.h, x, ctl.full_kv);
    };
    auto load_inputs = [&](int c) {
      const At x = place(c);
      expect(ctl.full_i, 2 * kTile + (p.g_dt == DR_BF16 ? 16384 : 32768));
      tc::tma_load_4d(sb + LK_R, &P.tg, 0, x.t0, x.h, x.b, tc::smem_u32(&ctl.full_i));
      load_panels(P.to, LK_O, x.h, x, ctl.full_i);
      load_part(ctl.full_i, LK_T, tile(c, 1), kTile);
    };
    // the token vectors of a chunk, lane = token and token + 32
    float b0 = 0.f, b1 = 0.f, k0 = 0.f, k1 = 0.f, q0 = 0.f, q1 = 0.f;
    auto load_vectors = [&](int c) {
      const At x = place(c);
      const int rows = min(kC, p.map.T - x.t0);
      const int64_t at = p.map.base(x.b, x.h, 1) + (int64_t)x.t0 * p.map.tok(1), tok = p.map.tok(1);
      b0 = b1 = 0.f;
      if (lane < rows && in(at + lane * tok)) b0 = p.beta[at + lane * tok];
      if (lane + 32 < rows && in(at + (lane + 32) * tok)) b1 = p.beta[at + (lane + 32) * tok];
      const float* nrm = tile(c, 0) + kXNorms + lane;
      k0 = nrm[0]; k1 = nrm[kXNormRow]; q0 = nrm[2 * kXNormRow]; q1 = nrm[3 * kXNormRow];
    };
    auto store_vectors = [&]() {   // before the inputs' barrier is armed: who waits for that sees them
      ctl.beta[lane] = b0; ctl.beta[lane + 32] = b1;
      ctl.rk[lane] = k0; ctl.rk[lane + 32] = k1;
      ctl.rq[lane] = q0; ctl.rq[lane + 32] = q1;
      __syncwarp();
    };
    int c = list.next(p, P.chunks, lane);
    if (c < P.chunks) {
      load_vectors(c);
      store_vectors();
      if (tc::elect_one()) {
        load_inputs(c);
        load_kv(c);
        load_s_upper(c);
        load_s_lower(c);
        load_d_upper(c);
        load_d_lower(c);
      }
      __syncwarp();
    }
    uint32_t ph = 0;
#pragma unroll 1
    for (int next; c < P.chunks; c = next, ph ^= 1) {
      asm volatile("" : "+r"(sb), "+r"(tb));   // the descriptors are formed for each chunk: kept over the loop they would be spilled
      next = list.next(p, P.chunks, lane);
      asm volatile("bar.sync 7, 544;" ::: "memory");
      tc::tc_fence_after();
      constexpr uint32_t hi_lo[3] = {0, 1, 0}, lo_hi[3] = {0, 0, 1};   // terms of A and of B in the three products
      if (tc::elect_one()) {
        const uint64_t sT = tc::smem_desc(sb + LK_S, 4096, 128), kd = tc::smem_desc(sb + LK_N, 128, 2048);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
#pragma unroll
          for (int x = 0; x < 3; ++x)
            tc::mma_ss(tb + tKS, adv(sT, hi_lo[x] * 2048 + ks * 8192), adv(kd, lo_hi[x] * kTile + ks * 256), tc::idesc_bf16(128, 64, 1, 1), ks + x > 0);
      }
      __syncwarp();
      asm volatile("bar.sync 2, 544;" ::: "memory");
      tc::tc_fence_after();
      if (tc::elect_one()) {
        const uint64_t dT = tc::smem_desc(sb + LK_D, 4096, 128), kd = tc::smem_desc(sb + LK_R, 128, 2048), od = tc::smem_desc(sb + LK_O, 128, 2048);
        const uint64_t odT = tc::smem_desc(sb + LK_O, 2048, 128), ad = tc::smem_desc(sb + LK_T, 128, 1024), sd = tc::smem_desc(sb + LK_S, 128, 4096);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
#pragma unroll
          for (int x = 0; x < 3; ++x)
            tc::mma_ss(tb + tKD, adv(dT, hi_lo[x] * 2048 + ks * 8192), adv(kd, lo_hi[x] * kTile + ks * 256), tc::idesc_bf16(128, 64, 1, 1), ks + x > 0);
#pragma unroll
        for (int ks = 3; ks >= 0; --ks)
#pragma unroll
          for (int x = 0; x < 2; ++x) tc::mma_ss(tb + tAO, adv(odT, ks * 4096), adv(ad, x * 8192 + ks * 256), tc::idesc_bf16(128, 16 * (ks + 1), 0, 1), ks < 3 || x > 0);
        commit(0);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
#pragma unroll
          for (int x = 0; x < 2; ++x) tc::mma_ss(tb + tQ1, adv(sd, x * 2048 + ks * 256), adv(od, ks * 256), tc::idesc_bf16(128, 64, 0, 1), ks + x > 0);
        if (next < P.chunks) {   // what the next chunk reads
          const At x = place(next);
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            l2_panel(&P.tq, 64 * e, x.hq, x.t0, x.b);
            l2_panel(&P.tk, 64 * e, x.hq, x.t0, x.b);
            l2_panel(&P.tv, 64 * e, x.h, x.t0, x.b);
            l2_panel(&P.to, 64 * e, x.h, x.t0, x.b);
          }
          l2_bulk(tile(next, 0), 3 * 16384);
          l2_panel(&P.tg, 0, x.t0, x.h, x.b);
        }
        wait_bar(0, ph);   // A has been read
        expect(ctl.full_t, kTile);
        load_part(ctl.full_t, LK_T, tile(c, 2), kTile);
      }
      __syncwarp();
      if (next < P.chunks) load_vectors(next);
      asm volatile("bar.sync 3, 544;" ::: "memory");
      tc::tc_fence_after();
      if (tc::elect_one()) {
        wait_at(ctl.full_t, ph);
        const uint64_t tk = tc::smem_desc(sb + LK_T, 1024, 128), tm = tc::smem_desc(sb + LK_T, 128, 1024);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          const uint32_t id = tc::idesc_bf16(128, 64 - 16 * ks, 0, 0);
          tc::mma_ts(tb + tVn + 16 * ks, tb + tR + 8 * ks, adv(tk, ks * 2304), id, 1);
          tc::mma_ts(tb + tVn + 16 * ks, tb + tR + 32 + 8 * ks, adv(tk, ks * 2304), id, 1);
          tc::mma_ts(tb + tVn + 16 * ks, tb + tR + 8 * ks, adv(tk, 8192 + ks * 2304), id, 1);
        }
#pragma unroll
        for (int ks = 3; ks >= 0; --ks) {
          const uint32_t id = tc::idesc_bf16(128, 16 * (ks + 1), 0, 1);
          tc::mma_ts(tb + tdR, tb + tV + 8 * ks, adv(tm, ks * 256), id, 1);
          tc::mma_ts(tb + tdR, tb + tV + 32 + 8 * ks, adv(tm, ks * 256), id, 1);
          tc::mma_ts(tb + tdR, tb + tV + 8 * ks, adv(tm, 8192 + ks * 256), id, 1);
        }
        commit(1);
        wait_bar(1, ph);   // T has been read
        expect(ctl.full_x, kTile);
        load_part(ctl.full_x, LK_T, tile(c, 0), kTile);
      }
      __syncwarp();
      asm volatile("bar.sync 4, 544;" ::: "memory");
      tc::tc_fence_after();
      if (tc::elect_one()) {
        const uint64_t od = tc::smem_desc(sb + LK_O, 128, 2048), nd = tc::smem_desc(sb + LK_N, 128, 2048);
        const uint64_t sd = tc::smem_desc(sb + LK_S, 128, 4096), dd = tc::smem_desc(sb + LK_D, 128, 4096);
        constexpr uint32_t id = tc::idesc_bf16(128, 64, 1, 1), ik = tc::idesc_bf16(128, 64, 0, 1);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
          tc::mma_ss(tb + tA, adv(od, ks * 256), adv(nd, ks * 256), id, ks > 0);
          tc::mma_ss(tb + tA, adv(od, ks * 256), adv(nd, kTile + ks * 256), id, 1);
          tc::mma_ss(tb + tM, adv(od, kTile + ks * 256), adv(nd, ks * 256), id, ks > 0);   // rows 64 ..: the low term of dR
        }
        commit(2);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
#pragma unroll
          for (int x = 0; x < 3; ++x)
            tc::mma_ss(tb + tKr1, adv(sd, hi_lo[x] * 2048 + ks * 256), adv(od, kTile + lo_hi[x] * kTile + ks * 256), ik, ks + x > 0);
        commit(3);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
#pragma unroll
          for (int x = 0; x < 3; ++x)
            tc::mma_ss(tb + tKc1, adv(dd, hi_lo[x] * 2048 + ks * 256), adv(nd, lo_hi[x] * kTile + ks * 256), ik, ks + x > 0);
        commit(4);
        wait_bar(3, ph);   // S0, dO, dR have been read
        {
          const At x = place(c);
          expect(ctl.full_q, kTile);
          load_panels(P.tq, LK_S, x.hq, x, ctl.full_q);
        }
        if (next < P.chunks) load_s_upper(next);
        wait_bar(4, ph);   // dS1, Vn
        if (next < P.chunks) load_d_upper(next);
      }
      __syncwarp();
      asm volatile("bar.sync 5, 544;" ::: "memory");
      tc::tc_fence_after();
      if (tc::elect_one()) {
        const uint64_t kd = tc::smem_desc(sb + LK_KD, 2048, 128), kg = tc::smem_desc(sb + LK_N, 2048, 128), qg = tc::smem_desc(sb + LK_QG, 2048, 128);
        const uint64_t pk = tc::smem_desc(sb + LK_P, 1024, 128), pm = tc::smem_desc(sb + LK_P, 128, 1024);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          const uint32_t id = tc::idesc_bf16(128, 64 - 16 * ks, 0, 0);
#pragma unroll
          for (int x = 0; x < 3; ++x) {
            tc::mma_ss(tb + tQ2 + 16 * ks, adv(kd, hi_lo[x] * kTile + ks * 4096), adv(pk, lo_hi[x] * 8192 + ks * 2304), id, ks + x > 0);
            tc::mma_ss(tb + tKr2 + 16 * ks, adv(kd, hi_lo[x] * kTile + ks * 4096), adv(pk, 16384 + lo_hi[x] * 8192 + ks * 2304), id, ks + x > 0);
          }
        }
#pragma unroll
        for (int ks = 3; ks >= 0; --ks) {
          const uint32_t id = tc::idesc_bf16(128, 16 * (ks + 1), 0, 1);
#pragma unroll
          for (int x = 0; x < 3; ++x) {
            tc::mma_ss(tb + tKc2, adv(qg, hi_lo[x] * kTile + ks * 4096), adv(pm, lo_hi[x] * 8192 + ks * 256), id, ks < 3 || x > 0);
            tc::mma_ss(tb + tKc3, adv(kg, hi_lo[x] * kTile + ks * 4096), adv(pm, 16384 + lo_hi[x] * 8192 + ks * 256), id, ks < 3 || x > 0);
          }
        }
        commit(5);
        if (next < P.chunks) {
          load_s_lower(next);
          wait_bar(5, ph);   // Qg and Kg have been read
          load_kv(next);
          load_d_lower(next);
        }
      }
      __syncwarp();
      asm volatile("bar.sync 6, 544;" ::: "memory");   // dv is staged, the sums are there
      {
        const At x = place(c);
        if (tc::elect_one()) {
#pragma unroll
          for (int e = 0; e < 2; ++e) tc::tma_store_4d(&P.tdv, sb + LK_R + kTile + 8192 * e, 64 * e, x.h, x.t0, x.b);
        }
        __syncwarp();
        const int rows = min(kC, p.map.T - x.t0);
        const int64_t at = p.map.base(x.b, x.h, 1) + (int64_t)x.t0 * p.map.tok(1), tok = p.map.tok(1);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int i = lane + 32 * e;
          if (i < rows && in(at + i * tok)) p.dbeta[at + i * tok] = (total(sum.x, i) - total(sum.row[2], i)) + total(sum.v, i);
        }
      }
      asm volatile("bar.sync 1, 544;" ::: "memory");   // dq, dk, dv are staged; everything but the next states, K and V is free
      if (tc::elect_one()) {
        const At x = place(c);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          if (p.map.Hq == p.map.H) {
            tc::tma_store_4d(&P.tdq, sb + LK_O + 8192 * e, 64 * e, x.h, x.t0, x.b);
            tc::tma_store_4d(&P.tdk, sb + LK_R + 8192 * e, 64 * e, x.h, x.t0, x.b);
          }
        }
        tc::bulk_commit();
      }
      __syncwarp();
      store_vectors();
      if (tc::elect_one()) {
        if (next < P.chunks) {
          tc::bulk_wait_read_all();
          load_inputs(next);
        } else {
          tc::bulk_wait_all();
        }
      }
      __syncwarp();
    }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kLkWorkerRegs));
    uint32_t ph = 0;
#pragma unroll 1
    for (int c = list.next(p, P.chunks, lane); c < P.chunks; c = list.next(p, P.chunks, lane), ph ^= 1) {
      // (what follows from the thread's place is formed for each chunk: kept over the loop it would be spilled, and there is no L1 to speak of)
      int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
      asm volatile("" : "+r"(warp), "+r"(lane));
      warp = __shfl_sync(0xffffffffu, warp, 0);
      const int qd = warp & 3, cg = warp >> 2, row = 32 * qd + lane;   // this thread's channel (or row of [dO; dR]) and sixteen tokens from 16 cg
      const uint32_t ta = tb + ((uint32_t)(32 * qd) << 16) + 16 * cg;
      const int own = 2 * cg * 2048 + (row >> 3) * 128 + (row & 7) * 16;   // this channel's eight tokens in the [8 tokens][8 channels] tiles; + 2048: the next eight
      // its entry of token 16 cg in the swizzled panels; token 16 cg + e: ^ (e & 7) << 4, + 128 e
      const uint32_t el = (row >> 6) * 8192 + 16 * cg * 128 + ((row >> 3) & 7) * 16 + (row & 7) * 2;
      auto entry = [&](int base, int e) { return reinterpret_cast<__nv_bfloat16*>(smem + base + (el ^ ((e & 7) << 4)) + 128 * e); };
      auto raw2 = [&](int base, int e) {   // two tokens
        return (uint32_t)__bfloat16_as_ushort(*entry(base, 2 * e)) | ((uint32_t)__bfloat16_as_ushort(*entry(base, 2 * e + 1)) << 16);
      };
      auto four = [&](const float (&a)[64], int e) { return *reinterpret_cast<const float4*>(a + 16 * cg + e); };
      auto half = [](uint32_t u, int f) { return f & 1 ? mma::hi_f(u) : mma::lo_f(u); };
      auto hand_over = [](int id) {
        tc::fence_async_smem();
        tc::tc_fence_before();
        asm volatile("bar.arrive %0, 544;" ::"r"(id) : "memory");
      };
      auto workers_sync = []() { asm volatile("bar.sync 8, 512;" ::: "memory"); };
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
      // sixteen tokens of this channel -> the two terms of a tile
      auto put = [&](int base, const float (&y)[16]) {
  #pragma unroll
        for (int x = 0; x < 2; ++x) {
          uint32_t hi[4], lo[4];
  #pragma unroll
          for (int e = 0; e < 4; ++e) split2(y[8 * x + 2 * e], y[8 * x + 2 * e + 1], hi[e], lo[e]);
          *reinterpret_cast<uint4*>(smem + base + own + x * 2048) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
          *reinterpret_cast<uint4*>(smem + base + kTile + own + x * 2048) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        }
      };
      // ---- G over this thread's tokens (log2 units); K, V, dO (warp = eight channels) -> registers ----------------------------------------------
      float G[16];
      uint32_t kp[8], vp[8], od[8];
      wait_at(ctl.full_kv, ph);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        kp[e] = raw2(LK_N, e);
        vp[e] = raw2(LK_N + kTile, e);
      }
      wait_at(ctl.full_i, ph);
      if (p.g_dt == DR_BF16) {
#pragma unroll
        for (int e = 0; e < 16; ++e) G[e] = bf(reinterpret_cast<const __nv_bfloat16*>(smem + LK_R) + (16 * cg + e) * kD + row);
      } else {
#pragma unroll
        for (int e = 0; e < 16; ++e) G[e] = reinterpret_cast<const float*>(smem + LK_R)[(16 * cg + e) * kD + row];
      }
#pragma unroll
      for (int e = 0; e < 16; ++e) G[e] = G[e] * kLog2e + (e ? G[e - 1] : 0.f);
      ctl.g[cg][row] = G[15];
      {
        const uint32_t src = sb + LK_O + (warp >> 3) * 8192 + (lane & 7) * 128 + (((warp & 7) ^ (lane & 7)) << 4);
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          uint32_t r[4];
          mma::ldsm4t(r, src + (4 * x + (lane >> 3)) * 1024);
#pragma unroll
          for (int m = 0; m < 4; ++m) od[4 * x + m] = r[m];
        }
      }
      // A lane's pieces of eight columns of the states are skewed by the row, and rows 4 .. 7 read the halves of a piece in the other order: no bank
      // conflicts on either side
      const int r8 = lane & 7, turn = r8 >> 2;
      workers_sync();
      // ---- G from the chunk's start; dO^T; Kg, the terms of S0; then Kd, dS1 --------------------------------------------------------------
      float GL;
      {
        float pre = 0.f;
        GL = 0.f;
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          if (s == cg) pre = GL;
          GL += ctl.g[s][row];
        }
#pragma unroll
        for (int e = 0; e < 16; ++e) G[e] += pre;
      }
      // k^ or q^ times the decay from the chunk's start, or to its end
      auto decayed = [&](float (&y)[16], const uint32_t (&x)[8], const float (&r)[64], bool to_end) {
#pragma unroll
        for (int e4 = 0; e4 < 16; e4 += 4) {
          const float4 r4 = four(r, e4);
          const float f[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
          for (int e = e4; e < e4 + 4; ++e) y[e] = f[e & 3] * half(x[e >> 1], e) * ex2(to_end ? GL - G[e] : G[e]);
        }
      };
      // the terms of a state in place of its rows
      auto split_state = [&](int base) {
        float4 x[8];
#pragma unroll
        for (int it = 0; it < 4; ++it) {
          const uint8_t* src = smem + base + warp * 4096 + r8 * 512 + ((4 * it + (lane >> 3) + r8) & 15) * 32;
          x[2 * it] = *reinterpret_cast<const float4*>(src + 16 * turn);
          x[2 * it + 1] = *reinterpret_cast<const float4*>(src + 16 - 16 * turn);
        }
        __syncwarp();
#pragma unroll
        for (int it = 0; it < 4; ++it) {
          uint32_t u[4], l[4];
          split2(x[2 * it].x, x[2 * it].y, u[0], l[0]);
          split2(x[2 * it].z, x[2 * it].w, u[1], l[1]);
          split2(x[2 * it + 1].x, x[2 * it + 1].y, u[2], l[2]);
          split2(x[2 * it + 1].z, x[2 * it + 1].w, u[3], l[3]);
          uint8_t* dst = smem + base + warp * 4096 + ((4 * it + (lane >> 3) + r8) & 15) * 128 + r8 * 16;
          *reinterpret_cast<uint4*>(dst) = turn ? make_uint4(u[2], u[3], u[0], u[1]) : make_uint4(u[0], u[1], u[2], u[3]);
          *reinterpret_cast<uint4*>(dst + 2048) = turn ? make_uint4(l[2], l[3], l[0], l[1]) : make_uint4(l[0], l[1], l[2], l[3]);
        }
      };
#pragma unroll
      for (int m = 0; m < 8; ++m) *reinterpret_cast<uint32_t*>(smem + LK_O + m * 2048 + warp * 128 + lane * 4) = od[m];
      float y[16];
      decayed(y, kp, ctl.rk, false);
      put(LK_N, y);
      wait_at(ctl.full_s, ph);
      wait_at(ctl.full_d, ph);
      float ts = 0.f;   // <dS1, S0> of channel 8 warp + (lane & 7)
#pragma unroll
      for (int it = 0; it < 8; ++it) {
        const int at = warp * 4096 + r8 * 512 + ((4 * (it >> 1) + (lane >> 3) + r8) & 15) * 32 + 16 * ((it & 1) ^ turn);
        const float4 s = *reinterpret_cast<const float4*>(smem + LK_S + at), d = *reinterpret_cast<const float4*>(smem + LK_D + at);
        ts += (s.x * d.x + s.y * d.y) + (s.z * d.z + s.w * d.w);
      }
      ts += __shfl_xor_sync(0xffffffffu, ts, 8);
      ts += __shfl_xor_sync(0xffffffffu, ts, 16);
      split_state(LK_S);
      hand_over(7);
      decayed(y, kp, ctl.rk, true);
      put(LK_R, y);
      // (G waits in tensor memory wherever it is not needed: registers are what these phases are short of)
      auto park = [&](uint32_t col) {
        uint32_t u[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) u[e] = __float_as_uint(G[e]);
        tc::tmem_st16(ta + col, u);
        tc::tc_wait_st();
      };
      auto fetch = [&](uint32_t col) {
        uint32_t u[16];
        tc::tmem_ld16(ta + col, u);
        tc::tc_wait_ld();
#pragma unroll
        for (int e = 0; e < 16; ++e) G[e] = __uint_as_float(u[e]);
      };
      park(tVn);
      split_state(LK_D);
      hand_over(2);
      // ---- R and dVn, as two terms in tensor memory ----------------------------------------------------------------------------------
      wait_bar(0, ph);
      tc::tc_fence_after();
      {
        fetch(tVn);   // (R goes there)
        uint32_t u[16], l[16];
        tc::tmem_ld16(ta + tKS, u);
        tc::tc_wait_ld();
#pragma unroll
        for (int e4 = 0; e4 < 16; e4 += 4) {
          const float4 b4 = four(ctl.beta, e4);
          const float bt[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
          for (int e = e4; e < e4 + 4; ++e) y[e] = bt[e & 3] * (half(vp[e >> 1], e) - __uint_as_float(u[e]));
        }
        const uint32_t tt = ta - 8 * cg;   // eight columns for sixteen tokens
        uint32_t hi[8], lo[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) split2(y[2 * e], y[2 * e + 1], hi[e], lo[e]);
        tc::tmem_st8(tt + tR, hi);
        tc::tmem_st8(tt + tR + 32, lo);
#pragma unroll
        for (int e = 0; e < 16; ++e) u[e] = __float_as_uint(y[e]);
        tc::tmem_st16(ta + tVn, u);
        tc::tmem_ld16(ta + tKD, u);
        tc::tmem_ld16(ta + tAO, l);
        tc::tc_wait_ld();
#pragma unroll
        for (int e = 0; e < 16; ++e) u[e] = __float_as_uint(__uint_as_float(u[e]) + __uint_as_float(l[e]));
        tc::tmem_st16(ta + tdR, u);
#pragma unroll
        for (int e = 0; e < 8; ++e) split2(__uint_as_float(u[2 * e]), __uint_as_float(u[2 * e + 1]), hi[e], lo[e]);
        tc::tmem_st8(tt + tV, hi);
        tc::tmem_st8(tt + tV + 32, lo);
        tc::tc_wait_st();
      }
      hand_over(3);
      // ---- Vn, dR -> tiles -----------------------------------------------------------------------------------------------------------------
      wait_bar(1, ph);
      tc::tc_fence_after();
      park(tV);
      {
        uint32_t u[16], w[16];
        tc::tmem_ld16(ta + tVn, u);
        tc::tmem_ld16(ta + tdR, w);
        tc::tc_wait_ld();
#pragma unroll
        for (int e = 0; e < 16; ++e) y[e] = __uint_as_float(u[e]);
        put(LK_N, y);
#pragma unroll
        for (int e = 0; e < 16; ++e) y[e] = __uint_as_float(w[e]);
        put(LK_R, y);
      }
      hand_over(4);
      // ---- P = dA (rows 0 .. 63 of the product), Px = dX and dM . X (rows 64 ..); Kd, Kg, Qg once more -----------------------------------------
      float xs = 0.f;
      const bool second = row >= 64;
      {
        const int i = row & 63;
        wait_bar(2, ph);
        tc::tc_fence_after();
        uint32_t a[16];
        tc::tmem_ld16(ta + tA, a);
        const int last = i - 1 - 16 * cg;   // below the diagonal
        if (second) {
          uint32_t a2[16];
          tc::tmem_ld16(ta + tM, a2);
          tc::tc_wait_ld();
          const float bt = ctl.beta[i];
          wait_at(ctl.full_x, ph);
#pragma unroll
          for (int f = 0; f < 4; ++f) {
            const float4 x4 = *reinterpret_cast<const float4*>(smem + LK_T + ((4 * cg + f) * 64 + i) * 16);   // X carries its decay factor
            const float x[4] = {x4.x, x4.y, x4.z, x4.w};
#pragma unroll
            for (int e = 4 * f; e < 4 * f + 4; ++e) {
              const float dm = -(__uint_as_float(a[e]) + __uint_as_float(a2[e]));
              xs += e <= last ? dm * x[e & 3] : 0.f;
              y[e] = e <= last ? bt * dm : 0.f;
            }
          }
        } else {
          tc::tc_wait_ld();
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            y[e] = e <= last ? __uint_as_float(a[e]) : 0.f;
            if (e == last + 1) dA[i] = __uint_as_float(a[e]);
          }
        }
        float m = 0.f;
#pragma unroll
        for (int e = 0; e < 16; ++e) m = fmaxf(m, fabsf(y[e]));
        const uint32_t most = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
        if (lane == 0) atomicMax(&ctl.top[ph][second], most);
        workers_sync();   // X has been read: Kd goes over it
        if (tid < 2) ctl.top[ph ^ 1][tid] = 0u;   // for the next chunk
        const float s = lift(ctl.top[ph][second]);
        wait_bar(3, ph);   // dO and dR have been read
        uint8_t* dst = smem + LK_P + (second ? 16384 : 0) + 2 * cg * 1024 + (i >> 3) * 128 + (i & 7) * 16;
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          uint32_t u[4], l[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) split2(s * y[8 * hf + 2 * e], s * y[8 * hf + 2 * e + 1], u[e], l[e]);
          *reinterpret_cast<uint4*>(dst + hf * 1024) = make_uint4(u[0], u[1], u[2], u[3]);
          *reinterpret_cast<uint4*>(dst + 8192 + hf * 1024) = make_uint4(l[0], l[1], l[2], l[3]);
        }
      }
      fetch(tV);
      decayed(y, kp, ctl.rk, true);
      put(LK_KD, y);
      uint32_t qp[8];
      wait_at(ctl.full_q, ph);
#pragma unroll
      for (int e = 0; e < 8; ++e) qp[e] = raw2(LK_S, e);
      wait_bar(4, ph);   // Vn and dS1 have been read
      decayed(y, kp, ctl.rk, false);
      put(LK_N, y);
      decayed(y, qp, ctl.rq, false);
      put(LK_QG, y);
      hand_over(5);
      // ---- dV = beta dR, dR . V (while the last products run) ---------------------------------------------------------------------------------
      uint32_t dv[8];
      float vs;
      {
        uint32_t u[16];
        tc::tmem_ld16(ta + tdR, u);
        tc::tc_wait_ld();
#pragma unroll
        for (int e4 = 0; e4 < 16; e4 += 4) {
          const float4 b4 = four(ctl.beta, e4);
          const float bt[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
          for (int e = e4; e < e4 + 4; ++e) {
            const float d = __uint_as_float(u[e]);
            y[e] = d * half(vp[e >> 1], e);
            u[e] = __float_as_uint(bt[e & 3] * d);
          }
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) dv[e] = mma::pack(__uint_as_float(u[2 * e]), __uint_as_float(u[2 * e + 1]));
        vs = reduce16(y);
        park(tdR);
      }
      // ---- dq^, dk^, dG and their sums; dq^ and dk^ wait in tensor memory for the sums over all channels ----------------------------------------
      wait_bar(5, ph);
      tc::tc_fence_after();
      if (second) sum.x[cg][row & 63] = xs;
      if (!(lane & 1)) sum.v[qd][16 * cg + (lane >> 1)] = vs;
      if (lane < 8) sum.ts[8 * warp + lane] = ts;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        *entry(LK_R + kTile, 2 * e) = __ushort_as_bfloat16((unsigned short)(dv[e] & 0xffffu));
        *entry(LK_R + kTile, 2 * e + 1) = __ushort_as_bfloat16((unsigned short)(dv[e] >> 16));
      }
      float ex = 0.f;   // dKt . Kt
      {
        const float el = ex2(GL), eli = ex2(-GL), fp = drop(ctl.top[ph][0]), fx = drop(ctl.top[ph][1]);
        // sums of eight values over the lanes: lane l ends up with value l >> 2
        auto reduce8 = [&](float (&w)[8]) -> float {
#pragma unroll
          for (int o = 16, m = 4; o > 2; o >>= 1, m >>= 1)
#pragma unroll
            for (int i = 0; i < m; ++i) {
              const bool high = lane & o;
              const float send = high ? w[i] : w[i + m], keep = high ? w[i + m] : w[i];
              w[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
          const float x = w[0] + __shfl_xor_sync(0xffffffffu, w[0], 2);
          return x + __shfl_xor_sync(0xffffffffu, x, 1);
        };
        auto row_sum = [&](int i, int hf, float (&w)[8]) {
          const float x = reduce8(w);
          if (!(lane & 3)) sum.row[i][qd][16 * cg + 8 * hf + (lane >> 2)] = x;
        };
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          uint32_t u[8], w[8], gg[8];
          float eg[8], dg[8], s8[8];
          tc::tmem_ld8(ta + tdR + 8 * hf, gg);
          tc::tmem_ld8(ta + tQ1 + 8 * hf, u);
          tc::tmem_ld8(ta + tQ2 + 8 * hf, w);
          tc::tc_wait_ld();
#pragma unroll
          for (int e4 = 0; e4 < 8; e4 += 4) {
            const float4 q4 = four(ctl.rq, 8 * hf + e4), k4 = four(ctl.rk, 8 * hf + e4), a4 = four(dA, 8 * hf + e4);
            const float rq[4] = {q4.x, q4.y, q4.z, q4.w}, rk[4] = {k4.x, k4.y, k4.z, k4.w}, da[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
            for (int e = e4; e < e4 + 4; ++e) {
              const int j = 8 * hf + e;
              eg[e] = ex2(__uint_as_float(gg[e]));
              const float x = eg[e] * (__uint_as_float(u[e]) + (__uint_as_float(w[e]) * eli) * fp), qh = rq[e & 3] * half(qp[j >> 1], j);
              const float all = x + da[e & 3] * (rk[e & 3] * half(kp[j >> 1], j));
              dg[e] = qh * x;
              s8[e] = qh * all;
              u[e] = __float_as_uint(all);
            }
          }
          tc::tmem_st8(ta + tQ1 + 8 * hf, u);
          row_sum(0, hf, s8);
          uint32_t z[8];
          tc::tmem_ld8(ta + tKr1 + 8 * hf, u);
          tc::tmem_ld8(ta + tKr2 + 8 * hf, w);
          tc::tc_wait_ld();
#pragma unroll
          for (int e4 = 0; e4 < 8; e4 += 4) {
            const float4 r4 = four(ctl.rk, 8 * hf + e4), b4 = four(ctl.beta, 8 * hf + e4);
            const float r[4] = {r4.x, r4.y, r4.z, r4.w}, bt[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
            for (int e = e4; e < e4 + 4; ++e) {
              const int j = 8 * hf + e;
              const float kh = r[e & 3] * half(kp[j >> 1], j), g1 = __uint_as_float(u[e]);
              const float x = eg[e] * ((__uint_as_float(w[e]) * eli) * fx - bt[e & 3] * g1);
              dg[e] += kh * x;
              s8[e] = eg[e] * g1 * kh;
              u[e] = __float_as_uint(x);   // dk^_row
            }
          }
          row_sum(2, hf, s8);
          tc::tmem_ld8(ta + tKc2 + 8 * hf, w);
          tc::tmem_ld8(ta + tKc3 + 8 * hf, z);
          tc::tc_wait_ld();
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const float em = ex2(-__uint_as_float(gg[e]));
            s8[e] = (em * __uint_as_float(w[e])) * fp + (em * __uint_as_float(z[e])) * fx;
            gg[e] = __float_as_uint(em);
          }
          tc::tmem_ld8(ta + tKc1 + 8 * hf, w);
          tc::tc_wait_ld();
#pragma unroll
          for (int e4 = 0; e4 < 8; e4 += 4) {
            const float4 q4 = four(ctl.rq, 8 * hf + e4), k4 = four(ctl.rk, 8 * hf + e4), a4 = four(dA, 8 * hf + e4);
            const float rq[4] = {q4.x, q4.y, q4.z, q4.w}, rk[4] = {k4.x, k4.y, k4.z, k4.w}, da[4] = {a4.x, a4.y, a4.z, a4.w};
#pragma unroll
            for (int e = e4; e < e4 + 4; ++e) {
              const int j = 8 * hf + e;
              const float kh = rk[e & 3] * half(kp[j >> 1], j), g3 = (__uint_as_float(gg[e]) * el) * __uint_as_float(w[e]);
              const float kc = g3 + s8[e], x = (__uint_as_float(u[e]) + kc) + da[e & 3] * (rq[e & 3] * half(qp[j >> 1], j));
              ex += g3 * kh;
              dg[e] -= kh * kc;
              u[e] = __float_as_uint(x);
              s8[e] = kh * x;
            }
          }
          tc::tmem_st8(ta + tKr1 + 8 * hf, u);
          row_sum(1, hf, s8);
#pragma unroll
          for (int e = 0; e < 8; ++e) u[e] = __float_as_uint(dg[e]);
          tc::tmem_st8(ta + tdR + 8 * hf, u);   // over G
          tc::tc_wait_st();
        }
      }
      float up[16];   // dG
      {
        uint32_t u[16];
        tc::tmem_ld16(ta + tdR, u);
        tc::tc_wait_ld();
#pragma unroll
        for (int e = 0; e < 16; ++e) up[e] = __uint_as_float(u[e]);
      }
      // dG: suffix sums over the sixteen tokens
#pragma unroll
      for (int e = 14; e >= 0; --e) up[e] += up[e + 1];
      sum.g[cg][row] = up[0];
      sum.ex[cg][row] = ex;
      tc::fence_async_smem();
      asm volatile("bar.sync 6, 544;" ::: "memory");   // the sums of all warps, dv
      // ---- dg; the chain rule's factors, dq, dk -------------------------------------------------------------------------------------------------
      {
        const int unit = c / p.N, rows = min(kC, p.map.T - (c % p.N) * kC) - 16 * cg;
        const int64_t gk_tok = p.map.tok(kD), gk_at = p.map.base(unit / p.map.H, unit % p.map.H, kD) + ((c % p.N) * kC + 16 * cg) * gk_tok + row;
        float post = ((sum.ex[0][row] + sum.ex[1][row]) + (sum.ex[2][row] + sum.ex[3][row])) + sum.ts[row] * ex2(GL);
#pragma unroll
        for (int s = 3; s > 0; --s)
          if (s > cg) post += sum.g[s][row];
#pragma unroll
        for (int e = 0; e < 16; ++e)
          if (e < rows && in_bounds(P.status, gk_at + e * gk_tok, P.n_tok * kD)) p.dg[gk_at + e * gk_tok] = up[e] + post;
      }
      {   // each warp for its own sixteen tokens: q in the lower lanes, k in the upper ones
        // y = s x / (|x| + eps), y^ = s x r:  dx = s r dy - y^ (y^ . dy) / (s |x|)
        const int i = 16 * cg + (lane & 15);
        const float r = lane < 16 ? ctl.rq[i] : ctl.rk[i], s = lane < 16 ? p.scale : 1.f, nrm = s / r - 1e-6f;   // |x|
        sum.f[warp][lane] = p.l2norm && nrm > 0.f ? r / (s * nrm) * total(sum.row[lane >> 4], i) : 0.f;
        __syncwarp();
      }
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t u[8], w[8];
        tc::tmem_ld8(ta + tQ1 + 8 * hf, u);
        tc::tmem_ld8(ta + tKr1 + 8 * hf, w);
        tc::tc_wait_ld();
        if (p.map.Hq != p.map.H) {   // grouped heads: dq^, dk^ per head for the finalize kernel
          const int64_t at = ((int64_t)c * kC + 16 * cg + 8 * hf) * kD + row, half_n = (int64_t)P.chunks * (kC * kD);
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            if (in_bounds(P.status, at + e * kD, half_n) && in_bounds(P.status, half_n + at + e * kD, P.n_part)) {
              p.part[at + e * kD] = __uint_as_float(u[e]);
              p.part[half_n + at + e * kD] = __uint_as_float(w[e]);
            }
          }
        } else {
          float rq[8], rk[8], fq[8], fk[8];
#pragma unroll
          for (int e = 0; e < 8; e += 4) {
            *reinterpret_cast<float4*>(rq + e) = four(ctl.rq, 8 * hf + e);
            *reinterpret_cast<float4*>(rk + e) = four(ctl.rk, 8 * hf + e);
            *reinterpret_cast<float4*>(fq + e) = *reinterpret_cast<const float4*>(sum.f[warp] + 8 * hf + e);
            *reinterpret_cast<float4*>(fk + e) = *reinterpret_cast<const float4*>(sum.f[warp] + 16 + 8 * hf + e);
          }
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const int j = 8 * hf + e;
            *entry(LK_O, j) = __float2bfloat16_rn(rq[e] * __uint_as_float(u[e]) - fq[e] * half(qp[j >> 1], j));
            *entry(LK_R, j) = __float2bfloat16_rn(rk[e] * __uint_as_float(w[e]) - fk[e] * half(kp[j >> 1], j));
          }
        }
      }
      tc::tc_fence_before();
      tc::fence_async_smem();
      asm volatile("bar.sync 1, 544;" ::: "memory");
    }
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
