// The backward's pre-pass for per-channel decays (KDA) on tcgen05: X, A, T, N and Y of a chunk from q, k, g and beta.  Formulas and names:
// headers of dr_bwd.cuh and dr_bwd_chunk.cuh.
//
// float32 operands are two bf16 terms, three products per pair: 17 bits of every entry, float32's exponents (see dr_bwd_local_kda.cuh).  With
// Kg = k^ e^G, Qg = q^ e^G, Ki = k^ e^{-G}:
//   1  [X; A] = [Kg; Qg] Ki^T, then T by blocks
//   2  W^T = Kg^T (T diag(beta))^T
//   3  Y^T = Qg^T - W^T A^T,  N = -W^T Ki diag(e^{G_L})
// The factors of a pair multiply to the pair's own decay whatever each of them is, so a chunk may decay by what their exponents have room for: 2^40
// in any channel (kWideKda).  Others, and chunks with a positive log decay, are left to pre_kernel, which refers the decays to 16-row
// blocks; the forward's first kernel, which forms the same sums before this one starts, marks them (launch_bwd_forward).
//
// One persistent CTA per SM: sixteen warps that work, one that issues.  A worker warp owns four rows of the chunk up to the tiles, a lane four
// channels of them; a thread of an epilogue one row of a product.  Rows arrive by TMA a chunk ahead, as soon as the tiles of the chunk before
// are formed; A and T leave by bulk copies, X, N and Y as whole 128-byte lines.
//
// What bounds it: B=2, T=4096, H=16 (2048 chunks): 160 us on 116 SMs, 17 K cycles per chunk, where pre_kernel takes 266 us on 148 (65 K for two chunks at a
// time: 15 K loads, 23 K for X and A, 18 K for W, Y and N).  The phases of one chunk follow each other,
// sixteen warps on one: the tensor pipe has 4 K cycles of work.  210 KB of memory per chunk are 8 K cycles at the copy rate on all SMs.
// Gradients against float64 as with pre_kernel (T's tf32 merges decide): see dr_bwd_local_kda.cuh.
#pragma once

namespace dr {
namespace bwdc {

// Kg, Qg hi, then lo: panels of 64 channels [Kg 64 rows; Qg 64 rows]; Ki hi, lo: panels [64 rows]; all in the 128-byte swizzle.  k, q (swizzled
// panels) and g as they arrive; A and T as local_sm100_kda_kernel's tiles; decay of each four rows [16][128]; X and its inverse [64][68], then
// T diag(beta) as such a tile
constexpr int PK_A = 0, PK_KI = 65536, PK_K = PK_KI + 32768, PK_Q = PK_K + kTile, PK_G = PK_Q + kTile, PK_AT = PK_G + 32768, PK_T = PK_AT + kTile;
constexpr int PK_X = PK_T + kTile, PK_TOT = PK_X + 64 * LDT * 4, PK_CTL = PK_TOT + 16 * 128 * 4;
struct PkCtl {
  uint64_t bar[4], full, free;
  alignas(16) float el[128];
  float beta[2][64];
  uint32_t tmem_base;
  int abort;
};
constexpr int PK_TOTAL = PK_CTL + sizeof(PkCtl);
static_assert(PK_TOTAL <= 232448 && PK_CTL % 16 == 0 && PK_X % 1024 == 0, "shared memory");
struct alignas(64) PreParams {
  CUtensorMap tq, tk, tg;   // panels of q and k; boxes of 64 rows of g
  Params p;
  int chunks;
  int32_t* status;
  int64_t n_tok;   // entries of the arrays with one number per token (index checks of the debug build)
};

static __global__ void __launch_bounds__(kLtThreads, 1) pre_sm100_kda_kernel(const __grid_constant__ PreParams P) {
  const Params& p = P.p;
  extern __shared__ __align__(1024) uint8_t pk_smem[];
  uint8_t* const smem = pk_smem;
  PkCtl& ctl = *reinterpret_cast<PkCtl*>(smem + PK_CTL);
  float* const sX = reinterpret_cast<float*>(smem + PK_X);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  if (warp == 16) {
    tc::tmem_alloc(tc::smem_u32(&ctl.tmem_base), 512);
    tc::tmem_relinquish();
  }
  if (tid == 0) {
    for (int i = 0; i < 4; ++i) tc::mbar_init(tc::smem_u32(&ctl.bar[i]), 1);
    tc::mbar_init(tc::smem_u32(&ctl.full), 1);
    tc::mbar_init(tc::smem_u32(&ctl.free), 1);
    tc::fence_mbar_init();
    ctl.abort = 0;
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
  ChunkList list;
  list.start(p, P.chunks, lane);
  // tensor memory: [X; A], W^T, its two terms, W^T A^T, N
  constexpr uint32_t tXA = 0, tW = 64, tWt = 128, tWA = 192, tN = 256;

  if (warp == 16) {
    // (only the low word changes: the address field does not carry into the other)
    auto adv = [](uint64_t d, uint32_t bytes) { return (d & 0xffffffff00000000ull) | ((uint32_t)d + (bytes >> 4)); };
    auto commit = [&](int i) { tc::mma_commit(tc::smem_u32(&ctl.bar[i])); };
    auto load = [&](int c, uint32_t turn) {
      const int unit = c / p.N, b = unit / p.map.H, h = unit % p.map.H, hq = p.map.hq(h), t0 = (c % p.N) * kC, rows = min(kC, p.map.T - t0);
      const int64_t at = p.map.base(b, h, 1) + (int64_t)t0 * p.map.tok(1), tok = p.map.tok(1);
      auto in = [&](int i) { return i < rows && in_bounds(P.status, at + i * tok, P.n_tok); };
      ctl.beta[turn][lane] = in(lane) ? p.beta[at + lane * tok] : 0.f;
      ctl.beta[turn][lane + 32] = in(lane + 32) ? p.beta[at + (lane + 32) * tok] : 0.f;
      __syncwarp();   // (before the barrier is armed: who waits for it sees them)
      if (tc::elect_one()) {
        const uint32_t bar = tc::smem_u32(&ctl.full);
        tc::mbar_arrive_expect_tx(bar, 2 * kTile + (p.g_dt == DR_BF16 ? 16384 : 32768));
        tc::tma_load_4d(sb + PK_G, &P.tg, 0, t0, h, b, bar);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          tc::tma_load_4d(sb + PK_K + 8192 * e, &P.tk, 64 * e, hq, t0, b, bar);
          tc::tma_load_4d(sb + PK_Q + 8192 * e, &P.tq, 64 * e, hq, t0, b, bar);
        }
      }
      __syncwarp();
    };
    int c = list.next(p, P.chunks, lane);
    if (c < P.chunks) load(c, 0);
    list_wide(p, P.chunks, lane);
    uint32_t turn = 0;
    constexpr uint32_t hi_lo[3] = {0, 1, 0}, lo_hi[3] = {0, 0, 1};   // terms of the left and of the right operand in the three products
#pragma unroll 1
    for (int next; c < P.chunks; c = next, turn ^= 1) {
      asm volatile("" : "+r"(sb), "+r"(tb));
      next = list.next(p, P.chunks, lane);
      asm volatile("bar.sync 2, 544;" ::: "memory");
      tc::tc_fence_after();
      if (tc::elect_one()) {
        const uint64_t ad = tc::smem_desc_sw128(sb + PK_A, 128, 1024), bd = tc::smem_desc_sw128(sb + PK_KI, 128, 1024);
#pragma unroll
        for (int ks = 0; ks < 8; ++ks)
#pragma unroll
          for (int x = 0; x < 3; ++x)
            tc::mma_ss(tb + tXA, adv(ad, hi_lo[x] * 32768 + (ks >> 2) * 16384 + (ks & 3) * 32), adv(bd, lo_hi[x] * kTile + (ks >> 2) * 8192 + (ks & 3) * 32),
                       tc::idesc_bf16(128, 64, 0, 0), ks + x > 0);
        commit(0);
      }
      __syncwarp();
      if (next < P.chunks) load(next, turn ^ 1);
      float* xat = p.xat + (int64_t)c * (3 * 64 * 64);
      asm volatile("bar.sync 3, 544;" ::: "memory");
      if (tc::elect_one()) tc::bulk_s2g(xat + 4096, sb + PK_AT, kTile);
      __syncwarp();
      asm volatile("bar.sync 4, 544;" ::: "memory");
      tc::tc_fence_after();
      if (tc::elect_one()) {
        const uint64_t ad = tc::smem_desc_sw128(sb + PK_A, 16384, 1024), bd = tc::smem_desc(sb + PK_X, 1024, 128);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
#pragma unroll
          for (int x = 0; x < 3; ++x)
            tc::mma_ss(tb + tW + 16 * ks, adv(ad, hi_lo[x] * 32768 + ks * 2048), adv(bd, lo_hi[x] * 8192 + ks * 2304), tc::idesc_bf16(128, 64 - 16 * ks, 1, 0), ks + x > 0);
        commit(1);
        tc::bulk_s2g(xat + 8192, sb + PK_T, kTile);
        tc::bulk_commit();
      }
      __syncwarp();
      asm volatile("bar.sync 5, 544;" ::: "memory");
      tc::tc_fence_after();
      if (tc::elect_one()) {
        const uint64_t ad = tc::smem_desc(sb + PK_AT, 1024, 128), kd = tc::smem_desc_sw128(sb + PK_KI, 8192, 1024);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
#pragma unroll
          for (int x = 0; x < 3; ++x)
            tc::mma_ts(tb + tWA + 16 * ks, tb + tWt + 32 * hi_lo[x] + 8 * ks, adv(ad, lo_hi[x] * 8192 + ks * 2304), tc::idesc_bf16(128, 64 - 16 * ks, 0, 0), ks + x > 0);
        commit(2);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
#pragma unroll
          for (int x = 0; x < 3; ++x)
            tc::mma_ts(tb + tN, tb + tWt + 32 * hi_lo[x] + 8 * ks, adv(kd, lo_hi[x] * kTile + ks * 2048), tc::idesc_bf16(128, 128, 0, 1), ks + x > 0);
        commit(3);
        tc::bulk_wait_read_all();
        sm100::mbar_arrive(tc::smem_u32(&ctl.free));   // A and T have left
      }
      __syncwarp();
    }
    tc::bulk_wait_all();
  } else {
    auto workers_sync = []() { asm volatile("bar.sync 8, 512;" ::: "memory"); };
    auto hand_over = [](int id) {
      tc::fence_async_smem();
      tc::tc_fence_before();
      asm volatile("bar.arrive %0, 544;" ::"r"(id) : "memory");
    };
    uint32_t ph = 0;
#pragma unroll 1
    for (int c = list.next(p, P.chunks, lane); c < P.chunks; c = list.next(p, P.chunks, lane), ph ^= 1) {
      int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
      asm volatile("" : "+r"(warp), "+r"(lane));
      warp = __shfl_sync(0xffffffffu, warp, 0);
      float* xat = p.xat + (int64_t)c * (3 * 64 * 64);
      // ---- the warp's four rows: prefix sums over them, norm factors ---------------------------------------------------------------------------
      // byte of this lane's four channels in row 4 warp + r of a panel: + 128 r, piece ^ row
      const int piece = (lane & 15) >> 1, own = (4 * warp) * 128 + (lane & 1) * 8;
      auto at = [&](int base, int panel, int r) {
        return reinterpret_cast<uint2*>(smem + base + (lane >> 4) * panel + own + r * 128 + ((piece ^ ((4 * warp + r) & 7)) << 4));
      };
      float4 G[4];
      float rk[4], rq[4];
      wait_at(ctl.full, ph);
      {
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          float4 x;
          if (p.g_dt == DR_BF16) {
            const uint2 u = *reinterpret_cast<const uint2*>(smem + PK_G + (4 * warp + r) * 256 + lane * 8);
            x = make_float4(mma::lo_f(u.x), mma::hi_f(u.x), mma::lo_f(u.y), mma::hi_f(u.y));
          } else {
            x = *reinterpret_cast<const float4*>(smem + PK_G + (4 * warp + r) * 512 + lane * 16);
          }
          acc.x += x.x * kLog2e; acc.y += x.y * kLog2e; acc.z += x.z * kLog2e; acc.w += x.w * kLog2e;
          G[r] = acc;
        }
        *reinterpret_cast<float4*>(smem + PK_TOT + warp * 512 + lane * 16) = acc;
        float ss[8];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const uint2 q = *at(PK_Q, 8192, r), k = *at(PK_K, 8192, r);
          const float q0 = mma::lo_f(q.x), q1 = mma::hi_f(q.x), q2 = mma::lo_f(q.y), q3 = mma::hi_f(q.y);
          const float k0 = mma::lo_f(k.x), k1 = mma::hi_f(k.x), k2 = mma::lo_f(k.y), k3 = mma::hi_f(k.y);
          ss[r] = q0 * q0 + q1 * q1 + q2 * q2 + q3 * q3;
          ss[4 + r] = k0 * k0 + k1 * k1 + k2 * k2 + k3 * k3;
        }
#pragma unroll
        for (int o = 16, m = 4; o > 2; o >>= 1, m >>= 1)
#pragma unroll
          for (int i = 0; i < m; ++i) {
            const bool high = lane & o;
            const float send = high ? ss[i] : ss[i + m], keep = high ? ss[i + m] : ss[i];
            ss[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
          }
        ss[0] += __shfl_xor_sync(0xffffffffu, ss[0], 2);
        ss[0] += __shfl_xor_sync(0xffffffffu, ss[0], 1);   // lane l: q rows l >> 2, from lane 16 on k rows
        const float s = lane < 16 ? p.scale : 1.f, m = p.l2norm ? s / (sqrtf(ss[0]) + 1e-6f) : s;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          rq[r] = __shfl_sync(0xffffffffu, m, 4 * r);
          rk[r] = __shfl_sync(0xffffffffu, m, 16 + 4 * r);
        }
        if (!(lane & 3)) {
          const int i = 4 * warp + ((lane >> 2) & 3);
          const int place = kXNorms + ((lane < 16 ? 2 : 0) + (i >> 5)) * kXNormRow + (i & 31);
          if (in_bounds(P.status, (int64_t)c * (3 * 64 * 64) + place, (int64_t)P.chunks * (3 * 64 * 64))) xat[place] = m;
        }
      }
      workers_sync();
      {
        float4 pre = make_float4(0.f, 0.f, 0.f, 0.f), run = pre;
#pragma unroll
        for (int s = 0; s < 16; ++s) {
          if (s == warp) pre = run;
          const float4 x = *reinterpret_cast<const float4*>(smem + PK_TOT + s * 512 + lane * 16);
          run.x += x.x; run.y += x.y; run.z += x.z; run.w += x.w;
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) G[r] = make_float4(G[r].x + pre.x, G[r].y + pre.y, G[r].z + pre.z, G[r].w + pre.w);
        if (warp == 0) {
          const float4 e = make_float4(ex2(run.x), ex2(run.y), ex2(run.z), ex2(run.w));
          *reinterpret_cast<float4*>(ctl.el + 4 * lane) = e;
          if (in_bounds_run(P.status, (int64_t)c * 128 + 4 * lane, 4, (int64_t)P.chunks * 128)) *reinterpret_cast<float4*>(p.el + (int64_t)c * 128 + 4 * lane) = e;
        }
      }
      {
        // ---- the tiles -----------------------------------------------------------------------------------------------------------------------
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const uint2 q = *at(PK_Q, 8192, r), k = *at(PK_K, 8192, r);
          const float gg[4] = {G[r].x, G[r].y, G[r].z, G[r].w};
          const float kh[4] = {rk[r] * mma::lo_f(k.x), rk[r] * mma::hi_f(k.x), rk[r] * mma::lo_f(k.y), rk[r] * mma::hi_f(k.y)};
          const float qh[4] = {rq[r] * mma::lo_f(q.x), rq[r] * mma::hi_f(q.x), rq[r] * mma::lo_f(q.y), rq[r] * mma::hi_f(q.y)};
          float a[4], b[4], d[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float x = ex2(gg[e]);
            a[e] = kh[e] * x;
            b[e] = qh[e] * x;
            d[e] = kh[e] * ex2(-gg[e]);
          }
          auto put = [&](int base, int panel, int lo, const float (&x)[4]) {
            uint2 u, l;
            split2(x[0], x[1], u.x, l.x);
            split2(x[2], x[3], u.y, l.y);
            *at(base, panel, r) = u;
            *at(base + lo, panel, r) = l;
          };
          put(PK_A, 16384, 32768, a);
          put(PK_A + 8192, 16384, 32768, b);
          put(PK_KI, 8192, kTile, d);
        }
      }
      hand_over(2);
      const int qd = warp & 3, cg = warp >> 2, row = 32 * qd + lane;   // this thread's row of a product and sixteen of its columns from 16 cg
      const uint32_t ta = tb + ((uint32_t)(32 * qd) << 16) + 16 * cg;
      // ---- X (rows 0 .. 63), A (rows 64 ..) --------------------------------------------------------------------------------------------------------
      {
        wait_at(ctl.bar[0], ph);
        tc::tc_fence_after();
        uint32_t u[16];
        tc::tmem_ld16(ta + tXA, u);
        tc::tc_wait_ld();
        const bool second = row >= 64;
        const int i = row & 63, last = (second ? i : i - 1) - 16 * cg;   // X is strictly below the diagonal
        float x[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) x[e] = e <= last ? __uint_as_float(u[e]) : 0.f;
        if (!second) {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float4 y = make_float4(x[4 * e], x[4 * e + 1], x[4 * e + 2], x[4 * e + 3]);
            *reinterpret_cast<float4*>(sX + i * LDT + 16 * cg + 4 * e) = y;
            if (cg <= (i >> 4) && in_bounds(P.status, (int64_t)c * (3 * 64 * 16) + (4 * cg + e) * 64 + i, (int64_t)P.chunks * (3 * 64 * 16)))
              reinterpret_cast<float4*>(xat)[(4 * cg + e) * 64 + i] = y;   // columns in fours
          }
        }
        workers_sync();   // (X for the inverse)
        if (second) {
          wait_at(ctl.free, ph ^ 1);   // the chunk before's has left
#pragma unroll
          for (int hf = 0; hf < 2; ++hf) {
            uint32_t h[4], l[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) split2(x[8 * hf + 2 * e], x[8 * hf + 2 * e + 1], h[e], l[e]);
            uint4* dst = reinterpret_cast<uint4*>(smem + PK_AT) + (2 * cg + hf) * 64 + i;
            dst[0] = make_uint4(h[0], h[1], h[2], h[3]);
            dst[512] = make_uint4(l[0], l[1], l[2], l[3]);
          }
        }
        hand_over(3);
      }
      // ---- T in place (eight warps), then T - I and T diag(beta) as tiles ----------------------------------------------------------------------------
      const float* beta = ctl.beta[ph];
      if (warp < 8) sm100::block_inverse_64(sX, beta, sX, 32 * warp + lane);
      workers_sync();
      {
        const int i = 32 * warp + lane, r = 8 * ((i >> 3) & 7) + (i & 7), cc = 8 * (i >> 6);
        float x[8], y[8];
        *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(sX + r * LDT + cc);
        *reinterpret_cast<float4*>(x + 4) = *reinterpret_cast<const float4*>(sX + r * LDT + cc + 4);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          x[e] = cc + e <= r ? x[e] : 0.f;
          y[e] = x[e] * beta[cc + e];
        }
        workers_sync();   // T has been read
        wait_at(ctl.free, ph ^ 1);
        uint32_t h[4], l[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) split2(cc + 2 * e < r ? x[2 * e] : 0.f, cc + 2 * e + 1 < r ? x[2 * e + 1] : 0.f, h[e], l[e]);
        reinterpret_cast<uint4*>(smem + PK_T)[i] = make_uint4(h[0], h[1], h[2], h[3]);
        reinterpret_cast<uint4*>(smem + PK_T)[512 + i] = make_uint4(l[0], l[1], l[2], l[3]);
#pragma unroll
        for (int e = 0; e < 4; ++e) split2(y[2 * e], y[2 * e + 1], h[e], l[e]);
        reinterpret_cast<uint4*>(smem + PK_X)[i] = make_uint4(h[0], h[1], h[2], h[3]);
        reinterpret_cast<uint4*>(smem + PK_X)[512 + i] = make_uint4(l[0], l[1], l[2], l[3]);
      }
      hand_over(4);
      // ---- W^T: row = channel; its terms in tensor memory -------------------------------------------------------------------------------------
      {
        wait_at(ctl.bar[1], ph);
        tc::tc_fence_after();
        uint32_t u[16];
        tc::tmem_ld16(ta + tW, u);
        tc::tc_wait_ld();
        uint32_t h[8], l[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) split2(__uint_as_float(u[2 * e]), __uint_as_float(u[2 * e + 1]), h[e], l[e]);
        tc::tmem_st8(ta - 8 * cg + tWt, h);
        tc::tmem_st8(ta - 8 * cg + tWt + 32, l);
        tc::tc_wait_st();
      }
      hand_over(5);
      // ---- Y^T = Qg^T - W^T A^T ------------------------------------------------------------------------------------------------------------------
      {
        float y[16];
        const uint32_t el = (row >> 6) * 16384 + 8192 + 16 * cg * 128 + ((row >> 3) & 7) * 16 + (row & 7) * 2;
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const uint8_t* src = smem + PK_A + (el ^ ((e & 7) << 4)) + 128 * e;
          y[e] = bf(reinterpret_cast<const __nv_bfloat16*>(src)) + bf(reinterpret_cast<const __nv_bfloat16*>(src + 32768));
        }
        wait_at(ctl.bar[2], ph);
        tc::tc_fence_after();
        uint32_t u[16];
        tc::tmem_ld16(ta + tWA, u);
        tc::tc_wait_ld();
        const int64_t dst = (int64_t)c * kHalf4 + (row >> 3) * 64 + 2 * cg * 8 + (row & 7);   // see store_f32
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (in_bounds(P.status, dst + (e & 1) * (kHalf4 / 2) + (e >> 1) * 8, (int64_t)P.chunks * kHalf4))
            p.yf[dst + (e & 1) * (kHalf4 / 2) + (e >> 1) * 8] = make_float4(y[4 * e] - __uint_as_float(u[4 * e]), y[4 * e + 1] - __uint_as_float(u[4 * e + 1]),
                                                                   y[4 * e + 2] - __uint_as_float(u[4 * e + 2]), y[4 * e + 3] - __uint_as_float(u[4 * e + 3]));
      }
      // ---- N = -W^T Ki diag(e^{G_L}): thread = 32 columns -----------------------------------------------------------------------------------------
      {
        wait_at(ctl.bar[3], ph);
        tc::tc_fence_after();
        const int64_t dst = (2 * (int64_t)c + (cg >> 1)) * kHalf4 + (row >> 3) * 64 + 4 * (cg & 1) * 8 + (row & 7);
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          uint32_t u[16];
          tc::tmem_ld16(ta + 16 * cg + tN + 16 * x, u);
          tc::tc_wait_ld();
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float4 d = *reinterpret_cast<const float4*>(ctl.el + 32 * cg + 16 * x + 4 * e);
            const int64_t at = dst + (e & 1) * (kHalf4 / 2) + (2 * x + (e >> 1)) * 8;
            if (in_bounds(P.status, at, 2 * (int64_t)P.chunks * kHalf4))
              p.nf[at] = make_float4(-__uint_as_float(u[4 * e]) * d.x, -__uint_as_float(u[4 * e + 1]) * d.y, -__uint_as_float(u[4 * e + 2]) * d.z,
                            -__uint_as_float(u[4 * e + 3]) * d.w);
          }
        }
      }
      workers_sync();   // e^{G_L} and the rows' totals have been read
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
