// RWKV-7 (diagonal plus low rank) and RWKV-6 scans, eight tokens per step of the state, on the warp-level tensor cores in
// float32 precision (three tf32 products per pair, dr_tf32.cuh); K = 64, value columns in multiples of 64, bf16 or float32 storage.
//
// With W_i the product of the block's decays up to token i, h the state at its start and u_i = a_i^T h_{i-1}:
//     u_i = (a_i W_{i-1})^T h + sum_{j<i} ak_ij v_j + ab_ij u_j        ak_ij = sum_c a_i (W_{i-1} / W_j) k_j,  ab: with b_j
//     o_i = (q_i W_i)^T h     + sum_{j<=i} qk_ij v_j + qb_ij u_j        qk_ij = sum_c q_i (W_i / W_j) k_j,      qb: with b_j
//     h'  = W_7 h + sum_j (W_7 / W_j k_j) v_j^T + (W_7 / W_j b_j) u_j^T
// so U = T D_a + (T ak) V with T = (I - ab)^-1 [8 x 8].  RWKV-6 (o_i reads h_{i-1}, a bonus u q.k on the current token, no a, b) is
// the same without U.
//
// Eight warps keep the state transposed in accumulators (16 value columns x 32 keys each; the two warps of a column block
// exchange their partial dots).  An accumulator is, register for register, an A operand whose contraction runs over its columns: h
// feeds the dots, their result feeds T, U feeds the update, and nothing of the state touches memory.  Three groups of four warps
// (RWKV-6: four) stage the blocks ahead in turn: raw rows from a ring of asynchronous copies, decay products, the row vectors and
// the 8 x 8 coefficients.  A filled stage is handed over by a named barrier, arrived on by its group and waited for by the state's
// warps; an emptied one by an mbarrier (see kEmptyTries).
//
// What bounds it: the chain of a block through the dots, U and the update, 2.6 K cycles with the schedulers 55 % and the tensor pipe 35 %
// busy (B=8, T=4096, H=16: 868 us with four warps of 64 keys and products in source order, 820 with them free to move, 785
// with eight warps, 761 with the B operands split once by the staging warps; two staging groups instead of three: 872; 690 with
// running products in blocks of too strong a decay; 681 with the stages handed back by mbarriers).
// The token recurrence it replaces here ran
// at 540 cycles per token whatever its instruction count or prefetch depth: one dependent reduce-and-update chain per token, and
// 260 shared-memory wavefronts per token to feed 160 multiply-adds per thread (a 16-byte load fills a quarter of a warp per
// wavefront, broadcast or not).  A four-token form on the CUDA cores stayed at that roof (1.18 ms against 1.14).
#pragma once

#include "dr_linrec.cuh"
#include "dr_mma.cuh"
#include "dr_sm100_common.cuh"
#include "dr_tcgen05.cuh"
#include "dr_tf32.cuh"

namespace dr {
namespace rwkv {

using mma::AFrag;
using mma::BFrag;
constexpr int kK = 64, kTB = 8, kGroups = 3, kRing = 3, kStages = 4, kCons = 256;
// Staging groups.  RWKV-6 has less of a chain per block (no U), so there a fourth pays: B=8, T=4096, H=16 764 -> 718 us, B=2, T=500 97.9 ->
// 92.7; RWKV-7 681 -> 692.  float32 rows leave room for three.
template <int KIND, bool BF> constexpr int groups_of = KIND == LR_RWKV6 && BF ? 4 : kGroups;
template <int KIND, bool BF> constexpr int threads_of = kCons + 128 * groups_of<KIND, BF>;
constexpr int kHand = kCons + 128;   // threads of a hand-over barrier: the consumers and one staging group
constexpr int LDR = 72;    // row vectors [token][key], read as B operands along the key axis
constexpr int LDU = 66;    // update vectors [token pair][key], read across tokens
constexpr int LDH = 68;    // values [token][column], read across tokens

template <int KIND, bool BF>
struct Ring {
  static constexpr int NV = KIND == LR_DPLR ? 5 : 3;            // q k w [a b]
  static constexpr int ES = BF ? 2 : 4;
  static constexpr int kVec = kTB * kK * ES;                    // bytes of one vector's block
  static constexpr int kTasks = (NV + 1) * kVec / 512;          // warps' worth of 16-byte pieces (v last)
  static constexpr int kSlot = (NV + 1) * kVec;
};

// What the consumers read as B operands is stored split into its two tf32 terms, once, by the staging warps (four warps of value
// columns read each; splitting it there was a third of their instructions), in the order of a fragment: one 16-byte read each.
struct Stage {
  float2 row[16][LDR];      // (hi, lo); 0-7: q W (RWKV-6: q W_{i-1});  8-15: a W_{i-1}
  float4 upd[8][LDU];       // token pairs (hi, hi, lo, lo); 0-3: W_7 / W_j k;  4-7: W_7 / W_j b
  float4 qk[32], qb[32], T[32], P[32];   // [i][j / 2], (hi, hi, lo, lo) of j, j + 1; P = T ak
  float v[kTB][LDH];
  float w[kK];              // W_7
};
__device__ __forceinline__ float2 split(float x) {
  const float hi = __uint_as_float((__float_as_uint(x) + 0x1000u) & 0xffffe000u);
  return make_float2(hi, x - hi);
}
__device__ __forceinline__ float4 split2(float x, float y) {
  const float2 a = split(x), b = split(y);
  return make_float4(a.x, b.x, a.y, b.y);
}
__device__ __forceinline__ BFrag<true> frag(float4 x) {   // of a pair stored by split2
  BFrag<true> b;
  b.h[0] = __float_as_uint(x.x); b.h[1] = __float_as_uint(x.y);
  b.l[0] = __float_as_uint(x.z); b.l[1] = __float_as_uint(x.w);
  return b;
}
__device__ __forceinline__ void put(float4* m, int i, int j, float x) {   // one entry of an 8 x 8 coefficient matrix
  const float2 a = split(x);
  float* at = reinterpret_cast<float*>(m + 4 * i + (j >> 1)) + (j & 1);
  at[0] = a.x; at[2] = a.y;
}

using Exchange = float[2][4][2][2][32][4];   // [block parity][16 value columns][key half][q, a][lane][entry]: partial dots

struct Scratch {            // of one staging group
  float inv[16][LDR];       // k / W_j, b / W_j
  float ab[64], ak[64], T[64];
  int wide;
};
template <int KIND, bool BF>
constexpr int kGroupBytes = ((int)sizeof(Scratch) + 15) / 16 * 16 + kRing * Ring<KIND, BF>::kSlot;
template <int KIND, bool BF>   // then one mbarrier per stage
constexpr int kEmptyAt = kStages * (int)sizeof(Stage) + (int)sizeof(Exchange) + groups_of<KIND, BF> * kGroupBytes<KIND, BF>;
template <int KIND, bool BF>
constexpr int kSmemBytes = kEmptyAt<KIND, BF> + kStages * 8;
static_assert(kEmptyAt<LR_DPLR, false> % 8 == 0 && kEmptyAt<LR_RWKV6, true> % 8 == 0 && kSmemBytes<LR_DPLR, false> <= 232448 && kSmemBytes<LR_RWKV6, true> <= 232448, "227 KB per CTA");

__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory"); }
constexpr int kBarFull = 1, kBarGroup = 1 + kStages, kBarPair = kBarGroup + groups_of<LR_RWKV6, true>;
static_assert(kBarPair + 4 <= 16, "named barriers");
// With three groups a stage passes from group to group (kStages is no multiple of kGroups), so "the consumers have left stage s for the n-th time" is
// phase n of an mbarrier: a named barrier has no phases, and two groups would meet on it in either order.  The group of block blk
// waits for phase blk / kStages - 1.  It cannot be a phase behind (phase blk / kStages needs blk staged first), nor a phase ahead:
// its last block, blk - kGroups, was staged after every warp had left blk - kGroups - kStages, so after it had arrived for the phase
// before.
// Measured against the named barriers it replaces (which could be passed out of order): RWKV-7 B=8, T=4096, H=16 685 -> 681 us, B=1,
// T=2048, H=8 345 -> 342; RWKV-6 B=4, T=2048, H=16 380 -> 386.  Every thread of the group waits: one waiting for the others took
// 2.2 % more.  Three stages, each of one group, with named barriers: 710, 356, 430.
constexpr uint32_t kEmptyTries = 1u << 20;   // and about a second of clock

// a float32-precise product whose terms go to three accumulators (hi hi, lo hi, hi lo)
__device__ __forceinline__ void fma3(float (&d)[3][4], const AFrag<true>& a, const BFrag<true>& b) {
  mma::tf32(d[1], a.l, b.h);
  mma::tf32(d[2], a.h, b.l);
  mma::tf32(d[0], a.h, b.h);
}

template <int KIND, bool BF>
__global__ void __launch_bounds__(threads_of<KIND, BF>, 1) rwkv_chunk_kernel(const LinRecParams p) {
  pdl_entry();
  using R = Ring<KIND, BF>;
  constexpr bool LR = KIND == LR_DPLR;
  constexpr int kGroups = groups_of<KIND, BF>;
  constexpr int NV = R::NV;
  extern __shared__ __align__(16) uint8_t smem[];
  static_assert(sizeof(Stage) % 16 == 0, "stages stay aligned");
  Stage* s_st = reinterpret_cast<Stage*>(smem);
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int nvs = p.V / 64, unit = blockIdx.x / nvs, v0 = (blockIdx.x % nvs) * 64;
  const int b = unit / p.H, h = unit % p.H, T = p.T, nblk = (T + kTB - 1) / kTB;
  const uint32_t empty = tc::smem_u32(smem + kEmptyAt<KIND, BF>);
  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) tc::mbar_init(empty + 8 * i, kCons / 32);
    tc::fence_mbar_init();
  }
  __syncthreads();

  if (threadIdx.x >= kCons) {
    // =========================== staging =========================================================================================
    const int grp = (threadIdx.x - kCons) >> 7, tid = threadIdx.x & 127, warp = tid >> 5;
    uint8_t* mine = smem + kStages * sizeof(Stage) + sizeof(Exchange) + grp * kGroupBytes<KIND, BF>;
    Scratch& X = *reinterpret_cast<Scratch*>(mine);
    uint8_t* ring = mine + (sizeof(Scratch) + 15) / 16 * 16;
    constexpr int kRounds = (R::kTasks + 3) / 4;
    const uint8_t* src[kRounds];
    int64_t step[kRounds], at0[kRounds], size[kRounds];   // (the last two: index checks of the debug build)
    int rtok[kRounds];
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
      const int byte = (warp + 4 * r) * 512 + lane * 16, j = byte / R::kVec, off = byte % R::kVec;
      const LrVec* vecs[5] = {&p.q, &p.k, &p.w, &p.a, &p.b};
      const void* ptr = p.v.p;
      int64_t st = p.v.st, at = p.v.at(b, h, 0) + v0, n = p.v.n;
#pragma unroll
      for (int jj = 0; jj < NV; ++jj)
        if (jj == j) { ptr = vecs[jj]->p; st = vecs[jj]->st; at = vecs[jj]->at(b, h, 0); n = vecs[jj]->n; }
      rtok[r] = off / (kK * R::ES);
      src[r] = reinterpret_cast<const uint8_t*>(ptr) + (at + rtok[r] * st) * R::ES + off % (kK * R::ES);
      step[r] = (int64_t)kTB * st * R::ES;
      at0[r] = at + rtok[r] * st + off % (kK * R::ES) / R::ES;
      size[r] = n;
    }
    auto issue = [&](int blk) {   // blocks of this group: blk = grp, grp + kGroups, ...
      if (blk * kTB < T) {
        const uint32_t slot = tc::smem_u32(ring + (blk / kGroups % kRing) * R::kSlot) + (uint32_t)(warp * 512 + lane * 16);
#pragma unroll
        for (int r = 0; r < kRounds; ++r) {
          if (warp + 4 * r < R::kTasks) {
            const bool ok = blk * kTB + rtok[r] < T && in_bounds_run(p.status, at0[r] + blk * (step[r] / R::ES), 16 / R::ES, size[r]);
            tc::cp_async16(slot + 2048u * r, src[r] + (ok ? blk * step[r] : 0), ok);
          }
        }
      }
      tc::cp_async_commit();
    };
    auto sync128 = [&]() { bar_sync(kBarGroup + grp, 128); };
    auto raw = [&](const uint8_t* slot, int j, int tok, int c) -> float {
      const uint8_t* a = slot + j * R::kVec + (tok * kK + c) * R::ES;
      return BF ? __uint_as_float((uint32_t)*reinterpret_cast<const uint16_t*>(a) << 16) : *reinterpret_cast<const float*>(a);
    };
    const int ch = tid & 63, role = tid >> 6;   // role 0: q rows and k vectors; role 1: a rows and b vectors (RWKV-6: values)
    const float u_ch = !LR ? p.u[(int64_t)h * kK + ch] : 0.f;
#pragma unroll
    for (int i = 0; i < kRing; ++i) issue(grp + kGroups * i);
    for (int blk = grp; blk < nblk; blk += kGroups) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kRing - 1) : "memory");
      if (tid == 0) X.wide = 0;
      if (blk >= kStages &&   // the consumers have left this stage
          !tc::mbar_wait_compact(empty + 8 * (blk % kStages), (blk / kStages - 1) & 1, kEmptyTries) && p.status)
        atomicOr(p.status, DR_DEV_TIMEOUT);
      sync128();   // every thread's pieces of this block have landed
      const uint8_t* slot = ring + (blk / kGroups % kRing) * R::kSlot;
      Stage& S = s_st[blk % kStages];
      const int t0 = blk * kTB;
      if (LR || role == 0) {
        float w[8], y[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float x = raw(slot, 2, i, ch);
          w[i] = t0 + i < T ? (LR ? expf(x) : expf(-expf(x))) : 1.f;   // tokens past the end: decay 1, zero vectors
        }
        float W = 1.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          float x;
          if (LR) x = role == 0 ? raw(slot, 0, i, ch) * p.scale : raw(slot, 3, i, ch);
          else x = t0 + i < T ? p.scale / (1.f + __expf(-raw(slot, 0, i, ch))) : 0.f;   // sigmoid(r) scale
          if (LR && role == 0) W *= w[i];
          S.row[8 * role + i][ch] = split(x * W);
          if (!(LR && role == 0)) W *= w[i];
          y[i] = raw(slot, LR && role == 1 ? 4 : 1, i, ch);
        }
        if (role == 0) {
          S.w[ch] = W;
          if (!(W >= 5.4e-20f)) X.wide = 1;   // 2^-64: too wide for the form with 1 / W_j below
        }
        float D = 1.f;
#pragma unroll
        for (int j = 7; j >= 0; j -= 2) {
          const float hi = y[j] * D;
          D *= w[j];
          S.upd[4 * role + (j >> 1)][ch] = split2(y[j - 1] * D, hi);
          D *= w[j - 1];
        }
        float I = 1.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          I *= __fdividef(1.f, w[j]);
          X.inv[8 * role + j][ch] = y[j] * I;
        }
      }
      // values (RWKV-6: by the threads without row work)
      if (LR) {
#pragma unroll
        for (int e = 0; e < 4; ++e) S.v[(tid >> 6) + 2 * e][ch] = raw(slot, NV, (tid >> 6) + 2 * e, ch);
      } else if (role == 1) {
#pragma unroll
        for (int e = 0; e < 8; ++e) S.v[e][ch] = raw(slot, NV, e, ch);
      }
      sync128();
      // ---- coefficients: rows q (and a) against k / W (warp 0) and b / W (warp 1) ----------------------------------------------------
      if (X.wide) {
        // too strong a decay: the decays between two tokens multiplied up.  Four lanes per (row kind, vector kind, j), sixteen channels
        // each, the product running over i (with every pair on its own, and its exponentials, such a block took 35 us)
        if (role == 0) {
#pragma unroll
          for (int i = 0; i < 8; ++i) {   // the decays take the place of k / W_j, which is not used
            const float x = raw(slot, 2, i, ch);
            X.inv[i][ch] = t0 + i < T ? (LR ? expf(x) : expf(-expf(x))) : 1.f;
          }
        }
        sync128();
        const int item = tid >> 2, isa = item >> 4, which = (item >> 3) & 1, j = item & 7;
        if (LR || item < 8) {
          const bool incl = LR && !isa;   // q reads the state after token i's decay; a (and RWKV-6) the one before
          float acc[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[i] = 0.f;
          for (int c = tid & 3; c < kK; c += 4) {
            float x = raw(slot, which ? 4 : 1, j, c);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float w = i > j ? X.inv[i][c] : 1.f;
              if (incl) x *= w;
              float q = raw(slot, isa ? 3 : 0, i, c);
              if (!isa) q = LR ? q * p.scale : p.scale / (1.f + __expf(-q));
              acc[i] += q * x;
              if (!incl) x *= w;
            }
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], 1);
            acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], 2);
            if ((tid & 3) == 0) {
              const float v = (incl ? i >= j : i > j) && t0 + i < T ? acc[i] : 0.f;
              if (isa) (which ? X.ab : X.ak)[8 * i + j] = v;
              else put(which ? S.qb : S.qk, i, j, v);
            }
          }
        }
      } else if (warp < (LR ? 2 : 1)) {
        float d[4] = {0.f, 0.f, 0.f, 0.f}, d2[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int ks = 0; ks < 8; ++ks) {
          const float4 x0 = *reinterpret_cast<const float4*>(&S.row[g][8 * ks + 2 * t]);
          const float4 x1 = LR ? *reinterpret_cast<const float4*>(&S.row[8 + g][8 * ks + 2 * t]) : make_float4(0.f, 0.f, 0.f, 0.f);
          const float2 y = *reinterpret_cast<const float2*>(&X.inv[8 * warp + g][8 * ks + 2 * t]);
          AFrag<true> a;
          a.h[0] = __float_as_uint(x0.x); a.h[1] = __float_as_uint(x1.x); a.h[2] = __float_as_uint(x0.z); a.h[3] = __float_as_uint(x1.z);
          a.l[0] = __float_as_uint(x0.y); a.l[1] = __float_as_uint(x1.y); a.l[2] = __float_as_uint(x0.w); a.l[3] = __float_as_uint(x1.w);
          BFrag<true> bb;
          bb.set(y.x, y.y);
          mma::fma<true>((ks & 1) ? d2 : d, a, bb);
        }
        float q[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int i = g, j = 2 * t + e;
          const float a = d[2 + e] + d2[2 + e];
          q[e] = (LR ? j <= i : j < i) ? d[e] + d2[e] : 0.f;
          if (LR) (warp ? X.ab : X.ak)[8 * i + j] = j < i ? a : 0.f;
        }
        (warp ? S.qb : S.qk)[lane] = split2(q[0], q[1]);
      }
      if (LR) {
        sync128();
        // T = (I - ab)^-1 by columns (eight lanes), P = T ak
        if (warp == 0) {
          if (lane < 8) {
            float x[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              x[i] = i == lane ? 1.f : 0.f;
#pragma unroll
              for (int j = 0; j < 8; ++j)
                if (j < i) x[i] += X.ab[8 * i + j] * x[j];
              X.T[8 * i + lane] = x[i];
              put(S.T, i, lane, x[i]);
            }
          }
          __syncwarp();
#pragma unroll
          for (int e = lane; e < 64; e += 32) {
            float acc = 0.f;
#pragma unroll
            for (int j = 0; j < 8; ++j) acc += X.T[(e & ~7) + j] * X.ak[8 * j + (e & 7)];
            put(S.P, e >> 3, e & 7, acc);
          }
        }
      } else {
        // the bonus on the current token: u q.k, eight sums over the channels (two warps' halves meet through X.ab)
        if (role == 0) {
          float x[8];
#pragma unroll
          for (int i = 0; i < 8; ++i)
            x[i] = t0 + i < T ? p.scale / (1.f + __expf(-raw(slot, 0, i, ch))) * u_ch * raw(slot, 1, i, ch) : 0.f;
#pragma unroll
          for (int m = 4; m >= 1; m >>= 1) {
            const bool up = lane & m;
#pragma unroll
            for (int i = 0; i < m; ++i) {
              const float send = up ? x[i] : x[i + m], keep = up ? x[i + m] : x[i];
              x[i] = keep + __shfl_xor_sync(0xffffffffu, send, m);
            }
          }
          x[0] += __shfl_xor_sync(0xffffffffu, x[0], 8);
          x[0] += __shfl_xor_sync(0xffffffffu, x[0], 16);
          if (lane < 8) X.ab[8 * warp + lane] = x[0];
        }
        sync128();
        if (tid < 8) put(S.qk, tid, tid, X.ab[tid] + X.ab[8 + tid]);
      }
      bar_arrive(kBarFull + blk % kStages, kHand);
      sync128();           // the raw block has been read by every thread
      issue(blk + kGroups * kRing);
    }
    return;
  }

  // =========================== the state: warp = 16 value columns, 32 keys ==============================================================
  const int cw = threadIdx.x >> 5, pair = cw & 3, half = cw >> 2, vb = 16 * pair, kb = 32 * half;
  Exchange& ex = *reinterpret_cast<Exchange*>(smem + kStages * sizeof(Stage));
  float S[4][4];   // tile nt: columns vb + g, + 8 (rows), keys kb + 8 nt + 2 t, + 1
  const float* h0 = p.h0 ? p.h0 + (int64_t)unit * kK * p.V + v0 + vb + g : nullptr;
#pragma unroll
  for (int nt = 0; nt < 4; ++nt)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int64_t at = (int64_t)(kb + 8 * nt + 2 * t + (e & 1)) * p.V + 8 * (e >> 1);
      S[nt][e] = h0 && in_bounds(p.status, (h0 - p.h0) + at, p.n_state) ? h0[at] : 0.f;
    }
  const int64_t o_at = (int64_t)b * p.o_sb + (int64_t)h * p.o_sh + v0 + vb + g;
  for (int blk = 0; blk < nblk; ++blk) {
    bar_sync(kBarFull + blk % kStages, kHand);
    const Stage& St = s_st[blk % kStages];
    const bool out = (blk & 1) == half;   // this warp's turn to form the block's output
    // this half's part of the dots of q (and a) with h, transposed: rows = columns of v, columns = tokens.  The three terms of
    // a float32 product go to accumulators of their own: four dependent products deep instead of twelve
    float dq[3][4], da[3][4];
#pragma unroll
    for (int x = 0; x < 3; ++x) { dq[x][0] = dq[x][1] = dq[x][2] = dq[x][3] = 0.f; da[x][0] = da[x][1] = da[x][2] = da[x][3] = 0.f; }
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      AFrag<true> a;
      a.set(S[ks][0], S[ks][2], S[ks][1], S[ks][3]);
      auto row = [&](int r) {   // two keys, each (hi, lo)
        const float4 y = *reinterpret_cast<const float4*>(&St.row[r][kb + 8 * ks + 2 * t]);
        return frag(make_float4(y.x, y.z, y.y, y.w));
      };
      fma3(dq, a, row(g));
      if constexpr (LR) fma3(da, a, row(8 + g));
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) { dq[0][e] += dq[1][e] + dq[2][e]; da[0][e] += da[1][e] + da[2][e]; }
    auto& mine = ex[blk & 1][pair][half];
    const auto& other = ex[blk & 1][pair][half ^ 1];
    *reinterpret_cast<float4*>(mine[0][lane]) = make_float4(dq[0][0], dq[0][1], dq[0][2], dq[0][3]);
    if constexpr (LR) *reinterpret_cast<float4*>(mine[1][lane]) = make_float4(da[0][0], da[0][1], da[0][2], da[0][3]);
    // decay of h and the values' update: independent of the dots
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
      const float2 w = *reinterpret_cast<const float2*>(&St.w[kb + 8 * nt + 2 * t]);
      S[nt][0] *= w.x; S[nt][1] *= w.y; S[nt][2] *= w.x; S[nt][3] *= w.y;
    }
    AFrag<true> av;   // V^T: rows = columns of v, k = tokens (bf16 values are exact in one term)
    av.set(St.v[2 * t][vb + g], St.v[2 * t][vb + g + 8], St.v[2 * t + 1][vb + g], St.v[2 * t + 1][vb + g + 8]);
    auto mul_v = [&](float (&d)[4], const BFrag<true>& bb) {
      if constexpr (BF) {
        mma::tf32(d, av.h, bb.l);
        mma::tf32(d, av.h, bb.h);
      } else {
        mma::fma<true>(d, av, bb);
      }
    };
    auto small = [&](const float4* m) { return frag(m[lane]); };   // an 8 x 8 coefficient matrix [i][j] as B operand (k = j, n = i)
    float o[4] = {0.f, 0.f, 0.f, 0.f}, u[3][4];
#pragma unroll
    for (int x = 0; x < 3; ++x) u[x][0] = u[x][1] = u[x][2] = u[x][3] = 0.f;
    if constexpr (LR) mul_v(u[0], small(St.P));
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {   // h += V^T (W_7 / W_j k)
      mul_v(S[nt], frag(St.upd[t][kb + 8 * nt + g]));
    }
    if (out) mul_v(o, small(St.qk));
    bar_sync(kBarPair + pair, 64);   // (two buffers: a warp is at most one block ahead of its partner)
    if (out) {
      const float4 x = *reinterpret_cast<const float4*>(other[0][lane]);
      o[0] += dq[0][0] + x.x; o[1] += dq[0][1] + x.y; o[2] += dq[0][2] + x.z; o[3] += dq[0][3] + x.w;
    }
    if constexpr (LR) {
      const float4 x = *reinterpret_cast<const float4*>(other[1][lane]);
      AFrag<true> aa;
      aa.set(da[0][0] + x.x, da[0][2] + x.z, da[0][1] + x.y, da[0][3] + x.w);
      fma3(u, aa, small(St.T));
      AFrag<true> au;
      au.set(u[0][0] + (u[1][0] + u[2][0]), u[0][2] + (u[1][2] + u[2][2]), u[0][1] + (u[1][1] + u[2][1]), u[0][3] + (u[1][3] + u[2][3]));
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {   // h += U^T (W_7 / W_j b)
        mma::fma<true>(S[nt], au, frag(St.upd[4 + t][kb + 8 * nt + g]));
      }
      if (out) mma::fma<true>(o, au, small(St.qb));
    }
    __syncwarp();
    if (lane == 0) sm100::mbar_arrive(empty + 8 * (blk % kStages));
    if (out) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int tok = blk * kTB + 2 * t + (e & 1);
        if (tok < T && in_bounds(p.status, o_at + (int64_t)tok * p.o_st + 8 * (e >> 1), p.n_o))
          st_elem(p.o, o_at + (int64_t)tok * p.o_st + 8 * (e >> 1), BF ? DR_BF16 : DR_F32, o[e]);
      }
    }
  }
  if (p.hT) {
    float* hT = p.hT + (int64_t)unit * kK * p.V + v0 + vb + g;
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int64_t at = (int64_t)(kb + 8 * nt + 2 * t + (e & 1)) * p.V + 8 * (e >> 1);
        if (in_bounds(p.status, (hT - p.hT) + at, p.n_state)) hT[at] = S[nt][e];
      }
  }
}

// 16-byte-aligned rows of K = 64 and whole 64-column slices; a decode step (one block) stays with the token kernel.  While every slice
// has an SM the blocks win from the second on (8 to 144 slices: 7.2 against 9.4 us at T = 9, 8.1 against 10.7 at 16, 17 against 25
// at 64).  This kernel fills an SM, the token recurrence's CTAs share one: in several waves the blocks win late, at about 20 tokens per
// wave (two waves: 17.8 against 16.8 us at T = 24, 24.3 against 27.0 at 48; three: 37.6 against 35.2 at 48, 76.6 against 80.4 at 128;
// seven: 105 against 95 at 64, 180 against 178 at 128, 622 against 670 at 512).
// RWKV-6 has no reduction on its token chain, and the token recurrence stays level or ahead in several waves (256 slices: 747
// against 759 us at T = 2048, 194 against 198 at 512).
inline bool eligible(int kind, bool bf, const LinRecParams& p, int sms) {
  const int64_t waves = sms > 0 ? ((int64_t)p.B * p.H * (p.V / 64) + sms - 1) / sms : 1;
  if (waves > 1 && (kind != LR_DPLR || p.T < 20 * waves)) return false;
  const int ep = bf ? 8 : 4;
  auto ok = [&](const LrVec& v) { return (reinterpret_cast<uintptr_t>(v.p) & 15) == 0 && v.sb % ep == 0 && v.sh % ep == 0 && v.st % ep == 0; };
  return p.K == kK && p.V % 64 == 0 && p.T > kTB && p.s_v == 1 && ok(p.q) && ok(p.k) && ok(p.w) && ok(p.v) &&
         (kind != LR_DPLR || (ok(p.a) && ok(p.b)));
}

template <int KIND, bool BF>
inline cudaError_t launch_t(const LinRecParams& p, cudaStream_t stream) {
  constexpr int bytes = kSmemBytes<KIND, BF>;
  auto kern = rwkv_chunk_kernel<KIND, BF>;
  thread_local int attr_dev = -1;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (attr_dev != dev) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    attr_dev = dev;
  }
  return launch_pdl(kern, dim3((unsigned)((int64_t)p.B * p.H * (p.V / 64))), dim3(threads_of<KIND, BF>), bytes, stream, p);
}
inline cudaError_t launch(int kind, bool bf, const LinRecParams& p, cudaStream_t stream) {
  if (kind == LR_DPLR) return bf ? launch_t<LR_DPLR, true>(p, stream) : launch_t<LR_DPLR, false>(p, stream);
  return bf ? launch_t<LR_RWKV6, true>(p, stream) : launch_t<LR_RWKV6, false>(p, stream);
}

}  // namespace rwkv
}  // namespace dr
