// Shared device/host helpers for the delta-rule kernels.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

#include "deltarule_sm100.h"

namespace dr {

// Programmatic dependent launch.  A kernel of a layer's token step runs 2-4 us, of which the start (launch, first instruction,
// first miss) is most: launch_pdl lets the grid start while its predecessor in the stream still runs, and every kernel launched
// so calls pdl_entry() before it touches global memory: it waits there until the predecessor has completed and its writes are
// visible, and lets its own successor start early in turn.  Nothing is read or written before the wait, so the order of effects
// on the stream is what it was.
__device__ __forceinline__ void pdl_entry() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <class... Params, class... Args>
inline cudaError_t launch_pdl(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// Addressing of one (batch, head) sequence inside a [B,H,T,D] or [B,T,H,D] tensor.
// Element index of token t, feature d is  base(b,h,D) + t * tok(D) + d.
struct SeqMap {
  int B, H, T;
  int bthd;  // 0: [B,H,T,D]   1: [B,T,H,D]
  int Hq;    // heads of q and k (grouped value attention: head h of v, o reads q/k head h / (H / Hq)); Hq == H: none
  __host__ __device__ inline int64_t base(int b, int h, int D) const {
    return bthd ? ((int64_t)b * T * H + h) * D : ((int64_t)b * H + h) * (int64_t)T * D;
  }
  __host__ __device__ inline int64_t tok(int D) const { return bthd ? (int64_t)H * D : D; }
  // the same for q and k
  __host__ __device__ inline int hq(int h) const { return Hq == H ? h : h / (H / Hq); }
  __host__ __device__ inline int64_t base_qk(int b, int h, int D) const {
    return bthd ? ((int64_t)b * T * Hq + hq(h)) * D : ((int64_t)b * Hq + hq(h)) * (int64_t)T * D;
  }
  __host__ __device__ inline int64_t tok_qk(int D) const { return bthd ? (int64_t)Hq * D : D; }
};

__device__ __forceinline__ float ld_elem(const void* p, int64_t i, int dt) {
  return dt == DR_BF16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i])
                       : reinterpret_cast<const float*>(p)[i];
}

__device__ __forceinline__ void st_elem(void* p, int64_t i, int dt, float x) {
  if (dt == DR_BF16)
    reinterpret_cast<__nv_bfloat16*>(p)[i] = __float2bfloat16_rn(x);
  else
    reinterpret_cast<float*>(p)[i] = x;
}

// Index checks of the debug build (-DDR_BOUNDS_CHECK, linearnexus_b200/libdeltarule_sm100_bounds.so): the kernels that
// index global memory by hand ask in_bounds() before an access; an index outside [0, n) sets DR_DEV_BOUNDS in the
// status word and the access is skipped -- never a trap, never a fault.  The release build compiles the checks away.
#ifdef DR_BOUNDS_CHECK
__device__ __forceinline__ bool in_bounds(int32_t* status, int64_t i, int64_t n) {
  if (i >= 0 && i < n) return true;
  if (status) atomicOr(status, DR_DEV_BOUNDS);
  return false;
}
#else
__device__ __forceinline__ bool in_bounds(int32_t*, int64_t, int64_t) { return true; }
#endif
// the same for `len` entries from i on (one vector access)
__device__ __forceinline__ bool in_bounds_run(int32_t* status, int64_t i, int len, int64_t n) {
  return in_bounds(status, i, n) && in_bounds(status, i + len - 1, n);
}

__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// Parameters every forward kernel takes (plain struct passed by value).
struct FwdParams {
  const void* q;
  const void* k;
  const void* v;
  const void* g;      // null for DR_DELTA
  const float* beta;
  const float* h0;    // null: zero state
  void* o;
  float* hT;          // null: not wanted
  int32_t* status;    // device status word or null
  float* ckpt;        // null, or [B*H][N][K][V]: state at the start of every chunk (backward)
  SeqMap map;
  int K, V, C;
  int variant, qkv_dt, g_dt, out_dt, l2norm;
  float scale;
  // element counts of the caller's arrays (what the index checks of the debug build compare against)
  int64_t n_qk, n_v, n_gk, n_tok, n_state, n_ckpt;
  __host__ void set_extents() {
    const int64_t bh = (int64_t)map.B * map.H, bhq = (int64_t)map.B * map.Hq;
    n_qk = bhq * map.T * K;
    n_v = bh * map.T * V;
    n_gk = bh * map.T * K;
    n_tok = bh * map.T;
    n_state = bh * K * V;
    n_ckpt = C > 0 ? bh * ((map.T + C - 1) / C) * K * V : 0;
  }
};

// The sequences of a packed batch that one launch works on, longest first (a CTA takes one sequence and head; CTAs
// start in this order, so the long sequences are under way while the short ones fill the remaining SMs).  Travels as
// a kernel parameter: no device memory, no copy.
constexpr int kMaxSeqs = 192;   // per launch; with the tensor maps the parameters stay below 4 KB
struct SeqTable {
  int n, chunks;             // sequences; chunks of all of them together
  int32_t start[kMaxSeqs];   // first token
  int32_t len[kMaxSeqs];
  int32_t index[kMaxSeqs];   // position in the caller's list (which state is its own)
  int32_t first[kMaxSeqs];   // chunks of the sequences before it in the table
};

}  // namespace dr
