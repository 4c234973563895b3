// Translation unit of the forward in transition form.
#include "dr_fwd_trans.cuh"
#include "dr_launch.h"

namespace dr {

int64_t trans_workspace_bytes(int64_t units, int T, int D) { return trans::workspace_bytes(units, T, D); }
cudaError_t launch_chunk_trans(const FwdParams& p, void* workspace, int sms, cudaStream_t stream) {
  if (p.K == 64) return trans::launch_d<64, true>(p, workspace, sms, stream);
  // bf16 rows at D = 128 stand in for kernels with bf16 operands: one tf32 product is more precise than those
  return p.qkv_dt == DR_BF16 ? trans::launch_d<128, false>(p, workspace, sms, stream) : trans::launch_d<128, true>(p, workspace, sms, stream);
}

}  // namespace dr
