// Translation unit of the forward in transition form.
#include "dr_fwd_trans.cuh"
#include "dr_launch.h"

namespace dr {

int64_t trans_workspace_bytes(int64_t units, int T, int D, bool bf16_tensor) {
  return bf16_tensor ? trans_bf16_workspace_bytes(units, T) : trans::workspace_bytes(units, T, D);
}
cudaError_t launch_chunk_trans(const FwdParams& p, bool bf16_tensor, void* workspace, int sms, cudaStream_t stream) {
  if (bf16_tensor) return launch_chunk_trans_bf16(p, workspace, sms, stream);
  return p.K == 64 ? trans::launch_d<64>(p, workspace, sms, stream) : trans::launch_d<128>(p, workspace, sms, stream);
}

}  // namespace dr
