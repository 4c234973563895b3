// Translation unit of the tensor-core forwards.
#include "dr_chunk_sm100.cuh"
#include "dr_kda_sm100.cuh"
#include "dr_launch.h"

namespace dr {

cudaError_t launch_chunk_fused(const FwdParams& p, cudaStream_t stream) { return sm100::launch_chunk(p, stream); }
cudaError_t launch_chunk_fused_packed(const FwdParams& p, const SeqTable& seqs, cudaStream_t stream) {
  return sm100::launch_chunk_packed(p, seqs, stream);
}
int64_t split_workspace_bytes(int64_t units, int T) { return kda::workspace_bytes(units, T); }
cudaError_t launch_chunk_split(const FwdParams& p, void* workspace, cudaStream_t stream, int* launches, cudaEvent_t after_intra, WideMarks marks) {
  return kda::launch_chunk(p, workspace, stream, launches, after_intra, marks);
}
cudaError_t launch_chunk_split_packed(const FwdParams& p, const SeqTable& seqs, void* workspace, cudaStream_t stream) {
  return kda::launch_chunk_packed(p, seqs, workspace, stream);
}

int64_t trans_bf16_workspace_bytes(int64_t units, int T) { return kda::trans_workspace_bytes(units, T); }
cudaError_t launch_chunk_trans_bf16(const FwdParams& p, void* workspace, int sms, cudaStream_t stream) {
  return kda::launch_trans(p, workspace, sms, stream);
}

}  // namespace dr
