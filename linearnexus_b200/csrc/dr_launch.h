// Launchers of the kernels that are compiled in translation units of their own (dr_fwd.cu: the tensor-core forwards,
// dr_trans.cu: the forward
// in transition form, dr_bwd.cu: the backward), so that the library's units build side by side.
#pragma once

#include "dr_common.cuh"

namespace dr {

// fused tcgen05 forward (Gated DeltaNet / DeltaNet; K = V = 128, chunk 64, bf16); packed: every sequence of the table
cudaError_t launch_chunk_fused(const FwdParams& p, cudaStream_t stream);
cudaError_t launch_chunk_fused_packed(const FwdParams& p, const SeqTable& seqs, cudaStream_t stream);
// two-kernel forward (any variant); the workspace holds split_workspace_bytes
int64_t split_workspace_bytes(int64_t units, int T);
// after_intra: recorded on `stream` between the two kernels (null: not)
// Where the chunk-parallel pass notes (1 or 0) of each chunk whether a channel decays by more than `limit` (log2) or a log decay is positive; at[2 .. 4]
// are set to zero.
struct WideMarks { float* at; int64_t stride; float limit; };
cudaError_t launch_chunk_split(const FwdParams& p, void* workspace, cudaStream_t stream, int* launches, cudaEvent_t after_intra = nullptr,
                               WideMarks marks = WideMarks{});
cudaError_t launch_chunk_split_packed(const FwdParams& p, const SeqTable& seqs, void* workspace, cudaStream_t stream);

// forward in transition form (two kernels; K = V = 64 or 128); bf16_tensor: the bf16-operand kernels (dr_fwd.cu; bf16 q, k, v,
// K = V = 128, chunk 64), else float32 precision for any storage type
int64_t trans_workspace_bytes(int64_t units, int T, int D, bool bf16_tensor);
cudaError_t launch_chunk_trans(const FwdParams& p, bool bf16_tensor, void* workspace, int sms, cudaStream_t stream);
int64_t trans_bf16_workspace_bytes(int64_t units, int T);
cudaError_t launch_chunk_trans_bf16(const FwdParams& p, void* workspace, int sms, cudaStream_t stream);

// backward (see dr_bwd.cuh)
int64_t bwd_workspace_bytes(const DrDesc* d);
cudaError_t launch_bwd_forward(const DrDesc* d, const void* q, const void* k, const void* v, const void* g, const float* beta,
                               const float* h0, void* o, float* hT, void* workspace, int32_t* status, cudaStream_t stream,
                               int* launches, bool own_stream = true);
cudaError_t launch_bwd_adjoint(const DrDesc* d, const void* q, const void* k, const void* v, const void* g, const float* beta,
                               const void* d_o, const float* d_hT, void* dq, void* dk, void* dv, float* dbeta, float* dg,
                               float* dh0, void* workspace, int32_t* status, cudaStream_t stream, int* launches,
                               const void* g_forward = nullptr);   // the decays that launch_bwd_forward had (null: aligned ones, see dr_chunk_fwd_saving)
// forward recomputation + adjoint
cudaError_t launch_bwd(const DrDesc* d, const void* q, const void* k, const void* v, const void* g, const float* beta,
                       const float* h0, const void* d_o, const float* d_hT, void* dq, void* dk, void* dv, float* dbeta, float* dg,
                       float* dh0, void* workspace, int32_t* status, cudaStream_t stream, int* launches, bool own_stream = true);

}  // namespace dr
