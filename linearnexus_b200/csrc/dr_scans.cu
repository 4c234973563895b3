// Translation unit of the scans: the delta-rule recurrence and the RWKV-7 / RWKV-6 / Mamba-2 scans, token by token or in
// chunk form by shape and storage type.
#include "dr_linrec.cuh"
#include "dr_rwkv_chunk.cuh"
#include "dr_recurrent.cuh"
#include "dr_ssd_chunk.cuh"
#include "dr_ssd_sm100.cuh"

namespace dr {

cudaError_t launch_linrec(int kind, bool io_bf16, const LinRecParams& p, int sms, cudaStream_t stream) {
  if (kind == LR_SSD && io_bf16 && ssd::eligible(p)) return ssdu::ahead(p) ? ssdu::launch(p, stream) : ssd::launch(p, sms, stream);
  if (kind != LR_SSD && rwkv::eligible(kind, io_bf16, p, sms)) return rwkv::launch(kind, io_bf16, p, stream);
  return launch_linrec_tokens(kind, io_bf16, p, stream);
}

}  // namespace dr
