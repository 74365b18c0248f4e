// msm_batch_g1.cu -- G1 (Fq) instantiation of the batched MSM (msm_batch.cuh).
// Products of operators are calls, as in the single MSM (msm_g1.cu).
#define CSB_MUL_NOINLINE
#include "msm_batch.cuh"

namespace csb {

cudaError_t msm_batch_g1(const MsmBatch& b, void* w, size_t wb, cudaStream_t st) {
  return msm_detail::batch_impl<Fq>(b, w, wb, st);
}

}  // namespace csb
