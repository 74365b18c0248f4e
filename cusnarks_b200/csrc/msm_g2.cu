// msm_g2.cu -- G2 (Fq2) instantiation of the MSM pipeline.
// Fq2 products are calls here, in the accumulation too: the batch-affine rounds are slower with
// theirs inlined (2^20 fixed-base terms 7.48 ms, inlined 8.00), the rest is alike (2^17 generic
// terms 2.89 ms both).  The lane groups inline theirs (Fp::mul_raw).
#define CSB_MUL_NOINLINE
#include "msm_impl.cuh"

namespace csb {

cudaError_t msm_g2(const uint32_t* s, const uint32_t* p, uint32_t n, uint32_t* out, void* w,
                   size_t wb, const MsmConfig& cfg, cudaStream_t st) {
  return msm_detail::msm_impl<Fq2, false>(s, p, n, out, w, wb, cfg, st);
}

cudaError_t msm_fixed_g2(const uint32_t* s, const uint32_t* table, uint32_t n, uint32_t* out, void* w,
                         size_t wb, const MsmConfig& cfg, cudaStream_t st) {
  return msm_detail::msm_impl<Fq2, true>(s, table, n, out, w, wb, cfg, st);
}

cudaError_t msm_fixed_table_g2(const uint32_t* points, uint32_t n, int c, uint32_t* table, void* w,
                               size_t wb, cudaStream_t st) {
  return msm_detail::fixed_table_impl<Fq2>(points, n, c, table, w, wb, st);
}

}  // namespace csb
