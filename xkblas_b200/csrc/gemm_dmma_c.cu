// gemm_dmma_c.cu -- the plain tile GEMM for float complex storage.
#include "gemm_dmma.cuh"

namespace xkb {
int gemm_dmma_c(const xkb_gemm_args* a, cudaStream_t st, const int* run_if) {
  return dispatch_type<float2>(a, st, run_if);
}
}  // namespace xkb
