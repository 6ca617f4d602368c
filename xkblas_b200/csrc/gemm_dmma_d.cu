// gemm_dmma_d.cu -- the plain tile GEMM for double storage.
#include "gemm_dmma.cuh"

namespace xkb {
int gemm_dmma_d(const xkb_gemm_args* a, cudaStream_t st, const int* run_if) {
  return dispatch_type<double>(a, st, run_if);
}
}  // namespace xkb
