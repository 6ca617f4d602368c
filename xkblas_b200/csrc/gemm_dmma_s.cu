// gemm_dmma_s.cu -- the plain tile GEMM for float storage.
#include "gemm_dmma.cuh"

namespace xkb {
int gemm_dmma_s(const xkb_gemm_args* a, cudaStream_t st, const int* run_if) {
  return dispatch_type<float>(a, st, run_if);
}
}  // namespace xkb
