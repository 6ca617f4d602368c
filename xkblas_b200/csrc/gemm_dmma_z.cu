// gemm_dmma_z.cu -- the plain tile GEMM for double complex storage.
#include "gemm_dmma.cuh"

namespace xkb {
int gemm_dmma_z(const xkb_gemm_args* a, cudaStream_t st, const int* run_if) {
  return dispatch_type<double2>(a, st, run_if);
}
}  // namespace xkb
