// gemm_dmma.cu -- the plain FP64 tile GEMM for sm_100a.
//
// Replaces the reference's per-tile cuBLAS bodies (blas/ztask_gemm.c:176-216,
// cublasZgemm at :206; the triangle-masked variants used for gemmt / syrk /
// herk / syr2k / her2k diagonal tiles, ztask_gemmt.c:213, ztask_syrk.c:130,
// ztask_herk.c:130).  One launch covers the whole matrix instead of one
// NB x NB tile per task.
//
// Design (B200; kernels in gemm_dmma.cuh, operand tiles in dmma_tile.cuh):
//   * TMA 2-D tile loads (cp.async.bulk.tensor, 128-byte swizzle) fill a
//     4-stage shared-memory ring guarded by mbarriers (full: transaction
//     bytes, empty: one arrive per MMA warp); a copy warp drives the ring,
//     four warps run FP64 DMMA tensor-core MMAs (mma.sync m16n8k8 f64);
//   * operands of any storage type (s/d/c/z) are loaded as raw tiles and
//     widened to double when fragments are read, so every precision computes
//     in FP64 and rounds once on store; complex products are four real MMAs;
//   * 64 x 64 tiles, three CTAs per SM, or 32 x 32 tiles, five per SM (complex
//     32 x 32, three), so that one CTA's epilogue and fill run beside the
//     others' MMAs and the last wave is short; split-K for few tiles with a
//     long K (plan_tiles);
//   * alpha/beta, the triangle mask and the Hermitian real-diagonal rule are
//     applied in the register epilogue; tiles wholly outside the triangle
//     exit before touching memory;
//   * every barrier wait is bounded (xkb_dev.cuh) and records an error word.
// Bound: the FP64 tensor pipe.  8192^3 real 30.8 ms = 35.7 TFLOP/s, 96 % of
// the 37.2 TFLOP/s DMMA nominal (before, 128 x 128 tiles one CTA per SM:
// 35.5); K = 512 updates of 8192^2 34.5 TFLOP/s (29.5).
#include <cstdio>
#include <cstdlib>

#include <algorithm>

#include "dmma_common.cuh"
#include "xkb_dev.cuh"

namespace xkb {

// C <- alpha op(A) op(B) + beta C for one storage type, operands aligned for
// TMA (gemm_dmma_s.cu, _d, _c, _z)
int gemm_dmma_s(const xkb_gemm_args* a, cudaStream_t st, const int* run_if);
int gemm_dmma_d(const xkb_gemm_args* a, cudaStream_t st, const int* run_if);
int gemm_dmma_c(const xkb_gemm_args* a, cudaStream_t st, const int* run_if);
int gemm_dmma_z(const xkb_gemm_args* a, cudaStream_t st, const int* run_if);

// C <- beta*C on the masked part (beta == 0 writes zeros without reading).
template <class T>
__global__ void k_scale(int M, int N, double br, double bi, T* Cv, long ldc, int uplo,
                        int herm_diag, long diag) {
  using S = typename St<T>::S;
  S* C = reinterpret_cast<S*>(Cv);
  const size_t total = (size_t)M * (size_t)N;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total;
       e += (size_t)gridDim.x * blockDim.x) {
    const int row = (int)(e % (size_t)M), col = (int)(e / (size_t)M);
    if (!in_mask(uplo, diag, row, col)) continue;
    const size_t idx = (size_t)row + (size_t)col * (size_t)ldc;
    if constexpr (St<T>::CPLX) {
      double cr = 0, ci = 0;
      if (br != 0.0 || bi != 0.0) {
        const double xr = (double)C[2 * idx], xi = (double)C[2 * idx + 1];
        cr = br * xr - bi * xi;
        ci = br * xi + bi * xr;
      }
      if (herm_diag && (long)row + diag == (long)col) ci = 0.0;
      C[2 * idx] = (S)cr;
      C[2 * idx + 1] = (S)ci;
    } else {
      C[idx] = (br != 0.0) ? (S)(br * (double)C[idx]) : (S)0;
    }
  }
}

// Copy a rows x cols column-major array (element size es) into a packed
// array with leading dimension ldd.  Used to give TMA a 16-byte aligned view
// of an operand whose base or leading dimension is not 16-byte aligned.
template <class W>
__global__ void k_repack(int rows_w, int cols, const W* __restrict__ src, long lds_w,
                         W* __restrict__ dst, long ldd_w, const int* run_if) {
  if (run_if && *run_if == 0) return;
  const size_t total = (size_t)rows_w * (size_t)cols;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total;
       e += (size_t)gridDim.x * blockDim.x) {
    const size_t i = e % (size_t)rows_w, j = e / (size_t)rows_w;
    dst[i + j * (size_t)ldd_w] = src[i + j * (size_t)lds_w];
  }
}

static bool tma_ok(const void* p, long ld, int es) {
  return reinterpret_cast<uintptr_t>(p) % 16 == 0 && ((size_t)ld * es) % 16 == 0;
}

// Packed copy of a stored operand (rows x cols, element size es); *out is a
// stream-ordered allocation the caller frees on the same stream.
static int repack(const void* src, long ld, int rows, int cols, int es, void** out, long* ldo,
                  cudaStream_t st, const int* run_if) {
  const long ldp = (long)(((size_t)rows * es + 15) / 16 * 16 / es);
  if (cudaMallocAsync(out, std::max<size_t>((size_t)ldp * cols * es, 16), st) != cudaSuccess)
    return XKB_ENOMEM;
  *ldo = ldp;
  const size_t total = (size_t)rows * cols;
  const unsigned grid = (unsigned)std::max<size_t>(
      1, std::min<size_t>((total + 255) / 256, (size_t)sm_count() * 16));
  const long long tv = evlog_kern_begin(st, "k_repack");
  if (es % 8 == 0 && reinterpret_cast<uintptr_t>(src) % 8 == 0)
    k_repack<double><<<grid, 256, 0, st>>>(rows * (es / 8), cols,
                                           static_cast<const double*>(src), ld * (es / 8),
                                           static_cast<double*>(*out), ldp * (es / 8), run_if);
  else
    k_repack<float><<<grid, 256, 0, st>>>(rows * (es / 4), cols, static_cast<const float*>(src),
                                          ld * (es / 4), static_cast<float*>(*out),
                                          ldp * (es / 4), run_if);
  evlog_kern_end(tv, st);
  count_launch();
  return cudaPeekAtLastError() == cudaSuccess ? XKB_OK : XKB_ECUDA;
}

template <class T>
static int launch_scale(int M, int N, const double* beta, void* C, long ldc, int uplo,
                        int herm_diag, long diag, cudaStream_t st) {
  const size_t total = (size_t)M * (size_t)N;
  if (total == 0) return XKB_OK;
  long blocks = (long)((total + 255) / 256);
  if (blocks > 4L * sm_count() * 8) blocks = 4L * sm_count() * 8;
  const long long tv = evlog_kern_begin(st, "k_scale");
  k_scale<T><<<(unsigned)blocks, 256, 0, st>>>(M, N, beta[0], St<T>::CPLX ? beta[1] : 0.0,
                                               reinterpret_cast<T*>(C), ldc, uplo, herm_diag,
                                               diag);
  evlog_kern_end(tv, st);
  count_launch();
  return cudaPeekAtLastError() == cudaSuccess ? XKB_OK : XKB_ECUDA;
}

}  // namespace xkb

using namespace xkb;

extern "C" int xkb_cuda_scale(int dtype, int M, int N, const double* beta, void* C, long ldc,
                              int uplo, int herm_diag, long diag, void* stream) {
  if (M < 0 || N < 0 || !beta) return XKB_EINVAL;
  if (M == 0 || N == 0) return XKB_OK;
  cudaStream_t st = resolve_stream(stream);
  switch (dtype) {
    case XKB_S: return launch_scale<float>(M, N, beta, C, ldc, uplo, herm_diag, diag, st);
    case XKB_D: return launch_scale<double>(M, N, beta, C, ldc, uplo, herm_diag, diag, st);
    case XKB_C: return launch_scale<float2>(M, N, beta, C, ldc, uplo, herm_diag, diag, st);
    case XKB_Z: return launch_scale<double2>(M, N, beta, C, ldc, uplo, herm_diag, diag, st);
  }
  return XKB_EINVAL;
}

namespace xkb {
// The whole-matrix product; run_if not null: the kernel runs only where the
// device word is non-zero (operand repacking, if any, runs regardless).
static int gemm_impl(const xkb_gemm_args* a, cudaStream_t st, const int* run_if) {
  if (!a || a->M < 0 || a->N < 0 || a->K < 0) return XKB_EINVAL;
  if (a->dtype < XKB_S || a->dtype > XKB_Z) return XKB_EINVAL;
  if (a->opA < XKB_OP_N || a->opA > XKB_OP_C || a->opB < XKB_OP_N || a->opB > XKB_OP_C)
    return XKB_EINVAL;
  if (a->M == 0 || a->N == 0) return XKB_OK;
  const bool cplx = (a->dtype == XKB_C || a->dtype == XKB_Z);
  const bool alpha_zero = a->alpha[0] == 0.0 && (!cplx || a->alpha[1] == 0.0);
  if (a->K == 0 || alpha_zero)
    return run_if ? XKB_EINVAL
                  : xkb_cuda_scale(a->dtype, a->M, a->N, a->beta, a->C, a->ldc, a->uplo,
                                   a->herm_diag, a->diag, st);
  if (!run_if && (a->dtype == XKB_S || a->dtype == XKB_C)) {
    const int e = gemm_exact(a, st);
    if (e != XKB_ERANGE && e != XKB_ENOMEM) return e;
  }
  const int slot = trace_begin(run_if ? "dmma_fallback" : "dmma_gemm", a->dtype, a->M, a->N,
                               a->K, 0, st);
  trace_mark(slot, 1, st);
  // the tensor-map loads need 16-byte aligned bases and leading dimensions:
  // other operands are first copied to packed, aligned arrays (C is read and
  // written with plain loads and stores, any alignment)
  const int es = (a->dtype == XKB_S) ? 4 : (a->dtype == XKB_Z ? 16 : 8);
  if (reinterpret_cast<uintptr_t>(a->A) % 4 || reinterpret_cast<uintptr_t>(a->B) % 4 ||
      reinterpret_cast<uintptr_t>(a->C) % 4)
    return XKB_EINVAL;
  xkb_gemm_args pa = *a;
  void* packA = nullptr;
  void* packB = nullptr;
  int r = XKB_OK;
  if (!tma_ok(a->A, a->lda, es))
    r = repack(a->A, a->lda, a->opA == XKB_OP_N ? a->M : a->K,
               a->opA == XKB_OP_N ? a->K : a->M, es, &packA, &pa.lda, st, run_if);
  if (r == XKB_OK && !tma_ok(a->B, a->ldb, es))
    r = repack(a->B, a->ldb, a->opB == XKB_OP_N ? a->K : a->N,
               a->opB == XKB_OP_N ? a->N : a->K, es, &packB, &pa.ldb, st, run_if);
  if (packA) pa.A = packA;
  if (packB) pa.B = packB;
  if (r == XKB_OK) {
    r = XKB_EINVAL;
    switch (a->dtype) {
      case XKB_S: r = gemm_dmma_s(&pa, st, run_if); break;
      case XKB_D: r = gemm_dmma_d(&pa, st, run_if); break;
      case XKB_C: r = gemm_dmma_c(&pa, st, run_if); break;
      case XKB_Z: r = gemm_dmma_z(&pa, st, run_if); break;
    }
  }
  if (packA) cudaFreeAsync(packA, st);
  if (packB) cudaFreeAsync(packB, st);
  trace_mark(slot, 2, st);
  trace_mark(slot, 3, st);
  return r;
}

int gemm_if(const xkb_gemm_args* a, const int* run_if, cudaStream_t st) {
  return gemm_impl(a, st, run_if);
}
}  // namespace xkb

extern "C" int xkb_cuda_gemm(const xkb_gemm_args* a, void* stream) {
  return gemm_impl(a, resolve_stream(stream), nullptr);
}
