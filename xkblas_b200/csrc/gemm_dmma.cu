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

// Copies of up to two column-major arrays, one per blockIdx.z: rows x cols
// words of W, wpe words per element, optionally only the elements of a
// triangle.  A block takes 256 rows x 8 columns (no index division: with one
// per element the copy ran at a third of the memory rate; 8 loads in flight
// per thread).
struct CopyWords {
  const void* src;
  void* dst;
  long lds, ldd;  // words
  int rows, cols, wpe, uplo;
};
template <class W>
__global__ void __launch_bounds__(256) k_repack(const CopyWords d0, const CopyWords d1,
                                                const int* run_if) {
  pdl_wait();
  pdl_launch();
  if (run_if && *run_if == 0) return;
  const CopyWords& d = blockIdx.z ? d1 : d0;
  const int r = blockIdx.x * 256 + threadIdx.x;
  if (r >= d.rows) return;
  const W* src = static_cast<const W*>(d.src);
  W* dst = static_cast<W*>(d.dst);
  const int er = d.wpe == 1 ? r : d.wpe == 2 ? r >> 1 : r >> 2;
  for (int c0 = blockIdx.y * 8; c0 < d.cols; c0 += gridDim.y * 8) {
    W v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (c0 + q < d.cols && in_mask(d.uplo, 0, er, c0 + q))
        v[q] = src[(size_t)r + (size_t)(c0 + q) * (size_t)d.lds];
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (c0 + q < d.cols && in_mask(d.uplo, 0, er, c0 + q))
        dst[(size_t)r + (size_t)(c0 + q) * (size_t)d.ldd] = v[q];
  }
}

int copy_arrays(const CopyArray* d, int n, int es, cudaStream_t st, const int* run_if) {
  if (n < 1 || n > 2) return n == 0 ? XKB_OK : XKB_EINVAL;
  bool wide = es % 8 == 0;
  for (int i = 0; i < n; ++i)
    wide = wide && reinterpret_cast<uintptr_t>(d[i].src) % 8 == 0 &&
           reinterpret_cast<uintptr_t>(d[i].dst) % 8 == 0;
  const int wb = wide ? 8 : 4, wpe = es / wb;
  CopyWords w[2];
  int mr = 0, mc = 0;
  for (int i = 0; i < n; ++i) {
    w[i] = {d[i].src, d[i].dst, d[i].lds * wpe, d[i].ldd * wpe, d[i].rows * wpe, d[i].cols, wpe,
            d[i].uplo};
    mr = std::max(mr, w[i].rows);
    mc = std::max(mc, w[i].cols);
  }
  if (n == 1) w[1] = w[0];
  const dim3 g((unsigned)((mr + 255) / 256), (unsigned)std::min((mc + 7) / 8, 32768), (unsigned)n);
  const long long tv = evlog_kern_begin(st, "k_repack");
  launch_pdl(wide ? k_repack<double> : k_repack<float>, g, dim3(256), 0, st, w[0], w[1], run_if);
  evlog_kern_end(tv, st);
  count_launch();
  return cudaPeekAtLastError() == cudaSuccess ? XKB_OK : XKB_ECUDA;
}

bool tma_ok(const void* p, long ld, int es) {
  return reinterpret_cast<uintptr_t>(p) % 16 == 0 && ((size_t)ld * es) % 16 == 0;
}

// Leading dimension of a packed, 16-byte aligned copy.
long packed_ld(long rows, int es) { return (long)(((size_t)rows * es + 15) / 16 * 16 / es); }

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
// The whole-matrix product; run_if not null: its kernels (an operand copy among
// them) do nothing unless the device word is non-zero.  XKB_ENOMEM is returned
// before the kernel that writes C is launched.
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
  if (reinterpret_cast<uintptr_t>(a->A) % 4 || reinterpret_cast<uintptr_t>(a->B) % 4 ||
      reinterpret_cast<uintptr_t>(a->C) % 4)
    return XKB_EINVAL;
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
  xkb_gemm_args pa = *a;
  void* pack = nullptr;  // one allocation and one launch for both operands
  int r = XKB_OK;
  const bool okA = tma_ok(a->A, a->lda, es), okB = tma_ok(a->B, a->ldb, es);
  if (!okA || !okB) {
    const int ra = a->opA == XKB_OP_N ? a->M : a->K, ca = a->opA == XKB_OP_N ? a->K : a->M;
    const int rb = a->opB == XKB_OP_N ? a->K : a->N, cb = a->opB == XKB_OP_N ? a->N : a->K;
    // the same array as both operands (a rank-k update) is copied once
    const bool same = a->A == a->B && a->lda == a->ldb && ra == rb && ca == cb;
    const long la = packed_ld(ra, es), lb = packed_ld(rb, es);
    const size_t za = okA ? 0 : ((size_t)la * ca * es + 255) / 256 * 256;
    const size_t zb = okB || same ? 0 : (size_t)lb * cb * es;
    if (!scratch_alloc(&pack, za + zb, st)) return XKB_ENOMEM;
    CopyArray d[2];
    int n = 0;
    if (!okA) {
      d[n++] = {a->A, pack, a->lda, la, ra, ca, XKB_FULL};
      pa.A = pack;
      pa.lda = la;
    }
    if (same) {
      pa.B = pa.A;
      pa.ldb = pa.lda;
    } else if (!okB) {
      pa.B = static_cast<char*>(pack) + za;
      pa.ldb = lb;
      d[n++] = {a->B, const_cast<void*>(pa.B), a->ldb, lb, rb, cb, XKB_FULL};
    }
    r = copy_arrays(d, n, es, st, run_if);
  }
  if (r == XKB_OK) {
    r = XKB_EINVAL;
    switch (a->dtype) {
      case XKB_S: r = gemm_dmma_s(&pa, st, run_if); break;
      case XKB_D: r = gemm_dmma_d(&pa, st, run_if); break;
      case XKB_C: r = gemm_dmma_c(&pa, st, run_if); break;
      case XKB_Z: r = gemm_dmma_z(&pa, st, run_if); break;
    }
  }
  if (pack) cudaFreeAsync(pack, st);
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
