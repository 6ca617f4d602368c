// trsm_leaf.cuh -- FP64 solve of one diagonal block of a triangular system
// (n <= 64 unknowns) against up to 64 right-hand sides by the MMA warps of the
// tile-task executor (sched.cu); leaf_at is shared with the whole-matrix
// solver (trsm.cu).  It is the body the reference hands to cublasZtrsm for a
// diagonal tile (blas/ztask_trsm.c:162-180).
//
// op(T), the right-hand sides and the inverses of the block's 8 x 8 diagonal
// sub-blocks lie in shared memory.  A warp owns 16 (complex 8) right-hand
// sides and walks the block in steps of 8 unknowns without waiting for another
// warp: Y = inv(T_ss) X_s by one DMMA (formed as Y^T, whose accumulators are
// the B fragment the update needs), then the rank-8 update of the unknowns
// still to solve by DMMA, as in k_trsm_block (trsm.cu).  What bounds it is
// latency: 8 steps of two dependent DMMAs and their shared-memory trips.  The
// substitution it replaces (a shuffle, a product and 16 dependent updates per
// unknown) took 40 to 60 us per block, most of a chain's time; it stays for
// ill-conditioned sub-blocks and for values that are not finite.
#pragma once
#include "dmma_common.cuh"

namespace xkb {

constexpr int kLeafRows = 64;

// Largest condition number (1-norm) of an 8 x 8 sub-block that is applied by
// its inverse.  The product's componentwise backward error grows with it:
// over 6000 random blocks the inverse's was 0.7 to 0.8 eps (median; largest
// 2.0) up to 8 and substitution's 1.1 to 1.2 (2.3); 1.4 (15) at 32 to 64,
// 21 (420) at 1e3 to 1e4, where substitution stays below 1.8.  Blocks with a
// dominant diagonal lie at 1 to 3.
constexpr double kLeafCond = 8.0;

template <class T>
struct LeafShape {
  static constexpr bool CP = St<T>::CPLX;
  static constexpr int PL = CP ? 2 : 1;
  static constexpr int LD = kLeafRows + 2;   // column stride of T and X, = 2 mod 16
  static constexpr int CW = CP ? 8 : 16;     // right-hand sides per warp
  static constexpr int COLS = 4 * CW;        // and per pass of the four warps
  static constexpr size_t T_D = (size_t)PL * kLeafRows * LD;  // doubles
  static constexpr size_t X_D = (size_t)PL * COLS * LD;
  static constexpr size_t V_D = (size_t)PL * (kLeafRows / 8) * 64;
  static constexpr size_t SMEM = sizeof(double) * (T_D + X_D + V_D + kLeafRows / 8);
};

// Barrier of the NT threads that run the solve (the CTA may hold others).
template <int NT>
__device__ __forceinline__ void leaf_sync() {
  asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory");
}

// element (row i, right-hand side c) of B: rhs_rows ? B[c + i ldb] : B[i + c ldb]
__device__ __forceinline__ size_t leaf_at(int i, int c, long ldb, bool rhs_rows) {
  return rhs_rows ? (size_t)c + (size_t)i * (size_t)ldb : (size_t)i + (size_t)c * (size_t)ldb;
}

// Unknowns b .. b + 7 of a warp's right-hand sides by substitution, a lane per
// right-hand side (Vr, Vi: the sub-block's inverse, whose diagonal is the
// reciprocals): an unknown that is Inf or NaN reaches those after it only,
// where a product with the inverse takes it to all eight through its zeros.
template <class T, bool LOWER>
__device__ __noinline__ void leaf_substitute(const double* Tr, const double* Ti, const double* Vr,
                                             const double* Vi, int b, double* xr, double* xi) {
  using Sh = LeafShape<T>;
  constexpr bool CP = Sh::CP;
  const int lane = threadIdx.x & 31;
  if (lane < Sh::CW) {
    double* x = xr + lane * Sh::LD + b;
    double* z = xi + lane * Sh::LD + b;
    for (int q = 0; q < 8; ++q) {
      const int j = LOWER ? q : 7 - q;
      const double dr = Vr[9 * j], di = CP ? Vi[9 * j] : 0.0;
      double vr = x[j], vi = 0.0;
      if (CP) {
        const double wr = vr * dr - z[j] * di;
        vi = vr * di + z[j] * dr;
        vr = wr;
        z[j] = vi;
      } else {
        vr *= dr;
      }
      x[j] = vr;
      const double* tr = Tr + (b + j) * Sh::LD + b;
      const double* ti = Ti + (b + j) * Sh::LD + b;
      for (int i = LOWER ? j + 1 : 0; i < (LOWER ? 8 : j); ++i) {
        x[i] -= CP ? tr[i] * vr - ti[i] * vi : tr[i] * vr;
        if (CP) z[i] -= tr[i] * vi + ti[i] * vr;
      }
    }
  }
  __syncwarp();
}

// X = (ar, ai) op(T)^-1 B in place for B's nrhs columns (ldb), by 128 threads:
// T(i,j) = A[swap ? j + i lda : i + j lda], conjugated when conj, unit: ones
// on its diagonal.  Operands are read through L2.
template <class T, bool LOWER>
__device__ __forceinline__ void leaf_solve(const typename St<T>::S* A, long lda, int n, bool swap,
                                           bool conj, bool unit, typename St<T>::S* B, long ldb,
                                           int nrhs, double ar, double ai, double* sm) {
  using Sh = LeafShape<T>;
  using S = typename St<T>::S;
  constexpr bool CP = Sh::CP;
  constexpr int LD = Sh::LD, W = CP ? 2 : 1, NT = 128;
  double* Tr = sm;  // T(i, j) at T[j * LD + i], zero outside the strict triangle
  double* Ti = Tr + (CP ? kLeafRows * LD : 0);
  double* Xr = sm + Sh::T_D;  // X[c * LD + i]
  double* Xi = Xr + (CP ? Sh::COLS * LD : 0);
  double* Vr = Xr + Sh::X_D;  // inverse of sub-block m: V[m * 64 + i * 8 + j]
  double* Vi = Vr + (CP ? (kLeafRows / 8) * 64 : 0);
  double* cond = Vr + Sh::V_D;  // condition number of sub-block m
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t = lane & 3;
  const int nsub = (n + 7) / 8;

  // ---- op(T): loads in groups of 8 before their stores ----
#pragma unroll 1
  for (int k0 = 0; k0 < kLeafRows * kLeafRows / NT; k0 += 8) {
    double vr[8], vi[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int e = tid + (k0 + k) * NT, a0 = e & (kLeafRows - 1), a1 = e / kLeafRows;
      const int i = swap ? a1 : a0, j = swap ? a0 : a1;
      vr[k] = vi[k] = 0.0;
      if (i < n && j < n && (LOWER ? j < i : j > i)) {
        const size_t idx = (size_t)a0 + (size_t)a1 * (size_t)lda;
        vr[k] = (double)__ldcg(A + W * idx);
        if (CP) vi[k] = (double)__ldcg(A + W * idx + W - 1);
      }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int e = tid + (k0 + k) * NT, a0 = e & (kLeafRows - 1), a1 = e / kLeafRows;
      const int o = (swap ? a0 : a1) * LD + (swap ? a1 : a0);
      Tr[o] = vr[k];
      if (CP) Ti[o] = conj ? -vi[k] : vi[k];
    }
  }
  leaf_sync<NT>();
  // ---- inverses of the 8 x 8 sub-blocks: thread (m, kk) column kk of
  // inv(T_m), by substitution against a unit vector; past n the identity ----
  if (tid < kLeafRows) {
    const int m = tid >> 3, kk = tid & 7, d = 8 * m + kk;
    double rk = 1.0, ik = 0.0, st = 1.0;  // st, sv: column sums of |T| and |inv(T)|
    if (!unit && d < n) {
      const size_t idx = (size_t)d + (size_t)d * (size_t)lda;
      const double dr = (double)__ldcg(A + W * idx);
      if (CP) {
        const double di = (conj ? -1.0 : 1.0) * (double)__ldcg(A + W * idx + W - 1);
        const double den = dr * dr + di * di;
        rk = dr / den;
        ik = -di / den;
        st = fabs(dr) + fabs(di);
      } else {
        rk = 1.0 / dr;
        st = fabs(dr);
      }
    }
    double zr[8], zi[8], sv = 0.0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      zr[i] = i == kk ? 1.0 : 0.0;
      zi[i] = 0.0;
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int jj = LOWER ? q : 7 - q;
      const double dr = __shfl_sync(0xffffffffu, rk, (lane & ~7) | jj);
      const double di = CP ? __shfl_sync(0xffffffffu, ik, (lane & ~7) | jj) : 0.0;
      if (LOWER ? jj >= kk : jj <= kk) {
        const double vr = zr[jj] * dr - zi[jj] * di, vi = zr[jj] * di + zi[jj] * dr;
        zr[jj] = vr;
        zi[jj] = vi;
        const double* col = Tr + (8 * m + jj) * LD + 8 * m;
        const double* coi = Ti + (8 * m + jj) * LD + 8 * m;
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (LOWER ? i > jj : i < jj) {
            const double tr = col[i], ti = CP ? coi[i] : 0.0;
            zr[i] -= tr * vr - ti * vi;
            if (CP) zi[i] -= tr * vi + ti * vr;
          }
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      Vr[m * 64 + i * 8 + kk] = zr[i];
      if (CP) Vi[m * 64 + i * 8 + kk] = zi[i];
      sv += fabs(zr[i]) + (CP ? fabs(zi[i]) : 0.0);
      st += fabs(Tr[d * LD + 8 * m + i]) + (CP ? fabs(Ti[d * LD + 8 * m + i]) : 0.0);
    }
    if (d >= n) st = sv = 0.0;  // the identity past n is no part of T
#pragma unroll
    for (int o = 4; o; o >>= 1) {
      sv = fmax(sv, __shfl_xor_sync(0xffffffffu, sv, o));
      st = fmax(st, __shfl_xor_sync(0xffffffffu, st, o));
    }
    if (kk == 0) cond[m] = sv * st;
  }
  leaf_sync<NT>();
  // sub-blocks applied by their inverse (bit m)
  const unsigned well =
      __ballot_sync(0xffffffffu, lane < kLeafRows / 8 && cond[lane & 7] <= kLeafCond);
  // ---- this warp's right-hand sides, nothing shared with the other warps ----
  double* xr = Xr + warp * Sh::CW * LD;
  double* xi = Xi + warp * Sh::CW * LD;
#pragma unroll 1
  for (int c0 = warp * Sh::CW; c0 < nrhs; c0 += Sh::COLS) {
    // X by the inverses of the well-conditioned sub-blocks; where a value is not
    // finite, which shows in that unknown's Y (an inverse's diagonal is not
    // zero), again from B by substitution throughout
    unsigned inv = well;
#pragma unroll 1
    for (;;) {
      int top = 0;  // largest exponent field of the Y (as integers: off the FP64 pipe)
#pragma unroll 1
      for (int q0 = 0; q0 < Sh::CW; q0 += 4) {
        double br[8], bi[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int i = lane + 32 * (k & 1), c = c0 + q0 + (k >> 1);
          br[k] = bi[k] = 0.0;
          if (i < n && c < nrhs) {
            const size_t idx = leaf_at(i, c, ldb, false);
            br[k] = (double)__ldcg(B + W * idx);
            if (CP) bi[k] = (double)__ldcg(B + W * idx + W - 1);
          }
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const int o = (q0 + (k >> 1)) * LD + lane + 32 * (k & 1);
          xr[o] = ar * br[k] - ai * bi[k];
          if (CP) xi[o] = ar * bi[k] + ai * br[k];
        }
      }
      __syncwarp();
      const int k0 = 2 * t, k1 = k0 + 1;
#pragma unroll 1
      for (int s = 0; s < nsub; ++s) {
        const int m = LOWER ? s : nsub - 1 - s, b = 8 * m;
        double yr[4] = {0.0, 0.0, 0.0, 0.0}, yi[4] = {0.0, 0.0, 0.0, 0.0};
        if (inv >> m & 1u) {
          // Y^T = X_s^T inv(T_ss)^T (k indices 2t, 2t + 1 on both sides)
          constexpr bool hi = Sh::CW > 8;  // right-hand sides g + 8 exist
          const double* v = Vr + m * 64 + g * 8;
          const double* x = xr + g * LD + b;
          const double a_r[4] = {x[k0], hi ? x[8 * LD + k0] : 0.0, x[k1], hi ? x[8 * LD + k1] : 0.0};
          const double b_r[2] = {v[k0], v[k1]};
          if constexpr (CP) {
            const double* w = Vi + m * 64 + g * 8;
            const double* z = xi + g * LD + b;
            const double a_i[4] = {z[k0], 0.0, z[k1], 0.0};
            const double n_i[4] = {-a_i[0], 0.0, -a_i[2], 0.0};
            const double b_i[2] = {w[k0], w[k1]};
            dmma_k8(yr, a_r, b_r);
            dmma_k8(yr, n_i, b_i);
            dmma_k8(yi, a_r, b_i);
            dmma_k8(yi, a_i, b_r);
          } else {
            dmma_k8(yr, a_r, b_r);
          }
          __syncwarp();  // every lane has read X_s
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const int c = g + ((v >> 1) << 3);
            if (c < Sh::CW) {
              xr[c * LD + b + k0 + (v & 1)] = yr[v];
              if (CP) xi[c * LD + b + k0 + (v & 1)] = yi[v];
            }
            top = max(top, __double2hiint(yr[v]) & 0x7fffffff);
            if (CP) top = max(top, __double2hiint(yi[v]) & 0x7fffffff);
          }
        } else {
          leaf_substitute<T, LOWER>(Tr, Ti, Vr + m * 64, Vi + m * 64, b, xr, xi);
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            const int c = g + ((v >> 1) << 3);
            yr[v] = c < Sh::CW ? xr[c * LD + b + k0 + (v & 1)] : 0.0;
            if (CP) yi[v] = c < Sh::CW ? xi[c * LD + b + k0 + (v & 1)] : 0.0;
          }
        }
        // rows still to solve -= T(rows, b .. b+7) Y
        const int u0 = LOWER ? b + 8 : 0, u1 = LOWER ? 8 * nsub : b;
#pragma unroll 1
        for (int m0 = u0; m0 < u1; m0 += 16) {
          // rows past u1 (a last half tile) are read in range and not stored
          const int ra = m0 + g, rb = min(m0 + g + 8, kLeafRows - 1);
          const double* t0 = Tr + (b + k0) * LD;
          const double* t1 = t0 + LD;
          const double a_r[4] = {-t0[ra], -t0[rb], -t1[ra], -t1[rb]};
          double a_i[4] = {0.0, 0.0, 0.0, 0.0}, n_i[4] = {0.0, 0.0, 0.0, 0.0};
          if constexpr (CP) {
            const double* s0 = Ti + (b + k0) * LD;
            const double* s1 = s0 + LD;
            a_i[0] = -s0[ra], a_i[1] = -s0[rb], a_i[2] = -s1[ra], a_i[3] = -s1[rb];
#pragma unroll
            for (int v = 0; v < 4; ++v) n_i[v] = -a_i[v];
          }
#pragma unroll
          for (int n0 = 0; n0 < Sh::CW; n0 += 8) {
            const double b_r[2] = {n0 ? yr[2] : yr[0], n0 ? yr[3] : yr[1]};
            double cr[4], ci[4];
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              const int o = (n0 + 2 * t + (v & 1)) * LD + (v >> 1 ? rb : ra);
              cr[v] = xr[o];
              ci[v] = CP ? xi[o] : 0.0;
            }
            if constexpr (CP) {
              const double b_i[2] = {yi[0], yi[1]};
              dmma_k8(cr, a_r, b_r);
              dmma_k8(cr, n_i, b_i);
              dmma_k8(ci, a_r, b_i);
              dmma_k8(ci, a_i, b_r);
            } else {
              dmma_k8(cr, a_r, b_r);
            }
#pragma unroll
            for (int v = 0; v < 4; ++v) {
              const int row = m0 + g + ((v >> 1) << 3);
              const int o = (n0 + 2 * t + (v & 1)) * LD + row;
              if (row < u1) {
                xr[o] = cr[v];
                if (CP) xi[o] = ci[v];
              }
            }
          }
        }
        __syncwarp();
      }
      if (inv == 0 || __all_sync(0xffffffffu, top < 0x7ff00000)) break;
      inv = 0;
    }
#pragma unroll 4
    for (int q = 0; q < 2 * Sh::CW; ++q) {
      const int i = lane + 32 * (q & 1), c = c0 + (q >> 1);
      if (i < n && c < nrhs) {
        const size_t idx = leaf_at(i, c, ldb, false);
        B[W * idx] = static_cast<S>(xr[(q >> 1) * LD + i]);
        if (CP) B[W * idx + W - 1] = static_cast<S>(xi[(q >> 1) * LD + i]);
      }
    }
    __syncwarp();
  }
}

}  // namespace xkb
