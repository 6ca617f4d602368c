// gemm_dmma.cuh -- kernels of the plain FP64 tile GEMM and their launch (see
// gemm_dmma.cu); included by one source per storage type (gemm_dmma_s.cu,
// _d, _c, _z), so that the instantiations compile side by side.
#pragma once
#include <algorithm>
#include <cstdlib>

#include "dmma_tile.cuh"
#include "xkb_dev.cuh"

namespace xkb {

struct GemmParams {
  int M, N, K;
  void* C;
  long ldc;
  double ar, ai, br, bi;
  int uplo, herm_diag;
  long diag;
  int conjA, conjB;
  int vec;  // C's row pairs are aligned for one access each
  int tiles_m, tiles_n, ktiles;
  const int* run_if;  // not null: the launch does nothing unless *run_if != 0
  // split-K: the k-tiles of every C tile are shared by ksplit CTAs, slice s
  // taking [s kt_slice, (s+1) kt_slice); each writes its raw accumulators to
  // ws and k_gemm_splitk sums the slices in order and runs the epilogue
  int ksplit, kt_slice;
  double* ws;
};

// Tile of CTA `bid` (< tiles_m tiles_n) in the grouped rasterisation: 8 tile
// rows share a band of B columns in L2.  False if it lies wholly outside the
// triangle mask (nothing to do).
template <int BM, int BN>
__device__ __forceinline__ bool dmma_tile(const GemmParams& p, int bid, int& m0, int& n0) {
  const int GROUP = 8;
  const int span = GROUP * p.tiles_n;
  const int first_m = (bid / span) * GROUP;
  const int gsz = min(p.tiles_m - first_m, GROUP);
  const int tm = first_m + (bid % span) % gsz;
  const int tn = (bid % span) / gsz;
  m0 = tm * BM;
  n0 = tn * BN;
  if (p.uplo == XKB_LOWER && (long)(m0 + BM - 1) + p.diag < (long)n0) return false;
  if (p.uplo == XKB_UPPER && (long)m0 + p.diag > (long)(n0 + BN - 1)) return false;
  return true;
}

// CTA tile of BM x BN for WM x WN MMA warps, MINB CTAs per SM, STAGES ring
// stages.  CPRE: the C values that beta multiplies are loaded before the main
// loop (small tiles: the registers are free and the load's latency hides).
template <class T_, int BM_, int BN_, int WM_, int WN_, int MINB_, int STAGES_, bool CPRE_ = false>
struct Cfg {
  static constexpr bool CPRE = CPRE_;
  using T = T_;
  static constexpr int BM = BM_, BN = BN_, WM = WM_, WN = WN_, MINB = MINB_, STAGES = STAGES_;
  static constexpr int WARPS = WM * WN;           // MMA warps
  static constexpr int THREADS = 32 * WARPS;     // their threads
  static constexpr int CTA = THREADS + 32;       // and the copy warp
  static constexpr int WTM = BM / WM, WTN = BN / WN;  // warp tile
  static constexpr int MF = WTM / 16, NF = WTN / 8;   // MMA fragments of a warp
  static constexpr int NACC = St<T>::CPLX ? 8 : 4;
  static constexpr int NREG = MF * NF * NACC;  // accumulators of a thread
  static constexpr int BK = 128 / (int)sizeof(T);
  static constexpr uint32_t A_BYTES = BM * 128, B_BYTES = BN * 128;
  static constexpr uint32_t STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr size_t SMEM = STAGES * (size_t)STAGE_BYTES + 2 * STAGES * 8 + 1024;
  static_assert(WTM % 16 == 0 && WTN % 16 == 0, "16-row and 16-column fragment blocks");
};

// The pair of C elements of this thread in fragment (mf, nf), column slot
// i & 1: rows row, row + PS (see OpTile) of column col; `one`, `two`: which of
// them lie in C and the triangle mask.
template <class C_, bool A_KC, bool B_KC>
__device__ __forceinline__ void dmma_elem(const GemmParams& p, int m0, int n0, int mf, int nf,
                                          int i, int& row, int& col, bool& one, bool& two) {
  using T = typename C_::T;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wm = warp / C_::WN, wn = warp % C_::WN;
  const int g = lane >> 2, t = lane & 3;
  row = m0 + wm * C_::WTM + mf * 16 + OpTile<T, A_KC>::prow(g, 0);
  col = n0 + wn * C_::WTN + (nf >> 1) * 16 + OpTile<T, B_KC>::prow(2 * t + (i & 1), nf & 1);
  one = row < p.M && col < p.N && in_mask(p.uplo, p.diag, row, col);
  constexpr int PS = OpTile<T, A_KC>::PS;
  two = row + PS < p.M && col < p.N && in_mask(p.uplo, p.diag, row + PS, col);
}

// The C values of fragment (mf, nf) that beta multiplies: cv[i] in
// accumulator order (imaginary parts at cv[4 + i]; 0 where nothing is
// stored).  The epilogue loads a whole row of fragments before it stores
// any: C is read and written through one pointer, so a load placed after a
// store could not be issued before that store completes.
template <class C_, bool A_KC, bool B_KC>
__device__ __forceinline__ void dmma_load_frag(const GemmParams& p, int m0, int n0, int mf,
                                               int nf, double* cv) {
  using T = typename C_::T;
  using S = typename St<T>::S;
  const S* C = reinterpret_cast<const S*>(p.C);
  const bool use_beta = (p.br != 0.0) || (p.bi != 0.0);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    double re[2] = {0.0, 0.0}, im[2] = {0.0, 0.0};
    if (use_beta) {
      int row, col;
      bool one, two;
      dmma_elem<C_, A_KC, B_KC>(p, m0, n0, mf, nf, i, row, col, one, two);
      ld_pair<T>(C + St<T>::W * ((size_t)row + (size_t)col * (size_t)p.ldc), p.vec, one, two, re,
                 im);
    }
    cv[i] = re[0];
    cv[2 + i] = re[1];
    if (St<T>::CPLX) {
      cv[4 + i] = im[0];
      cv[6 + i] = im[1];
    }
  }
}

// alpha/beta, mask, Hermitian diagonal, store of the fragment (mf, nf) of
// one thread's accumulators (a: its NACC registers; cv: from dmma_load_frag).
template <class C_, bool A_KC, bool B_KC>
__device__ __forceinline__ void dmma_store_frag(const GemmParams& p, int m0, int n0, int mf,
                                                int nf, const double* a, const double* cv) {
  using T = typename C_::T;
  using S = typename St<T>::S;
  S* C = reinterpret_cast<S*>(p.C);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    int row, col;
    bool one, two;
    dmma_elem<C_, A_KC, B_KC>(p, m0, n0, mf, nf, i, row, col, one, two);
    double re[2], im[2] = {0.0, 0.0};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int v = 2 * h + i;
      if constexpr (St<T>::CPLX) {
        re[h] = p.ar * a[v] - p.ai * a[4 + v];
        im[h] = p.ar * a[4 + v] + p.ai * a[v];
        re[h] += p.br * cv[v] - p.bi * cv[4 + v];
        im[h] += p.br * cv[4 + v] + p.bi * cv[v];
        if (p.herm_diag && (long)(row + h * OpTile<T, A_KC>::PS) + p.diag == (long)col) im[h] = 0.0;
      } else {
        re[h] = fma(p.br, cv[v], p.ar * a[v]);
      }
    }
    st_pair<T>(C + St<T>::W * ((size_t)row + (size_t)col * (size_t)p.ldc), p.vec, one, two, re,
               im);
  }
}

// alpha/beta, mask, Hermitian diagonal, store of one thread's accumulators,
// one row of fragments at a time: all of the row's loads, then its stores.
template <class C_, bool A_KC, bool B_KC>
__device__ __forceinline__ void dmma_epilogue(const GemmParams& p, int m0, int n0,
                                              const double* acc) {
#pragma unroll
  for (int mf = 0; mf < C_::MF; ++mf) {
    double cv[C_::NF][C_::NACC];
#pragma unroll
    for (int nf = 0; nf < C_::NF; ++nf)
      dmma_load_frag<C_, A_KC, B_KC>(p, m0, n0, mf, nf, cv[nf]);
#pragma unroll
    for (int nf = 0; nf < C_::NF; ++nf)
      dmma_store_frag<C_, A_KC, B_KC>(p, m0, n0, mf, nf, acc + (mf * C_::NF + nf) * C_::NACC,
                                      cv[nf]);
  }
}

// Fragments of one k step of a warp: its rows of op(A) and columns of op(B).
template <class C_, bool A_KC, bool B_KC>
struct Frags {
  using T = typename C_::T;
  double ar[C_::MF][2][2], ai[C_::MF][2][2];      // [16-row block][h][k slot]
  double br[C_::NF / 2][2][2], bi[C_::NF / 2][2][2];
  // fA, fB: sign flips of the imaginary parts (conj)
  __device__ __forceinline__ void load_b(const uint8_t* sb, int kc, int c0, int g, int t,
                                         unsigned fB) {
#pragma unroll
    for (int q = 0; q < C_::NF / 2; ++q) {
      OpTile<T, B_KC>::load(sb, c0 + 16 * q, kc, g, t, br[q], bi[q]);
      if (St<T>::CPLX) {
#pragma unroll
        for (int x = 0; x < 4; ++x) bi[q][x >> 1][x & 1] = xor_sign(bi[q][x >> 1][x & 1], fB);
      }
    }
  }
  __device__ __forceinline__ void load_a(const uint8_t* sa, int mf, int kc, int r0, int g, int t,
                                         unsigned fA) {
    OpTile<T, A_KC>::load(sa, r0 + 16 * mf, kc, g, t, ar[mf], ai[mf]);
    if (St<T>::CPLX) {
#pragma unroll
      for (int x = 0; x < 4; ++x) ai[mf][x >> 1][x & 1] = xor_sign(ai[mf][x >> 1][x & 1], fA);
    }
  }
  __device__ __forceinline__ void mma(int mf, double (&acc)[C_::MF][C_::NF][C_::NACC]) const {
    const double a_r[4] = {ar[mf][0][0], ar[mf][1][0], ar[mf][0][1], ar[mf][1][1]};
    if constexpr (St<T>::CPLX) {
      const double a_i[4] = {ai[mf][0][0], ai[mf][1][0], ai[mf][0][1], ai[mf][1][1]};
      const double n_i[4] = {-a_i[0], -a_i[1], -a_i[2], -a_i[3]};
#pragma unroll
      for (int nf = 0; nf < C_::NF; ++nf) {
        double* a = acc[mf][nf];
        double (&re)[4] = *reinterpret_cast<double(*)[4]>(a);
        double (&im)[4] = *reinterpret_cast<double(*)[4]>(a + 4);
        dmma_k8(re, a_r, br[nf >> 1][nf & 1]);
        dmma_k8(im, a_r, bi[nf >> 1][nf & 1]);
        dmma_k8(re, n_i, bi[nf >> 1][nf & 1]);
        dmma_k8(im, a_i, br[nf >> 1][nf & 1]);
      }
    } else {
#pragma unroll
      for (int nf = 0; nf < C_::NF; ++nf) {
        double (&d)[4] = *reinterpret_cast<double(*)[4]>(acc[mf][nf]);
        dmma_k8(d, a_r, br[nf >> 1][nf & 1]);
      }
    }
  }
};

// The stages [gc, gc + KT) of the ring: waits for each, runs this warp's MMAs
// and releases it.  False if a bounded wait gave up.
template <class C_, bool A_KC, bool B_KC>
__device__ __forceinline__ bool dmma_mainloop(uint8_t* base, uint64_t* full, uint64_t* empty,
                                              int gc, int KT,
                                              double (&acc)[C_::MF][C_::NF][C_::NACC], int r0,
                                              int c0, unsigned fA, unsigned fB) {
  constexpr int STG = C_::STAGES, KS = C_::BK / 8;
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  // every lane observes the phase itself (acquire of the TMA bytes); the
  // vote reconverges the warp before the .aligned MMAs
  auto wait_full = [&](int j) {
    const bool got = mbar_wait(&full[j % STG], (j / STG) & 1, kErrFullWait);
    return __all_sync(0xffffffffu, got) != 0;
  };
  // the stage was read through the generic proxy and will be rewritten by
  // TMA (async proxy): order the reads before its release
  auto release = [&](int j) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[j % STG]);
  };
  for (int j = gc; j < gc + KT; ++j) {
    if (!wait_full(j)) return false;
    const uint8_t* sa = base + (j % STG) * C_::STAGE_BYTES;
#pragma unroll
    for (int kc = 0; kc < KS; ++kc) {
      Frags<C_, A_KC, B_KC> f;
      f.load_b(sa + C_::A_BYTES, kc, c0, g, t, fB);
#pragma unroll
      for (int mf = 0; mf < C_::MF; ++mf) {
        f.load_a(sa, mf, kc, r0, g, t, fA);
        f.mma(mf, acc);
      }
    }
    release(j);
  }
  return true;
}

// TMA of one stage, issued by the copy warp: lane 0 expects the bytes, then
// lane l copies box l (op(A)'s boxes first).  A k-contiguous operand is one
// box of BM (BN) lines; the other layout one box per panel of BK rows.
template <class C_, bool A_KC, bool B_KC>
__device__ __forceinline__ void issue_stage(uint8_t* sa, const CUtensorMap* tmA,
                                            const CUtensorMap* tmB, int m0, int n0, int k0,
                                            uint64_t* full) {
  constexpr int W = St<typename C_::T>::W, BK = C_::BK;
  constexpr int NA = A_KC ? 1 : C_::BM / BK, NB = B_KC ? 1 : C_::BN / BK;
  static_assert(NA + NB <= 32, "one box per lane");
  const int lane = threadIdx.x & 31;
  uint8_t* sb = sa + C_::A_BYTES;
  if (lane == 0) mbar_expect_tx(full, C_::STAGE_BYTES);
  __syncwarp();
  if (lane < NA) {
    if (A_KC) tma_load_2d(sa, tmA, k0 * W, m0, full);
    else tma_load_2d(sa + lane * BK * 128, tmA, (m0 + lane * BK) * W, k0, full);
  } else if (lane < NA + NB) {
    const int l = lane - NA;
    if (B_KC) tma_load_2d(sb, tmB, k0 * W, n0, full);
    else tma_load_2d(sb + l * BK * 128, tmB, (n0 + l * BK) * W, k0, full);
  }
}

// Copies of ring positions [0, n): the copy warp.  A warp of its own: when an
// MMA warp also issued them (about 700 cycles a stage for the expect, the
// boxes and the wait for a free stage), it held back the whole CTA -- alone on
// an SM, 64 x 64 tiles ran at 0.51 and 32 x 32 tiles at 0.25 of the DMMA rate.
template <class C_, class Issue>
__device__ __forceinline__ void dmma_copy_warp(uint64_t* empty, int n, Issue issue) {
  constexpr int STG = C_::STAGES;
  for (int j = 0; j < n; ++j) {
    if (j >= STG) {
      const bool free_ = mbar_wait(&empty[j % STG], (j / STG - 1) & 1, kErrEmptyWait);
      if (!__all_sync(0xffffffffu, free_)) return;
    }
    issue(j);
  }
}

// A_KC: op(A) != N, else rows contiguous.  B_KC: op(B) == N.
template <class C_, bool A_KC, bool B_KC>
__global__ void __launch_bounds__(C_::CTA, C_::MINB)
    k_gemm_dmma(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                const GemmParams p) {
  constexpr int STG = C_::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(base + STG * C_::STAGE_BYTES);
  uint64_t* empty = full + STG;

  const int ntiles = p.tiles_m * p.tiles_n;
  const int slice = (int)blockIdx.x / ntiles;  // 0 unless split-K
  const int bid = (int)blockIdx.x - slice * ntiles;
  int m0, n0;
  if (!dmma_tile<C_::BM, C_::BN>(p, bid, m0, n0)) {
    // a tile outside the triangle leaves at once (behind the wait it cost a
    // masked K = 256 update 9 %); block 0 waits all the same, so that the grid
    // never ends before its predecessor
    if (blockIdx.x == 0) pdl_wait();
    return;
  }
  const int warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) {
    tma_prefetch(&tmA);
    tma_prefetch(&tmB);
    for (int s = 0; s < STG; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], C_::WARPS);
    }
    fence_barrier_init();
  }
  pdl_wait();
  pdl_launch();
  // a launch predicated on a device word (the Ozaki data rule's plain
  // fallback): every thread reads the same word, so the whole CTA leaves
  // before touching shared memory, barriers or C
  if (p.run_if && *p.run_if == 0) return;
  __syncthreads();

  // this CTA's stages: [kt0, kt0 + KT)
  const int kt0 = slice * p.kt_slice;
  const int KT = p.ksplit > 1 ? max(0, min(p.ktiles - kt0, p.kt_slice)) : p.ktiles;
  auto issue = [&](int it) {
    const int s = it % STG;
    issue_stage<C_, A_KC, B_KC>(base + s * C_::STAGE_BYTES, &tmA, &tmB, m0, n0,
                                (kt0 + it) * C_::BK, &full[s]);
  };
  if (warp == C_::WARPS) {
    dmma_copy_warp<C_>(empty, KT, issue);
    return;
  }

  const int r0 = (warp / C_::WN) * C_::WTM, c0 = (warp % C_::WN) * C_::WTN;
  double acc[C_::MF][C_::NF][C_::NACC];
#pragma unroll
  for (int i = 0; i < C_::MF; ++i)
#pragma unroll
    for (int j = 0; j < C_::NF; ++j)
#pragma unroll
      for (int v = 0; v < C_::NACC; ++v) acc[i][j][v] = 0.0;
  double cv[C_::CPRE ? C_::MF : 1][C_::NF][C_::NACC];
  if constexpr (C_::CPRE) {
    if (p.ksplit <= 1) {
#pragma unroll
      for (int mf = 0; mf < C_::MF; ++mf)
#pragma unroll
        for (int nf = 0; nf < C_::NF; ++nf)
          dmma_load_frag<C_, A_KC, B_KC>(p, m0, n0, mf, nf, cv[mf][nf]);
    }
  }

  const unsigned fA = p.conjA ? 0x80000000u : 0u, fB = p.conjB ? 0x80000000u : 0u;
  if (!dmma_mainloop<C_, A_KC, B_KC>(base, full, empty, 0, KT, acc, r0, c0, fA, fB))
    return;
  const double* accp = &acc[0][0][0];
  if (p.ksplit > 1) {
    // raw partial sums of this slice, register-major: for each register the
    // block's threads write consecutive doubles (coalesced)
    double* w = p.ws + ((size_t)slice * ntiles + bid) * (size_t)(C_::NREG * C_::THREADS) +
                threadIdx.x;
#pragma unroll
    for (int r = 0; r < C_::NREG; ++r) w[(size_t)r * C_::THREADS] = accp[r];
    return;
  }
  if constexpr (C_::CPRE) {
#pragma unroll
    for (int mf = 0; mf < C_::MF; ++mf)
#pragma unroll
      for (int nf = 0; nf < C_::NF; ++nf)
        dmma_store_frag<C_, A_KC, B_KC>(p, m0, n0, mf, nf, acc[mf][nf], cv[mf][nf]);
  } else {
    dmma_epilogue<C_, A_KC, B_KC>(p, m0, n0, accp);
  }
}

// Sum of n partial-sum slots (slot q at w0 + q * stride, NACC values
// kThreads apart) in slot order, loaded four slots at a time so that one
// memory latency covers four slots (the order of the additions, and so the
// result, is that of a slot-by-slot loop).
template <int NACC, int kThreads>
__device__ __forceinline__ void sum_slots(const double* w0, size_t stride, int n,
                                          double (&acc)[NACC]) {
#pragma unroll
  for (int v = 0; v < NACC; ++v) acc[v] = 0.0;
  for (int s0 = 0; s0 < n; s0 += 4) {
    double wv[4][NACC];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int v = 0; v < NACC; ++v)
        wv[q][v] = s0 + q < n ? w0[(size_t)(s0 + q) * stride + (size_t)v * kThreads] : 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (s0 + q < n) {
#pragma unroll
        for (int v = 0; v < NACC; ++v) acc[v] += wv[q][v];
      }
  }
}

// Split-K reduction: block (tile, fragment f) sums fragment f of the tile's
// slices in slice order (deterministic) with the GEMM kernel's
// thread-to-element map, then stores it as the unsplit epilogue does.  One
// block per (tile, fragment) spreads the reads of the slices over many SMs.
template <class C_, bool A_KC, bool B_KC>
__global__ void __launch_bounds__(C_::THREADS) k_gemm_splitk(const GemmParams p) {
  pdl_wait();
  pdl_launch();
  if (p.run_if && *p.run_if == 0) return;
  constexpr int NACC = C_::NACC, STRIDE = C_::NREG * C_::THREADS;
  const int ntiles = p.tiles_m * p.tiles_n;
  const int bid = blockIdx.x;
  const int f = blockIdx.y;  // fragment (mf, nf) = (f / NF, f % NF)
  int m0, n0;
  if (!dmma_tile<C_::BM, C_::BN>(p, bid, m0, n0)) return;
  double cv[NACC], acc[NACC];
  dmma_load_frag<C_, A_KC, B_KC>(p, m0, n0, f / C_::NF, f % C_::NF, cv);  // in flight meanwhile
  const double* w0 =
      p.ws + (size_t)bid * STRIDE + (size_t)(f * NACC) * C_::THREADS + threadIdx.x;
  sum_slots<NACC, C_::THREADS>(w0, (size_t)ntiles * STRIDE, p.ksplit, acc);
  dmma_store_frag<C_, A_KC, B_KC>(p, m0, n0, f / C_::NF, f % C_::NF, acc, cv);
}

// ---------------------------------------------------------------------------
// host side
// ksplit > 1: split-K over that many slices.
template <class C_, bool A_KC, bool B_KC>
static int launch_dmma(const xkb_gemm_args* a, cudaStream_t st, const int* run_if, int ksplit) {
  using T = typename C_::T;
  using S = typename St<T>::S;
  constexpr int W = St<T>::W, BM = C_::BM, BN = C_::BN, BK = C_::BK;
  const int es = (int)sizeof(S);
  CUtensorMap tA, tB;
  // A stored (A_KC ? K x M : M x K), B stored (B_KC ? K x N : N x K); boxes
  // of 128 bytes along the contiguous dimension
  const uint64_t a_rows = A_KC ? a->K : a->M, a_cols = A_KC ? a->M : a->K;
  const uint64_t b_rows = B_KC ? a->K : a->N, b_cols = B_KC ? a->N : a->K;
  if (!encode_tmap_2d(&tA, St<T>::DT, es, a->A, a_rows * W, a_cols, (uint64_t)a->lda * W,
                      BK * W, A_KC ? BM : BK, CU_TENSOR_MAP_SWIZZLE_128B))
    return XKB_EINVAL;
  if (!encode_tmap_2d(&tB, St<T>::DT, es, a->B, b_rows * W, b_cols, (uint64_t)a->ldb * W,
                      BK * W, B_KC ? BN : BK, CU_TENSOR_MAP_SWIZZLE_128B))
    return XKB_EINVAL;
  GemmParams p;
  p.M = a->M;
  p.N = a->N;
  p.K = a->K;
  p.C = a->C;
  p.ldc = a->ldc;
  p.ar = a->alpha[0];
  p.ai = St<T>::CPLX ? a->alpha[1] : 0.0;
  p.br = a->beta[0];
  p.bi = St<T>::CPLX ? a->beta[1] : 0.0;
  p.uplo = a->uplo;
  p.herm_diag = a->herm_diag;
  p.diag = a->diag;
  p.conjA = (a->opA == XKB_OP_C);
  p.conjB = (a->opB == XKB_OP_C);
  // row pairs of C (even rows first) move as one access when every pair is
  // aligned: 8 bytes for float, 16 otherwise
  const uintptr_t al = sizeof(T) == 4 ? 8 : 16;
  p.vec = reinterpret_cast<uintptr_t>(a->C) % al == 0 && ((size_t)a->ldc * sizeof(T)) % al == 0;
  p.tiles_m = (a->M + BM - 1) / BM;
  p.tiles_n = (a->N + BN - 1) / BN;
  p.ktiles = (a->K + BK - 1) / BK;
  p.run_if = run_if;
  p.ksplit = std::max(1, ksplit);
  p.kt_slice = (p.ktiles + p.ksplit - 1) / p.ksplit;
  p.ksplit = (p.ktiles + p.kt_slice - 1) / p.kt_slice;  // no empty slice
  p.ws = nullptr;
  constexpr int FRAGS = C_::MF * C_::NF;
  const long ntiles = (long)p.tiles_m * p.tiles_n;
  auto kern = k_gemm_dmma<C_, A_KC, B_KC>;
  static bool attr_done = false;  // one per instantiation
  if (!attr_done) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)C_::SMEM) != cudaSuccess)
      return XKB_ECUDA;
    attr_done = true;
  }
  if (p.ksplit > 1 &&
      !scratch_alloc(reinterpret_cast<void**>(&p.ws),
                     (size_t)p.ksplit * ntiles * C_::NREG * C_::THREADS * 8, st))
    p.ksplit = 1;  // no workspace: every tile walks the whole k range
  const long long tv = evlog_kern_begin(st, p.ksplit > 1 ? "k_gemm_dmma+k_gemm_splitk"
                                                         : "k_gemm_dmma");
  cudaError_t le =
      launch_pdl(kern, dim3((unsigned)(ntiles * p.ksplit)), dim3(C_::CTA), C_::SMEM, st, tA, tB, p);
  if (p.ksplit > 1) {
    const dim3 rg((unsigned)ntiles, (unsigned)FRAGS);
    if (le == cudaSuccess)
      le = launch_pdl(k_gemm_splitk<C_, A_KC, B_KC>, rg, dim3(C_::THREADS), 0, st, p);
    cudaFreeAsync(p.ws, st);
  }
  evlog_kern_end(tv, st);
  count_launch(p.ksplit > 1 ? 2 : 1);
  return le == cudaSuccess && cudaPeekAtLastError() == cudaSuccess ? XKB_OK : XKB_ECUDA;
}

template <class C_>
static int dispatch_ops(const xkb_gemm_args* a, cudaStream_t st, const int* run_if,
                        int ksplit) {
  const bool akc = a->opA != XKB_OP_N, bkc = a->opB == XKB_OP_N;
  if (akc && bkc) return launch_dmma<C_, true, true>(a, st, run_if, ksplit);
  if (akc && !bkc) return launch_dmma<C_, true, false>(a, st, run_if, ksplit);
  if (!akc && bkc) return launch_dmma<C_, false, true>(a, st, run_if, ksplit);
  return launch_dmma<C_, false, false>(a, st, run_if, ksplit);
}

// Tile and split of one call, by a model of its time on the SMs: n tiles
// spread over the SMs make q = ceil(n / SMs) on the fullest one, R of them at
// a time; r resident CTAs reach the fraction e[r] of an SM's DMMA rate (alone,
// a CTA's four MMA warps wait for their own fragments); `base`, `wave` and
// `tile` microseconds are added once, per wave of R (fill, drain, epilogue)
// and per tile; split-K adds its reduction.  The constants fit these times
// (B200, us; before: 128 x 128 tiles one CTA per SM, split-K and stream-K over
// them, 64 x 64 tiles with unswizzled operands):
//   8192^2 x 512: 64 x 64 1983, 32 x 32 2121 (before 2330)
//   7680^2 lower x 256: 532, 521 (597)     2048^2 x 512: 131, 138 (183)
//   2048^3: 502, 532 (646)     3001 x 517 x 777: 90, 83 (121)
//   3000^2 x 300: 172, 179     1500^3: 217, 214     4096^2 x 128 lower: 108, 94
//   1024^3: 114, 72, split 4 x 64 x 64 78 (93)    512^3: 29, 16 (35)
//   512^2 x 4096: 183, 92, split 4 x 32 x 32 80 (86)
//   1000 x 900 x 3000: 217, 203, split 3 x 64 x 64 189 (217)
//   complex 1200 x 900 x 1100: 327, split 2 312 (642)
// Stream-K over the same tiles (every CTA an equal share of the k steps) lost
// to the better of these everywhere measured, by 2 to 40 %.
struct TilePlan {
  bool small;  // the 32 x 32 tile
  int ksplit;
};
struct TileCost {
  int R;
  double e[5], base, wave, tile;
};

inline double tile_cost(long n, double unit_us, const TileCost& c) {
  const long sms = sm_count();
  const long q = (n + sms - 1) / sms, full = q / c.R, rem = q % c.R;
  return unit_us * ((double)(full * c.R) / c.e[c.R - 1] + (rem ? (double)rem / c.e[rem - 1] : 0.0)) +
         c.base + c.wave * (double)(full + (rem ? 1 : 0)) + c.tile * (double)q;
}

template <class T>
static TilePlan plan_tiles(const xkb_gemm_args* a) {
  constexpr bool CPLX = St<T>::CPLX;
  static const TileCost c64{3, {0.74, 0.90, 0.985}, 8.5, 3.2, 0.0},
      c64s{3, {0.74, 0.90, 0.985}, 1.0, 1.2, 0.0},  // a slice: no C, no epilogue
      c32{5, {0.42, 0.68, 0.76, 0.80, 0.93}, 1.5, 0.0, 0.3},
      cz{3, {0.63, 0.84, 0.89}, 1.5, 1.0, 0.0};
  auto tiles = [&](int b) {
    const long tm = (a->M + b - 1) / b, tn = (a->N + b - 1) / b;
    return a->uplo == XKB_FULL ? tm * tn : (tm * tn + std::max(tm, tn)) / 2;
  };
  // tuning table: 64 x 64 tiles from this many 128 x 128 blocks of C on
  // (XKBLAS_GEMM_TILE=big|small: always / never), for sweeps and tests; the
  // split stays the model's.  Saved tables hold no such line: one threshold
  // made 4096^2 x 128 lower 108 us (94), 1000 x 900 x 3000 203 (189)
  static const char* force = getenv("XKBLAS_GEMM_TILE");
  const double big = force ? (force[0] == 'b' ? 0.0 : 1e18) : tune("gemm_tile64_min_blocks", -1.0);
  const bool fixed = !CPLX && big >= 0.0;
  const bool want_small =
      (double)((a->M + 127) / 128) * (double)((a->N + 127) / 128) < big;
  TilePlan best{true, 1};
  double tbest = 1e300;
  for (int c = CPLX ? 1 : 0; c < 2; ++c) {
    const bool small = c == 1;
    if (fixed && small != want_small) continue;
    const int b = small ? 32 : 64;
    const long n = tiles(b);
    // microseconds of one tile at the SM's full rate (64 FMA a cycle)
    const double unit = (double)b * b * (CPLX ? 4.0 : 1.0) * (double)a->K / 64.0 / 1965.0;
    for (int ks = 1; ks <= 32; ks = ks < 4 ? ks + 1 : ks + ks / 2) {
      if (ks > 1 && (a->K < 128 * ks || n * ks > 32 * (long)sm_count())) break;
      double t = tile_cost(n * ks, unit / ks, CPLX ? cz : small ? c32 : ks > 1 ? c64s : c64);
      // reduction: a launch, and every slice written and read once (L2)
      if (ks > 1) t += 4.0 + (double)n * b * b * (CPLX ? 32.0 : 16.0) * ks * 1e-7;
      if (t < tbest) {
        tbest = t;
        best = {small, ks};
      }
    }
  }
  if (tune("gemm_splitk", 1.0) == 0.0) best.ksplit = 1;
  return best;
}

template <class T>
static int dispatch_type(const xkb_gemm_args* a, cudaStream_t st, const int* run_if) {
  const TilePlan pl = plan_tiles<T>(a);
  if constexpr (St<T>::CPLX) {
    return dispatch_ops<Cfg<T, 32, 32, 2, 2, 3, 4>>(a, st, run_if, pl.ksplit);
  } else {
    if (pl.small) return dispatch_ops<Cfg<T, 32, 32, 2, 2, 5, 4, true>>(a, st, run_if, pl.ksplit);
    return dispatch_ops<Cfg<T, 64, 64, 2, 2, 3, 4>>(a, st, run_if, pl.ksplit);
  }
}

}  // namespace xkb
