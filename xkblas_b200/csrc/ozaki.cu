// ozaki.cu -- FP64-accurate contraction on INT8 tensor cores (Ozaki scheme II).
//
// No counterpart in the reference (whose tile bodies call cuBLAS DGEMM,
// blas/ztask_gemm.c:206); selected by xkblas_set_modemath(XKBLAS_TENSOR_OP_MATH)
// or XKBLAS_DEFAULT_MATH=TC, the reference's switch for tensor-core math
// (blas/xkblas.h:100-107, blas/ztask_gemm.c:182-196).
//
// Method (Ozaki, Uchino, Imamura, "Ozaki Scheme II: a GEMM-oriented emulation
// of floating-point matrix multiplication using an integer modular
// technique", 2025), restated:
//   1. each row i of op(A) is scaled by 2^mu_i and each column j of op(B) by
//      2^nu_j and rounded to integers A', B' (|A'|,|B'| < 2^62), with the
//      shifts chosen from the 2-norms so that |A' B'| (Cauchy-Schwarz) stays
//      below P/2, P = p_1 ... p_n the product of the moduli;
//   2. for every modulus p_l (pairwise coprime, <= 256) the symmetric
//      residues A' mod p_l, B' mod p_l fit in int8 and their product is
//      computed EXACTLY on the tensor cores (tcgen05.mma kind::i8, INT32
//      accumulation in TMEM; K * 128^2 < 2^31 for K <= 131072), then reduced
//      mod p_l;
//   3. the n residues of each C entry are recombined by the Chinese remainder
//      theorem on the FP64 pipe (CRT weights split into an exact high part
//      and a rounded low part, the quotient by P exact; see crt_value),
//      mapped to the symmetric range and scaled back by 2^-(mu_i + nu_j);
//      alpha/beta are applied in FP64.
// With n = 16 moduli P ~ 2^125.4, so each operand keeps ~61 bits relative to
// its row / column 2-norm: the contraction error is below FP64 DGEMM's.
//
// Kernels: k_oz_norm (per-row / per-column scaling), k_oz_residues (scale,
// round, reduce to int8 planes in the K-major layout TMA reads), k_oz_gemm
// (TMA -> 4-stage smem ring -> tcgen05.mma -> TMEM -> mod-p epilogue, one
// launch for all moduli), k_oz_crt (reconstruction + alpha/beta + mask).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <type_traits>
#include <vector>

#include "xkb_dev.cuh"

namespace xkb {
namespace oz {

constexpr int kMaxMod = 16;  // moduli of a real product
constexpr int kMaxC = 17;    // moduli of a complex product (two planes each)
constexpr int kMaxPl = 2 * kMaxC;  // residue planes of an operand

struct Consts {
  int nmod;
  int H;                       // scaled operands stay below 2^H in 2-norm
  int p[kMaxMod];
  uint32_t wlo[kMaxMod], whi[kMaxMod];  // bytes of 2^(8t) mod p, t = 0..3, 4..7
  uint32_t off[kMaxMod];                // p - (2^62 mod p): undoes the +2^62 offset
  uint32_t offh[kMaxMod];               // off + floor(p/2): symmetric residues
  uint32_t magic[kMaxMod];              // ceil(2^32 / p): exact quotients below 2^21
  int half[kMaxMod];                    // floor(p/2)
  // CRT weights w = (P/p)((P/p)^-1 mod p) mod P split as w = w1 + w2: w1 the
  // bits of w from 2^csplit up (exact double, <= 41 significant bits), w2
  // the rest rounded to double; P = P1 + P2 the same way
  double w1[kMaxMod], w2[kMaxMod];
  double P1d, P2d, Pd, invPd;
};

// ---------------------------------------------------------------------------
// host: moduli and CRT constants
typedef unsigned __int128 u128;

static std::vector<int> moduli_list() {
  std::vector<int> m;
  for (int c = 256; c >= 2 && (int)m.size() < kMaxMod; --c) {
    bool ok = true;
    for (int q : m) {
      int a = c, b = q;
      while (b) {
        int t = a % b;
        a = b;
        b = t;
      }
      if (a != 1) {
        ok = false;
        break;
      }
    }
    if (ok) m.push_back(c);
  }
  return m;
}

static u128 mulmod(u128 a, u128 b, u128 m) {  // a, b < m < 2^127
  u128 r = 0;
  a %= m;
  while (b) {
    if (b & 1) {
      r += a;
      if (r >= m) r -= m;
    }
    a += a;
    if (a >= m) a -= m;
    b >>= 1;
  }
  return r;
}

static int inv_mod(int a, int p) {  // a^-1 mod p, gcd(a,p) = 1
  int t = 0, nt = 1, r = p, nr = ((a % p) + p) % p;
  while (nr) {
    int q = r / nr, tmp = t - q * nt;
    t = nt;
    nt = tmp;
    tmp = r - q * nr;
    r = nr;
    nr = tmp;
  }
  return t < 0 ? t + p : t;
}

static double log2P(int n) {
  std::vector<int> m = moduli_list();
  double s = 0;
  for (int i = 0; i < n; ++i) s += std::log2((double)m[i]);
  return s;
}

static bool make_consts(int n, Consts* c) {
  if (n < 2 || n > kMaxMod) return false;
  std::vector<int> m = moduli_list();
  std::memset(c, 0, sizeof(*c));
  c->nmod = n;
  u128 P = 1;
  for (int i = 0; i < n; ++i) P *= (u128)m[i];
  // budget: ||A'_i||_2 ||B'_j||_2 <= 2^(2H) (1+tiny) < P/2
  c->H = (int)std::floor((log2P(n) - 1.0) / 2.0) - 1;
  // split point of the CRT weights: sum_l r_l w1_l < 4080 P < 2^(bits(P)+12)
  // must be an integer multiple of 2^csplit below 2^(53+csplit)
  int bitsP = 0;
  for (u128 t = P; t; t >>= 1) ++bitsP;
  const int csplit = std::max(0, bitsP + 12 - 53);
  const u128 low = csplit ? (((u128)1 << csplit) - 1) : 0;
  for (int i = 0; i < n; ++i) {
    const int p = m[i];
    c->p[i] = p;
    uint32_t lo = 0, hi = 0;
    for (int t = 0; t < 8; ++t) {
      uint64_t w = 1;
      for (int s = 0; s < 8 * t; ++s) w = (w * 2) % (uint64_t)p;
      if (t < 4) lo |= (uint32_t)w << (8 * t);
      else hi |= (uint32_t)w << (8 * (t - 4));
    }
    c->wlo[i] = lo;
    c->whi[i] = hi;
    uint64_t t62 = 1;
    for (int s2 = 0; s2 < 62; ++s2) t62 = (t62 * 2) % (uint64_t)p;
    c->off[i] = (uint32_t)((uint64_t)p - t62);
    c->half[i] = p / 2;
    c->offh[i] = c->off[i] + (uint32_t)(p / 2);
    c->magic[i] = (uint32_t)(((1ull << 32) + (uint64_t)p - 1) / (uint64_t)p);
    const u128 Mi = P / (u128)p;
    const int inv = inv_mod((int)(Mi % (u128)p), p);
    const u128 w = mulmod(Mi, (u128)inv, P);
    c->w1[i] = std::ldexp((double)(uint64_t)(w >> csplit), csplit);  // < 2^41 units: exact
    c->w2[i] = (double)(w & low);
  }
  c->P1d = std::ldexp((double)(uint64_t)(P >> csplit), csplit);
  c->P2d = (double)(P & low);
  c->Pd = (double)P;
  c->invPd = 1.0 / c->Pd;
  return true;
}

// ---------------------------------------------------------------------------
// Complex products.  Modulo an odd p whose prime factors are all 1 mod 4, -1
// has a square root j, and a + ib -> (a + jb, a - jb) maps the complex
// integers mod p onto pairs of integers mod p with the product taken entry by
// entry.  So a complex contraction costs TWO real INT8 products per modulus
// (four with the operands concatenated as [Re | Im]), and the residues of its
// real and imaginary parts are (c+ + c-) / 2 and (c+ - c-) / (2j).  The factors
// 1/2 and 1/(2j) go into the CRT weights.  These moduli are smaller (the
// seventeen largest such pairwise coprime ones from 241 down), so a call of n
// real moduli's budget H takes n + 1 of them: 16 for n = 15, 17 for n = 16.
constexpr int kCMod[kMaxC] = {241, 233, 229, 221, 205, 197, 193, 181, 173,
                              157, 149, 137, 113, 109, 101, 97,  89};

struct CResConsts {  // of the residue kernel
  int p[kMaxC], half[kMaxC];
  uint32_t wlo[kMaxC], whi[kMaxC];  // bytes of 2^(8t) mod p
  uint32_t jlo[kMaxC], jhi[kMaxC];  // bytes of j 2^(8t) mod p
  uint32_t off[kMaxC], offj[kMaxC];  // undo the +2^62 offset of Re (plus half) and of Im
  uint32_t cp[kMaxC];                // a multiple of p above j Im's largest sum
  uint32_t magic[kMaxC];
};
struct CCrtConsts {  // of the recombination with n moduli, weights split as in Consts
  double w1[kMaxC], w2[kMaxC];  // real part: times c+ + c-
  double v1[kMaxC], v2[kMaxC];  // imaginary part: times c+ - c-
  double P1d, P2d, invPd;
};
struct CCrtTab {
  CCrtConsts c[kMaxC + 1];  // by moduli count
};

static double log2Pc(int n) {
  double s = 0;
  for (int i = 0; i < n; ++i) s += std::log2((double)kCMod[i]);
  return s;
}

static uint32_t pack_weights(uint64_t f, int p, int t0) {
  uint32_t r = 0;
  for (int t = t0; t < t0 + 4; ++t) {
    uint64_t w = f % (uint64_t)p;
    for (int q = 0; q < 8 * t; ++q) w = (w * 2) % (uint64_t)p;
    r |= (uint32_t)w << (8 * (t - t0));
  }
  return r;
}

static int sqrt_minus_one(int p) {
  for (int j = 1; j < p; ++j)
    if ((j * j) % p == p - 1) return j;
  return 0;
}

static const CResConsts& cres_consts() {
  static const CResConsts c = [] {
    CResConsts r;
    for (int i = 0; i < kMaxC; ++i) {
      const int p = kCMod[i], j = sqrt_minus_one(p);
      uint64_t t62 = 1;
      for (int q = 0; q < 62; ++q) t62 = (t62 * 2) % (uint64_t)p;
      r.p[i] = p;
      r.half[i] = p / 2;
      r.wlo[i] = pack_weights(1, p, 0);
      r.whi[i] = pack_weights(1, p, 4);
      r.jlo[i] = pack_weights((uint64_t)j, p, 0);
      r.jhi[i] = pack_weights((uint64_t)j, p, 4);
      r.off[i] = (uint32_t)((uint64_t)p - t62) + (uint32_t)(p / 2);
      r.offj[i] = (uint32_t)((uint64_t)p - (t62 * (uint64_t)j) % (uint64_t)p);
      r.cp[i] = (uint32_t)(((1 << 20) + p - 1) / p * p);
      r.magic[i] = (uint32_t)(((1ull << 32) + (uint64_t)p - 1) / (uint64_t)p);
    }
    return r;
  }();
  return c;
}

static const CCrtTab& ccrt_tab() {
  static const CCrtTab tab = [] {
    CCrtTab t;
    std::memset(&t, 0, sizeof(t));
    for (int n = 2; n <= kMaxC; ++n) {
      CCrtConsts& c = t.c[n];
      u128 P = 1;
      for (int i = 0; i < n; ++i) P *= (u128)kCMod[i];
      // sum_l (c+ + c-) w1 < 17 * 510 P < 2^(bits(P)+14)
      int bitsP = 0;
      for (u128 q = P; q; q >>= 1) ++bitsP;
      const int cs = std::max(0, bitsP + 14 - 53);
      const u128 low = cs ? (((u128)1 << cs) - 1) : 0;
      for (int i = 0; i < n; ++i) {
        const int p = kCMod[i], j = sqrt_minus_one(p);
        const u128 Mi = P / (u128)p;
        const int im = inv_mod((int)(Mi % (u128)p), p);
        const int fr = (int)((long)im * inv_mod(2, p) % p);
        const int fi = (int)((long)im * inv_mod(2 * j % p, p) % p);
        const u128 w = Mi * (u128)fr, v = Mi * (u128)fi;  // below P
        c.w1[i] = std::ldexp((double)(uint64_t)(w >> cs), cs);
        c.w2[i] = (double)(w & low);
        c.v1[i] = std::ldexp((double)(uint64_t)(v >> cs), cs);
        c.v2[i] = (double)(v & low);
      }
      c.P1d = std::ldexp((double)(uint64_t)(P >> cs), cs);
      c.P2d = (double)(P & low);
      c.invPd = 1.0 / (double)P;
    }
    return t;
  }();
  return tab;
}

// ---------------------------------------------------------------------------
// 1. scaling exponents and the moduli count.  View the operand as L "rows"
//    of length K, element (l,k) at X[l*sl + k*sk] (one of sl, sk is 1).
//    Partial sums over k-chunks go to part[chunk][l] = (sum of squares,
//    max |x|, sum |x|, nonzero count); k_oz_stat finalises each row.
constexpr int kNormChunk = 512;

// The moduli count of a call, chosen on the device (k_oz_pick) and read by
// every later kernel of the call: n moduli (0: the plain FP64 kernel runs
// instead), H the exponent budget of the scaled operands for that count.
struct OzSel {
  int n, H, fallback;
  int np;  // moduli actually multiplied: n, or a complex product's larger count
};

// Counters over all contractions of the process (xkb_ozaki_counts).
static __device__ unsigned long long g_oz_calls, g_oz_mod_sum, g_oz_fallbacks;
static __device__ int g_oz_last = -1;
// and over the single-precision products (xkb_exact_counts)
static __device__ unsigned long long g_ex_calls, g_ex_plain;
static __device__ int g_ex_last = -1;

// Exponent of the lowest set bit of a float that is not 0.
__device__ __forceinline__ int lsb_exp(float x) {
  const int b = __float_as_int(x), e = (b >> 23) & 0xff, m = b & 0x7fffff;
  return e ? e - 150 + __ffs(m | 0x800000) - 1 : -150 + __ffs(m);
}

// KC: k contiguous (sk == 1).  Single-precision operands (exact products, see
// k_oz_pick): the third sum is the lowest bit of the row's entries instead.
template <bool KC, class E>
__global__ void __launch_bounds__(256) k_oz_norm(int L, int K, const E* X, long ld, int cplx,
                                                  double4* part) {
  constexpr bool EXACT = sizeof(E) == 4;
  // block: 32 rows x 8 lanes along k (KC: warp-cooperative along k instead)
  const int chunk = blockIdx.y;
  const int k0 = chunk * kNormChunk, k1 = min(K, k0 + kNormChunk);
  double ss = 0.0, mx = 0.0, s1 = 0.0, nz = 0.0;
  int lo = 1000000, cnt = 0;
  auto merge = [](double a, double b) { return EXACT ? fmin(a, b) : a + b; };
  auto acc = [&](E x) {
    const double v = (double)x;
    ss = fma(v, v, ss);
    mx = fmax(mx, fabs(v));
    if constexpr (EXACT) {
      if (x != 0.0f) lo = min(lo, lsb_exp(x));
    } else {
      s1 += fabs(v);
      cnt += v != 0.0;
    }
  };
  // eight elements (complex: pairs) in flight; zeros past the end add nothing
  auto run = [&](int kb, int step, size_t base, size_t stride) {
    for (int k = kb; k < k1; k += 8 * step) {
      E a[8], b[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int kk = k + q * step;
        a[q] = b[q] = (E)0;
        if (kk < k1) {
          const size_t i = base + (size_t)kk * stride;
          if (cplx) {
            a[q] = X[2 * i];
            b[q] = X[2 * i + 1];
          } else {
            a[q] = X[i];
          }
        }
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        acc(a[q]);
        if (cplx) acc(b[q]);
      }
    }
    if (EXACT) s1 = (double)lo;
    nz = (double)cnt;
  };
  if constexpr (KC) {
    // one warp per row: lanes stride along contiguous k
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int l = blockIdx.x * 8 + warp;
    if (l < L) run(k0 + lane, 32, (size_t)l * ld, 1);
    else if (EXACT) s1 = 1.0e6;
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      ss += __shfl_xor_sync(0xffffffffu, ss, o);
      mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      s1 = merge(s1, __shfl_xor_sync(0xffffffffu, s1, o));
      nz += __shfl_xor_sync(0xffffffffu, nz, o);
    }
    if (lane == 0 && l < L) part[(size_t)chunk * L + l] = make_double4(ss, mx, s1, nz);
  } else {
    // l contiguous: 32 consecutive rows per warp-row, 8 k-lanes
    __shared__ double4 red[8][32];
    const int tl = threadIdx.x & 31, tk = threadIdx.x >> 5;
    const int l = blockIdx.x * 32 + tl;
    if (l < L) run(k0 + tk, 8, (size_t)l, (size_t)ld);
    red[tk][tl] = make_double4(ss, mx, s1, nz);
    __syncthreads();
    if (tk == 0 && l < L) {
      double4 t = red[0][tl];
      for (int i = 1; i < 8; ++i) {
        t.x += red[i][tl].x;
        t.y = fmax(t.y, red[i][tl].y);
        t.z = merge(t.z, red[i][tl].z);
        t.w += red[i][tl].w;
      }
      part[(size_t)chunk * L + l] = t;
    }
  }
}

// 2^e as a double for -1022 <= e <= 1023 (exact, no libm call)
__device__ __forceinline__ double pow2(int e) {
  return __longlong_as_double((long long)(1023 + e) << 52);
}

// Row codes written by k_oz_stat: the exponent e of a bound nrm < 2^e of the
// row's 2-norm, or one of two sentinels.  The shift of the row is H - e.
constexpr int kShiftNonFinite = -100000;  // the row holds Inf/NaN: results NaN
constexpr int kCodeZero = 100000;         // all-zero row: shift 0

__device__ __forceinline__ int shift_of(int code, int H) {
  if (code == kShiftNonFinite) return kShiftNonFinite;
  if (code == kCodeZero) return 0;
  return max(-1000, min(1000, H - code));  // scaled values stay finite
}

// Per row: the code above, and the row's concentration
// rho = sqrt(nnz) ||x||_2 / ||x||_1 (1 for entries of one magnitude, up to
// sqrt(nnz) for one dominant entry), whose maximum over the rows goes to
// *rmax (a non-negative float compared as its bits).
// exact (single precision): *rmax is the largest number of bits from a row's
// lowest set bit up to its norm's exponent instead (infinite when a row holds
// Inf / NaN): with at least that budget H the scaled rows are integers.
__global__ void k_oz_stat(int L, int K, int nchunks, const double4* part, int* code,
                          unsigned* rmax, int exact) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  float rho = 0.0f;
  if (l < L) {
    double ss = 0.0, mx = 0.0, s1 = exact ? 1.0e6 : 0.0, nz = 0.0;
    for (int c = 0; c < nchunks; ++c) {  // fixed order: deterministic
      const double4 v = part[(size_t)c * L + l];
      ss += v.x;
      mx = fmax(mx, v.y);
      s1 = exact ? fmin(s1, v.z) : s1 + v.z;
      nz += v.w;
    }
    if (!isfinite(mx) || isnan(ss)) {
      code[l] = kShiftNonFinite;
      if (exact) rho = __int_as_float(0x7f800000);
    } else if (mx == 0.0) {
      code[l] = kCodeZero;
    } else {
      // bound on the row 2-norm (the sum of squares may overflow for huge entries)
      double nrm = isfinite(ss) ? sqrt(ss) : mx * sqrt((double)K);
      nrm = fmax(nrm, mx) * (1.0 + 1e-12);
      int e;
      frexp(nrm, &e);  // nrm < 2^e
      code[l] = e;
      if (exact) rho = (float)(e - (int)s1);
      // scale-free form: sqrt(nnz) * (nrm / mx) / (s1 / mx), all ratios <= nnz
      const double r = sqrt(nz) * (nrm / mx) / fmax(s1 / mx, 1.0);
      if (!exact) rho = (float)fmin(r, 3.0e38);
    }
  }
  // warp maximum, one atomic per warp
#pragma unroll
  for (int o = 16; o; o >>= 1) rho = fmaxf(rho, __shfl_xor_sync(0xffffffffu, rho, o));
  if ((threadIdx.x & 31) == 0 && rho > 0.0f) atomicMax(rmax, __float_as_uint(rho));
}

// Moduli-count rule.  The scaled, rounded operands lose at most half a unit
// per nonzero entry; with errors of random sign the contraction error
// relative to sum_k |a_ik||b_kj| is about 0.58 rho_i sigma_j 2^-H, and its
// maximum over many entries about four times that (rho, sigma: the
// concentrations of row i of op(A) and column j of op(B)).  The smallest
// count with 2.31 rho_max sigma_max 2^-H <= 2^-53 keeps the result within
// FP64 rounding; if the largest count cannot, the call runs the plain FP64
// kernel instead (fallback = 1), or, where that is not allowed, the largest
// count.  fixed > 0: that count, no data rule.
// Exact products (single-precision operands): the smallest count whose budget
// scales every row and column to integers without rounding, so that the
// product is the exact one; else the plain kernel.
struct PickP {
  int fixed, lo, hi, allow_fallback, exact;
  int H[kMaxMod + 1];        // exponent budget per count
  int np[kMaxMod + 1];       // moduli multiplied per count
  int Hx[kMaxC + 1];         // exact: budget per moduli multiplied
};

__global__ void k_oz_pick(const unsigned* rmax, OzSel* sel, const PickP q) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  int n = q.fixed, fb = 0;
  if (q.exact) {
    const float need = fmaxf(__uint_as_float(rmax[0]), __uint_as_float(rmax[1]));
    int h = 0;
    n = 0;
#pragma unroll
    for (int c = kMaxC; c >= 2; --c)
      if (c >= q.lo && c <= q.hi && (float)q.Hx[c] >= need) n = c, h = q.Hx[c];
    sel->n = n;
    sel->H = h;
    sel->fallback = n == 0;
    sel->np = n;
    atomicAdd(&g_ex_calls, 1ull);
    if (n == 0) atomicAdd(&g_ex_plain, 1ull);
    g_ex_last = n;
    return;
  }
  if (n <= 0) {
    const double ra = fmax(1.0, (double)__uint_as_float(rmax[0]));
    const double rb = fmax(1.0, (double)__uint_as_float(rmax[1]));
    const double need = 53.0 + log2(2.31 * ra * rb);
    n = 0;
#pragma unroll
    for (int c = kMaxMod; c >= 2; --c)  // constant indices: no local copy of q.H
      if (c >= q.lo && c <= q.hi && (double)q.H[c] >= need) n = c;
    if (n == 0) {
      if (q.allow_fallback) fb = 1;
      else n = q.hi;
    }
  }
  sel->n = n;
  sel->H = n ? q.H[n] : 0;
  sel->fallback = fb;
  int np = 0;
#pragma unroll
  for (int c = kMaxMod; c >= 2; --c)
    if (c == n) np = q.np[c];
  sel->np = np;
  atomicAdd(&g_oz_calls, 1ull);
  atomicAdd(&g_oz_mod_sum, (unsigned long long)n);
  if (fb) atomicAdd(&g_oz_fallbacks, 1ull);
  g_oz_last = n;
}

// ---------------------------------------------------------------------------
// 2. residues: planes[m][l][k] (int8, row stride Kpad) for l < Lpad, k < Kpad
//    (zero padding), from X (L x K view, KC: k contiguous).  Complex operands
//    (cplx = 1) are handled by the caller through the concatenated views.
// Residue planes 1 .. min(CNT, n) - 1 of four consecutive elements whose
// offset values a' = a + 2^62 have 32-bit halves lo, hi (plane 0 is written
// by the caller).
template <int CNT>
__device__ __forceinline__ void res_planes(const Consts& c, const uint32_t (&lo)[4],
                                           const uint32_t (&hi)[4], int8_t* dst, size_t plane,
                                           int n) {
#pragma unroll
  for (int m = 1; m < CNT; ++m) {
    if (m >= n) break;
    const uint32_t p = (uint32_t)c.p[m];
    uint32_t r[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      // s = a' mod p + h (mod p) from the bytes of a': offh + sum_t byte_t
      // (2^(8t) mod p) < 2^21; q = floor(s / p) exactly by the 32-bit
      // reciprocal ceil(2^32 / p) (error s * 2^-32 < 1/p); s - q p - h is
      // the symmetric residue in [-h, h]
      uint32_t sacc = __dp4a(lo[v], c.wlo[m], c.offh[m]);
      sacc = __dp4a(hi[v], c.whi[m], sacc);
      const uint32_t q = __umulhi(sacc, c.magic[m]);
      r[v] = sacc - q * p - (uint32_t)c.half[m];
    }
    *reinterpret_cast<uint32_t*>(dst + (size_t)m * plane) =
        __byte_perm(__byte_perm(r[0], r[1], 0x0040), __byte_perm(r[2], r[3], 0x0040), 0x5410);
  }
}

template <bool KC, int NM, class E>
__global__ void __launch_bounds__(256) k_oz_residues(int L, int K, const E* X, long ld,
                                                      const int* code, const OzSel* sel,
                                                      const Consts c, int8_t* planes, long Lpad,
                                                      long Kpad) {
  // X element (l,k) = X[KC ? k + l*ld : l + k*ld];
  // planes 0 .. sel->n - 1 are written (NM: the most the call may use)
  const int nm = sel->n, H = sel->H;
  if (nm == 0) return;  // the plain kernel computes this call
  __shared__ double tile[64][65];
  const int l0 = blockIdx.x * 64, k0 = blockIdx.y * 64;
  {
    // all 16 loads of a thread in flight before the shared stores
    double v[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const int e = threadIdx.x + q * 256;
      const int ll = KC ? e >> 6 : e & 63, kk = KC ? e & 63 : e >> 6;
      const int l = l0 + ll, k = k0 + kk;
      v[q] = 0.0;
      if (l < L && k < K) {
        const size_t idx = KC ? (size_t)k + (size_t)l * ld : (size_t)l + (size_t)k * ld;
        v[q] = (double)X[idx];
      }
    }
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const int e = threadIdx.x + q * 256;
      const int ll = KC ? e >> 6 : e & 63, kk = KC ? e & 63 : e >> 6;
      tile[ll][kk] = v[q];
    }
  }
  __syncthreads();
  const size_t plane = (size_t)Lpad * (size_t)Kpad;
  for (int it = threadIdx.x; it < 64 * 16; it += 256) {
    const int ll = it >> 4, kq = (it & 15) * 4;
    const int l = l0 + ll;
    const int s = (l < L) ? shift_of(code[l], H) : 0;
    // a' = a + 2^62 >= 0 (|a| < 2^62); residues of a' are shifted back by the
    // per-modulus constant folded into c.off (no sign handling per modulus)
    const double sc = (s == kShiftNonFinite) ? 0.0 : pow2(s / 2) * pow2(s - s / 2);
    long long a[4];
    uint32_t lo[4], hi[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const double x = tile[ll][kq + v] * sc;  // exact power-of-two scaling
      a[v] = llrint(x);
      const unsigned long long u = (unsigned long long)a[v] + (1ull << 62);
      lo[v] = (uint32_t)u;
      hi[v] = (uint32_t)(u >> 32);
    }
    int8_t* dst = planes + (size_t)l * Kpad + k0 + kq;
    // p_0 = 256: the two's complement low byte (the offset 2^62 is 0 mod 256)
    *reinterpret_cast<uint32_t*>(dst) =
        __byte_perm(__byte_perm(lo[0], lo[1], 0x0040), __byte_perm(lo[2], lo[3], 0x0040), 0x5410);
    // planes 1 .. nm-1, unrolled for the plan's largest count and the one
    // below it (the data rule's two counts); other counts take a loop
    if (nm == NM) res_planes<NM>(c, lo, hi, dst, plane, NM);
    else if (NM > 2 && nm == NM - 1)
      res_planes<(NM > 2 ? NM - 1 : NM)>(c, lo, hi, dst, plane, NM - 1);
    else res_planes<NM>(c, lo, hi, dst, plane, nm);
  }
}

// Residue planes of a complex operand: planes 2m and 2m + 1 hold a + jb and
// a - jb mod p_m of every element a + ib (sign = -1: of its conjugate); element
// (l, k) = X[2 (KC ? k + l ld : l + k ld)].  The grid covers Lpad x Kpad.
template <bool KC, class E>
__global__ void __launch_bounds__(256) k_oz_residues_c(int L, int K, const E* X, long ld,
                                                        double sign, const int* code,
                                                        const OzSel* sel, const CResConsts c,
                                                        int8_t* planes, long Lpad, long Kpad) {
  using E2 = typename std::conditional<sizeof(E) == 4, float2, double2>::type;
  const int nm = sel->np, H = sel->H;
  if (nm == 0) return;
  __shared__ double tr[64][33], ti[64][33];
  const int l0 = blockIdx.x * 64, k0 = blockIdx.y * 32;
  {
    E2 v[8];  // all loads of a thread in flight before the shared stores
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int e = threadIdx.x + q * 256;
      const int l = l0 + (KC ? e >> 5 : e & 63), k = k0 + (KC ? e & 31 : e >> 6);
      v[q].x = v[q].y = (E)0;
      if (l < L && k < K) {
        const size_t idx = KC ? (size_t)k + (size_t)l * ld : (size_t)l + (size_t)k * ld;
        v[q].x = X[2 * idx];
        v[q].y = X[2 * idx + 1];
      }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int e = threadIdx.x + q * 256;
      tr[KC ? e >> 5 : e & 63][KC ? e & 31 : e >> 6] = (double)v[q].x;
      ti[KC ? e >> 5 : e & 63][KC ? e & 31 : e >> 6] = sign * (double)v[q].y;
    }
  }
  __syncthreads();
  const size_t plane = (size_t)Lpad * (size_t)Kpad;
#pragma unroll 1
  for (int it = threadIdx.x; it < 64 * 8; it += 256) {
    const int ll = it >> 3, kq = (it & 7) * 4;
    const int l = l0 + ll;
    const int s = (l < L) ? shift_of(code[l], H) : 0;
    const double sc = (s == kShiftNonFinite) ? 0.0 : pow2(s / 2) * pow2(s - s / 2);
    uint32_t rl[4], rh[4], il[4], ih[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) {  // offset values a + 2^62, b + 2^62
      const unsigned long long u =
          (unsigned long long)llrint(tr[ll][kq + v] * sc) + (1ull << 62);
      const unsigned long long w =
          (unsigned long long)llrint(ti[ll][kq + v] * sc) + (1ull << 62);
      rl[v] = (uint32_t)u, rh[v] = (uint32_t)(u >> 32);
      il[v] = (uint32_t)w, ih[v] = (uint32_t)(w >> 32);
    }
    int8_t* dst = planes + (size_t)l * Kpad + k0 + kq;
#pragma unroll
    for (int m = 0; m < kMaxC; ++m) {
      if (m >= nm) break;
      const uint32_t p = (uint32_t)c.p[m], h = (uint32_t)c.half[m], mg = c.magic[m];
      uint32_t rp[4], rm[4];
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        // sums of bytes times 2^(8t) mod p: below 2^22 with the offsets, so
        // umulhi by ceil(2^32 / p) is the exact quotient
        const uint32_t sa = __dp4a(rh[v], c.whi[m], __dp4a(rl[v], c.wlo[m], c.off[m]));
        const uint32_t sj = __dp4a(ih[v], c.jhi[m], __dp4a(il[v], c.jlo[m], c.offj[m]));
        const uint32_t a = sa + sj, b = sa + (c.cp[m] - sj);
        rp[v] = a - __umulhi(a, mg) * p - h;
        rm[v] = b - __umulhi(b, mg) * p - h;
      }
      *reinterpret_cast<uint32_t*>(dst + (size_t)(2 * m) * plane) = __byte_perm(
          __byte_perm(rp[0], rp[1], 0x0040), __byte_perm(rp[2], rp[3], 0x0040), 0x5410);
      *reinterpret_cast<uint32_t*>(dst + (size_t)(2 * m + 1) * plane) = __byte_perm(
          __byte_perm(rm[0], rm[1], 0x0040), __byte_perm(rm[2], rm[3], 0x0040), 0x5410);
    }
  }
}

// ---------------------------------------------------------------------------
// 3. INT8 tensor-core GEMM: persistent CTAs (one per SM) walking the
//    (modulus, 128 x 256 C tile) list.  Warp 0: TMA producer into a 4-stage
//    ring; warp 1: TMEM allocator (512 columns = two 256-column accumulators)
//    and single-thread MMA issuer; warps 2-5: epilogue.  The accumulator is
//    double buffered, so the epilogue of tile i (TMEM -> registers -> mod p ->
//    uint8 plane) runs while the MMAs of tile i+1 fill the other buffer.
constexpr int BM = 128, BN = 256, BKB = 128;  // BKB: k bytes per stage
constexpr int S = 4;
constexpr uint32_t A_STAGE = BM * BKB, B_STAGE = BN * BKB;
constexpr int kGemmThreads = 192;
constexpr uint32_t kTmemCols = 512;  // two accumulators of BN columns
constexpr int kEpiWarps = 4;

struct GemmP {
  int tiles_m, tiles_n, kblocks, nmod;  // nmod: planes of the operand buffers (the most used)
  const OzSel* sel;                     // planes multiplied: mult sel->np (<= nmod)
  int mult;                             // planes per modulus: 1, complex 2
  const int* list;  // not null: list[0] tiles (list[1 ..]) of every plane are in the triangle
  int bxor;  // plane z of op(A) meets plane z ^ bxor of op(B) (1: B is A's conjugate)
  int group;  // raster: M tiles per group (tiles in flight share A / B panels in L2)
  uint8_t* R;
  long Mpad, Npad;
  int uplo;
  long diag;
  int p[kMaxPl];
  uint32_t bias[kMaxPl], magic[kMaxPl];  // of the epilogue's mod p
};

__device__ __forceinline__ uint64_t desc_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);  // start address
  d |= (uint64_t)1 << 16;                    // leading byte offset (unused, K-major swizzled)
  d |= (uint64_t)(1024 >> 4) << 32;          // stride byte offset: 8 rows x 128 B
  d |= (uint64_t)1 << 46;                    // descriptor version (sm_100)
  d |= (uint64_t)2 << 61;                    // 128-byte swizzle
  return d;
}

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tc_mma_i8(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t idesc,
                                          uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
      "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* m, int x, int y, int z,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}

// tile t of the (modulus-major, grouped raster) list; false if the tile lies
// wholly outside the written triangle
__device__ __forceinline__ bool oz_tile(const GemmP& p, int t, int& mod, int& m0, int& n0) {
  const int tiles_mn = p.list ? p.list[0] : p.tiles_m * p.tiles_n;
  mod = t / tiles_mn;
  int r = t - mod * tiles_mn;
  if (p.list) r = p.list[1 + r];
  const int GROUP = p.group;
  const int span = GROUP * p.tiles_n;
  const int first_m = (r / span) * GROUP;
  const int gsz = min(p.tiles_m - first_m, GROUP);
  const int tm = first_m + (r % span) % gsz;
  const int tn = (r % span) / gsz;
  m0 = tm * BM;
  n0 = tn * BN;
  if (p.uplo == XKB_LOWER && (long)(m0 + BM - 1) + p.diag < (long)n0) return false;
  if (p.uplo == XKB_UPPER && (long)m0 + p.diag > (long)(n0 + BN - 1)) return false;
  return true;
}

// The tiles of one plane that meet the triangle, in raster order (one block of
// 1024 threads).  Walking all tiles with a fixed stride and skipping those
// outside gave the CTAs uneven shares: 4 to 10 % of a ZHERK 8192, by the
// raster group.
__global__ void __launch_bounds__(1024) k_oz_tiles(const GemmP p, int* list) {
  __shared__ int sums[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int base = 0;
  for (int r0 = 0; r0 < p.tiles_m * p.tiles_n; r0 += 1024) {
    const int r = r0 + (int)threadIdx.x;
    int mod, m0, n0;
    const bool in = r < p.tiles_m * p.tiles_n && oz_tile(p, r, mod, m0, n0);
    const unsigned b = __ballot_sync(0xffffffffu, in);
    if (lane == 0) sums[warp] = __popc(b);
    __syncthreads();
    int before = base, all = 0;
    for (int w = 0; w < 32; ++w) {
      if (w < warp) before += sums[w];
      all += sums[w];
    }
    if (in) list[1 + before + __popc(b & ((1u << lane) - 1u))] = r;
    base += all;
    __syncthreads();
  }
  if (threadIdx.x == 0) list[0] = base;
}

__device__ __forceinline__ void tmem_ld32(uint32_t (&v)[32], uint32_t addr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,"
      "%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
        "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
        "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]),
        "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]),
        "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(addr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Epilogue of one warp: its 32 TMEM lanes (rows) x 256 columns of an
// accumulator -> mod p -> uint8 plane R[column / 16][row][column % 16] (blocks
// of 16 columns: a lane's 16 bytes lie beside its neighbours', here and when
// the CRT reads them), 32 columns per lane at a time; drained() is called
// once every column is in registers.  The residue by integers: u = acc + bias is non-negative (bias:
// the multiple of p from 2^31 on; |acc| < 2^31 - 2^24 for p < 256, and for
// p = 256 wrapping is exact), q = umulhi(u, ceil(2^32 / p)) is floor(u / p)
// or one more, so r = u - q p or that plus p.  (By FP64 -- two conversions
// and a floor per element, a byte store per element -- the epilogue took
// longer than the MMAs below K of about 1500.)
template <class F>
__device__ __forceinline__ void oz_epilogue(const GemmP& p, int mod, int row, int n0,
                                            uint32_t tbase, F drained) {
  const uint32_t pm = (uint32_t)p.p[mod], bias = p.bias[mod], magic = p.magic[mod];
  uint8_t* dst = p.R + (size_t)mod * (size_t)p.Mpad * (size_t)p.Npad +
                 (size_t)n0 * (size_t)p.Mpad + (size_t)row * 16;
  const size_t blk = (size_t)p.Mpad * 16;  // bytes of a block of 16 columns
#pragma unroll 1
  for (int c = 0; c < 256 / 32; ++c) {
    uint32_t v[32];
    tmem_ld32(v, tbase + (uint32_t)(c * 32));
    if (c == 256 / 32 - 1) {
      tc_fence_before();
      __syncwarp();
      drained();
    }
    uint32_t w[8];
#pragma unroll
    for (int e = 0; e < 32; ++e) {
      const uint32_t u = v[e] + bias;
      const uint32_t r = u - __umulhi(u, magic) * pm;
      v[e] = min(r, r + pm);
    }
#pragma unroll
    for (int e = 0; e < 8; ++e)
      w[e] = __byte_perm(__byte_perm(v[4 * e], v[4 * e + 1], 0x0040),
                         __byte_perm(v[4 * e + 2], v[4 * e + 3], 0x0040), 0x5410);
    // streaming stores: the planes are read once, by the CRT kernel; they
    // should not evict the operand panels from L2
    __stcs(reinterpret_cast<uint4*>(dst), make_uint4(w[0], w[1], w[2], w[3]));
    __stcs(reinterpret_cast<uint4*>(dst + blk), make_uint4(w[4], w[5], w[6], w[7]));
    dst += 2 * blk;
  }
}

__global__ void __launch_bounds__(kGemmThreads, 1)
    k_oz_gemm(const __grid_constant__ CUtensorMap tA, const __grid_constant__ CUtensorMap tB,
              const GemmP p) {
  extern __shared__ uint8_t sm_raw[];
  uint8_t* sm =
      reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(sm_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sA = sm;
  uint8_t* sB = sm + S * A_STAGE;
  uint64_t* full = reinterpret_cast<uint64_t*>(sB + S * B_STAGE);
  uint64_t* empty = full + S;
  uint64_t* accf = empty + S;  // [2] accumulator ready
  uint64_t* acce = accf + 2;   // [2] accumulator drained
  uint32_t* tslot = reinterpret_cast<uint32_t*>(acce + 2);

  const int total =
      (p.list ? p.list[0] : p.tiles_m * p.tiles_n) * min(p.sel->np * p.mult, p.nmod);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&accf[b], 1);
      mbar_init(&acce[b], kEpiWarps);
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tslot)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    tc_fence_before();
  }
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tslot);
  const int KB = p.kblocks;

  if (warp == 0) {
    if (lane == 0) {  // ---- TMA producer
      tma_prefetch(&tA);
      tma_prefetch(&tB);
      uint32_t it = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
        int mod, m0, n0;
        if (!oz_tile(p, t, mod, m0, n0)) continue;
        for (int kb = 0; kb < KB; ++kb, ++it) {
          const int s = it % S;
          const uint32_t ph = (it / S) & 1;
          if (!mbar_wait(&empty[s], ph ^ 1, kErrEmptyWait)) {
            ok = false;
            break;
          }
          mbar_expect_tx(&full[s], A_STAGE + B_STAGE);
          tma_load_3d(sA + s * A_STAGE, &tA, kb * BKB, m0, mod, &full[s]);
          tma_load_3d(sB + s * B_STAGE, &tB, kb * BKB, n0, mod ^ p.bxor, &full[s]);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {  // ---- MMA issuer
      // kind::i8: D s32 (2 << 4), A s8 (1 << 7), B s8 (1 << 10), K-major A/B,
      // N >> 3 at bit 17, M >> 4 at bit 24
      const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) |
                             ((uint32_t)(BM >> 4) << 24);
      uint32_t it = 0, tl = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
        int mod, m0, n0;
        if (!oz_tile(p, t, mod, m0, n0)) continue;
        const int b = tl & 1;
        const uint32_t aph = (tl >> 1) & 1;
        if (!mbar_wait(&acce[b], aph ^ 1, kErrAccWait)) break;  // buffer drained
        tc_fence_after();
        const uint32_t d = tmem + (uint32_t)(b * BN);
        for (int kb = 0; kb < KB; ++kb, ++it) {
          const int s = it % S;
          const uint32_t ph = (it / S) & 1;
          if (!mbar_wait(&full[s], ph, kErrFullWait)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a0 = smem_u32(sA + s * A_STAGE), b0 = smem_u32(sB + s * B_STAGE);
#pragma unroll
          for (int k = 0; k < BKB / 32; ++k)
            tc_mma_i8(d, desc_sw128(a0 + 32 * k), desc_sw128(b0 + 32 * k), idesc,
                      (kb | k) != 0 ? 1u : 0u);
          tc_commit(&empty[s]);  // stage s free once these MMAs have read it
        }
        tc_commit(&accf[b]);  // accumulator b complete (also drains an aborted loop)
        ++tl;
      }
    }
  } else {
    // ---- epilogue: warps 2..5, TMEM lanes 32*(warp%4) .. +31
    const int q = warp & 3;
    uint32_t tl = 0;
    for (int t = blockIdx.x; t < total; t += gridDim.x) {
      int mod, m0, n0;
      if (!oz_tile(p, t, mod, m0, n0)) continue;
      const int b = tl & 1;
      const uint32_t aph = (tl >> 1) & 1;
      const bool got = mbar_wait(&accf[b], aph, kErrAccWait);
      if (!__all_sync(0xffffffffu, got)) break;  // uniform and converged for tcgen05.ld
      tc_fence_after();
      const int row = m0 + q * 32 + lane;
      const uint32_t tbase = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * BN);
      oz_epilogue(p, mod, row, n0, tbase, [&] {
        if (lane == 0) mbar_arrive(&acce[b]);
      });
      ++tl;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(kTmemCols)
                 : "memory");
  }
}

// ---------------------------------------------------------------------------
// 3b. The same product on CTA pairs (a cluster of 2): tcgen05.mma.cta_group::2
//     computes a 256 x 256 tile per pair, each CTA holding 128 rows of A and
//     128 rows of B (its half of N) in shared memory and 128 rows of the
//     accumulator in its TMEM.  Per CTA and stage: 16 KB of A + 16 KB of B
//     for the work that takes 16 + 32 KB in the single-CTA kernel, so a third
//     less operand traffic from L2 per MMA.  Both CTAs load their halves with
//     TMA; the loads signal the even CTA's stage barrier, the even CTA
//     issues the MMAs and commits to the barriers of both CTAs, and
//     the odd CTA's epilogue warps release the accumulator on the even CTA's
//     barrier.
constexpr int BM2 = 256, BN2 = 256;                 // pair tile
constexpr int S2 = 6;                               // stages
constexpr uint32_t H_STAGE = 128 * BKB;             // one 128-row operand half per stage
constexpr uint32_t kPeerMask = 0xFEFFFFFFu;         // shared::cluster address of the even CTA

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t mapa_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::
                   : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr)
               : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair(void* dst, const CUtensorMap* m, int x, int y,
                                                 int z, uint32_t bar_even) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(x), "r"(y), "r"(z), "r"(bar_even)
      : "memory");
}
__device__ __forceinline__ void tc_mma_i8_pair(uint32_t tmem, uint64_t ad, uint64_t bd,
                                               uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem),
      "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
      : "memory");
}
// commit the MMAs issued so far to the barrier at this offset in both CTAs
// (one commit per CTA, addressed through the cluster window)
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar) {
#pragma unroll
  for (uint32_t r = 0; r < 2; ++r)
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::
                     "r"(mapa_rank(smem_u32(bar), r))
                 : "memory");
}

__device__ __forceinline__ bool oz_tile2(const GemmP& p, int t, int& mod, int& m0, int& n0) {
  const int tiles_mn = p.tiles_m * p.tiles_n;
  mod = t / tiles_mn;
  const int r = t - mod * tiles_mn;
  const int GROUP = p.group;
  const int span = GROUP * p.tiles_n;
  const int first_m = (r / span) * GROUP;
  const int gsz = min(p.tiles_m - first_m, GROUP);
  const int tm = first_m + (r % span) % gsz;
  const int tn = (r % span) / gsz;
  m0 = tm * BM2;
  n0 = tn * BN2;
  if (p.uplo == XKB_LOWER && (long)(m0 + BM2 - 1) + p.diag < (long)n0) return false;
  if (p.uplo == XKB_UPPER && (long)m0 + p.diag > (long)(n0 + BN2 - 1)) return false;
  return true;
}

__global__ void __launch_bounds__(kGemmThreads, 1)
    k_oz_gemm2(const __grid_constant__ CUtensorMap tA, const __grid_constant__ CUtensorMap tB,
               const GemmP p) {
  extern __shared__ uint8_t sm_raw[];
  uint8_t* sm =
      reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(sm_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sA = sm;
  uint8_t* sB = sm + S2 * H_STAGE;
  uint64_t* full = reinterpret_cast<uint64_t*>(sB + S2 * H_STAGE);
  uint64_t* empty = full + S2;
  uint64_t* accf = empty + S2;  // [2] accumulator ready (both CTAs)
  uint64_t* acce = accf + 2;    // [2] accumulator drained (even CTA: both epilogues)
  uint32_t* tslot = reinterpret_cast<uint32_t*>(acce + 2);

  const uint32_t rank = cluster_rank();
  const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
  const int total = p.tiles_m * p.tiles_n * min(p.sel->np * p.mult, p.nmod);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S2; ++s) {
      mbar_init(&full[s], 1);  // the even CTA expects the bytes of both CTAs' loads
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&accf[b], 1);
      mbar_init(&acce[b], 2 * kEpiWarps);
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tslot)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    tc_fence_before();
  }
  __syncthreads();
  cluster_sync();  // barriers of both CTAs initialised before any cross-CTA signal
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tslot);
  const int KB = p.kblocks;

  if (warp == 0) {
    if (lane == 0) {  // ---- TMA producer (both CTAs): this CTA's halves of A and B
      tma_prefetch(&tA);
      tma_prefetch(&tB);
      uint32_t it = 0;
      bool ok = true;
      for (int t = pair; t < total && ok; t += npairs) {
        int mod, m0, n0;
        if (!oz_tile2(p, t, mod, m0, n0)) continue;
        for (int kb = 0; kb < KB; ++kb, ++it) {
          const int s = it % S2;
          const uint32_t ph = (it / S2) & 1;
          if (!mbar_wait(&empty[s], ph ^ 1, kErrEmptyWait)) {
            ok = false;
            break;
          }
          // the even CTA's stage barrier (the pair-form TMA names it with the
          // peer bit cleared) counts the four halves.  The odd CTA signals it
          // by its bytes only: a remote arrive per stage held its producer
          // back for longer than the stage's MMAs
          if (rank == 0) mbar_expect_tx(&full[s], 4 * H_STAGE);
          const uint32_t fe = smem_u32(&full[s]) & kPeerMask;
          tma_load_3d_pair(sA + s * H_STAGE, &tA, kb * BKB, m0 + 128 * (int)rank, mod, fe);
          tma_load_3d_pair(sB + s * H_STAGE, &tB, kb * BKB, n0 + 128 * (int)rank, mod ^ p.bxor,
                           fe);
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {  // ---- MMA issuer (even CTA)
      // kind::i8: D s32, A s8, B s8, K-major; N = 256, M = 256 (the pair)
      const uint32_t idesc = (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN2 >> 3) << 17) |
                             ((uint32_t)(BM2 >> 4) << 24);
      uint32_t it = 0, tl = 0;
      bool ok = true;
      for (int t = pair; t < total && ok; t += npairs) {
        int mod, m0, n0;
        if (!oz_tile2(p, t, mod, m0, n0)) continue;
        const int b = tl & 1;
        const uint32_t aph = (tl >> 1) & 1;
        if (!mbar_wait(&acce[b], aph ^ 1, kErrAccWait)) break;  // drained in both CTAs
        tc_fence_after();
        const uint32_t d = tmem + (uint32_t)(b * BN2);
        for (int kb = 0; kb < KB; ++kb, ++it) {
          const int s = it % S2;
          const uint32_t ph = (it / S2) & 1;
          if (!mbar_wait(&full[s], ph, kErrFullWait)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a0 = smem_u32(sA + s * H_STAGE), b0 = smem_u32(sB + s * H_STAGE);
#pragma unroll
          for (int k = 0; k < BKB / 32; ++k)
            tc_mma_i8_pair(d, desc_sw128(a0 + 32 * k), desc_sw128(b0 + 32 * k), idesc,
                           (kb | k) != 0 ? 1u : 0u);
          tc_commit_pair(&empty[s]);  // stage s free in both CTAs once read
        }
        tc_commit_pair(&accf[b]);  // accumulator b complete in both CTAs
        ++tl;
      }
    }
  } else {
    // ---- epilogue (both CTAs): warps 2..5, TMEM lanes 32*(warp%4) .. +31
    const int q = warp & 3;
    const uint32_t ae0 = mapa_rank(smem_u32(&acce[0]), 0), ae1 = mapa_rank(smem_u32(&acce[1]), 0);
    uint32_t tl = 0;
    for (int t = pair; t < total; t += npairs) {
      int mod, m0, n0;
      if (!oz_tile2(p, t, mod, m0, n0)) continue;
      const int b = tl & 1;
      const uint32_t aph = (tl >> 1) & 1;
      const bool got = mbar_wait(&accf[b], aph, kErrAccWait);
      if (!__all_sync(0xffffffffu, got)) break;  // uniform and converged for tcgen05.ld
      tc_fence_after();
      const int row = m0 + 128 * (int)rank + q * 32 + lane;
      const uint32_t tbase = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * BN2);
      oz_epilogue(p, mod, row, n0, tbase, [&] {
        if (lane == 0) mbar_arrive_cluster(b ? ae1 : ae0);
      });
      ++tl;
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();  // both CTAs done with the pair's TMEM and barriers
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(kTmemCols)
                 : "memory");
  }
}

// ---------------------------------------------------------------------------
// 4. CRT reconstruction + scaling + alpha/beta, 16 columns of one row per thread.
struct CrtP {
  int M, N;
  const uint8_t* R;
  long Mpad, Npad;
  const int* mu;     // row codes of op(A) (k_oz_stat)
  const int* nu;     // column codes of op(B)
  const OzSel* sel;  // the call's moduli count and exponent budget
  void* C;
  long ldc;
  double ar, ai, br, bi;  // real: ar, br used
  int uplo, herm_diag;
  long diag;
};

// Recombination on the FP64 pipe.  S = sum_l r_l w_l < 4080 P; the shifts
// keep |C'| <= P/8, so the wanted value is S - qP with q = round(S / P).
// With w = w1 + w2 (w1: multiples of 2^csplit, <= 41 significant bits):
//  - S1 = sum r_l w1_l is exact (8-bit x 41-bit products, multiples of
//    2^csplit, sum below 2^(53+csplit));
//  - q = rint(S1 / P) is exact: S2 / P < 2^-28 and S / P lies within 1/8 of
//    an integer (q < 2^12);
//  - S1 - q P1 is exact (a 53-bit product, the difference a multiple of
//    2^csplit below 2^(42+csplit));
//  - S2 - q P2 carries absolute errors of order 2^(csplit-37) plus the
//    rounding of w2 (2^43 at 16 moduli), far below the 2^(2H-61) sqrt(K)
//    already left by rounding the scaled operands to integers.
// r_l becomes a double by one byte permutation (4096 + r_l) and an FP64 add: a
// conversion from int per residue takes longer than the sums.
// 2 FP64 FMAs per modulus and element (a 128-bit integer sum would take 4
// 64-bit integer multiply-adds).  The weights are constant loads, not operands
// of an FP64 FMA, so each is used for eight elements at once.

// x * 2^e for the shift range used here (|e| <= 2000), exact unless the
// result under/overflows
__device__ __forceinline__ double scale2(double x, int e) {
  // x normal and x 2^e normal: add e to the exponent field
  const int hi = __double2hiint(x);
  const int ex = (hi >> 20) & 0x7ff;
  if (ex != 0 && (unsigned)(ex + e - 1) < 2046u)
    return __hiloint2double(hi + (int)((unsigned)e << 20), __double2loint(x));
  const int e1 = e / 2, e2 = e - e1;
  return x * pow2(e1) * pow2(e2);
}

// byte b of w as a double: bytes 40 B0 r 00 are the high word of 4096 + r
__device__ __forceinline__ double crt_byte(uint32_t w, int b) {
  return __hiloint2double((int)__byte_perm(w, 0x40B00000u, 0x7604 + (b << 4)), 0) - 4096.0;
}

// A warp takes 16 rows x 16 columns: lane l row l / 2 and columns 8 (l % 2)
// .. + 7, so that each plane is read 256 contiguous bytes at a time and C's
// columns 128.
constexpr int kCrtRows = 16, kCrtCols = 16 * 8;  // of a block of eight warps

// The eight columns j0 + e of this thread: pre(i, j, e) for each (the loads of
// what f combines, issued together and before any store), then
// f(i, j, e, value); columns outside C or the triangle mask are left out.
template <int NM, class G, class F>
__device__ __forceinline__ void crt_cols(const CrtP& p, const Consts& c, int H, G pre, F f) {
  const size_t plane = (size_t)p.Mpad * (size_t)p.Npad;
  const int lane = threadIdx.x & 31;
  const int i0 = blockIdx.x * kCrtRows, i = i0 + (lane >> 1);
  const int jw = blockIdx.y * kCrtCols + (int)(threadIdx.x >> 5) * 16;  // the warp's columns
  const int j0 = jw + 8 * (lane & 1);
  const bool mask = p.uplo != XKB_FULL;
  // a block of 16 rows x 16 columns wholly outside the triangle
  if (p.uplo == XKB_LOWER && (long)i0 + kCrtRows - 1 + p.diag < (long)jw) return;
  if (p.uplo == XKB_UPPER && (long)i0 + p.diag > (long)jw + 15) return;
  if (i >= p.M || j0 >= p.N) return;
  uint2 words[NM];
  const uint8_t* src = p.R + (size_t)jw * (size_t)p.Mpad + (size_t)i * 16 + (size_t)(8 * (lane & 1));
#pragma unroll
  for (int m = 0; m < NM; ++m)
    words[m] = __ldcs(reinterpret_cast<const uint2*>(src + (size_t)m * plane));
  const int last = p.N - j0;  // columns of this thread inside C
  const bool whole = !mask && jw + 16 <= p.N;  // the warp's
  auto in = [&](int e) {
    if (whole) return true;
    if (e >= last) return false;
    if (!mask) return true;
    return p.uplo == XKB_LOWER ? (long)i + p.diag >= (long)(j0 + e)
                               : (long)i + p.diag <= (long)(j0 + e);
  };
  double s1[8], s2[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) s1[e] = s2[e] = 0.0;
#pragma unroll
  for (int m = 0; m < NM; ++m) {
    const double w1 = c.w1[m], w2 = c.w2[m];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const double rv = crt_byte(e < 4 ? words[m].x : words[m].y, e & 3);
      s1[e] = fma(rv, w1, s1[e]);
      s2[e] = fma(rv, w2, s2[e]);
    }
  }
#pragma unroll
  for (int e = 0; e < 8; ++e)
    if (in(e)) pre(i, j0 + e, e);
  const int mui = shift_of(p.mu[i], H);
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    if (!in(e)) continue;
    const double q = rint(s1[e] * c.invPd);
    const double v = fma(-q, c.P1d, s1[e]) + fma(-q, c.P2d, s2[e]);
    const int nuj = shift_of(p.nu[j0 + e], H);
    f(i, j0 + e, e, (mui == kShiftNonFinite || nuj == kShiftNonFinite)
                        ? __longlong_as_double(0x7ff8000000000000ll)
                        : scale2(v, -(mui + nuj)));
  }
}

template <int NM>
__device__ __forceinline__ void crt_body(const CrtP& p, const Consts& c, int H) {
  const bool beta = p.br != 0.0;
  double* C = static_cast<double*>(p.C);
  double cr[8];
  crt_cols<NM>(
      p, c, H,
      [&](int i, int j, int e) {
        if (beta) cr[e] = C[(size_t)i + (size_t)j * p.ldc];
      },
      [&](int i, int j, int e, double y) {
        double out = p.ar * y;
        if (beta) out = fma(p.br, cr[e], out);
        C[(size_t)i + (size_t)j * p.ldc] = out;
      });
}

// Complex recombination: a warp takes 8 rows x 16 columns, a lane row l / 4
// and the four columns 4 (l % 4) .. + 3; both parts of an element come from
// the planes 2m (c+) and 2m + 1 (c-) in one pass: c+ + c- meets the real
// part's weights, c+ - c- the imaginary part's.  Bounds as in the real form:
// the sums stay below 17 * 510 P < 2^(53+csplit), |q| < 2^14, and |C'| <= P/4
// leaves q = rint(S1 / P) exact.
constexpr int kCrtRowsC = 8;

template <int NM>
__device__ __forceinline__ void crt_body_c(const CrtP& p, const CCrtConsts& c, int H) {
  const size_t plane = (size_t)p.Mpad * (size_t)p.Npad;
  const int lane = threadIdx.x & 31;
  const int i0 = blockIdx.x * kCrtRowsC, i = i0 + (lane >> 2);
  const int jw = blockIdx.y * kCrtCols + (int)(threadIdx.x >> 5) * 16;
  const int j0 = jw + 4 * (lane & 3);
  if (p.uplo == XKB_LOWER && (long)i0 + kCrtRowsC - 1 + p.diag < (long)jw) return;
  if (p.uplo == XKB_UPPER && (long)i0 + p.diag > (long)jw + 15) return;
  if (i >= p.M || j0 >= p.N) return;
  uint32_t wp[NM], wm[NM];
  const uint8_t* src = p.R + (size_t)jw * (size_t)p.Mpad + (size_t)i * 16 + (size_t)(4 * (lane & 3));
#pragma unroll
  for (int m = 0; m < NM; ++m) {
    wp[m] = __ldcs(reinterpret_cast<const uint32_t*>(src + (size_t)(2 * m) * plane));
    wm[m] = __ldcs(reinterpret_cast<const uint32_t*>(src + (size_t)(2 * m + 1) * plane));
  }
  double r1[4], r2[4], x1[4], x2[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    r1[e] = r2[e] = x1[e] = x2[e] = 0.0;
  }
#pragma unroll
  for (int m = 0; m < NM; ++m) {
    const double w1 = c.w1[m], w2 = c.w2[m], v1 = c.v1[m], v2 = c.v2[m];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const double a = crt_byte(wp[m], e), b = crt_byte(wm[m], e);
      const double su = a + b, di = a - b;
      r1[e] = fma(su, w1, r1[e]);
      r2[e] = fma(su, w2, r2[e]);
      x1[e] = fma(di, v1, x1[e]);
      x2[e] = fma(di, v2, x2[e]);
    }
  }
  const bool beta = p.br != 0.0 || p.bi != 0.0;
  const bool mask = p.uplo != XKB_FULL;
  double* C = static_cast<double*>(p.C);
  auto in = [&](int e) {
    if (j0 + e >= p.N) return false;
    if (!mask) return true;
    return p.uplo == XKB_LOWER ? (long)i + p.diag >= (long)(j0 + e)
                               : (long)i + p.diag <= (long)(j0 + e);
  };
  double cr[4], ci[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    cr[e] = ci[e] = 0.0;
    if (beta && in(e)) {
      const size_t idx = (size_t)i + (size_t)(j0 + e) * p.ldc;
      cr[e] = C[2 * idx];
      ci[e] = C[2 * idx + 1];
    }
  }
  const int mui = shift_of(p.mu[i], H);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    if (!in(e)) continue;
    const int nuj = shift_of(p.nu[j0 + e], H);
    const double qr = rint(r1[e] * c.invPd), qi = rint(x1[e] * c.invPd);
    double xr = fma(-qr, c.P1d, r1[e]) + fma(-qr, c.P2d, r2[e]);
    double xi = fma(-qi, c.P1d, x1[e]) + fma(-qi, c.P2d, x2[e]);
    if (mui == kShiftNonFinite || nuj == kShiftNonFinite) {
      xr = xi = __longlong_as_double(0x7ff8000000000000ll);
    } else {
      xr = scale2(xr, -(mui + nuj));
      xi = scale2(xi, -(mui + nuj));
    }
    double vr = p.ar * xr - p.ai * xi;
    double vi = p.ar * xi + p.ai * xr;
    if (beta) {
      vr += p.br * cr[e] - p.bi * ci[e];
      vi += p.br * ci[e] + p.bi * cr[e];
    }
    if (p.herm_diag && (long)i + p.diag == (long)(j0 + e)) vi = 0.0;
    const size_t idx = (size_t)i + (size_t)(j0 + e) * p.ldc;
    C[2 * idx] = vr;
    C[2 * idx + 1] = vi;
  }
}

// CRT kernels.  A fixed count: one instance per count.  A count chosen on the
// device between 15 and 16 (the data rule's range, k_oz_pick): one kernel
// holding both reconstructions, each block taking the one sel->n names; the
// single-precision and complex kernels hold every count a call may come to.
// A call the pick sent to the plain kernel (sel->n == 0) writes nothing here.
template <int NM>
__global__ void __launch_bounds__(256, 3) k_oz_crt(const CrtP p, const Consts c) {
  const OzSel s = *p.sel;
  if (s.n != NM) return;
  crt_body<NM>(p, c, s.H);
}
__global__ void __launch_bounds__(256, 3) k_oz_crt_15_16(const CrtP p, const Consts c15,
                                                         const Consts c16) {
  const OzSel s = *p.sel;
  if (s.n == 15) crt_body<15>(p, c15, s.H);
  else if (s.n == 16) crt_body<16>(p, c16, s.H);
}

// Exact products (single precision).  A row whose entries are small beside
// the operand's largest may meet a column the same way, and its C' is then far
// below the 2^(csplit-36) that the two-part weights leave: here the weights
// have three parts of 41 (complex 39, 39, 40) bits and every sum is exact.
// Real: r_l < 2^8 and at most 15 moduli, P < 2^118: with c1 = bits(P) - 41,
// c2 = max(0, c1 - 41) <= 36, the sums S1, S2, S3 of r_l times the parts are
// multiples of 2^c1, 2^c2, 1 below 2^(53 + c1), 2^(53 + c2), 2^53, and so are
// S_i - q P_i (q = rint(S1 / P) < 2^12 as above, the products 53 bits).  Their
// sum is formed with one compensated addition: relative error 2^-52.
constexpr int kExactLo = 8, kExactHi = 15;    // moduli of an exact product
constexpr int kExactLoC = 9, kExactHiC = 16;  // and of a complex one
struct Crt3 {
  double w[3][kMaxC];  // times r, complex: the real part's, times c+ + c-
  double v[3][kMaxC];  // complex: the imaginary part's, times c+ - c-
  double P[3], invP;
};
struct Crt3Tab {
  Crt3 c[kExactHi - kExactLo + 1];
};
static_assert(kExactHi - kExactLo == kExactHiC - kExactLoC, "one table type");

static void split3(u128 x, int c1, int c2, double* p0, double* p1, double* p2) {
  *p0 = std::ldexp((double)(uint64_t)(x >> c1), c1);
  x &= (((u128)1) << c1) - 1;
  *p1 = std::ldexp((double)(uint64_t)(x >> c2), c2);
  x &= c2 ? (((u128)1) << c2) - 1 : 0;
  *p2 = (double)(uint64_t)x;
}

static const Crt3Tab& crt3_tab(bool cplx) {
  auto make = [](bool cx) {
    Crt3Tab t;
    std::memset(&t, 0, sizeof(t));
    const std::vector<int> rm = moduli_list();
    const int lo = cx ? kExactLoC : kExactLo, hi = cx ? kExactHiC : kExactHi;
    for (int n = lo; n <= hi; ++n) {
      Crt3& c = t.c[n - lo];
      auto mod = [&](int i) { return cx ? kCMod[i] : rm[i]; };
      u128 P = 1;
      for (int i = 0; i < n; ++i) P *= (u128)mod(i);
      int bitsP = 0;
      for (u128 q = P; q; q >>= 1) ++bitsP;
      const int w = cx ? 39 : 41;
      const int c1 = std::max(1, bitsP - w), c2 = std::max(0, c1 - w);
      for (int i = 0; i < n; ++i) {
        const int p = mod(i);
        const u128 Mi = P / (u128)p;
        const int im = inv_mod((int)(Mi % (u128)p), p);
        const int f = cx ? (int)((long)im * inv_mod(2, p) % p) : im;
        split3(Mi * (u128)f, c1, c2, &c.w[0][i], &c.w[1][i], &c.w[2][i]);
        if (cx) {
          const int j = sqrt_minus_one(p);
          const int fi = (int)((long)im * inv_mod(2 * j % p, p) % p);
          split3(Mi * (u128)fi, c1, c2, &c.v[0][i], &c.v[1][i], &c.v[2][i]);
        }
      }
      split3(P, c1, c2, &c.P[0], &c.P[1], &c.P[2]);
      c.invP = 1.0 / (double)P;
    }
    return t;
  };
  static const Crt3Tab real = make(false), comp = make(true);
  return cplx ? comp : real;
}

// The value of the exact sums s[0..2].
__device__ __forceinline__ double crt3_value(const double (&s)[3], const Crt3& c) {
  const double q = rint(s[0] * c.invP);
  const double d0 = fma(-q, c.P[0], s[0]), d1 = fma(-q, c.P[1], s[1]),
               d2 = fma(-q, c.P[2], s[2]);
  const double t = d0 + d1, z = t - d0;  // t + e = d0 + d1
  const double e = (d0 - (t - z)) + (d1 - z);
  return t + (e + d2);
}
// A warp takes 8 rows x 16 columns, a lane row l / 4 and the four columns
// 4 (l % 4) .. + 3 (as crt_body_c).
template <int NM, bool CPLX>
__device__ __forceinline__ void crt_body_x(const CrtP& p, const Crt3& c, int H) {
  constexpr int PL = CPLX ? 2 : 1;
  const size_t plane = (size_t)p.Mpad * (size_t)p.Npad;
  const int lane = threadIdx.x & 31;
  const int i0 = blockIdx.x * kCrtRowsC, i = i0 + (lane >> 2);
  const int jw = blockIdx.y * kCrtCols + (int)(threadIdx.x >> 5) * 16;
  const int j0 = jw + 4 * (lane & 3);
  if (p.uplo == XKB_LOWER && (long)i0 + kCrtRowsC - 1 + p.diag < (long)jw) return;
  if (p.uplo == XKB_UPPER && (long)i0 + p.diag > (long)jw + 15) return;
  if (i >= p.M || j0 >= p.N) return;
  uint32_t word[PL * NM];
  const uint8_t* src = p.R + (size_t)jw * (size_t)p.Mpad + (size_t)i * 16 + (size_t)(4 * (lane & 3));
#pragma unroll
  for (int m = 0; m < PL * NM; ++m)
    word[m] = __ldcs(reinterpret_cast<const uint32_t*>(src + (size_t)m * plane));
  double r[4][3], x[4][3];
#pragma unroll
  for (int e = 0; e < 4; ++e)
#pragma unroll
    for (int q = 0; q < 3; ++q) r[e][q] = x[e][q] = 0.0;
#pragma unroll
  for (int m = 0; m < NM; ++m) {
    const double w0 = c.w[0][m], w1 = c.w[1][m], w2 = c.w[2][m];
    const double v0 = CPLX ? c.v[0][m] : 0.0, v1 = CPLX ? c.v[1][m] : 0.0,
                 v2 = CPLX ? c.v[2][m] : 0.0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      double su = crt_byte(word[PL * m], e);
      if constexpr (CPLX) {
        const double b = crt_byte(word[2 * m + 1], e), di = su - b;
        su += b;
        x[e][0] = fma(di, v0, x[e][0]);
        x[e][1] = fma(di, v1, x[e][1]);
        x[e][2] = fma(di, v2, x[e][2]);
      }
      r[e][0] = fma(su, w0, r[e][0]);
      r[e][1] = fma(su, w1, r[e][1]);
      r[e][2] = fma(su, w2, r[e][2]);
    }
  }
  const bool beta = p.br != 0.0 || p.bi != 0.0;
  const bool mask = p.uplo != XKB_FULL;
  float* C = static_cast<float*>(p.C);
  const int mui = shift_of(p.mu[i], H);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int j = j0 + e;
    if (j >= p.N) break;
    if (mask && (p.uplo == XKB_LOWER ? (long)i + p.diag < (long)j : (long)i + p.diag > (long)j))
      continue;
    const int sh = -(mui + shift_of(p.nu[j], H));
    const size_t idx = (size_t)i + (size_t)j * p.ldc;
    const double xr = scale2(crt3_value(r[e], c), sh);
    if constexpr (CPLX) {
      const double xi = scale2(crt3_value(x[e], c), sh);
      double vr = p.ar * xr - p.ai * xi;
      double vi = p.ar * xi + p.ai * xr;
      if (beta) {
        const double cr = (double)C[2 * idx], ci = (double)C[2 * idx + 1];
        vr += p.br * cr - p.bi * ci;
        vi += p.br * ci + p.bi * cr;
      }
      if (p.herm_diag && (long)i + p.diag == (long)j) vi = 0.0;
      C[2 * idx] = (float)vr;
      C[2 * idx + 1] = (float)vi;
    } else {
      double out = p.ar * xr;
      if (beta) out = fma(p.br, (double)C[idx], out);
      C[idx] = (float)out;
    }
  }
}
template <int NM, bool CPLX>
__device__ __forceinline__ void crt_any_x(const CrtP& p, const Crt3Tab& t, const OzSel& s) {
  constexpr int LO = CPLX ? kExactLoC : kExactLo, HI = CPLX ? kExactHiC : kExactHi;
  if (s.np == NM) crt_body_x<NM, CPLX>(p, t.c[NM - LO], s.H);
  else if constexpr (NM < HI) crt_any_x<NM + 1, CPLX>(p, t, s);
}
template <bool CPLX>
__global__ void __launch_bounds__(256, 2) k_oz_crt_x(const CrtP p,
                                                     const __grid_constant__ Crt3Tab t) {
  const OzSel s = *p.sel;
  crt_any_x<CPLX ? kExactLoC : kExactLo, CPLX>(p, t, s);
}

template <int NM>
__device__ __forceinline__ void crt_any_c(const CrtP& p, const CCrtTab& t, const OzSel& s) {
  if (s.np == NM) crt_body_c<NM>(p, t.c[NM], s.H);
  else if constexpr (NM < kMaxC) crt_any_c<NM + 1>(p, t, s);
}
__global__ void __launch_bounds__(256, 2) k_oz_crt_c(const CrtP p,
                                                     const __grid_constant__ CCrtTab t) {
  const OzSel s = *p.sel;
  if (s.np >= 2) crt_any_c<2>(p, t, s);
}

// lo == hi: that count; (lo, hi) == (15, 16): the count the device chose.
static int launch_crt(cudaStream_t st, const CrtP& cp, const Consts* lo, const Consts* hi) {
  if (!lo || !hi) return XKB_EINVAL;
  const dim3 g((unsigned)((cp.M + kCrtRows - 1) / kCrtRows),
               (unsigned)((cp.N + kCrtCols - 1) / kCrtCols));
  const long long tv = evlog_kern_begin(st, "k_oz_crt");
  if (lo->nmod != hi->nmod) {
    if (lo->nmod != 15 || hi->nmod != 16) return XKB_EINVAL;
    k_oz_crt_15_16<<<g, 256, 0, st>>>(cp, *lo, *hi);
  } else {
    switch (hi->nmod) {
#define XKB_CRT_CASE(NM) \
  case NM:               \
    k_oz_crt<NM><<<g, 256, 0, st>>>(cp, *hi); break;
      XKB_CRT_CASE(2) XKB_CRT_CASE(3) XKB_CRT_CASE(4) XKB_CRT_CASE(5) XKB_CRT_CASE(6)
      XKB_CRT_CASE(7) XKB_CRT_CASE(8) XKB_CRT_CASE(9) XKB_CRT_CASE(10) XKB_CRT_CASE(11)
      XKB_CRT_CASE(12) XKB_CRT_CASE(13) XKB_CRT_CASE(14) XKB_CRT_CASE(15) XKB_CRT_CASE(16)
#undef XKB_CRT_CASE
      default: return XKB_EINVAL;
    }
  }
  evlog_kern_end(tv, st);
  count_launch();
  return cudaPeekAtLastError() == cudaSuccess ? XKB_OK : XKB_ECUDA;
}

// ---------------------------------------------------------------------------
// host orchestration
static size_t rup(size_t v, size_t a) { return (v + a - 1) / a * a; }

static const Consts* consts_for(int n) {
  static Consts cache[kMaxMod + 1];
  static bool have[kMaxMod + 1] = {false};
  static std::mutex mu;
  std::lock_guard<std::mutex> g(mu);
  if (n < 2 || n > kMaxMod) return nullptr;
  if (!have[n]) {
    if (!make_consts(n, &cache[n])) return nullptr;
    have[n] = true;
  }
  return &cache[n];
}

// Operand descriptor: an L x K "row" view (rows of op(A), or columns of
// op(B)) of a matrix.
struct View {
  const void* X;
  long ld;    // leading dimension in elements
  bool kc;    // k contiguous
  int dtype;  // XKB_S .. XKB_Z
  bool conj;
};

// Device words of one call: the moduli selection and the two concentration
// maxima (rows of op(A), columns of op(B)); zeroed before the norms.
struct CallWords {
  OzSel sel;
  unsigned rmax[2];
  unsigned pad[2];
};

// The counts a call may use: a fixed count (lo = hi), or the data rule's
// range [lo, 16] with lo = max(15, the tuning table's count for K's band).
struct ModPlan {
  int lo = 0, hi = 0;
  bool fixed = true;
  const Consts* clo = nullptr;
  const Consts* chi = nullptr;
};

static bool plan_moduli(int nmod, long K, ModPlan* pl) {
  if (nmod > 0) {
    pl->lo = pl->hi = nmod;
    pl->fixed = true;
  } else {
    const int tuned = tune_band("ozaki_moduli_k<=", K);
    pl->lo = std::min(kMaxMod, std::max(15, (tuned >= 2 && tuned <= kMaxMod) ? tuned : 0));
    pl->hi = kMaxMod;
    pl->fixed = false;
  }
  pl->clo = consts_for(pl->lo);
  pl->chi = consts_for(pl->hi);
  return pl->clo && pl->chi;
}

// Row statistics of an L x K operand view: codes (k_oz_stat) and the
// concentration maximum into *rmax.
template <class E>
static void norm_kernel(const View& v, int L, int K, int cplx, double4* part, cudaStream_t st) {
  const unsigned nch = (unsigned)((K + kNormChunk - 1) / kNormChunk);
  const E* X = static_cast<const E*>(v.X);
  if (v.kc)
    k_oz_norm<true, E><<<dim3((unsigned)((L + 7) / 8), nch), 256, 0, st>>>(L, K, X, v.ld, cplx,
                                                                           part);
  else
    k_oz_norm<false, E><<<dim3((unsigned)((L + 31) / 32), nch), 256, 0, st>>>(L, K, X, v.ld, cplx,
                                                                              part);
}
static int launch_norm(const View& v, int L, int K, double4* part, int* code, unsigned* rmax,
                       cudaStream_t st) {
  const int cplx = v.dtype == XKB_C || v.dtype == XKB_Z;
  const int exact = v.dtype == XKB_S || v.dtype == XKB_C;
  const long long tv = evlog_kern_begin(st, "k_oz_norm+k_oz_stat");
  if (exact) norm_kernel<float>(v, L, K, cplx, part, st);
  else norm_kernel<double>(v, L, K, cplx, part, st);
  k_oz_stat<<<(unsigned)((L + 255) / 256), 256, 0, st>>>(
      L, K, (K + kNormChunk - 1) / kNormChunk, part, code, rmax, exact);
  evlog_kern_end(tv, st);
  count_launch(2);
  return cudaPeekAtLastError() == cudaSuccess ? XKB_OK : XKB_ECUDA;
}

// Smallest complex moduli count whose P/4 holds |C'| <= 2^(2H).
static int cplx_count(int H) {
  for (int n = 2; n < kMaxC; ++n)
    if (log2Pc(n) - 2.0 >= 2.0 * H) return n;
  return kMaxC;
}

static int launch_pick(CallWords* w, const ModPlan& pl, bool allow_fallback, cudaStream_t st,
                       bool cplx = false, bool exact = false) {
  PickP q;
  std::memset(&q, 0, sizeof(q));
  q.fixed = pl.fixed ? pl.hi : 0;
  q.lo = pl.lo;
  q.hi = pl.hi;
  q.allow_fallback = allow_fallback ? 1 : 0;
  for (int n = 2; n <= kMaxMod; ++n) {
    const Consts* c = consts_for(n);
    if (!c) return XKB_EINVAL;
    q.H[n] = c->H;
    q.np[n] = cplx ? cplx_count(c->H) : n;
  }
  if (exact) {
    q.exact = 1;
    q.lo = cplx ? kExactLoC : kExactLo;
    q.hi = cplx ? kExactHiC : kExactHi;
    for (int n = 2; n <= q.hi; ++n)
      q.Hx[n] = cplx ? (int)std::floor((log2Pc(n) - 2.0) / 2.0) : consts_for(n)->H;
  }
  const long long tv = evlog_kern_begin(st, "k_oz_pick");
  k_oz_pick<<<1, 32, 0, st>>>(w->rmax, &w->sel, q);
  evlog_kern_end(tv, st);
  count_launch();
  return cudaPeekAtLastError() == cudaSuccess ? XKB_OK : XKB_ECUDA;
}

// Residue planes 0 .. sel->n - 1 of an operand view (c: the constants of the
// plan's largest count; the per-modulus constants are those of every count).
template <class E>
static int res_real(const View& v, int L, int K, const int* code, const OzSel* sel,
                    const Consts* c, int8_t* planes, long Lpad, long Kpad, long rows,
                    cudaStream_t st) {
  const dim3 g((unsigned)(rows / 64), (unsigned)(rup((size_t)K, 64) / 64));
  const E* X = static_cast<const E*>(v.X);
  const auto go = [&](auto nm) {
    constexpr int NM = decltype(nm)::value;
    if (v.kc)
      k_oz_residues<true, NM, E><<<g, 256, 0, st>>>(L, K, X, v.ld, code, sel, *c, planes, Lpad,
                                                    Kpad);
    else
      k_oz_residues<false, NM, E><<<g, 256, 0, st>>>(L, K, X, v.ld, code, sel, *c, planes, Lpad,
                                                     Kpad);
  };
  if constexpr (sizeof(E) == 4) {  // exact products plan for every count
    go(std::integral_constant<int, kExactHi>());
    return XKB_OK;
  } else {
    switch (c->nmod) {
#define XKB_RES_CASE(NM) \
  case NM: go(std::integral_constant<int, NM>()); return XKB_OK;
      XKB_RES_CASE(2) XKB_RES_CASE(3) XKB_RES_CASE(4) XKB_RES_CASE(5) XKB_RES_CASE(6)
      XKB_RES_CASE(7) XKB_RES_CASE(8) XKB_RES_CASE(9) XKB_RES_CASE(10) XKB_RES_CASE(11)
      XKB_RES_CASE(12) XKB_RES_CASE(13) XKB_RES_CASE(14) XKB_RES_CASE(15) XKB_RES_CASE(16)
#undef XKB_RES_CASE
      default: return XKB_EINVAL;
    }
  }
}
template <class E>
static void res_cplx(const View& v, int L, int K, const int* code, const OzSel* sel,
                     int8_t* planes, long Lpad, long Kpad, cudaStream_t st) {
  const dim3 g((unsigned)(Lpad / 64), (unsigned)(Kpad / 32));
  const E* X = static_cast<const E*>(v.X);
  const double sign = v.conj ? -1.0 : 1.0;
  if (v.kc)
    k_oz_residues_c<true, E><<<g, 256, 0, st>>>(L, K, X, v.ld, sign, code, sel, cres_consts(),
                                                planes, Lpad, Kpad);
  else
    k_oz_residues_c<false, E><<<g, 256, 0, st>>>(L, K, X, v.ld, sign, code, sel, cres_consts(),
                                                 planes, Lpad, Kpad);
}
static int launch_res(const View& v, int L, int K, const int* code, const OzSel* sel,
                      const Consts* c, int8_t* planes, long Lpad, long Kpad, cudaStream_t st,
                      long grid_rows = 0) {
  // grid covers Lpad (or grid_rows, for a block of rows of larger planes:
  // planes stay Lpad rows apart) x (K rounded to 64; complex: Kpad); rows
  // from L to the grid's end are written as zeros
  const long rows = grid_rows ? grid_rows : Lpad;
  const long long tv = evlog_kern_begin(st, "k_oz_residues");
  int e = XKB_OK;
  switch (v.dtype) {
    case XKB_S: e = res_real<float>(v, L, K, code, sel, c, planes, Lpad, Kpad, rows, st); break;
    case XKB_D: e = res_real<double>(v, L, K, code, sel, c, planes, Lpad, Kpad, rows, st); break;
    case XKB_C: res_cplx<float>(v, L, K, code, sel, planes, Lpad, Kpad, st); break;
    default: res_cplx<double>(v, L, K, code, sel, planes, Lpad, Kpad, st); break;
  }
  evlog_kern_end(tv, st);
  count_launch();
  if (e) return e;
  return cudaPeekAtLastError() == cudaSuccess ? XKB_OK : XKB_ECUDA;
}

static bool encode_planes(CUtensorMap* m, const int8_t* base, long Kpad, long Lpad, int nmod,
                          uint32_t box_rows, long plane_rows = 0) {
  return encode_tmap_3d_u8(m, base, (uint64_t)Kpad, (uint64_t)Lpad, (uint64_t)nmod, 128,
                           box_rows, (uint64_t)plane_rows);
}

// a_rows / b_rows: rows per plane of the A / B residue buffers (>= Mpad /
// Npad; equal when one buffer serves both operands).  a_stride / b_stride
// (0: the same): rows between consecutive planes, when Ap / Bp point at a
// block of rows of larger planes.
// c: the plan's largest count; null: a complex product of cplanes planes
// (bxor: see GemmP).  list: room for the tiles of a masked product (1 + one int
// per 128 x 256 tile), or null.
static int launch_gemm(const int8_t* Ap, long a_rows, const int8_t* Bp, long b_rows, long Mpad,
                       long Npad, long Kpad, const Consts* c, const OzSel* sel, uint8_t* R,
                       int uplo, long diag, cudaStream_t st, long a_stride = 0,
                       long b_stride = 0, int cplanes = 0, int bxor = 0,
                       int* list = nullptr) {
  CUtensorMap tA, tB;
  const int npl = c ? c->nmod : cplanes;
  if (a_rows < Mpad || b_rows < Npad) return XKB_EINVAL;
  if (!encode_planes(&tA, Ap, Kpad, a_rows, npl, BM, a_stride)) return XKB_EINVAL;
  if (!encode_planes(&tB, Bp, Kpad, b_rows, npl, BN, b_stride)) return XKB_EINVAL;
  GemmP p;
  std::memset(&p, 0, sizeof(p));
  p.mult = c ? 1 : 2;
  p.bxor = bxor;
  p.tiles_m = (int)(Mpad / BM);
  p.tiles_n = (int)(Npad / BN);
  p.kblocks = (int)(Kpad / BKB);
  p.nmod = npl;
  p.sel = sel;
  // raster group (tuning table oz_group_m, default 8 M tiles)
  p.group = std::max(1, std::min(p.tiles_m, (int)tune("oz_group_m", 8.0)));
  p.R = R;
  p.Mpad = Mpad;
  p.Npad = Npad;
  p.uplo = uplo;
  p.diag = diag;
  for (int m = 0; m < npl; ++m) {
    const uint32_t q = (uint32_t)(c ? c->p[m] : kCMod[m / 2]);
    p.p[m] = (int)q;
    p.magic[m] = (uint32_t)(((1ull << 32) + q - 1) / q);
    p.bias[m] = (uint32_t)(((1ull << 31) + q - 1) / q) * q;
  }
  const long total2 = (Mpad % BM2 == 0 && Npad % BN2 == 0)
                         ? (Mpad / BM2) * (Npad / BN2) * (long)npl : 0;
  if (total2 > 0 && tune("oz_2cta", 0.0) != 0.0 && sm_count() >= 2) {
    // CTA pairs: 256 x 256 tiles, each CTA loading 128-row halves of A and B
    CUtensorMap tB2;
    if (!encode_planes(&tB2, Bp, Kpad, b_rows, npl, 128, b_stride)) return XKB_EINVAL;
    p.tiles_m = (int)(Mpad / BM2);
    p.tiles_n = (int)(Npad / BN2);
    p.group = std::max(1, std::min(p.tiles_m, (int)tune("oz_group_m", 8.0)));
    const size_t smem2 = 1024 + S2 * (size_t)(2 * H_STAGE) + (2 * S2 + 4) * 8 + 16;
    static bool attr2 = false;
    if (!attr2) {
      if (cudaFuncSetAttribute(k_oz_gemm2, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)smem2) != cudaSuccess)
        return XKB_ECUDA;
      attr2 = true;
    }
    const long pairs = std::min<long>(total2, sm_count() / 2);
    cudaLaunchConfig_t cfg;
    std::memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3((unsigned)(2 * pairs));
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = smem2;
    cfg.stream = st;
    cudaLaunchAttribute la[1];
    la[0].id = cudaLaunchAttributeClusterDimension;
    la[0].val.clusterDim.x = 2;
    la[0].val.clusterDim.y = 1;
    la[0].val.clusterDim.z = 1;
    cfg.attrs = la;
    cfg.numAttrs = 1;
    const long long tv = evlog_kern_begin(st, "k_oz_gemm2");
    const cudaError_t le = cudaLaunchKernelEx(&cfg, k_oz_gemm2, tA, tB2, p);
    evlog_kern_end(tv, st);
    if (le != cudaSuccess) return XKB_ECUDA;
    count_launch();
    return cudaPeekAtLastError() == cudaSuccess ? XKB_OK : XKB_ECUDA;
  }
  const size_t smem = 1024 + S * (size_t)(A_STAGE + B_STAGE) + (2 * S + 4) * 8 + 16;
  static bool attr = false;
  if (!attr) {
    if (cudaFuncSetAttribute(k_oz_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
        cudaSuccess)
      return XKB_ECUDA;
    attr = true;
  }
  const long total = (long)p.tiles_m * p.tiles_n * npl;
  const unsigned grid = (unsigned)std::min<long>(total, sm_count());  // persistent
  const long long tv = evlog_kern_begin(st, "k_oz_gemm");
  if (list && uplo != XKB_FULL) {
    k_oz_tiles<<<1, 1024, 0, st>>>(p, list);
    p.list = list;
    count_launch();
  }
  k_oz_gemm<<<grid, kGemmThreads, smem, st>>>(tA, tB, p);
  evlog_kern_end(tv, st);
  count_launch();
  return cudaPeekAtLastError() == cudaSuccess ? XKB_OK : XKB_ECUDA;
}

int default_moduli(long K) {
  if (K <= 0 || K > 131072) return 0;  // exact INT32 accumulation limit
  // a count the autotuner measured for this K band (tuning table keys
  // "ozaki_moduli_k<=<K>"), when one covers K
  const int tuned = tune_band("ozaki_moduli_k<=", K);
  if (tuned >= 2 && tuned <= kMaxMod) return tuned;
  // keep >= 53 bits for the largest entry of a row whose entries are all of
  // the same magnitude: H - log2(K)/2 >= 53
  for (int n = 8; n <= kMaxMod; ++n) {
    const int H = (int)std::floor((log2P(n) - 1.0) / 2.0) - 1;
    if ((double)H - 0.5 * std::log2((double)K) >= 53.0) return n;
  }
  return kMaxMod;
}

}  // namespace oz
}  // namespace xkb

using namespace xkb;
using namespace xkb::oz;

extern "C" int xkb_ozaki_default_moduli(long K) { return default_moduli(K); }

extern "C" int xkb_ozaki_counts(unsigned long long* out, int* last, int reset) {
  if (!out) return XKB_EINVAL;
  // the counters are written by kernels on the library's non-blocking streams
  if (cudaDeviceSynchronize() != cudaSuccess) return XKB_ECUDA;
  if (cudaMemcpyFromSymbol(&out[0], g_oz_calls, sizeof(out[0])) != cudaSuccess ||
      cudaMemcpyFromSymbol(&out[1], g_oz_mod_sum, sizeof(out[1])) != cudaSuccess ||
      cudaMemcpyFromSymbol(&out[2], g_oz_fallbacks, sizeof(out[2])) != cudaSuccess)
    return XKB_ECUDA;
  if (last && cudaMemcpyFromSymbol(last, g_oz_last, sizeof(int)) != cudaSuccess) return XKB_ECUDA;
  if (reset) {
    const unsigned long long z = 0;
    const int none = -1;
    if (cudaMemcpyToSymbol(g_oz_calls, &z, sizeof z) != cudaSuccess ||
        cudaMemcpyToSymbol(g_oz_mod_sum, &z, sizeof z) != cudaSuccess ||
        cudaMemcpyToSymbol(g_oz_fallbacks, &z, sizeof z) != cudaSuccess ||
        cudaMemcpyToSymbol(g_oz_last, &none, sizeof none) != cudaSuccess)
      return XKB_ECUDA;
  }
  return XKB_OK;
}

extern "C" int xkb_exact_counts(unsigned long long* out, int* last, int reset) {
  if (!out) return XKB_EINVAL;
  if (cudaDeviceSynchronize() != cudaSuccess ||
      cudaMemcpyFromSymbol(&out[0], g_ex_calls, sizeof(out[0])) != cudaSuccess ||
      cudaMemcpyFromSymbol(&out[1], g_ex_plain, sizeof(out[1])) != cudaSuccess ||
      (last && cudaMemcpyFromSymbol(last, g_ex_last, sizeof(int)) != cudaSuccess))
    return XKB_ECUDA;
  const unsigned long long z = 0;
  const int none = -1;
  if (reset && (cudaMemcpyToSymbol(g_ex_calls, &z, sizeof z) != cudaSuccess ||
                cudaMemcpyToSymbol(g_ex_plain, &z, sizeof z) != cudaSuccess ||
                cudaMemcpyToSymbol(g_ex_last, &none, sizeof none) != cudaSuccess))
    return XKB_ECUDA;
  return XKB_OK;
}

// Real or complex Ozaki GEMM.  nmod > 0: that many moduli.  nmod == 0: the
// count is chosen on the device from the operands (k_oz_pick: 15 or 16, at
// least the tuning table's count for K's band); operands whose spread 16
// moduli cannot carry to FP64 accuracy are computed by the plain FP64
// kernel instead, launched here and predicated on the device's choice.
// Single precision (S, C): the exact product or the plain kernel.
// XKB_ENOMEM, XKB_ERANGE: nothing that writes C was queued.
// Scratch (stream-ordered, from the pool): residue planes of op(A) and
// op(B) for the largest count the call may use (nmod x Mpad x Kpad,
// nmod x Npad x Kpad int8; complex two planes per modulus, 34 for 16), residue
// planes of C (as many Mpad x Npad uint8), row codes, norm partials and the
// call's device words.
static int oz_run(const xkb_gemm_args* a, int nmod, cudaStream_t st) {
  const bool cplx = a->dtype == XKB_Z || a->dtype == XKB_C;
  const bool exact = a->dtype == XKB_S || a->dtype == XKB_C;
  const long Keff = cplx ? 2L * a->K : (long)a->K;
  if (Keff > 131072) return XKB_ERANGE;
  ModPlan pl;
  if (!plan_moduli(exact ? kExactHi : nmod, Keff, &pl)) return XKB_ERANGE;
  // planes: of the largest count the call may use
  const int nmax = cplx ? 2 * (exact ? kExactHiC : cplx_count(pl.chi->H)) : pl.hi;
  const Consts* c = cplx ? nullptr : pl.chi;
  const int M = a->M, N = a->N, K = a->K;
  const long Kpad = (long)rup(K, BKB);
  const long Mpad = (long)rup(M, BM2), Npad = (long)rup(N, BN);  // BM2: CTA-pair tiles
  const bool akc = a->opA != XKB_OP_N, bkc = a->opB == XKB_OP_N;
  const bool cA = a->opA == XKB_OP_C, cB = a->opB == XKB_OP_C;
  // C = A A^T or A A^H (or A^T A, A^H A): op(B)^T's rows are op(A)'s rows or,
  // complex, their conjugates (whose planes are op(A)'s, each pair swapped),
  // so one residue buffer serves both operands; it then holds
  // max(Mpad, Npad) rows per plane
  const bool same = (a->A == a->B) && (a->lda == a->ldb) && (akc == bkc) && M == N;
  const int bxor = cplx && same && cA != cB ? 1 : 0;
  const long Arows = same ? std::max(Mpad, Npad) : Mpad;
  const size_t szA = (size_t)nmax * Arows * Kpad, szB = same ? 0 : (size_t)nmax * Npad * Kpad;
  const size_t szR = (size_t)nmax * Mpad * Npad;
  const int nch = (K + kNormChunk - 1) / kNormChunk;
  const size_t szPart = 256 + sizeof(double4) * (size_t)nch * (size_t)std::max(M, N) * 2;
  int8_t *Ap = nullptr, *Bp = nullptr;
  uint8_t* R = nullptr;
  int *mu = nullptr, *nu = nullptr;
  unsigned char* pw = nullptr;  // CallWords, then the norm partials from byte 256
  auto alloc = [&](void** p, size_t n) {
    return scratch_alloc(p, n, st);
  };
  int* list = nullptr;  // the INT8 tiles of a masked product
  const size_t szL = a->uplo == XKB_FULL ? 0 : 4 * (1 + (size_t)(Mpad / BM) * (Npad / BN));
  bool ok = (!szL || alloc((void**)&list, szL)) && alloc((void**)&Ap, szA) && (same || alloc((void**)&Bp, szB)) &&
            alloc((void**)&R, szR) && alloc((void**)&mu, sizeof(int) * M) &&
            alloc((void**)&nu, sizeof(int) * N) && alloc((void**)&pw, szPart);
  int err = ok ? XKB_OK : XKB_ENOMEM;
  CallWords* w = reinterpret_cast<CallWords*>(pw);
  double4* part = reinterpret_cast<double4*>(pw + 256);
  const OzSel* sel = w ? &w->sel : nullptr;
  // operand views ----------------------------------------------------------
  // rows of op(A): opA == N -> A is M x K, row i = A[i + k*lda] (i contiguous)
  //                else     -> A is K x M, row i = A[k + i*lda] (k contiguous)
  // columns of op(B): opB == N -> B is K x N, col j = B[k + j*ldb] (k contig.)
  //                   else     -> B is N x K, col j = B[j + k*ldb]
  // (complex: the norm of a row is over its real and imaginary parts)
  const View va{a->A, a->lda, akc, a->dtype, cA}, vb{a->B, a->ldb, bkc, a->dtype, cB};
  const int slot = trace_begin("ozaki_gemm", a->dtype, M, N, K, pl.fixed ? pl.hi : 0, st);
  if (!err && cudaMemsetAsync(w, 0, sizeof(CallWords), st) != cudaSuccess) err = XKB_ECUDA;
  if (!err) err = launch_norm(va, M, K, part, mu, &w->rmax[0], st);
  if (!err)
    err = launch_norm(vb, N, K, part + (size_t)nch * std::max(M, N), nu, &w->rmax[1], st);
  if (!err) err = launch_pick(w, pl, !pl.fixed, st, cplx, exact);
  // The device may have sent the call to the plain FP64 kernel.  Its launch
  // comes before the recombination's (only one of the two writes C): where it
  // finds no scratch, nothing that writes C has been queued yet, and
  // XKB_ENOMEM leaves C as it was.
  if (!err && (exact || !pl.fixed)) err = gemm_if(a, &w->sel.fallback, st);
  if (!err) err = launch_res(va, M, K, mu, sel, pl.chi, Ap, Arows, Kpad, st);
  if (!err && !same) err = launch_res(vb, N, K, nu, sel, pl.chi, Bp, Npad, Kpad, st);
  if (!err && !cplx && Kpad > (long)rup(K, 64)) {
    // zero the k padding beyond the last 64-column block
    const size_t kz = rup(K, 64);
    if (cudaMemset2DAsync(Ap + kz, Kpad, 0, Kpad - kz, (size_t)nmax * Arows, st) != cudaSuccess ||
        (!same &&
         cudaMemset2DAsync(Bp + kz, Kpad, 0, Kpad - kz, (size_t)nmax * Npad, st) != cudaSuccess))
      err = XKB_ECUDA;
  }
  trace_mark(slot, 1, st);
  if (!err)
    err = launch_gemm(Ap, Arows, same ? Ap : Bp, same ? Arows : Npad, Mpad, Npad, Kpad, c, sel, R,
                      a->uplo, a->diag, st, 0, 0, nmax, bxor, list);
  trace_mark(slot, 2, st);
  if (!err) {
    CrtP cp;
    std::memset(&cp, 0, sizeof(cp));
    cp.M = M;
    cp.N = N;
    cp.R = R;
    cp.Mpad = Mpad;
    cp.Npad = Npad;
    cp.mu = mu;
    cp.nu = nu;
    cp.sel = sel;
    cp.C = a->C;
    cp.ldc = a->ldc;
    cp.ar = a->alpha[0];
    cp.ai = cplx ? a->alpha[1] : 0.0;
    cp.br = a->beta[0];
    cp.bi = cplx ? a->beta[1] : 0.0;
    cp.uplo = a->uplo;
    cp.herm_diag = a->herm_diag;
    cp.diag = a->diag;
    if (a->dtype == XKB_D) {
      err = launch_crt(st, cp, pl.clo, pl.chi);
    } else {
      const long long tv = evlog_kern_begin(st, "k_oz_crt");
      const unsigned gy = (unsigned)((N + kCrtCols - 1) / kCrtCols);
      const unsigned gc = (unsigned)((M + kCrtRowsC - 1) / kCrtRowsC);
      const dim3 g(gc, gy);
      if (a->dtype == XKB_S) k_oz_crt_x<false><<<g, 256, 0, st>>>(cp, crt3_tab(false));
      else if (a->dtype == XKB_C) k_oz_crt_x<true><<<g, 256, 0, st>>>(cp, crt3_tab(true));
      else k_oz_crt_c<<<g, 256, 0, st>>>(cp, ccrt_tab());
      evlog_kern_end(tv, st);
      count_launch();
      if (cudaPeekAtLastError() != cudaSuccess) err = XKB_ECUDA;
    }
  }
  if (!err && cudaPeekAtLastError() != cudaSuccess) err = XKB_ECUDA;
  trace_mark(slot, 3, st);
  if (list) cudaFreeAsync(list, st);
  if (Ap) cudaFreeAsync(Ap, st);
  if (Bp) cudaFreeAsync(Bp, st);
  if (R) cudaFreeAsync(R, st);
  if (mu) cudaFreeAsync(mu, st);
  if (nu) cudaFreeAsync(nu, st);
  if (pw) cudaFreeAsync(pw, st);
  return err;
}

extern "C" int xkb_cuda_ozaki_gemm(const xkb_gemm_args* a, int nmod, void* stream) {
  if (!a || (a->dtype != XKB_D && a->dtype != XKB_Z)) return XKB_EINVAL;
  if (a->M < 0 || a->N < 0 || a->K < 0) return XKB_EINVAL;
  if (a->M == 0 || a->N == 0) return XKB_OK;
  if (a->K == 0 || (a->alpha[0] == 0.0 && a->alpha[1] == 0.0))
    return xkb_cuda_gemm(a, stream);
  return oz_run(a, nmod, resolve_stream(stream));
}

namespace xkb {
// The exact form of a large single-precision product (S, C): FP64 work would
// leave the INT8 tensor cores idle.  Whether the operands allow it is decided
// on the device (k_oz_pick), else the plain kernel runs within the same call.
// XKB_ERANGE: not taken for this shape, XKB_ENOMEM: no scratch, either before
// anything that writes C; the caller then runs the plain kernel.  Taken from
// M N K = 3.4e9 on (C: a quarter of it).  Measured (B200, us, plain -> exact):
// S 1024^3 76 -> 108, 1500^3 214 -> 184, 2048^3 527 -> 270, 4096^3 3978 -> 1042
// (error against 64 bits 2.53e-8, the final rounding, on both); C 1024^3 258 ->
// 209, 2048^3 1976 -> 489.  Operands that do not fit pay the norm passes, the
// allocations and the empty launches: S 1800^3 376 -> 472, 2048^3 529 -> 593,
// 4096^3 3996 -> 4108; C 1000^3 258 -> 317, 2048^3 1980 -> 2055.
int gemm_exact(const xkb_gemm_args* a, cudaStream_t st) {
  const bool cplx = a->dtype == XKB_C;
  const double mn = std::min(a->M, a->N);
  if (tune("gemm_exact", 1.0) == 0.0 || mn < 512 || a->K < 512 ||
      (double)a->M * a->N * a->K * (cplx ? 4.0 : 1.0) < tune("gemm_exact_min", 3.4e9))
    return XKB_ERANGE;
  const double planes = cplx ? 2 * kExactHiC : kExactHi;
  if (planes * ((double)a->M * a->K + (double)a->N * a->K + (double)a->M * a->N) > 17.2e9)
    return XKB_ERANGE;  // at most 16 GiB of scratch
  return oz_run(a, 0, st);
}
}  // namespace xkb

// ===========================================================================
// Column-panel form of the real contraction, for callers that move op(B)
// and C across the host link panel by panel: op(A) is scaled and converted
// once; then for each column panel [n0, n1) of op(B) / C the stream waits on
// wait_ev[p] (the panel's operands are on the device), the panel's column
// shifts and residue planes are formed, multiplied on the INT8 tensor cores
// and recombined into C[:, n0:n1), and done_ev[p] is recorded (the panel's
// result is final).  Transfers of later panels and of finished results then
// overlap the arithmetic.  The caller orders op(A) before the call.
// Real, C full (no triangle mask); other calls use xkb_cuda_ozaki_gemm.
extern "C" int xkb_cuda_ozaki_gemm_panels(const xkb_gemm_args* a, int nmod, void* stream,
                                          int npanel, const long* bounds,
                                          void* const* wait_ev, void* const* done_ev) {
  if (!a || a->dtype != XKB_D || a->uplo != XKB_FULL || npanel < 1 || !bounds)
    return XKB_EINVAL;
  if (a->M < 0 || a->N < 0 || a->K < 0) return XKB_EINVAL;
  if (bounds[0] != 0 || bounds[npanel] != a->N) return XKB_EINVAL;
  for (int q = 0; q < npanel; ++q)
    if (bounds[q + 1] <= bounds[q]) return XKB_EINVAL;
  cudaStream_t st = resolve_stream(stream);
  auto wait = [&](int q) {
    if (wait_ev && wait_ev[q]) cudaStreamWaitEvent(st, static_cast<cudaEvent_t>(wait_ev[q]), 0);
  };
  auto done = [&](int q) {
    if (done_ev && done_ev[q]) cudaEventRecord(static_cast<cudaEvent_t>(done_ev[q]), st);
  };
  if (a->M == 0) {
    for (int q = 0; q < npanel; ++q) done(q);
    return XKB_OK;
  }
  if (a->K == 0 || a->alpha[0] == 0.0 || a->K > 131072) {  // no split product to pipeline
    for (int q = 0; q < npanel; ++q) wait(q);
    const int r = a->K > 131072 ? XKB_ERANGE : xkb_cuda_gemm(a, st);
    for (int q = 0; q < npanel; ++q) done(q);
    return r;
  }
  // op(A) is converted before op(B) arrives: the count is fixed for the call
  // (the tuning table's or the K rule's when nmod == 0)
  if (nmod == 0) nmod = default_moduli(a->K);
  ModPlan pl;
  if (!plan_moduli(nmod, a->K, &pl)) return XKB_ERANGE;
  const Consts* c = pl.chi;
  const int M = a->M, K = a->K;
  const long Kpad = (long)rup(K, BKB), Mpad = (long)rup(M, BM2);
  long wmax = 0;
  for (int q = 0; q < npanel; ++q) wmax = std::max(wmax, bounds[q + 1] - bounds[q]);
  const long Wpad = (long)rup((size_t)wmax, BN);
  const bool akc = a->opA != XKB_OP_N, bkc = a->opB == XKB_OP_N;
  const int nch = (int)((K + kNormChunk - 1) / kNormChunk);
  int8_t *Ap = nullptr, *Bp = nullptr;
  uint8_t* R = nullptr;
  int *mu = nullptr, *nu = nullptr;
  unsigned char* pw = nullptr;  // CallWords, then the norm partials from byte 256
  auto alloc = [&](void** p, size_t n) {
    return scratch_alloc(p, n, st);
  };
  bool ok = alloc((void**)&Ap, (size_t)nmod * Mpad * Kpad) &&
            alloc((void**)&Bp, (size_t)nmod * Wpad * Kpad) &&
            alloc((void**)&R, (size_t)nmod * Mpad * Wpad) && alloc((void**)&mu, sizeof(int) * M) &&
            alloc((void**)&nu, sizeof(int) * a->N) &&
            alloc((void**)&pw, 256 + sizeof(double4) * (size_t)nch * (size_t)std::max<long>(M, wmax));
  int err = ok ? XKB_OK : XKB_ENOMEM;
  CallWords* w = reinterpret_cast<CallWords*>(pw);
  double4* part = reinterpret_cast<double4*>(pw + 256);
  const OzSel* sel = w ? &w->sel : nullptr;
  const double* Ad = static_cast<const double*>(a->A);
  const double* Bd = static_cast<const double*>(a->B);
  const int slot = trace_begin("ozaki_panels", a->dtype, M, a->N, K, nmod, st);
  if (!err) {
    View va{Ad, a->lda, akc, XKB_D, false};
    if (cudaMemsetAsync(w, 0, sizeof(CallWords), st) != cudaSuccess) err = XKB_ECUDA;
    if (!err) err = launch_norm(va, M, K, part, mu, &w->rmax[0], st);
    if (!err) err = launch_pick(w, pl, false, st);
    if (!err) err = launch_res(va, M, K, mu, sel, c, Ap, Mpad, Kpad, st);
    if (!err && Kpad > (long)rup(K, 64)) {
      const size_t kz = rup(K, 64);
      if (cudaMemset2DAsync(Ap + kz, Kpad, 0, Kpad - kz, (size_t)nmod * Mpad, st) != cudaSuccess)
        err = XKB_ECUDA;
    }
  }
  trace_mark(slot, 1, st);
  for (int q = 0; q < npanel; ++q) {
    wait(q);
    const long n0 = bounds[q], nw = bounds[q + 1] - bounds[q];
    const long npad = (long)rup((size_t)nw, BN);
    if (!err) {
      // columns n0.. of op(B): opB == N -> B[k + j ldb]; else B[j + k ldb]
      View vb{bkc ? Bd + n0 * a->ldb : Bd + n0, a->ldb, bkc, XKB_D, false};
      err = launch_norm(vb, (int)nw, K, part, nu + n0, &w->rmax[1], st);
      if (!err) err = launch_res(vb, (int)nw, K, nu + n0, sel, c, Bp, npad, Kpad, st);
      if (!err && Kpad > (long)rup(K, 64)) {
        const size_t kz = rup(K, 64);
        if (cudaMemset2DAsync(Bp + kz, Kpad, 0, Kpad - kz, (size_t)nmod * npad, st) != cudaSuccess)
          err = XKB_ECUDA;
      }
      if (!err)
        err = launch_gemm(Ap, Mpad, Bp, npad, Mpad, npad, Kpad, c, sel, R, XKB_FULL, 0, st);
      if (!err) {
        CrtP cp;
        std::memset(&cp, 0, sizeof(cp));
        cp.M = M;
        cp.N = (int)nw;
        cp.R = R;
        cp.Mpad = Mpad;
        cp.Npad = npad;
        cp.mu = mu;
        cp.nu = nu + n0;
        cp.sel = sel;
        cp.C = static_cast<double*>(a->C) + n0 * a->ldc;
        cp.ldc = a->ldc;
        cp.ar = a->alpha[0];
        cp.br = a->beta[0];
        cp.uplo = XKB_FULL;
        err = launch_crt(st, cp, c, c);
      }
    }
    done(q);  // recorded on every path: waiters never hang on an error
  }
  trace_mark(slot, 2, st);
  trace_mark(slot, 3, st);
  if (Ap) cudaFreeAsync(Ap, st);
  if (Bp) cudaFreeAsync(Bp, st);
  if (R) cudaFreeAsync(R, st);
  if (mu) cudaFreeAsync(mu, st);
  if (nu) cudaFreeAsync(nu, st);
  if (pw) cudaFreeAsync(pw, st);
  return err;
}

// Row blocks of op(A) and column panels of op(B) landing in the order `seq`
// names; see include/xkb_cuda.h.  Every block is converted once, when it
// lands, into residue planes that hold all of op(A) (all of op(B)); the
// products of the newly landed block with all the blocks of the other
// operand converted before it form one rectangle of C -- one INT8 launch,
// one CRT -- whose completion is recorded on done_ev[k].  Row blocks and
// column panels each land in increasing order, so those rectangles are
// [row block i] x [0, the columns landed so far) or [0, the rows landed so
// far) x [panel j], and together they cover C once.
extern "C" int xkb_cuda_ozaki_gemm_blocks(const xkb_gemm_args* a, int nmod, void* stream, int nr,
                                          const long* rb, int nc, const long* cb, const int* seq,
                                          void* const* a_ev, void* const* b_ev,
                                          void* const* done_ev) {
  if (!a || a->dtype != XKB_D || a->uplo != XKB_FULL || nr < 1 || nc < 1 || !rb || !cb || !seq)
    return XKB_EINVAL;
  if (a->M < 0 || a->N < 0 || a->K < 0) return XKB_EINVAL;
  if (rb[0] != 0 || rb[nr] != a->M || cb[0] != 0 || cb[nc] != a->N) return XKB_EINVAL;
  // interior bounds on multiples of 256: block and panel offsets then fall on
  // INT8 tile and TMA boundaries of the residue planes
  for (int i = 0; i < nr; ++i)
    if (rb[i + 1] <= rb[i] || (i > 0 && rb[i] % 256 != 0)) return XKB_EINVAL;
  for (int j = 0; j < nc; ++j)
    if (cb[j + 1] <= cb[j] || (j > 0 && cb[j] % 256 != 0)) return XKB_EINVAL;
  {
    int ni = 0, nj = 0;  // each block once, row blocks and panels in increasing order
    for (int k = 0; k < nr + nc; ++k) {
      if (seq[k] < 0) {
        if (-1 - seq[k] != ni) return XKB_EINVAL;
        ++ni;
      } else {
        if (seq[k] != nj) return XKB_EINVAL;
        ++nj;
      }
    }
    if (ni != nr || nj != nc) return XKB_EINVAL;
  }
  cudaStream_t st = resolve_stream(stream);
  const int nseq = nr + nc;
  auto wait = [&](void* const* evs, int q) {
    if (evs && evs[q]) cudaStreamWaitEvent(st, static_cast<cudaEvent_t>(evs[q]), 0);
  };
  auto done = [&](int k) {
    if (done_ev && done_ev[k]) cudaEventRecord(static_cast<cudaEvent_t>(done_ev[k]), st);
  };
  if (a->M == 0 || a->K == 0 || a->alpha[0] == 0.0 || a->K > 131072) {
    // nothing to pipeline: every operand, then one plain product
    for (int k = 0; k < nseq; ++k) wait(seq[k] < 0 ? a_ev : b_ev, seq[k] < 0 ? -1 - seq[k] : seq[k]);
    const int r = a->K > 131072 ? XKB_ERANGE : (a->M == 0 ? XKB_OK : xkb_cuda_gemm(a, st));
    for (int k = 0; k < nseq; ++k) done(k);
    return r;
  }
  // blocks are converted before the other operand has landed: the count is
  // fixed for the call (the tuning table's or the K rule's when nmod == 0)
  if (nmod == 0) nmod = default_moduli(a->K);
  ModPlan pl;
  if (!plan_moduli(nmod, a->K, &pl)) return XKB_ERANGE;
  const Consts* c = pl.chi;
  const int M = a->M, N = a->N, K = a->K;
  const long Kpad = (long)rup(K, BKB), Mpad = (long)rup(M, BM2), Npad = (long)rup(N, BN2);
  long rmax = 0, cmax = 0;
  for (int i = 0; i < nr; ++i) rmax = std::max(rmax, rb[i + 1] - rb[i]);
  for (int j = 0; j < nc; ++j) cmax = std::max(cmax, cb[j + 1] - cb[j]);
  const bool akc = a->opA != XKB_OP_N, bkc = a->opB == XKB_OP_N;
  const int nch = (int)((K + kNormChunk - 1) / kNormChunk);
  int8_t *Ap = nullptr, *Bp = nullptr;
  uint8_t* R = nullptr;
  int *mu = nullptr, *nu = nullptr;
  unsigned char* pw = nullptr;  // CallWords, then the norm partials from byte 256
  auto alloc = [&](void** p, size_t n) {
    return scratch_alloc(p, n, st);
  };
  // the largest rectangle: all rows x one panel, or one row block x all columns
  const size_t rsz = std::max((size_t)Mpad * rup((size_t)cmax, BN), rup((size_t)rmax, BM) * (size_t)Npad);
  bool ok = alloc((void**)&Ap, (size_t)nmod * Mpad * Kpad) &&
            alloc((void**)&Bp, (size_t)nmod * Npad * Kpad) && alloc((void**)&R, (size_t)nmod * rsz) &&
            alloc((void**)&mu, sizeof(int) * M) && alloc((void**)&nu, sizeof(int) * N) &&
            alloc((void**)&pw, 256 + sizeof(double4) * (size_t)nch * (size_t)std::max(rmax, cmax));
  int err = ok ? XKB_OK : XKB_ENOMEM;
  CallWords* w = reinterpret_cast<CallWords*>(pw);
  double4* part = reinterpret_cast<double4*>(pw + 256);
  const OzSel* sel = w ? &w->sel : nullptr;
  const double* Ad = static_cast<const double*>(a->A);
  const double* Bd = static_cast<const double*>(a->B);
  const int slot = trace_begin("ozaki_blocks", a->dtype, M, N, K, nmod, st);
  if (!err) {
    if (cudaMemsetAsync(w, 0, sizeof(CallWords), st) != cudaSuccess) err = XKB_ECUDA;
    if (!err) err = launch_pick(w, pl, false, st);
    // k columns past K (to the INT8 k-block) are zero in every plane
    const size_t kz = rup(K, 64);
    if (!err && Kpad > (long)kz &&
        (cudaMemset2DAsync(Ap + kz, Kpad, 0, Kpad - kz, (size_t)nmod * Mpad, st) != cudaSuccess ||
         cudaMemset2DAsync(Bp + kz, Kpad, 0, Kpad - kz, (size_t)nmod * Npad, st) != cudaSuccess))
      err = XKB_ECUDA;
  }
  trace_mark(slot, 1, st);
  int ra = 0, cn = 0;  // row blocks / panels landed so far
  for (int k = 0; k < nseq; ++k) {
    long r0, r1, c0, c1;  // the rectangle of C this landing completes
    if (seq[k] < 0) {
      const int i = -1 - seq[k];
      wait(a_ev, i);
      r0 = rb[i];
      r1 = rb[i + 1];
      c0 = 0;
      c1 = cb[cn];
      if (!err) {
        // rows r0.. of op(A): opA == N -> A[i + k lda]; else A[k + i lda]
        View va{akc ? Ad + r0 * a->lda : Ad + r0, a->lda, akc, XKB_D, false};
        const int L = (int)(r1 - r0);
        err = launch_norm(va, L, K, part, mu + r0, &w->rmax[0], st);
        if (!err)
          err = launch_res(va, L, K, mu + r0, sel, c, Ap + r0 * Kpad, Mpad, Kpad, st,
                           (long)rup((size_t)L, 64));
      }
      ++ra;
    } else {
      const int j = seq[k];
      wait(b_ev, j);
      r0 = 0;
      r1 = rb[ra];
      c0 = cb[j];
      c1 = cb[j + 1];
      if (!err) {
        // columns c0.. of op(B): opB == N -> B[k + j ldb]; else B[j + k ldb]
        View vb{bkc ? Bd + c0 * a->ldb : Bd + c0, a->ldb, bkc, XKB_D, false};
        const int L = (int)(c1 - c0);
        err = launch_norm(vb, L, K, part, nu + c0, &w->rmax[1], st);
        if (!err)
          err = launch_res(vb, L, K, nu + c0, sel, c, Bp + c0 * Kpad, Npad, Kpad, st,
                           (long)rup((size_t)L, 64));
      }
      ++cn;
    }
    if (!err && r1 > r0 && c1 > c0) {
      const long mp = (long)rup((size_t)(r1 - r0), BM), np = (long)rup((size_t)(c1 - c0), BN);
      err = launch_gemm(Ap + r0 * Kpad, mp, Bp + c0 * Kpad, np, mp, np, Kpad, c, sel, R, XKB_FULL,
                        0, st, Mpad, Npad);
      if (!err) {
        CrtP cp;
        std::memset(&cp, 0, sizeof(cp));
        cp.M = (int)(r1 - r0);
        cp.N = (int)(c1 - c0);
        cp.R = R;
        cp.Mpad = mp;
        cp.Npad = np;
        cp.mu = mu + r0;
        cp.nu = nu + c0;
        cp.sel = sel;
        cp.C = static_cast<double*>(a->C) + r0 + c0 * a->ldc;
        cp.ldc = a->ldc;
        cp.ar = a->alpha[0];
        cp.br = a->beta[0];
        cp.uplo = XKB_FULL;
        err = launch_crt(st, cp, c, c);
      }
    }
    done(k);  // recorded on every path: waiters never hang on an error
  }
  trace_mark(slot, 2, st);
  trace_mark(slot, 3, st);
  if (Ap) cudaFreeAsync(Ap, st);
  if (Bp) cudaFreeAsync(Bp, st);
  if (R) cudaFreeAsync(R, st);
  if (mu) cudaFreeAsync(mu, st);
  if (nu) cudaFreeAsync(nu, st);
  if (pw) cudaFreeAsync(pw, st);
  return err;
}

// ===========================================================================
// Scratch-free variant of the real Ozaki contraction.
//
// Who needs it: callers that cannot ask the CUDA allocator for memory at call
// time -- for example a program that has already handed all free device
// memory to its own caching allocator (cudaMallocAsync would then fail), or a
// latency-bound loop that must not risk an allocation stalling or failing in
// the middle of a step.  xkb_cuda_ozaki_gemm takes its scratch (residue
// planes, shifts, norm partials) from the stream-ordered pool on every call;
// this entry point takes it from one fixed device array compiled into the
// library instead, and allocates nothing.
//
// Limits and rules:
//   * real double (XKB_D) only, M, N, K <= kNoAllocMaxDim (512); larger sizes
//     are refused with XKB_ERANGE before anything is launched;
//   * the array (kNoAllocBytes, about 12.6 MiB) lives in every GPU that
//     loads this library, for the life of the process;
//   * all calls share it: two calls whose kernels overlap on the GPU (other
//     streams, other host threads) race on it and corrupt each other --
//     serialise them;
//   * the array is placed in device memory when this file's CUDA module is
//     loaded, which with lazy module loading (the CUDA 12 default) happens
//     at its first use, not when the library is opened.  noalloc_prepare()
//     -- run by xkblas_init() for its device, or else by the first call of
//     this entry point on a device -- looks the array's address up with
//     cudaGetSymbolAddress (that device current), which loads the module, and
//     loads every kernel this entry point launches.  A caller that is about
//     to hand the free device memory to its own allocator therefore calls
//     xkblas_init() (or this entry point once) first; that first call should
//     also come before any stream capture;
//   * the address is cached per device together with the CUDA context's
//     unique ID; after cudaDeviceReset() the next call sees a new context and
//     looks the (reloaded) array up again.
// Nothing in the array has to start at zero: every byte a call reads is
// written earlier in the same call (planes padded by the residue kernel and a
// 2-D memset, row codes and partials fully rewritten, the call's moduli
// selection words cleared by a memset first).
namespace xkb {
namespace oz {
constexpr int kNoAllocMaxDim = 512;
// per-plane rows and k extent at the limit: max(rup(512,128), rup(512,256))
constexpr size_t kNoAllocRows = 512, kNoAllocK = 512;
constexpr size_t kNoAllocPlane = kNoAllocRows * kNoAllocK;              // bytes
constexpr size_t kNoAllocA = kMaxMod * kNoAllocPlane;                  // A planes
constexpr size_t kNoAllocB = kMaxMod * kNoAllocPlane;                  // B planes
constexpr size_t kNoAllocR = kMaxMod * kNoAllocRows * kNoAllocRows;    // C residues
constexpr size_t kNoAllocShift = 2 * 4 * kNoAllocRows;                 // mu, nu
constexpr size_t kNoAllocPart = sizeof(double4) * 2 * kNoAllocRows;    // 1 k-chunk
constexpr size_t kNoAllocBytes =
    kNoAllocA + kNoAllocB + kNoAllocR + kNoAllocShift + kNoAllocPart + 4096;

static __device__ __align__(256) unsigned char g_oz_noalloc_scratch[kNoAllocBytes];

// C <- beta C on the masked part (beta == 0 writes zeros without reading),
// for K == 0 or alpha == 0: kept in this file so that the scratch-free path
// launches only kernels of this module (loaded by noalloc_prepare).
__global__ void k_oz_beta(int M, int N, double beta, double* C, long ldc, int uplo, long diag) {
  const size_t total = (size_t)M * (size_t)N;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total;
       e += (size_t)gridDim.x * blockDim.x) {
    const long i = (long)(e % (size_t)M), j = (long)(e / (size_t)M);
    if (uplo == XKB_LOWER && i + diag < j) continue;
    if (uplo == XKB_UPPER && i + diag > j) continue;
    double* c = C + (size_t)i + (size_t)j * (size_t)ldc;
    *c = beta != 0.0 ? beta * *c : 0.0;
  }
}

// Kernels the scratch-free path launches, loaded up front (with lazy loading
// a kernel's code is otherwise placed in device memory at its first launch).
template <int NM>
static bool load_nm_kernels() {
  cudaFuncAttributes fa;
  return cudaFuncGetAttributes(&fa, k_oz_residues<true, NM, double>) == cudaSuccess &&
         cudaFuncGetAttributes(&fa, k_oz_residues<false, NM, double>) == cudaSuccess &&
         cudaFuncGetAttributes(&fa, k_oz_crt<NM>) == cudaSuccess;
}
static bool load_noalloc_kernels() {
  cudaFuncAttributes fa;
  bool ok = cudaFuncGetAttributes(&fa, k_oz_norm<true, double>) == cudaSuccess &&
            cudaFuncGetAttributes(&fa, k_oz_norm<false, double>) == cudaSuccess &&
            cudaFuncGetAttributes(&fa, k_oz_stat) == cudaSuccess &&
            cudaFuncGetAttributes(&fa, k_oz_pick) == cudaSuccess &&
            cudaFuncGetAttributes(&fa, k_oz_crt_15_16) == cudaSuccess &&
            cudaFuncGetAttributes(&fa, k_oz_gemm) == cudaSuccess &&
            cudaFuncGetAttributes(&fa, k_oz_beta) == cudaSuccess;
  ok = ok && load_nm_kernels<2>() && load_nm_kernels<3>() && load_nm_kernels<4>() &&
       load_nm_kernels<5>() && load_nm_kernels<6>() && load_nm_kernels<7>() &&
       load_nm_kernels<8>() && load_nm_kernels<9>() && load_nm_kernels<10>() &&
       load_nm_kernels<11>() && load_nm_kernels<12>() && load_nm_kernels<13>() &&
       load_nm_kernels<14>() && load_nm_kernels<15>() && load_nm_kernels<16>();
  return ok;
}

// Device address of the array for the current device, looked up when the
// device's context is seen for the first time (once per device, unless the
// context is reset).
static int noalloc_base(unsigned char** out) {
  static std::mutex mu;
  static unsigned char* ptr[64] = {nullptr};
  static unsigned long long ctx_of[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return XKB_ECUDA;
  std::lock_guard<std::mutex> g(mu);
  const unsigned long long id = context_id();
  if (!ptr[dev] || id == 0 || id != ctx_of[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_oz_noalloc_scratch) != cudaSuccess || !p ||
        !load_noalloc_kernels()) {
      cudaGetLastError();
      ptr[dev] = nullptr;
      return XKB_ECUDA;
    }
    ptr[dev] = static_cast<unsigned char*>(p);
    ctx_of[dev] = context_id();  // the lookup made the primary context current
  }
  *out = ptr[dev];
  return XKB_OK;
}
}  // namespace oz

int noalloc_prepare() {
  unsigned char* p = nullptr;
  return oz::noalloc_base(&p);
}
}  // namespace xkb

extern "C" int xkb_cuda_ozaki_gemm_noalloc(const xkb_gemm_args* a, int nmod, void* stream) {
  if (!a || a->dtype != XKB_D) return XKB_EINVAL;
  if (a->M < 0 || a->N < 0 || a->K < 0) return XKB_EINVAL;
  if (a->M > kNoAllocMaxDim || a->N > kNoAllocMaxDim || a->K > kNoAllocMaxDim) return XKB_ERANGE;
  if (a->M == 0 || a->N == 0) return XKB_OK;
  if (a->K > 0 && a->alpha[0] != 0.0 && (a->opA < XKB_OP_N || a->opA > XKB_OP_C ||
                                         a->opB < XKB_OP_N || a->opB > XKB_OP_C))
    return XKB_EINVAL;
  // nmod == 0: the data rule's count, at most 16 (there is no plain fallback
  // here: the plain kernel may need scratch for unaligned operands)
  ModPlan pl;
  if (!plan_moduli(nmod, a->K > 0 ? a->K : 1, &pl)) return XKB_ERANGE;
  const Consts* c = pl.chi;
  nmod = pl.hi;
  unsigned char* base = nullptr;
  int err = noalloc_base(&base);
  if (err) return err;
  cudaStream_t st = resolve_stream(stream);
  if (a->K == 0 || a->alpha[0] == 0.0) {  // beta C only
    const size_t total = (size_t)a->M * (size_t)a->N;
    const unsigned blocks = (unsigned)std::min<size_t>((total + 255) / 256, 1024);
    const long long tv = evlog_kern_begin(st, "k_oz_beta");
    k_oz_beta<<<blocks, 256, 0, st>>>(a->M, a->N, a->beta[0], static_cast<double*>(a->C), a->ldc,
                                      a->uplo, a->diag);
    evlog_kern_end(tv, st);
    count_launch();
    return cudaPeekAtLastError() == cudaSuccess ? XKB_OK : XKB_ECUDA;
  }
  const int M = a->M, N = a->N, K = a->K;
  const long Kpad = (long)rup(K, BKB), Mpad = (long)rup(M, BM), Npad = (long)rup(N, BN);
  const bool akc = a->opA != XKB_OP_N, bkc = a->opB == XKB_OP_N;
  const bool same = (a->A == a->B) && (a->lda == a->ldb) && (akc == bkc) && M == N;
  const long Arows = same ? std::max(Mpad, Npad) : Mpad;
  // carve the fixed array (all offsets 256-byte aligned)
  int8_t* Ap = reinterpret_cast<int8_t*>(base);
  int8_t* Bp = reinterpret_cast<int8_t*>(base + kNoAllocA);
  uint8_t* R = base + kNoAllocA + kNoAllocB;
  int* mu = reinterpret_cast<int*>(base + kNoAllocA + kNoAllocB + kNoAllocR);
  int* nu = mu + kNoAllocRows;
  unsigned char* tail = base + kNoAllocA + kNoAllocB + kNoAllocR + kNoAllocShift;
  double4* part = reinterpret_cast<double4*>(tail);
  CallWords* w = reinterpret_cast<CallWords*>(tail + kNoAllocPart);
  const OzSel* sel = &w->sel;
  const double* Ad = static_cast<const double*>(a->A);
  const double* Bd = static_cast<const double*>(a->B);
  const int slot = trace_begin("ozaki_noalloc", a->dtype, M, N, K, pl.fixed ? nmod : 0, st);
  View va{Ad, a->lda, akc, XKB_D, false}, vb{Bd, a->ldb, bkc, XKB_D, false};
  if (cudaMemsetAsync(w, 0, sizeof(CallWords), st) != cudaSuccess) err = XKB_ECUDA;
  if (!err) err = launch_norm(va, M, K, part, mu, &w->rmax[0], st);
  if (!err) err = launch_norm(vb, N, K, part + kNoAllocRows, nu, &w->rmax[1], st);
  if (!err) err = launch_pick(w, pl, false, st);
  if (!err) err = launch_res(va, M, K, mu, sel, c, Ap, Arows, Kpad, st);
  if (!err && !same) err = launch_res(vb, N, K, nu, sel, c, Bp, Npad, Kpad, st);
  if (!err && Kpad > (long)rup(K, 64)) {
    const size_t kz = rup(K, 64);
    if (cudaMemset2DAsync(Ap + kz, Kpad, 0, Kpad - kz, (size_t)nmod * Arows, st) != cudaSuccess ||
        (!same &&
         cudaMemset2DAsync(Bp + kz, Kpad, 0, Kpad - kz, (size_t)nmod * Npad, st) != cudaSuccess))
      err = XKB_ECUDA;
  }
  trace_mark(slot, 1, st);
  if (!err)
    err = same ? launch_gemm(Ap, Arows, Ap, Arows, Mpad, Npad, Kpad, c, sel, R, a->uplo, a->diag,
                             st)
               : launch_gemm(Ap, Mpad, Bp, Npad, Mpad, Npad, Kpad, c, sel, R, a->uplo, a->diag,
                             st);
  trace_mark(slot, 2, st);
  if (!err) {
    CrtP cp;
    std::memset(&cp, 0, sizeof(cp));
    cp.M = M;
    cp.N = N;
    cp.R = R;
    cp.Mpad = Mpad;
    cp.Npad = Npad;
    cp.mu = mu;
    cp.nu = nu;
    cp.sel = sel;
    cp.C = a->C;
    cp.ldc = a->ldc;
    cp.ar = a->alpha[0];
    cp.br = a->beta[0];
    cp.uplo = a->uplo;
    cp.diag = a->diag;
    err = launch_crt(st, cp, pl.clo, pl.chi);
  }
  trace_mark(slot, 3, st);
  return err;
}
