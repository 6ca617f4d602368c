// dmma_tile.cuh -- shared-memory operand tiles of the FP64 DMMA GEMM and
// their fragment loads.
//
// A stage holds BK = 128 / sizeof(T) k indices of op(A) (BM rows) and op(B)
// (BN columns), 128 bytes per row and operand, written by TMA with the
// 128-byte swizzle: the 16-byte chunk c of a 128-byte line lies at chunk
// c ^ (line & 7).
//   k contiguous (KC):  line = row, the line's 128 bytes = its BK k values;
//   otherwise:          panels of BK rows, line = k within the panel, the
//                       line's 128 bytes = the panel's BK rows.
// Both layouts are read with the widest load whose lanes fall on distinct
// banks.  Two free permutations make that possible without copying: which
// physical k a lane's two MMA k slots hold (the same for A and B, so sums
// are unchanged), and which physical row an MMA row (column of op(B)) is
// (undone where the accumulators are stored).  Where elements are 4 or 8
// bytes, MMA row g + 8h of a 16-row block is physical row 2 q(g) + h, so a
// lane's two accumulator rows are neighbours in memory and C moves in 8- and
// 16-byte accesses.
// Without the swizzle (rows at 128-byte or 1 KB strides) the A loads had
// 4-way and the B loads 2-way bank conflicts: hidden behind the DMMA pipe in
// 128 x 128 tiles, but 64 x 64 tiles then ran at 74 % of the big tiles' rate
// per SM.
#pragma once
#include "dmma_common.cuh"

namespace xkb {

template <class T, bool KC>
struct OpTile {
  static constexpr int ES = (int)sizeof(T);
  static constexpr int BK = 128 / ES;   // k per stage; rows per panel when !KC
  static constexpr int KS = BK / 8;     // MMA k steps per stage (double complex: 1)
  // rows between a lane's two accumulator rows: neighbours, or (16-byte
  // elements, one access each) MMA rows g and g + 8 where they are
  static constexpr int PS = ES == 16 ? 8 : 1;

  // physical row in a 16-row block of MMA row g + 8h
  static __device__ __forceinline__ int prow(int g, int h) {
    if (ES == 16) return g + 8 * h;
    const int q = ES == 8 && KC ? ((g >> 1) & 1) | ((g & 1) << 1) | (g & 4) : g;
    return 2 * q + h;
  }

  // byte offset of element (row r, k) in the tile
  static __device__ __forceinline__ int off(int r, int k) {
    if constexpr (KC) return r * 128 + ((k * ES) ^ ((r & 7) << 4));
    else return (r / BK) * (BK * 128) + k * 128 + (((r % BK) * ES) ^ ((k & 7) << 4));
  }
  // physical k of this lane's MMA k slot v (0, 1) in step kc
  static __device__ __forceinline__ int kof(int t, int v, int kc) {
    return kc * 8 + 2 * t + v;
  }

  // Rows [r0, r0 + 16) (r0 a multiple of 16), k step kc: re/im[h][v] = element
  // of MMA row g + 8h, k slot v.
  static __device__ __forceinline__ void load(const uint8_t* tile, int r0, int kc, int g, int t,
                                              double (&re)[2][2], double (&im)[2][2]) {
    if constexpr (ES == 16) {
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          const double2 x =
              *reinterpret_cast<const double2*>(tile + off(r0 + prow(g, h), kof(t, v, kc)));
          re[h][v] = x.x;
          im[h][v] = x.y;
        }
    } else if constexpr (KC) {  // one load: both k slots of a row
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint8_t* q = tile + off(r0 + prow(g, h), kof(t, 0, kc));
        if constexpr (St<T>::CPLX) {
          const float4 x = *reinterpret_cast<const float4*>(q);
          re[h][0] = x.x, im[h][0] = x.y, re[h][1] = x.z, im[h][1] = x.w;
        } else if constexpr (ES == 8) {
          const double2 x = *reinterpret_cast<const double2*>(q);
          re[h][0] = x.x, re[h][1] = x.y;
        } else {
          const float2 x = *reinterpret_cast<const float2*>(q);
          re[h][0] = x.x, re[h][1] = x.y;
        }
      }
    } else {  // one load: both rows of a k slot
#pragma unroll
      for (int v = 0; v < 2; ++v) {
        const uint8_t* q = tile + off(r0 + prow(g, 0), kof(t, v, kc));
        if constexpr (St<T>::CPLX) {
          const float4 x = *reinterpret_cast<const float4*>(q);
          re[0][v] = x.x, im[0][v] = x.y, re[1][v] = x.z, im[1][v] = x.w;
        } else if constexpr (ES == 8) {
          const double2 x = *reinterpret_cast<const double2*>(q);
          re[0][v] = x.x, re[1][v] = x.y;
        } else {
          const float2 x = *reinterpret_cast<const float2*>(q);
          re[0][v] = x.x, re[1][v] = x.y;
        }
      }
    }
  }
};

// x with its sign bit flipped where flip has bit 31 set (an integer
// operation: the FP64 pipe stays with the MMAs)
__device__ __forceinline__ double xor_sign(double x, unsigned flip) {
  return __hiloint2double(__double2hiint(x) ^ (int)flip, __double2loint(x));
}

// Two values of C, PS rows apart (see OpTile); one, two: which of them are
// wanted; vec: aligned for one access (16-byte elements: one each).
template <class T>
__device__ __forceinline__ void ld_pair(const typename St<T>::S* c, bool vec, bool one, bool two,
                                        double (&re)[2], double (&im)[2]) {
  using S = typename St<T>::S;
  constexpr int D = St<T>::W * OpTile<T, true>::PS;
  re[0] = re[1] = im[0] = im[1] = 0.0;
  if (vec && one && two) {
    if constexpr (sizeof(T) == 16) {
      const double2 a = reinterpret_cast<const double2*>(c)[0];
      const double2 b = *reinterpret_cast<const double2*>(c + D);
      re[0] = a.x, im[0] = a.y, re[1] = b.x, im[1] = b.y;
    } else if constexpr (St<T>::CPLX) {
      const float4 a = *reinterpret_cast<const float4*>(c);
      re[0] = a.x, im[0] = a.y, re[1] = a.z, im[1] = a.w;
    } else if constexpr (sizeof(S) == 8) {
      const double2 a = *reinterpret_cast<const double2*>(c);
      re[0] = a.x, re[1] = a.y;
    } else {
      const float2 a = *reinterpret_cast<const float2*>(c);
      re[0] = a.x, re[1] = a.y;
    }
    return;
  }
  if (one) {
    re[0] = (double)c[0];
    if (St<T>::CPLX) im[0] = (double)c[1];
  }
  if (two) {
    re[1] = (double)c[D];
    if (St<T>::CPLX) im[1] = (double)c[D + 1];
  }
}
template <class T>
__device__ __forceinline__ void st_pair(typename St<T>::S* c, bool vec, bool one, bool two,
                                        const double (&re)[2], const double (&im)[2]) {
  using S = typename St<T>::S;
  constexpr int D = St<T>::W * OpTile<T, true>::PS;
  if (vec && one && two) {
    if constexpr (sizeof(T) == 16) {
      reinterpret_cast<double2*>(c)[0] = make_double2(re[0], im[0]);
      *reinterpret_cast<double2*>(c + D) = make_double2(re[1], im[1]);
    } else if constexpr (St<T>::CPLX) {
      *reinterpret_cast<float4*>(c) =
          make_float4((float)re[0], (float)im[0], (float)re[1], (float)im[1]);
    } else if constexpr (sizeof(S) == 8) {
      *reinterpret_cast<double2*>(c) = make_double2(re[0], re[1]);
    } else {
      *reinterpret_cast<float2*>(c) = make_float2((float)re[0], (float)re[1]);
    }
    return;
  }
  if (one) {
    c[0] = static_cast<S>(re[0]);
    if (St<T>::CPLX) c[1] = static_cast<S>(im[0]);
  }
  if (two) {
    c[D] = static_cast<S>(re[1]);
    if (St<T>::CPLX) c[D + 1] = static_cast<S>(im[1]);
  }
}

}  // namespace xkb
