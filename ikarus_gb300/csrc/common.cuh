// Device helpers shared by the element, sparse and solver kernels (sm_103a).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace ikr {

// 2-point Gauss-Legendre abscissae on [0,1]: 1/2 -+ 1/(2 sqrt 3).  With them every Q1 shape-function
// factor at a Gauss point is one of these two numbers (1 - lo == hi).
constexpr double kGaussLo = 0.21132486540518711775;
constexpr double kGaussHi = 0.78867513459481288225;
constexpr double kGaussW = 0.125;  // 2x2x2 rule on the unit cube

// Gauss point q = x + 2y + 4z; Dune vertex v = (v&1, v>>1&1, v>>2&1).
// dN_v/dxi_d at Gauss point q = s_d(v) * prod_{d' != d} (bit_d'(v) == bit_d'(q) ? hi : lo).
template <typename T>
__device__ __forceinline__ void ref_gradient_at_gp(int v, int q, T dxi[3]) {
  const T f0 = (((v ^ q) & 1) == 0) ? T(kGaussHi) : T(kGaussLo);
  const T f1 = (((v ^ q) & 2) == 0) ? T(kGaussHi) : T(kGaussLo);
  const T f2 = (((v ^ q) & 4) == 0) ? T(kGaussHi) : T(kGaussLo);
  dxi[0] = ((v & 1) ? T(1) : T(-1)) * f1 * f2;
  dxi[1] = ((v & 2) ? T(1) : T(-1)) * f0 * f2;
  dxi[2] = ((v & 4) ? T(1) : T(-1)) * f0 * f1;
}
// The same for one Gauss point and all nodes, without FP64 instructions: |dN_v/dxi_d| takes four values per direction,
// by the node's bits in the other two directions (d = 0: bits 1, 2; 1: bits 0, 2; 2: bits 0, 1), its sign is bit d's.
struct GpFactors {
  double f[3][4];
  __device__ __forceinline__ explicit GpFactors(int q) {
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const int a = (q >> (d == 0 ? 1 : 0)) & 1, b = (q >> (d == 2 ? 1 : 2)) & 1;
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const int same = ((m & 1) == a) + ((m >> 1) == b);
        f[d][m] = same == 2 ? kGaussHi * kGaussHi : same == 1 ? kGaussHi * kGaussLo : kGaussLo * kGaussLo;
      }
    }
  }
  // dN_v/dxi_d (v and d compile-time)
  __device__ __forceinline__ double operator()(int v, int d) const {
    const int a = (v >> (d == 0 ? 1 : 0)) & 1, b = (v >> (d == 2 ? 1 : 2)) & 1;
    const double x = f[d][a + 2 * b];
    return (v >> d) & 1 ? x : -x;
  }
};
// The trilinear interpolation as butterflies over the eight lanes of an element: lane v holds the value at node v and gets
// that at Gauss point v, bit d of both being the side in direction d.  Along a direction the interpolation is
// own + Lo (other - own) and the derivative the difference of the two sides, so the three derivatives of a field take 12
// FP64 instructions instead of the 24 of a sum over the nodes, and the transposed operation 15 instead of 24 and the sum
// over the points.  All 32 lanes take part.
struct GpButterfly {
  uint32_t sign[3];  // the sign bit, set on the high side of a direction
  __device__ __forceinline__ explicit GpButterfly(int q) {
#pragma unroll
    for (int d = 0; d < 3; ++d) sign[d] = (uint32_t)((q >> d) & 1) << 31;
  }
  static __device__ __forceinline__ double other(double x, int d) { return __shfl_xor_sync(0xffffffffu, x, 1 << d); }
  static __device__ __forceinline__ double flip(double x, uint32_t s) {
    return __hiloint2double((int)((uint32_t)__double2hiint(x) ^ s), __double2loint(x));
  }
  static __device__ __forceinline__ double along(double x, int d) { return fma(kGaussLo, other(x, d) - x, x); }
  __device__ __forceinline__ void gradient(double u, double (&g)[3]) const {
    const double dz = other(u, 2) - u, t = fma(kGaussLo, dz, u);
    g[0] = along(flip(other(t, 0) - t, sign[0]), 1);
    g[1] = along(flip(other(t, 1) - t, sign[1]), 0);
    g[2] = along(along(flip(dz, sign[2]), 1), 0);
  }
  // sum over the points of q . dN_v/dxi
  __device__ __forceinline__ double onto_nodes(const double (&q)[3]) const {
    double s[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) s[d] = flip(q[d] + other(q[d], d), sign[d] ^ 0x80000000u);
    return along(along(s[0], 1) + along(s[1], 0), 2) + along(along(s[2], 1), 0);
  }
};
// dN_v/dxi at the element centre (1/2,1/2,1/2)
template <typename T>
__device__ __forceinline__ void ref_gradient_at_center(int v, T dxi[3]) {
  dxi[0] = ((v & 1) ? T(0.25) : T(-0.25));
  dxi[1] = ((v & 2) ? T(0.25) : T(-0.25));
  dxi[2] = ((v & 4) ? T(0.25) : T(-0.25));
}

template <typename T>
__device__ __forceinline__ T det3(const T m[3][3]) {
  return m[0][0] * (m[1][1] * m[2][2] - m[1][2] * m[2][1]) - m[0][1] * (m[1][0] * m[2][2] - m[1][2] * m[2][0]) +
         m[0][2] * (m[1][0] * m[2][1] - m[1][1] * m[2][0]);
}
// inverse of a 3x3 by cofactors; returns the determinant
template <typename T>
__device__ __forceinline__ T inv3(const T m[3][3], T r[3][3]) {
  const T c00 = m[1][1] * m[2][2] - m[1][2] * m[2][1];
  const T c01 = m[1][2] * m[2][0] - m[1][0] * m[2][2];
  const T c02 = m[1][0] * m[2][1] - m[1][1] * m[2][0];
  const T d = m[0][0] * c00 + m[0][1] * c01 + m[0][2] * c02;
  const T id = T(1) / d;
  r[0][0] = c00 * id;
  r[0][1] = (m[0][2] * m[2][1] - m[0][1] * m[2][2]) * id;
  r[0][2] = (m[0][1] * m[1][2] - m[0][2] * m[1][1]) * id;
  r[1][0] = c01 * id;
  r[1][1] = (m[0][0] * m[2][2] - m[0][2] * m[2][0]) * id;
  r[1][2] = (m[0][2] * m[1][0] - m[0][0] * m[1][2]) * id;
  r[2][0] = c02 * id;
  r[2][1] = (m[0][1] * m[2][0] - m[0][0] * m[2][1]) * id;
  r[2][2] = (m[0][0] * m[1][1] - m[0][1] * m[1][0]) * id;
  return d;
}

// butterfly sum over the 8 lanes that share an element (lanes 8k..8k+7 of a warp)
template <typename T>
__device__ __forceinline__ T sum8(T v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  v += __shfl_xor_sync(0xffffffffu, v, 4);
  return v;
}

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Voigt pairs in the order 11,22,33,23,13,12
__device__ __forceinline__ int voigt_a(int v) { return v < 3 ? v : (v == 3 ? 1 : 0); }
__device__ __forceinline__ int voigt_b(int v) { return v < 3 ? v : (v == 5 ? 1 : 2); }

}  // namespace ikr
