// Enhanced-assumed-strain Q1 hexahedra (sm_103a): the element kernel template, included by element_eas.cu
// (NeoHooke, StVenantKirchhoff, BlatzKo) and element_eas_hyper.cu (the hyperelastic framework).
//
// Reference: EnhancedAssumedStrains (ikarus/finiteelements/mechanics/enhancedassumedstrains.hh:225-434) with
// the strain functions easfunctions/{greenlagrangestrain,displacementgradient,displacementgradienttransposed}.hh
// and the ansatz spaces easvariants/{linearandglstrains,displacementgradient,helperfunctions}.hh.
//
// One element per block of 64 threads: eight lanes (lane = node I) for each of the eight Gauss points, because the work
// at a point is some 800 to 1 300 FP64 instructions a lane, many of them dependent, which GB300 starts one per 16 cycles and SM and finishes
// one per 60: an element whose points follow one another keeps a small mesh waiting for eight times that, and one lane
// factorising D keeps the other seven.  The loops over modes, columns and blocks are rolled: unrolled, the kernels had 120 to
// 280 KB of instructions, each run once, and now have 70 to 120.  Measured with assembly, residual and tangent, eight
// lanes per element and one launch per colour -> unrolled -> this: 10 elements (H9) 660 -> 60 -> 46 us and 1 030 -> 80 -> 67 us,
// 8 192 elements (E9) 2.34 -> 1.01 -> 0.75 ms and 3.86 -> 1.63 -> 1.35 ms.  E21, whose tangent takes 110 KB of shared memory,
// two blocks per SM, first and last form: 256 elements 6.53 -> 0.12 and 8.32 -> 0.14 ms, 16 384 elements 6.96 -> 4.74 and
// 8.88 -> 6.12 ms.
// The lanes of a point share F, S and the Voigt tangent C (each lane computes a few of its 36 entries into shared
// memory), and each lane computes the enhanced-strain columns E_alpha(:,k) and C E_alpha(:,k) for k = I, I+8, ...
// The points' shares of f, K, L, D and R~ are summed in a fixed order through shared memory.  D (n_alpha x n_alpha) is
// LU-factorised by a warp (partial pivoting, FP64), the 24 columns of D^{-1} L and D^{-1} R~ are solved with
// a lane each, and the condensed quantities
//   f_I -= L_I^T D^{-1} R~,   K_IJ -= L_I^T D^{-1} L_J        (enhancedassumedstrains.hh:291-296, 336-345)
// are formed by all 64 threads; K as the 40 blocks (I, I + d mod 8), d = 0..4, d = 1..3 transposed as well.
// D^{-1} R~ and D^{-1} L are cached per element (FP64) when the residual is formed, so the internal-state
// update alpha -= D^{-1} (R~ + L dd) (enhancedassumedstrains.hh:225-248) costs one pass over the cache.
// The kernel writes element vectors and matrices; assembly gathers them (element.cu), in element order.
//
// The enhancement modes are rank one.  H9: H_p = s_p a_r (x) a_c with p = 3r + c, s_p = (detJ0/detJ)(2 xi_c - 1)
// and a_k the k-th column of J0^{-T} (easvariants/displacementgradient.hh:136-161, helperfunctions.hh:27-36).
// Every enhanced-strain quantity is therefore written through (v, coef) with column i of the mode's
// displacement-gradient matrix equal to coef_i v:  H: v = a_r, coef = s a_c;   H9T (F_c0 H_p^T): v = F_c0 a_c,
// coef = s a_r.  GL (E9/E21): E_alpha(:,k) = (T0^{-1} / detJ) M0(:,k) with one nonzero per M0 column.
#pragma once
#include <cmath>

#include "common.cuh"
#include "hyperelastic.cuh"
#include "kernels.h"

namespace ikr {

namespace {

// E9 / E21 ansatz (easvariants/linearandglstrains.hh:252-327): column k has its single entry in row kRow[k],
// equal to the product of (2 xi_f - 1) over the listed factors (second factor -1 = none).
__constant__ int kRow[21] = {0, 1, 2, 3, 3, 4, 4, 5, 5, 3, 3, 4, 4, 5, 5, 0, 0, 1, 1, 2, 2};
__constant__ int kF1[21] = {0, 1, 2, 1, 2, 0, 2, 0, 1, 0, 0, 0, 1, 0, 1, 0, 0, 0, 1, 0, 1};
__constant__ int kF2[21] = {-1, -1, -1, -1, -1, -1, -1, -1, -1, 1, 2, 1, 2, 2, 2, 1, 2, 1, 2, 2, 2};

template <int NA>
struct EasCfg {
  static constexpr int NT = NA * (NA + 1) / 2; // packed upper triangle of D
  // shared memory of a Gauss point (doubles)
  static constexpr int O_DN = 0;               // 8 x 3   modified nodal gradients
  static constexpr int O_C6 = O_DN + 24;       // 36      Voigt tangent
  static constexpr int O_EA = O_C6 + 36;       // NA x 6  E_alpha columns
  static constexpr int O_CEA = O_EA + 6 * NA;  // NA x 6  C E_alpha columns
  static constexpr int O_S = O_CEA + 6 * NA;   // NA x 6  GL: ansatz coefficients / detJ times alpha; H/HT: v and coef
  static constexpr int POINT = O_S + 6 * NA;
  // of the element: the points' shares [share][point], shares in the order f or K, L, D, R~
  static constexpr int shares(bool want_k) { return (want_k ? 360 : 24) + 24 * NA + NT + (want_k ? 0 : NA); }
  // after the points: T0^{-1} (GL) or A0 and Fc0 A0 (H/HT), D, R~ and its solution, L, D^{-1} L, the row order
  static constexpr int O_GEO = 8 * POINT;
  static constexpr int O_D = O_GEO + 36;
  static constexpr int O_RT = O_D + NA * NA;
  static constexpr int O_L = O_RT + 2 * NA;    // NA x 24
  static constexpr int O_Y = O_L + 24 * NA;    // 24 x NA
  static constexpr int O_PERM = O_Y + 24 * NA; // NA
  static constexpr int O_INV = O_PERM + NA;    // NA      reciprocal pivots
  static constexpr int O_SHARE = O_INV + NA;
  static constexpr int total(bool want_k) { return O_SHARE + 8 * shares(want_k); }
};

__device__ __forceinline__ void packed_index(int t, int na, int& a, int& b) {
  a = 0;
  int rowlen = na;
  while (t >= rowlen) {
    t -= rowlen;
    ++a;
    --rowlen;
  }
  b = a + t;
}

// Voigt form of sym(F^T (coef (x) ... )) for a displacement-gradient variation whose column i is coef_i v:
// E[0] = coef0 g0, ..., E[3] = coef2 g1 + coef1 g2, with g_j = v . F(:,j)  (easfunctions/displacementgradient.hh:153-166)
__device__ __forceinline__ void sym_voigt(const double coef[3], const double v[3], const double F[3][3], double E[6]) {
  double g[3];
#pragma unroll
  for (int j = 0; j < 3; ++j) g[j] = v[0] * F[0][j] + v[1] * F[1][j] + v[2] * F[2][j];
  E[0] = coef[0] * g[0];
  E[1] = coef[1] * g[1];
  E[2] = coef[2] * g[2];
  E[3] = coef[2] * g[1] + coef[1] * g[2];
  E[4] = coef[2] * g[0] + coef[0] * g[2];
  E[5] = coef[1] * g[0] + coef[0] * g[1];
}

// B-operator (6x3) of the Green-Lagrange strain variation, rows as in easfunctions/displacementgradient.hh:135-145
__device__ __forceinline__ void bop(const double F[3][3], const double dN[3], double B[6][3]) {
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double g0 = F[a][0], g1 = F[a][1], g2 = F[a][2];
    B[0][a] = dN[0] * g0;
    B[1][a] = dN[1] * g1;
    B[2][a] = dN[2] * g2;
    B[3][a] = dN[2] * g1 + dN[1] * g2;
    B[4][a] = dN[2] * g0 + dN[0] * g2;
    B[5][a] = dN[1] * g0 + dN[0] * g1;
  }
}

// HYP: the hyperelastic framework's material point (hyperelastic.cuh) instead of the closed-form laws
template <int NA, int KIND, int MODE, bool HYP>
__global__ void __launch_bounds__(64) eas_element_kernel(ElemArgs a, const int32_t* __restrict__ list, int e_base) {
  using Cfg = EasCfg<NA>;
  constexpr bool WANT_R = MODE & kWantR;
  constexpr bool WANT_K = MODE & kWantK;
  static_assert(WANT_R != WANT_K && (MODE & kElemOut), "element vectors or element matrices");
  extern __shared__ double smem[];

  const int lane = threadIdx.x & 31;
  const int sub = threadIdx.x & 7;
  const int q = threadIdx.x >> 3;  // Gauss point
  double* sm = smem + (size_t)q * Cfg::POINT;
  const int li = blockIdx.x;
  const int e = list ? list[li] : e_base + li;
  const int ne = a.n_elems;
  const int node = a.conn[sub * ne + e];
  const int src = lane & ~7;

  double dX[3], dU[3], Ud[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double x = a.X[3 * node + c];
    Ud[c] = a.u ? a.u[3 * node + c] : 0.0;
    dX[c] = x - __shfl_sync(0xffffffffu, x, src);
    dU[c] = Ud[c] - __shfl_sync(0xffffffffu, Ud[c], src);
  }
  // centre data
  double A0[3][3] = {}, detJ0 = 0.0, dN0[3] = {0, 0, 0}, Fc0[3][3] = {}, Fa[3][3] = {};
  if (KIND == 1) {
    if (threadIdx.x < 36) smem[Cfg::O_GEO + threadIdx.x] = a.eas_geo[(size_t)threadIdx.x * ne + e];
  } else {
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) A0[i][j] = a.eas_geo[(size_t)(3 * i + j) * ne + e];
    detJ0 = a.eas_geo[(size_t)9 * ne + e];
    if (threadIdx.x < 9) smem[Cfg::O_GEO + threadIdx.x] = a.eas_geo[(size_t)threadIdx.x * ne + e];
    if (KIND == 3) {
#pragma unroll
      for (int k = 0; k < 3; ++k) dN0[k] = a.eas_geo[(size_t)(10 + 3 * sub + k) * ne + e];
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) Fc0[i][j] = sum8(dU[i] * dN0[j]) + (i == j ? 1.0 : 0.0);
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int c = 0; c < 3; ++c) Fa[i][c] = Fc0[i][0] * A0[0][c] + Fc0[i][1] * A0[1][c] + Fc0[i][2] * A0[2][c];
      if (threadIdx.x == 0) {
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int c = 0; c < 3; ++c) smem[Cfg::O_GEO + 9 + 3 * i + c] = Fa[i][c];
      }
    }
  }
  __syncthreads();

  const double lam = a.lam_e ? a.lam_e[e] : a.lam, mu = a.mu_e ? a.mu_e[e] : a.mu;
  int bad = 0;
  double* share = smem + Cfg::O_SHARE + q;  // share t of this point at share[8 t]
  constexpr int kL = WANT_K ? 360 : 24, kD = kL + 24 * NA, kR = kD + Cfg::NT;
  {
    double dxi[3];
    ref_gradient_at_gp<double>(sub, q, dxi);
    double J[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) J[i][j] = sum8(dX[i] * dxi[j]);
    double Ji[3][3];
    const double detJ = inv3(J, Ji);
    double dN[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) dN[k] = dxi[0] * Ji[0][k] + dxi[1] * Ji[1][k] + dxi[2] * Ji[2][k];
    double H[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) H[i][j] = sum8(dU[i] * dN[j]);

    // enhancement at this Gauss point
    const double rdet = 1.0 / detJ;
    double sx[3] = {};  // H/HT mode scales by the mode's column
    double Ht[3][3] = {};
    if (KIND == 1) {  // GL ansatz coefficients / detJ, by the lane that owns the column
#pragma unroll 1
      for (int k = sub; k < NA; k += 8) {
        const int f1 = kF1[k], f2 = kF2[k];
        double v = (q >> f1) & 1 ? 2.0 * kGaussHi - 1.0 : 2.0 * kGaussLo - 1.0;
        if (f2 >= 0) v *= (q >> f2) & 1 ? 2.0 * kGaussHi - 1.0 : 2.0 * kGaussLo - 1.0;
        v *= rdet;
        sm[Cfg::O_S + 2 * k] = v;
        sm[Cfg::O_S + 2 * k + 1] = v * a.alpha[(size_t)k * ne + e];
      }
      __syncwarp();
    } else {
      const double sc = detJ0 * rdet;
#pragma unroll
      for (int c = 0; c < 3; ++c) sx[c] = sc * ((q >> c) & 1 ? 2.0 * kGaussHi - 1.0 : 2.0 * kGaussLo - 1.0);
      // Ht = A0 M A0^T with M the scaled modes
      double T1[3][3] = {};
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const double w = a.alpha[(size_t)(3 * r + c) * ne + e] * sx[c];
#pragma unroll
          for (int i = 0; i < 3; ++i) T1[i][c] += A0[i][r] * w;
        }
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) Ht[i][j] = T1[i][0] * A0[j][0] + T1[i][1] * A0[j][1] + T1[i][2] * A0[j][2];
      if (KIND == 2) {
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = 0; j < 3; ++j) H[i][j] += Ht[i][j];
      } else {  // H = Hc + Fc0 Ht^T (displacementgradienttransposed.hh:353-368)
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = 0; j < 3; ++j) H[i][j] += Fc0[i][0] * Ht[j][0] + Fc0[i][1] * Ht[j][1] + Fc0[i][2] * Ht[j][2];
      }
    }
    double F[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) F[i][j] = H[i][j] + (i == j ? 1.0 : 0.0);
    // Green-Lagrange strain (Voigt, doubled shears) plus the GL enhancement M alpha
    double Ev[6];
    {
      double E[3][3];
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
          E[i][j] = 0.5 * (H[i][j] + H[j][i] + H[0][i] * H[0][j] + H[1][i] * H[1][j] + H[2][i] * H[2][j]);
      Ev[0] = E[0][0], Ev[1] = E[1][1], Ev[2] = E[2][2];
      Ev[3] = 2.0 * E[1][2], Ev[4] = 2.0 * E[0][2], Ev[5] = 2.0 * E[0][1];
    }
    if (KIND == 1) {  // lane r forms component r
      const double* T = smem + Cfg::O_GEO + 6 * min(sub, 5);
      double x = 0.0;
#pragma unroll 3
      for (int k = 0; k < NA; ++k) x += sm[Cfg::O_S + 2 * k + 1] * T[kRow[k]];
#pragma unroll
      for (int r = 0; r < 6; ++r) Ev[r] += __shfl_sync(0xffffffffu, x, src + r);
    }
    double S[6], Sm[3][3];
    if constexpr (HYP) {
      // Hyperelastic<Deviatoric<DF>, Volumetric<VF>> on C = 2E + I (hyper::evaluate; moduli needed for D and L)
      double C[3][3];
      C[0][0] = 2.0 * Ev[0] + 1.0, C[1][1] = 2.0 * Ev[1] + 1.0, C[2][2] = 2.0 * Ev[2] + 1.0;
      C[1][2] = C[2][1] = Ev[3];
      C[0][2] = C[2][0] = Ev[4];
      C[0][1] = C[1][0] = Ev[5];
      hyper::Point pt;
      bad |= hyper::evaluate(a.hyper, C, pt, true);
#pragma unroll
      for (int v = 0; v < 6; ++v) {
        const int i = voigt_a(v), j = voigt_b(v);
        S[v] = hyper::stress(pt, i, j);
        Sm[i][j] = Sm[j][i] = S[v];
      }
#pragma unroll 1
      for (int t = sub; t < 36; t += 8) {
        const int r = t / 6, c = t % 6;
        sm[Cfg::O_C6 + t] = hyper::modulus(pt, voigt_a(r), voigt_b(r), voigt_a(c), voigt_b(c));
      }
    } else if (a.material == 1) {
      // StVenantKirchhoff (svk.hh:96-163): S = lambda tr(E) + 2 mu E (Voigt shears mu * 2E_ij), constant moduli
      const double trE = Ev[0] + Ev[1] + Ev[2];
#pragma unroll
      for (int v = 0; v < 6; ++v) {
        const int i = voigt_a(v), j = voigt_b(v);
        S[v] = v < 3 ? lam * trE + 2.0 * mu * Ev[v] : mu * Ev[v];
        Sm[i][j] = Sm[j][i] = S[v];
      }
#pragma unroll 1
      for (int t = sub; t < 36; t += 8) {
        const int r = t / 6, c = t % 6;
        sm[Cfg::O_C6 + t] = (r < 3 && c < 3 ? lam : 0.0) + (r == c ? (r < 3 ? 2.0 * mu : mu) : 0.0);
      }
    } else if (a.material == 2) {
      // BlatzKo on C = 2E + I: S = mu (J C^-1 - C^-2), moduli mu [J Ci_ij Ci_kl - J (Ci_ik Ci_jl + Ci_il Ci_jk)
      // + Ci_ik Ci2_jl + Ci_il Ci2_jk + Ci2_ik Ci_jl + Ci2_il Ci_jk] with Ci2 = C^-2
      double C[3][3], Ci[3][3], Ci2[3][3];
      C[0][0] = 2.0 * Ev[0] + 1.0, C[1][1] = 2.0 * Ev[1] + 1.0, C[2][2] = 2.0 * Ev[2] + 1.0;
      C[1][2] = C[2][1] = Ev[3];
      C[0][2] = C[2][0] = Ev[4];
      C[0][1] = C[1][0] = Ev[5];
      const double detC = inv3(C, Ci);
      if (!(detC > 1e-10)) bad |= kStatusNonPositiveDetC;
      const double Jd = sqrt(detC);
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j) Ci2[i][j] = Ci[i][0] * Ci[0][j] + Ci[i][1] * Ci[1][j] + Ci[i][2] * Ci[2][j];
#pragma unroll
      for (int v = 0; v < 6; ++v) {
        const int i = voigt_a(v), j = voigt_b(v);
        S[v] = mu * (Jd * Ci[i][j] - Ci2[i][j]);
        Sm[i][j] = Sm[j][i] = S[v];
      }
#pragma unroll 1
      for (int t = sub; t < 36; t += 8) {
        const int r = t / 6, c = t % 6;
        const int i = voigt_a(r), j = voigt_b(r), k = voigt_a(c), l = voigt_b(c);
        sm[Cfg::O_C6 + t] = mu * (Jd * Ci[i][j] * Ci[k][l] - Jd * (Ci[i][k] * Ci[j][l] + Ci[i][l] * Ci[j][k]) +
                                  Ci[i][k] * Ci2[j][l] + Ci[i][l] * Ci2[j][k] + Ci2[i][k] * Ci[j][l] +
                                  Ci2[i][l] * Ci[j][k]);
      }
    } else {
      // NeoHooke on C = 2E + I (neohooke.hh:100-142)
      double C[3][3], Ci[3][3];
      C[0][0] = 2.0 * Ev[0] + 1.0, C[1][1] = 2.0 * Ev[1] + 1.0, C[2][2] = 2.0 * Ev[2] + 1.0;
      C[1][2] = C[2][1] = Ev[3];
      C[0][2] = C[2][0] = Ev[4];
      C[0][1] = C[1][0] = Ev[5];
      const double detC = inv3(C, Ci);
      if (!(detC > 1e-10)) bad |= kStatusNonPositiveDetC;
      const double lnJ = log(sqrt(detC));
#pragma unroll
      for (int v = 0; v < 6; ++v) {
        const int i = voigt_a(v), j = voigt_b(v);
        S[v] = mu * ((i == j ? 1.0 : 0.0) - Ci[i][j]) + lam * lnJ * Ci[i][j];
        Sm[i][j] = Sm[j][i] = S[v];
      }
      const double cc = mu - lam * lnJ;
#pragma unroll 1
      for (int t = sub; t < 36; t += 8) {
        const int r = t / 6, c = t % 6;
        const int i = voigt_a(r), j = voigt_b(r), k = voigt_a(c), l = voigt_b(c);
        sm[Cfg::O_C6 + t] = lam * Ci[i][j] * Ci[k][l] + cc * (Ci[i][k] * Ci[j][l] + Ci[i][l] * Ci[j][k]);
      }
    }
    // nodal gradients entering B and kg (HT adds Ht dN0, displacementgradienttransposed.hh:126-140)
    double dNm[3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
      dNm[k] = dN[k] + (KIND == 3 ? Ht[k][0] * dN0[0] + Ht[k][1] * dN0[1] + Ht[k][2] * dN0[2] : 0.0);
#pragma unroll
    for (int k = 0; k < 3; ++k) sm[Cfg::O_DN + 3 * sub + k] = dNm[k];
    const double w = kGaussW * detJ;
    double B[6][3];
    bop(F, dNm, B);
    if (WANT_R) {
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        double t = 0.0;
#pragma unroll
        for (int r = 0; r < 6; ++r) t += B[r][b] * S[r];
        share[8 * (3 * sub + b)] = w * t;
      }
    }
    __syncwarp();  // C6 and dNm of all nodes are in shared memory

    double V[6][3];  // C B_I
#pragma unroll
    for (int r = 0; r < 6; ++r)
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        double t = 0.0;
#pragma unroll
        for (int x = 0; x < 6; ++x) t += sm[Cfg::O_C6 + 6 * r + x] * B[x][b];
        V[r][b] = t;
      }
    if (WANT_K) {
      double SdN[3];
#pragma unroll
      for (int i = 0; i < 3; ++i) SdN[i] = Sm[i][0] * dNm[0] + Sm[i][1] * dNm[1] + Sm[i][2] * dNm[2];
#pragma unroll 1
      for (int d = 0; d < 5; ++d) {
        const int Jn = (sub + d) & 7;
        double dNJ[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) dNJ[k] = sm[Cfg::O_DN + 3 * Jn + k];
        double BJ[6][3];
        bop(F, dNJ, BJ);
        const double kg = SdN[0] * dNJ[0] + SdN[1] * dNJ[1] + SdN[2] * dNJ[2];
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
          for (int j = 0; j < 3; ++j) {
            double t = (i == j) ? kg : 0.0;
#pragma unroll
            for (int r = 0; r < 6; ++r) t += V[r][i] * BJ[r][j];
            share[8 * ((d * 8 + sub) * 9 + 3 * i + j)] = w * t;
          }
      }
    }

    // enhanced-strain columns owned by this lane
#pragma unroll 1
    for (int k = sub; k < NA; k += 8) {
      double Ea[6];
      if (KIND == 1) {
        const double sk = sm[Cfg::O_S + 2 * k];
#pragma unroll
        for (int r = 0; r < 6; ++r) Ea[r] = sk * smem[Cfg::O_GEO + 6 * r + kRow[k]];
      } else {
        const int r = k / 3, c = k - 3 * r;
        const double sk = c == 0 ? sx[0] : c == 1 ? sx[1] : sx[2];
        double v[3], coef[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          v[i] = KIND == 2 ? smem[Cfg::O_GEO + 3 * i + r] : smem[Cfg::O_GEO + 9 + 3 * i + c];
          coef[i] = sk * smem[Cfg::O_GEO + 3 * i + (KIND == 2 ? c : r)];
          sm[Cfg::O_S + 6 * k + i] = v[i];
          sm[Cfg::O_S + 6 * k + 3 + i] = coef[i];
        }
        sym_voigt(coef, v, F, Ea);
      }
#pragma unroll
      for (int r = 0; r < 6; ++r) {
        sm[Cfg::O_EA + 6 * k + r] = Ea[r];
        double t = 0.0;
#pragma unroll
        for (int x = 0; x < 6; ++x) t += sm[Cfg::O_C6 + 6 * r + x] * Ea[x];
        sm[Cfg::O_CEA + 6 * k + r] = t;
      }
    }
    __syncwarp();
    // L_I(k, :) += (C E_alpha(:,k))^T B_I + E_alpha,d (enhancedassumedstrains.hh:401-408)
    double SdNm[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) SdNm[i] = Sm[i][0] * dNm[0] + Sm[i][1] * dNm[1] + Sm[i][2] * dNm[2];
    double ac[3] = {};  // HT: a_c . dN0
    if (KIND == 3) {
#pragma unroll
      for (int c = 0; c < 3; ++c) ac[c] = A0[0][c] * dN0[0] + A0[1][c] * dN0[1] + A0[2][c] * dN0[2];
    }
#pragma unroll 1
    for (int k0 = 0; k0 < NA; k0 += 3)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const int k = k0 + c;
        double t[3];
#pragma unroll
        for (int b = 0; b < 3; ++b) {
          double x = 0.0;
#pragma unroll
          for (int r = 0; r < 6; ++r) x += sm[Cfg::O_CEA + 6 * k + r] * B[r][b];
          t[b] = x;
        }
        if (KIND != 1) {
          const double* v = sm + Cfg::O_S + 6 * k;
          const double* coef = v + 3;
          // H: v_b (coef . S dN); HT: v_b (coef . S dNm) + (F S hv)_b with hv = s a_r (a_c . dN0)
          const double cs = coef[0] * SdNm[0] + coef[1] * SdNm[1] + coef[2] * SdNm[2];
#pragma unroll
          for (int b = 0; b < 3; ++b) t[b] += v[b] * cs;
          if (KIND == 3) {
            double hv[3], Shv[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) hv[i] = coef[i] * ac[c];
#pragma unroll
            for (int i = 0; i < 3; ++i) Shv[i] = Sm[i][0] * hv[0] + Sm[i][1] * hv[1] + Sm[i][2] * hv[2];
#pragma unroll
            for (int b = 0; b < 3; ++b) t[b] += F[b][0] * Shv[0] + F[b][1] * Shv[1] + F[b][2] * Shv[2];
          }
        }
#pragma unroll
        for (int b = 0; b < 3; ++b) share[8 * (kL + 24 * k + 3 * sub + b)] = w * t[b];
      }
    // D share: (E_alpha^T C E_alpha + E_alpha,alpha) w detJ (enhancedassumedstrains.hh:400)
#pragma unroll 1
    for (int t = sub; t < Cfg::NT; t += 8) {
      int aa, bb;
      packed_index(t, NA, aa, bb);
      double x = 0.0;
#pragma unroll
      for (int r = 0; r < 6; ++r) x += sm[Cfg::O_EA + 6 * aa + r] * sm[Cfg::O_CEA + 6 * bb + r];
      if (KIND != 1) {  // (v^a . v^b)(coef^a . S coef^b)  (displacementgradient.hh:213-230)
        const double *va = sm + Cfg::O_S + 6 * aa, *vb = sm + Cfg::O_S + 6 * bb, *fa = va + 3, *fb = vb + 3;
        double Sfb[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) Sfb[i] = Sm[i][0] * fb[0] + Sm[i][1] * fb[1] + Sm[i][2] * fb[2];
        x += (va[0] * vb[0] + va[1] * vb[1] + va[2] * vb[2]) * (fa[0] * Sfb[0] + fa[1] * Sfb[1] + fa[2] * Sfb[2]);
      }
      share[8 * (kD + t)] = w * x;
    }
    // R~ share: E_alpha^T S w detJ (enhancedassumedstrains.hh:428)
    if (WANT_R) {
#pragma unroll 1
      for (int k = sub; k < NA; k += 8) {
        double x = 0.0;
#pragma unroll
        for (int r = 0; r < 6; ++r) x += sm[Cfg::O_EA + 6 * k + r] * S[r];
        share[8 * (kR + k)] = w * x;
      }
    }
  }
  __syncthreads();

  // ---- sums over the points, in a fixed order ---------------------------------------------------------------
  const double* shares = smem + Cfg::O_SHARE;
  auto total = [&](int t) {
    const double* x = shares + 8 * t;
    return ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
  };
  double* L = smem + Cfg::O_L;
  double* D = smem + Cfg::O_D;
  double* Y = smem + Cfg::O_Y;
  int* perm = reinterpret_cast<int*>(smem + Cfg::O_PERM);
#pragma unroll 1
  for (int t = threadIdx.x; t < 24 * NA; t += 64) L[t] = total(kL + t);
#pragma unroll 1
  for (int t = threadIdx.x; t < Cfg::NT; t += 64) {
    int aa, bb;
    packed_index(t, NA, aa, bb);
    D[NA * aa + bb] = D[NA * bb + aa] = total(kD + t);
  }
  if (threadIdx.x < NA) {
    if (WANT_R) smem[Cfg::O_RT + threadIdx.x] = total(kR + threadIdx.x);
    perm[threadIdx.x] = threadIdx.x;
  }
  __syncthreads();

  // ---- static condensation ------------------------------------------------------------------------------
  if (threadIdx.x < 32) {
    // LU with partial pivoting of D in place
    double* rpiv = smem + Cfg::O_INV;
#pragma unroll 1
    for (int k = 0; k < NA; ++k) {
      // the largest magnitude, of equal ones the first row: magnitudes are ordered as their bits
      const bool cand = lane >= k && lane < NA;
      const unsigned long long m = (unsigned long long)__double_as_longlong(fabs(cand ? D[NA * lane + k] : 0.0));
      const unsigned hi = (unsigned)(m >> 32), H = __reduce_max_sync(0xffffffffu, hi);
      const unsigned lo = hi == H ? (unsigned)m : 0u, Lo = __reduce_max_sync(0xffffffffu, lo);
      const int p = __ffs(__ballot_sync(0xffffffffu, cand && hi == H && lo == Lo)) - 1;
      if ((H | Lo) == 0u || H > 0x7ff00000u || (H == 0x7ff00000u && Lo != 0u)) {  // zero or NaN
        bad |= kStatusSingularD;
        if (lane == 0) D[NA * k + k] = rpiv[k] = 1.0;
        __syncwarp();
        continue;
      }
      if (p != k) {
        if (lane < NA) {
          const double t = D[NA * k + lane];
          D[NA * k + lane] = D[NA * p + lane];
          D[NA * p + lane] = t;
        }
        if (lane == 0) {
          const int t = perm[k];
          perm[k] = perm[p];
          perm[p] = t;
        }
        __syncwarp();
      }
      const double inv = 1.0 / D[NA * k + k];
      if (lane == 0) rpiv[k] = inv;
      if (lane > k && lane < NA) D[NA * lane + k] *= inv;
      __syncwarp();
#pragma unroll 1
      for (int i = k + 1 + (lane >> 3); i < NA; i += 4) {  // eight lanes a row
        const double l = D[NA * i + k];
#pragma unroll 1
        for (int j = k + 1 + (lane & 7); j < NA; j += 8) D[NA * i + j] -= l * D[NA * k + j];
      }
      __syncwarp();
    }
    // columns of D^{-1} L (lanes 0 .. 23) and D^{-1} R~ (lane 24)
    if (lane < (WANT_R ? 25 : 24)) {
      double z[NA];
#pragma unroll
      for (int k = 0; k < NA; ++k) z[k] = lane < 24 ? L[24 * perm[k] + lane] : smem[Cfg::O_RT + perm[k]];
#pragma unroll
      for (int i = 1; i < NA; ++i)
#pragma unroll
        for (int j = 0; j < i; ++j) z[i] -= D[NA * i + j] * z[j];
#pragma unroll
      for (int i = NA - 1; i >= 0; --i) {
#pragma unroll
        for (int j = i + 1; j < NA; ++j) z[i] -= D[NA * i + j] * z[j];
        z[i] *= rpiv[i];
      }
      double* out = lane < 24 ? Y + lane * NA : smem + Cfg::O_RT + NA;
#pragma unroll
      for (int k = 0; k < NA; ++k) out[k] = z[k];
    }
  }
  if (bad && a.status) atomicOr(a.status, bad);
  __syncthreads();

  if (WANT_R) {
    const double* y = smem + Cfg::O_RT + NA;
    if (a.eas_y) {  // condensation cache for the state update
      if (threadIdx.x < NA) a.eas_y[(size_t)threadIdx.x * ne + e] = y[threadIdx.x];
      for (int t = threadIdx.x; t < 24 * NA; t += 64) a.eas_Y[(size_t)t * ne + e] = Y[(t % 24) * NA + t / 24];
    }
    if (threadIdx.x < 24) {
      const int i = threadIdx.x;
      double f = total(i), t = 0.0;
#pragma unroll
      for (int k = 0; k < NA; ++k) t += L[24 * k + i] * y[k];
      f -= t;
      if (a.trac_idx) {
        const int tr = a.trac_idx[e];
        if (tr >= 0) f -= (a.load_factor_dev ? *a.load_factor_dev : a.load_factor) * a.trac[24 * tr + i];
      }
      if (a.ext) f -= a.ext[24 * (size_t)e + i];
      a.elem_vec[24 * (size_t)li + i] = f;
    }
  } else {
    double* out = a.elem_mat + 576 * (size_t)li;
#pragma unroll 1
    for (int t = threadIdx.x; t < 360; t += 64) {
      const int d = t / 72, I = (t / 9) & 7, i = (t % 9) / 3, j = t % 3, J = (I + d) & 7;
      double x = 0.0;
#pragma unroll
      for (int k = 0; k < NA; ++k) x += L[24 * k + 3 * I + i] * Y[(3 * J + j) * NA + k];
      const double v = total(t) - x;
      out[(3 * J + j) * 24 + 3 * I + i] = v;
      if (d >= 1 && d <= 3) out[(3 * I + i) * 24 + 3 * J + j] = v;
    }
  }
}

template <int NA, int KIND, int MODE, bool HYP>
void launch_t(const ElemArgs& a, const int32_t* list, int n_list, int e_base, cudaStream_t s) {
  auto kern = eas_element_kernel<NA, KIND, MODE, HYP>;
  constexpr int shm = (int)sizeof(double) * EasCfg<NA>::total(MODE & kWantK);
  if (shm > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, shm);
  kern<<<n_list, 64, shm, s>>>(a, list, e_base);
}

// element vectors or element matrices of the listed elements, in their order
template <int NA, int KIND, bool HYP>
void launch_kind(const ElemArgs& a, int mode, const int32_t* list, int n, int base, cudaStream_t s) {
  if (mode == (kWantR | kElemOut)) launch_t<NA, KIND, kWantR | kElemOut, HYP>(a, list, n, base, s);
  else if (mode == (kWantK | kElemOut)) launch_t<NA, KIND, kWantK | kElemOut, HYP>(a, list, n, base, s);
}

// the element launches of one material family (HYP: the hyperelastic framework)
template <bool HYP>
void launch_eas_family(const ElemArgs& a, int mode, const int32_t* list, int n, int base, cudaStream_t s) {
  if (n <= 0) return;
  if (a.eas_kind == 1 && a.n_alpha == 9) launch_kind<9, 1, HYP>(a, mode, list, n, base, s);
  else if (a.eas_kind == 1 && a.n_alpha == 21) launch_kind<21, 1, HYP>(a, mode, list, n, base, s);
  else if (a.eas_kind == 2) launch_kind<9, 2, HYP>(a, mode, list, n, base, s);
  else if (a.eas_kind == 3) launch_kind<9, 3, HYP>(a, mode, list, n, base, s);
}

}  // namespace
}  // namespace ikr
