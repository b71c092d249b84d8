// Boundary -> inclusion rows (BEMBuilderElastic3D.cpp:1511-1867) from moments of the derivatives
// of R over an element, for one (particle, element) pair.
//
// Every entry of the stress kernels and their first two gradients (get_for_stress_BEM*,
// restated per entry by codegen.gen_bem_stress_function) is a combination of derivatives of R = |y - P|: with
// G_ij = A d_ij / R - B R_,ij, p = 1/R (p_,a = 1/2 R_,aii) and R biharmonic,
//   Dst[kl][n] =  dlam d_kl (A - 2B) p_,nW + dmu [A (d_nk p_,lW + d_nl p_,kW) - 2B R_,nklW]
//   Dsu[kl][n] =  n_m { dlam d_kl 2 mu0 (A - 2B) p_,mnW + dmu [2 lam0 (A - 2B) d_mn p_,klW
//                 + mu0 (A (d_mk p_,nlW + d_ml p_,nkW + d_nk p_,mlW + d_nl p_,mkW) - 4B R_,mnklW)] }
// up to the signs (+-1)^|W| of differentiating at P.  So instead of forming the 6 x 3 kernels
// for every derivative tuple W at every Gauss point, the Gauss sums are taken of the derivatives
// themselves, times the shape functions and (for Dsu) times the normal's components: moments
//   M[a][c][j] = sum over Gauss points of R_,a N_j w J {1, n_0, n_1, n_2}[c],
// and the entries are combined from the moments once per pair.  Derivatives of equal index
// counts are one number: 10, 15, 21, 28 of order 3 to 6.
#pragma once
#include "gen_sphere_common.cuh"

namespace ibem {

// position of the derivative with index counts (c0, c1, c2), order n = c0 + c1 + c2, among all
// of orders 3 .. n
IBEM_HD IBEM_INLINE constexpr int bmo_base(int n) { return n == 3 ? 0 : n == 4 ? 10 : n == 5 ? 25 : 46; }
IBEM_HD IBEM_INLINE constexpr int bmo_idx(int n, int c0, int c2) { return bmo_base(n) + (n - c0) * (n - c0 + 1) / 2 + c2; }

// number of ways to pair 2 j of c equal indices: c! / (2^j j! (c - 2j)!)
IBEM_HD IBEM_INLINE constexpr double bmo_pairs(int c, int j) {
  double v = 1.0;
  for (int i = 0; i < 2 * j; ++i) v *= c - i;
  for (int i = 1; i <= j; ++i) v /= 2.0 * i;
  return v;
}

// All derivatives of R of orders 3 .. TOP at offset x: put(index, value).  R = sqrt(2u), u =
// |x|^2 / 2: with F[k] = d^k R / du^k, R_,a = sum over (j0, j1, j2) of the pairings of each axis
// times the remaining powers of x times F[n - j0 - j1 - j2].
// The index counts are template parameters: the pairing factors are then literals and F and the
// powers stay in registers.
template <int N, int C0, int C2, int J0, int J1, int J2, int TOP>
IBEM_HD IBEM_INLINE double bmo_term(const double (&px)[3][TOP + 1], const double (&F)[TOP + 1]) {
  constexpr double f = bmo_pairs(C2, J2);
  double v = px[2][C2 - 2 * J2] * F[N - J0 - J1 - J2];
  if constexpr (f != 1.0) v *= f;
  if constexpr (J2 < C2 / 2) v += bmo_term<N, C0, C2, J0, J1, J2 + 1, TOP>(px, F);
  return v;
}
template <int N, int C0, int C2, int J0, int J1, int TOP>
IBEM_HD IBEM_INLINE double bmo_sum(const double (&px)[3][TOP + 1], const double (&F)[TOP + 1]) {
  constexpr int C1 = N - C0 - C2;
  constexpr double f = bmo_pairs(C0, J0) * bmo_pairs(C1, J1);
  double v = px[0][C0 - 2 * J0] * px[1][C1 - 2 * J1];
  if constexpr (f != 1.0) v *= f;
  v *= bmo_term<N, C0, C2, J0, J1, 0, TOP>(px, F);
  if constexpr (J1 < C1 / 2) v += bmo_sum<N, C0, C2, J0, J1 + 1, TOP>(px, F);
  else if constexpr (J0 < C0 / 2) v += bmo_sum<N, C0, C2, J0 + 1, 0, TOP>(px, F);
  return v;
}
template <int N, int C0, int C2, int TOP, class Put>
IBEM_HD IBEM_INLINE void bmo_walk(const double (&px)[3][TOP + 1], const double (&F)[TOP + 1], Put& put) {
  put(bmo_idx(N, C0, C2), bmo_sum<N, C0, C2, 0, 0, TOP>(px, F));
  if constexpr (C2 < N - C0) bmo_walk<N, C0, C2 + 1, TOP>(px, F, put);
  else if constexpr (C0 > 0) bmo_walk<N, C0 - 1, 0, TOP>(px, F, put);
  else if constexpr (N < TOP) bmo_walk<N + 1, N + 1, 0, TOP>(px, F, put);
}
template <int TOP, class Put>
IBEM_HD IBEM_INLINE void bmo_derivatives(double x0, double x1, double x2, double ir, Put&& put) {
  double F[TOP + 1], px[3][TOP + 1];
  F[0] = 0.0;
  F[1] = ir;
#pragma unroll
  for (int k = 2; k <= TOP; ++k) F[k] = F[k - 1] * (ir * ir) * (double)(3 - 2 * k);
  const double x[3] = {x0, x1, x2};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    px[d][0] = 1.0;
#pragma unroll
    for (int k = 1; k <= TOP; ++k) px[d][k] = px[d][k - 1] * x[d];
  }
  bmo_walk<3, 3, 0, TOP>(px, F, put);
}

// Moments of one pair and one shape function: mom(c, index) reads M[index][c].  Index tuples
// are given by their sums of unit counts: an index i adds cnt(i) to a packed count.
IBEM_HD IBEM_INLINE constexpr int bmo_e(int i) { return i == 0 ? 1 : i == 1 ? 16 : 256; }
template <class Mom>
struct BmoEntries {
  Mom mom;
  double A, B, lam0, mu0, dlam, dmu;

  IBEM_HD IBEM_INLINE double R(int c, int n, int cnt) const { return mom(c, bmo_idx(n, cnt & 15, cnt >> 8)); }
  IBEM_HD IBEM_INLINE double p(int c, int n, int cnt) const {   // derivative of order n of 1/R
    return 0.5 * (R(c, n + 2, cnt + 2 * bmo_e(0)) + R(c, n + 2, cnt + 2 * bmo_e(1)) + R(c, n + 2, cnt + 2 * bmo_e(2)));
  }
  IBEM_HD IBEM_INLINE double S(int n, int cnt) const {          // sum_m n_m p_,m..
    return p(1, n + 1, cnt + bmo_e(0)) + p(2, n + 1, cnt + bmo_e(1)) + p(3, n + 1, cnt + bmo_e(2));
  }
  // traction and displacement entries of row (k, l), |W| = o with packed counts w, column dof n
  IBEM_HD IBEM_INLINE void entry(int k, int l, int o, int w, int n, double& st, double& su) const {
    const double q = A - 2.0 * B, sign = (o & 1) ? -1.0 : 1.0;
    const int ek = bmo_e(k), el = bmo_e(l), en = bmo_e(n);
    double t = dmu * (-2.0 * B) * R(0, 3 + o, en + ek + el + w);
    double u = p(n + 1, 2 + o, ek + el + w) * (2.0 * lam0 * q);
    double v = A * (p(k + 1, 2 + o, en + el + w) + p(l + 1, 2 + o, en + ek + w));
    const int a = en + ek + el + w;
    v -= 4.0 * B * (R(1, 4 + o, a + bmo_e(0)) + R(2, 4 + o, a + bmo_e(1)) + R(3, 4 + o, a + bmo_e(2)));
    if (n == k) {
      t += dmu * A * p(0, 1 + o, el + w);
      v += A * S(1 + o, el + w);
    }
    if (n == l) {
      t += dmu * A * p(0, 1 + o, ek + w);
      v += A * S(1 + o, ek + w);
    }
    u = dmu * (u + mu0 * v);
    if (k == l) {
      t += dlam * q * p(0, 1 + o, en + w);
      u += dlam * 2.0 * mu0 * q * S(1 + o, en + w);
    }
    st = -sign * t;
    su = sign * u;
  }
};

}  // namespace ibem
