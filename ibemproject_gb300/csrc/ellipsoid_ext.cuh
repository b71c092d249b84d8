// Pair block of an ellipsoidal source by a shorter route than ellipsoid.cuh's (included by it).
//
// In the principal frame every potential reduces to the integrals I_k after one or two
// derivatives, because U vanishes at lambda:
//   F1_k = int U prod t^k ds/Delta,     d_j F1_k = -2 y_j I_{k + e_j}
//   F2_k = int U^2 prod t^k ds/Delta,   d_j F2_k = -4 y_j F1_{k + e_j}
//   phi_1 = C F1_0,  phi_m = C a_m^2 y_m F1_m,
//   phi_mn = C [a_m^2 a_n^2 y_m y_n F1_mn + d_mn a_m^2 / 4 (F2_0 - a_m^2 F2_m)]
// so that the block's derivatives (of order 2 and more) need Taylor series of the I_k to third
// order only, and those are univariate in lambda: lambda(y + h) is solved for order by order
// from sum (y_m + h_m)^2 / (a_m^2 + lambda) = 1, whose coefficients are quadratics with three
// terms per axis in this frame.  The 20 values I_k come from Gauss-Legendre quadrature: with
// X the largest of x_m = a_m^2 + lambda, s = X (1/u^2 - 1) and kappa_m = 1 - x_m / X,
//   I_k = 2 X^(-1/2 - |k|) int_0^1 u^(2|k|) prod (1 - kappa_m u^2)^(-1/2 - k_m) du,
// an even analytic integrand, whose n-node error falls as rho^(-4n), rho = kappa^(-1/2) +
// (1/kappa - 1)^(1/2): 8 nodes give 1e-17 up to kappa = 0.2, which holds for every pair but
// close neighbours of flat sources; up to kappa = 0.96 more nodes, beyond that ellipsoid.cuh's
// general path.  Inside the source lambda stays 0 and the I_k are constants.  The tables of derivatives are rotated to the global
// frame by the matrices of the rotation on symmetric tensors of order 2 to 5, formed once per
// source.
//
// About 11,000 operations per block (quadrature 450, series 3,500, rotation 3,700, entries
// 2,500) where the general path takes 58,000.  Six realisations of 50 to 300 ellipsoids: 43 ->
// 11 ms for their blocks; its rounding is smaller too (in FP32, mean error of a block 1.1e-6 of
// its largest entry at contact, general path 8e-6).
#pragma once

#include "ell_gauss.cuh"

namespace ibem {
namespace ell {

// unique components of a symmetric tensor of order n: index of the counts (c0, c1, c2)
IBEM_HD constexpr int sidx(int n, int c0, int c2) { return (n - c0) * (n - c0 + 1) / 2 + c2; }
IBEM_HD constexpr int ssize(int n) { return (n + 1) * (n + 2) / 2; }

// Matrices of the rotation principal -> global on the unique components of symmetric tensors of
// order 2 to 5 (row-major), one after the other: T'_beta = sum_alpha M[beta][alpha] T_alpha.
IBEM_HD constexpr int rot_off(int n) { return n <= 2 ? 0 : n == 3 ? 36 : n == 4 ? 136 : 361; }
constexpr int kRotSize = 36 + 100 + 225 + 441;

// row (b0, b2) of order n from the rows of order n - 1: prev for n = 2 is the rotation itself
template <typename T>
IBEM_HD inline void rot_row(const T* Q, int n, int row, const T* prev, T* out) {
  int b0 = n, b2 = row;   // unpack the row's counts
  while (b2 > n - b0) {
    b2 -= n - b0 + 1;
    --b0;
  }
  const int b1 = n - b0 - b2;
  const int i = b0 > 0 ? 0 : (b1 > 0 ? 1 : 2);
  const int r0 = b0 - (i == 0), r2 = b2 - (i == 2);
  const T* pr = n == 2 ? nullptr : prev + sidx(n - 1, r0, r2) * ssize(n - 1);
  const int j1 = n == 2 ? (r0 ? 0 : (r2 ? 2 : 1)) : 0;   // the one index left at n = 2
  for (int a0 = 0; a0 <= n; ++a0)
    for (int a2 = 0; a2 <= n - a0; ++a2) {
      const int a1 = n - a0 - a2;
      T v = T(0);
      for (int j = 0; j < 3; ++j) {
        const int c0 = a0 - (j == 0), c1 = a1 - (j == 1), c2 = a2 - (j == 2);
        if (c0 < 0 || c1 < 0 || c2 < 0) continue;
        v += Q[3 * i + j] * (n == 2 ? Q[3 * j1 + (c0 ? 0 : (c2 ? 2 : 1))] : pr[sidx(n - 1, c0, c2)]);
      }
      out[sidx(n, a0, a2)] = v;
    }
}

// coefficients of I_k(lambda0 + delta) up to delta^3
template <typename T>
struct EllSeries {
  T c[20][4];
};

// the I_k by quadrature (kappa <= 0.96) and their lambda-derivatives at x_m = a_m^2 + lambda0
template <typename T>
IBEM_HD inline void ell_series(const T x[3], T kmax, EllSeries<T>& S) {
  const T X = vfmax(x[0], vfmax(x[1], x[2])), iX = T(1) / X;
  T kap[3], ik[20];
#pragma unroll
  for (int m = 0; m < 3; ++m) kap[m] = T(1) - x[m] * iX;
#pragma unroll
  for (int i = 0; i < 20; ++i) ik[i] = T(0);
  const int n = kmax <= T(0.2) ? 8 : (kmax <= T(0.55) ? 16 : (kmax <= T(0.85) ? 32 : 64));
  const int o = n - 8;   // 8, 16, 32 and 64 nodes start at 0, 8, 24 and 56
#pragma unroll 1
  for (int q = 0; q < n; ++q) {
    const T u2 = T(kGauss[o + q][0]);
    T d[3], g[3];
#pragma unroll
    for (int m = 0; m < 3; ++m) d[m] = T(1) - kap[m] * u2;
    const T d01 = d[0] * d[1], rs = vrsqrt(d01 * d[2]), r2 = rs * rs * u2;
    g[0] = r2 * (d[1] * d[2]);
    g[1] = r2 * (d[0] * d[2]);
    g[2] = r2 * d01;
    T p0 = T(kGauss[o + q][1]) * rs;
#pragma unroll
    for (int k1 = 0; k1 <= 3; ++k1) {
      T p1 = p0;
#pragma unroll
      for (int k2 = 0; k2 <= 3 - k1; ++k2) {
        T p2 = p1;
#pragma unroll
        for (int k3 = 0; k3 <= 3 - k1 - k2; ++k3) {
          ik[midx(k1, k2, k3)] += p2;
          if (k3 < 3 - k1 - k2) p2 *= g[2];
        }
        if (k2 < 3 - k1) p1 *= g[1];
      }
      if (k1 < 3) p0 *= g[0];
    }
  }
  T ix[3];
#pragma unroll
  for (int m = 0; m < 3; ++m) ix[m] = T(1) / x[m];
  const T rf = vrsqrt(x[0] * x[1] * x[2]), sc = T(2) * vrsqrt(X);
  const T scale[4] = {sc, sc * iX, sc * iX * iX, sc * iX * iX * iX};
  T f0 = rf;
#pragma unroll
  for (int k1 = 0; k1 <= 3; ++k1) {
    T f1 = f0;
#pragma unroll
    for (int k2 = 0; k2 <= 3 - k1; ++k2) {
      T f2 = f1;
#pragma unroll
      for (int k3 = 0; k3 <= 3 - k1 - k2; ++k3) {
        const T q0 = T(k1) + T(0.5), q1 = T(k2) + T(0.5), q2 = T(k3) + T(0.5);
        const T s1 = q0 * ix[0] + q1 * ix[1] + q2 * ix[2];
        const T s2 = q0 * ix[0] * ix[0] + q1 * ix[1] * ix[1] + q2 * ix[2] * ix[2];
        T* c = S.c[midx(k1, k2, k3)];
        c[0] = scale[k1 + k2 + k3] * ik[midx(k1, k2, k3)];
        c[1] = -f2;
        c[2] = T(0.5) * f2 * s1;
        c[3] = -f2 * (s1 * s1 + s2) / T(6);
        f2 *= ix[2];
      }
      f1 *= ix[1];
    }
    f0 *= ix[0];
  }
}

// powers of delta(h) = lambda(y + h) - lambda0 up to third order: d1 (degrees 1-3), d2 (2-3), d3 (3)
template <typename T>
struct EllDelta {
  T d1[20], d2[20], d3[20];
};
template <typename T>
IBEM_HD inline void ell_delta(const T y[3], const T x[3], EllDelta<T>& D) {
  T A1[3], A2[3], B1[3], B2[3], C1[3];
  T b0 = T(0), C0 = T(0), D0 = T(0);
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    const T t = T(1) / x[m], t2 = t * t, yy = y[m] * y[m];
    A1[m] = T(2) * y[m] * t;
    A2[m] = t;
    b0 += yy * t2;
    B1[m] = T(2) * y[m] * t2;
    B2[m] = t2;
    C0 += yy * t2 * t;
    C1[m] = T(2) * y[m] * t2 * t;
    D0 += yy * t2 * t2;
  }
  const T ib = T(1) / b0;
#pragma unroll
  for (int i = 0; i < 20; ++i) D.d1[i] = D.d2[i] = D.d3[i] = T(0);
#define IBEM_M1(i) midx((i) == 0, (i) == 1, (i) == 2)
#define IBEM_M2(i, j) midx(((i) == 0) + ((j) == 0), ((i) == 1) + ((j) == 1), ((i) == 2) + ((j) == 2))
#define IBEM_M3(i, j, k)                                                                             \
  midx(((i) == 0) + ((j) == 0) + ((k) == 0), ((i) == 1) + ((j) == 1) + ((k) == 1), ((i) == 2) + ((j) == 2) + ((k) == 2))
  T l[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    l[i] = A1[i] * ib;
    D.d1[IBEM_M1(i)] = l[i];
  }
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      D.d2[IBEM_M2(i, j)] += l[i] * l[j];
      D.d1[IBEM_M2(i, j)] += ib * (C0 * l[i] * l[j] - B1[i] * l[j]);
    }
#pragma unroll
  for (int i = 0; i < 3; ++i) D.d1[IBEM_M2(i, i)] += ib * A2[i];
  // third order: b0 d = -B1 d_2 - B2 d_1 + 2 C0 d_1 d_2 + C1 d_1^2 - D0 d_1^3
#pragma unroll
  for (int k = 0; k < 3; ++k)
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = i; j < 3; ++j) {
        const T q = D.d1[IBEM_M2(i, j)], ll = D.d2[IBEM_M2(i, j)];
        D.d2[IBEM_M3(i, j, k)] += T(2) * l[k] * q;
        D.d3[IBEM_M3(i, j, k)] += l[k] * ll;
        D.d1[IBEM_M3(i, j, k)] += ib * ((T(2) * C0 * l[k] - B1[k]) * q + (C1[k] - D0 * l[k]) * ll);
      }
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) D.d1[IBEM_M3(i, i, j)] -= ib * B2[i] * l[j];
#undef IBEM_M1
#undef IBEM_M2
#undef IBEM_M3
}

// coefficient i (of degree deg) of the series of I_k
template <typename T>
IBEM_HD IBEM_INLINE T ell_icoef(const T* c, const EllDelta<T>& D, int i, int deg) {
  if (deg == 0) return c[0];
  T v = c[1] * D.d1[i];
  if (deg >= 2) v += c[2] * D.d2[i];
  if (deg >= 3) v += c[3] * D.d3[i];
  return v;
}

// F1_k up to fourth order (the value itself is not formed): every coefficient from the
// derivative along its first axis
template <typename T>
IBEM_HD inline void ell_f1(const T y[3], const EllSeries<T>& S, const EllDelta<T>& D, int k1, int k2, int k3, T* F) {
  F[0] = T(0);
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    const T* c = S.c[midx(k1 + (j == 0), k2 + (j == 1), k3 + (j == 2))];
    T I[20];
#pragma unroll
    for (int d = 0; d <= 3; ++d)
#pragma unroll
      for (int a = 0; a <= (j == 0 ? d : 0); ++a)
#pragma unroll
        for (int b = 0; b <= (j == 2 ? 0 : d - a); ++b) I[midx(a, b, d - a - b)] = ell_icoef(c, D, midx(a, b, d - a - b), d);
#pragma unroll
    for (int d = 1; d <= 4; ++d)
#pragma unroll
      for (int a = (j == 0 ? 1 : 0); a <= (j == 0 ? d : 0); ++a)
#pragma unroll
        for (int b = (j == 1 ? 1 : 0); b <= (j == 2 ? 0 : d - a); ++b) {
          const int cc = d - a - b, n = j == 0 ? a : (j == 1 ? b : cc);
          T v = y[j] * I[midx(a - (j == 0), b - (j == 1), cc - (j == 2))];
          if (n >= 2) v += I[midx(a - 2 * (j == 0), b - 2 * (j == 1), cc - 2 * (j == 2))];
          F[midx(a, b, cc)] = v * T(-2.0 / n);
        }
  }
}

// o[deg d0 .. 4] = (y + h_m) F for a series F of which the degrees d0 - 1 .. 4 are set
template <typename T>
IBEM_HD inline void ell_times(T y, int m, const T* F, int d0, T scale, T* o) {
#pragma unroll 1
  for (int d = d0; d <= 4; ++d)
#pragma unroll 1
    for (int a = 0; a <= d; ++a)
#pragma unroll 1
      for (int b = 0; b <= d - a; ++b) {
        const int c = d - a - b, n = m == 0 ? a : (m == 1 ? b : c);
        T v = y * F[midx(a, b, c)];
        if (n > 0) v += F[midx(a - (m == 0), b - (m == 1), c - (m == 2))];
        o[midx(a, b, c)] = scale * v;
      }
}

// Derivatives of the potentials at the target, densities 1 and y'_p, as symmetric tensors:
// phi of orders 2 and 3, psi of orders 4 and 5.
template <typename T>
struct EllTables {
  T p2[4][6], p3[4][10], s4[4][15], s5[4][21];
};

template <typename T>
IBEM_HD inline T ell_factorials(int a, int b, int c) {
  const T f[5] = {T(1), T(1), T(2), T(6), T(24)};
  return f[a] * f[b] * f[c];
}

// in the principal frame, offset y, semi-axes a
template <typename T>
IBEM_HD inline void ell_ext_tables(const T y[3], const T a[3], T lam, bool inside, T kmax, EllTables<T>& W) {
  T x[3], a2[3];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    a2[m] = a[m] * a[m];
    x[m] = a2[m] + lam;
  }
  const T C = T(IBEM_PI) * a[0] * a[1] * a[2];
  // Taylor coefficients (degrees 2 to 4) of phi_1, phi_m, and (3 and 4) of phi_mn
  T f[4][35], g[6][35];
  {
    EllSeries<T> S;
    EllDelta<T> D;
    ell_series(x, kmax, S);
    if (inside) {   // lambda stays 0: the I_k are constants
#pragma unroll 1
      for (int i = 0; i < 20; ++i) D.d1[i] = D.d2[i] = D.d3[i] = T(0);
    } else {
      ell_delta(y, x, D);
    }
    T F1[3][35], F[35];
    ell_f1(y, S, D, 0, 0, 0, F);
#pragma unroll 1
    for (int i = 4; i < 35; ++i) f[0][i] = C * F[i];
#pragma unroll 1
    for (int m = 0; m < 3; ++m) {
      ell_f1(y, S, D, m == 0, m == 1, m == 2, F1[m]);
      ell_times(y[m], m, F1[m], 2, C * a2[m], f[1 + m]);
    }
    // F2_0, then F2_m, in the degrees 3 and 4: coefficient from the derivative along the first axis
    const T q4[5] = {T(0), T(-4), T(-2), T(-4.0 / 3.0), T(-1)};
    auto f2 = [&](const T* G0, const T* G1, const T* G2, int a_, int b_, int c_) {
      const int j = a_ > 0 ? 0 : (b_ > 0 ? 1 : 2), n = j == 0 ? a_ : (j == 1 ? b_ : c_);
      const T* G = j == 0 ? G0 : (j == 1 ? G1 : G2);
      T v = y[j] * G[midx(a_ - (j == 0), b_ - (j == 1), c_ - (j == 2))];
      if (n >= 2) v += G[midx(a_ - 2 * (j == 0), b_ - 2 * (j == 1), c_ - 2 * (j == 2))];
      return v * q4[n];
    };
    T FF[6][35];
#pragma unroll 1
    for (int m = 0; m < 3; ++m)
#pragma unroll 1
      for (int n = m; n < 3; ++n) {
        T* G = FF[sym_pair(m, n)];
        ell_f1(y, S, D, (m == 0) + (n == 0), (m == 1) + (n == 1), (m == 2) + (n == 2), G);
        T t[35];
        ell_times(y[m], m, G, 2, T(1), t);
        ell_times(y[n], n, t, 3, C * a2[m] * a2[n], g[sym_pair(m, n)]);
      }
#pragma unroll 1
    for (int d = 3; d <= 4; ++d)
#pragma unroll 1
      for (int p = 0; p <= d; ++p)
#pragma unroll 1
        for (int q = 0; q <= d - p; ++q) {
          const int r = d - p - q, id = midx(p, q, r);
          const T v0 = f2(F1[0], F1[1], F1[2], p, q, r);
#pragma unroll
          for (int m = 0; m < 3; ++m) {
            const T vm = f2(FF[sym_pair(m, 0)], FF[sym_pair(m, 1)], FF[sym_pair(m, 2)], p, q, r);
            g[sym_pair(m, m)][id] += C * a2[m] * T(0.25) * (v0 - a2[m] * vm);
          }
        }
  }
#pragma unroll 1
  for (int r = 0; r < 4; ++r) {
#pragma unroll 1
    for (int d = 2; d <= 3; ++d)
#pragma unroll 1
      for (int p = 0; p <= d; ++p)
#pragma unroll 1
        for (int q = 0; q <= d - p; ++q) {
          const int s = d - p - q;
          const T v = ell_factorials<T>(p, q, s) * f[r][midx(p, q, s)];
          if (d == 2) W.p2[r][sidx(2, p, s)] = v;
          else W.p3[r][sidx(3, p, s)] = v;
        }
    // psi_r of order d + 1 from x_k phi_r - phi_rk, k the first axis of the index
#pragma unroll 1
    for (int d = 4; d <= 5; ++d)
#pragma unroll 1
      for (int p = 0; p <= d; ++p)
#pragma unroll 1
        for (int q = 0; q <= d - p; ++q) {
          const int s = d - p - q, k = p > 0 ? 0 : (q > 0 ? 1 : 2);
          const int u = p - (k == 0), v = q - (k == 1), w = s - (k == 2), id = midx(u, v, w);
          const T* gk = r == 0 ? f[1 + k] : g[sym_pair(r - 1, k)];
          T val = y[k] * f[r][id] - gk[id];
          if ((k == 0 ? u : (k == 1 ? v : w)) > 0) val += f[r][midx(u - (k == 0), v - (k == 1), w - (k == 2))];
          val *= ell_factorials<T>(u, v, w);
          if (d == 4) W.s4[r][sidx(4, p, s)] = val;
          else W.s5[r][sidx(5, p, s)] = val;
        }
  }
}

// rotate one family of tensors (order N, four densities) to the global frame in place
template <typename T, int N>
IBEM_HD inline void ell_rotate(const T* Q, const T* M, T (&t)[4][(N + 1) * (N + 2) / 2]) {
  constexpr int n = (N + 1) * (N + 2) / 2;
#pragma unroll 1
  for (int half = 0; half < 2; ++half) {   // two densities at a time: their components stay in registers
    T v0[n], v1[n];
#pragma unroll
    for (int i = 0; i < n; ++i) {
      v0[i] = half == 0 ? t[0][i] : t[2][i];
      v1[i] = half == 0 ? t[1][i] : t[3][i];
    }
#pragma unroll 1
    for (int b = 0; b < n; ++b) {
      T s0 = T(0), s1 = T(0);
#pragma unroll
      for (int i = 0; i < n; ++i) {
        s0 += M[b * n + i] * v0[i];
        s1 += M[b * n + i] * v1[i];
      }
      t[2 * half][b] = s0;
      t[2 * half + 1][b] = s1;
    }
  }
#pragma unroll 1
  for (int i = 0; i < n; ++i) {   // the densities y'_m to x'_p
    const T a = t[1][i], b = t[2][i], c = t[3][i];
#pragma unroll
    for (int p = 0; p < 3; ++p) t[1 + p][i] = Q[3 * p] * a + Q[3 * p + 1] * b + Q[3 * p + 2] * c;
  }
}

// Entries of the block from the global tables (the layout and factors of ell_block24): sc the
// source's longest semi-axis, by which the tables' coordinates were scaled.
template <typename T>
IBEM_HD inline void ell_ext_entries(const EllTables<T>& W, const SphMat& mc, T sc, T* out) {
  const T nu = T(mc.tn2) / T(2), kd = T(mc.kd), n1 = T(1) - nu;
#pragma unroll 1
  for (int r = 0; r < 4; ++r) {   // collocation derivative: none, or r - 1
    const int e0 = r == 1, e2 = r == 3, o = r > 0;
#pragma unroll 1
    for (int rho = 0; rho < 4; ++rho) {
      const T* ph = o ? W.p3[rho] : W.p2[rho];
      const T* ps = o ? W.s5[rho] : W.s4[rho];
      T p[6], D[6][6];
#pragma unroll
      for (int t = 0; t < 6; ++t) {
        const int i = pair_i(t), j = pair_j(t);
        p[t] = ph[sidx(2 + o, (i == 0) + (j == 0) + e0, (i == 2) + (j == 2) + e2)];
      }
#pragma unroll
      for (int t = 0; t < 6; ++t)
#pragma unroll
        for (int u = t; u < 6; ++u) {
          const int i = pair_i(t), j = pair_j(t), k = pair_i(u), l = pair_j(u);
          T s4 = T(0);
          if (i == l) s4 += p[sym_pair(k, j)];
          if (j == l) s4 += p[sym_pair(k, i)];
          if (i == k) s4 += p[sym_pair(l, j)];
          if (j == k) s4 += p[sym_pair(l, i)];
          // the part that is symmetric in the two pairs
          const T v = ps[sidx(4 + o, (i == 0) + (j == 0) + (k == 0) + (l == 0) + e0, (i == 2) + (j == 2) + (k == 2) + (l == 2) + e2)] -
                      n1 * s4;
          D[t][u] = D[u][t] = v;
        }
      const T f = -kd * ((rho > 0) == (r > 0) ? T(1) : (rho > 0 ? sc : T(1) / sc));
      const T f2 = f * T(2) * T(mc.dmu), fl = f * T(mc.dlam);
      T q[6];
#pragma unroll
      for (int t = 0; t < 6; ++t) q[t] = T(2) * nu * p[t];
      const T qtr = q[0] + q[3] + q[5];
#pragma unroll
      for (int u = 0; u < 6; ++u) {
        const bool du = u == 0 || u == 3 || u == 5;
        const T map = du ? T(1) : T(2);
        T tr = D[0][u] + D[3][u] + D[5][u];
        if (du) tr -= qtr;
        const T trf = fl * tr * map;
        const int col = rho == 0 ? u : 6 + 3 * u + rho - 1;
#pragma unroll
        for (int t = 0; t < 6; ++t) {
          const bool dt = t == 0 || t == 3 || t == 5;
          const T v = f2 * map * (du ? D[t][u] - q[t] : D[t][u]);
          const int row = r == 0 ? t : 6 + 3 * t + r - 1;
          out[row * 24 + col] = dt ? v + trf : v;
        }
      }
    }
  }
}

// Block without the self term; M: the source's rotation matrices (kRotSize).  Returns false (out
// untouched) where the general path has to be taken: a source so flat and close (or entered) that
// the quadrature does not resolve it.
template <typename T>
IBEM_HD inline bool ell_block24_ext(const T d[3], const T Q[9], const T a[3], const T* M, const SphMat& mc, T* out) {
  const T sc = vfmax(a[0], vfmax(a[1], a[2])), isc = T(1) / sc;
  T y[3], as[3], a2[3];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    y[m] = (Q[m] * d[0] + Q[3 + m] * d[1] + Q[6 + m] * d[2]) * isc;
    as[m] = a[m] * isc;
    a2[m] = as[m] * as[m];
  }
  const T qin = y[0] * y[0] / a2[0] + y[1] * y[1] / a2[1] + y[2] * y[2] / a2[2];
  const bool inside = qin <= T(1);
  const T lam = inside ? T(0) : ell_lambda(y, a2);
  const T kmax = (T(1) - vfmin3(a2)) / (T(1) + lam);   // the longest scaled semi-axis is 1
  if (!(kmax <= T(0.96))) return false;
  EllTables<T> W;
  ell_ext_tables(y, as, lam, inside, kmax, W);
  ell_rotate<T, 2>(Q, M + rot_off(2), W.p2);
  ell_rotate<T, 3>(Q, M + rot_off(3), W.p3);
  ell_rotate<T, 4>(Q, M + rot_off(4), W.s4);
  ell_rotate<T, 5>(Q, M + rot_off(5), W.s5);
  ell_ext_entries(W, mc, sc, out);
  return true;
}

// the self term of the own block: C0 on the unknowns of equal order and moment
template <typename T>
IBEM_HD inline void ell_self_add(const SphMat& mc, T* out) {
#pragma unroll 1
  for (int t = 0; t < 6; ++t)
#pragma unroll 1
    for (int u = 0; u < 6; ++u) {
      const int i = pair_i(t), j = pair_j(t), m = pair_i(u), n = pair_j(u);
      T c0 = T(mc.mu0) * (T((i == m) * (j == n)) + T((i == n) * (j == m)));
      if (i == j && m == n) c0 += T(mc.lam0);
      c0 *= m == n ? T(1) : T(2);
      out[24 * t + u] += c0;
      for (int p = 0; p < 3; ++p) out[24 * (6 + 3 * t + p) + 6 + 3 * u + p] += c0;
    }
}

}  // namespace ell
}  // namespace ibem
