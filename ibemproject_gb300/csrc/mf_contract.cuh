// Product of one 24 x 24 sphere pair block with a coefficient vector, without forming the
// block (the matrix-free solver's inner loop).
//
// Rows of order 0 of the pair block (integratorElastic3D.cpp:341-454) are, for every source
// column, map[m][n] (kmu D_ij + klam d_ij Tr D) with D the Eshelby-type tensor without its
// 1 / (8 pi (1 - nu)) factor (integratorElastic3DHelper.cpp:2394-2442); rows of order 1
// (:455-567) are the same with one more derivative in the target position x_r (D_41, D_51).
// Summed against the source's coefficients x_h, the order-0 rows are therefore
//   y_ij = kmu r_ij + klam d_ij (r_00 + r_11 + r_22),   r = e / c,
// with e the strain that the source's eigenstrain x_h produces at the target centre (the
// post-processor's sum, postProcessorElastic3D.cpp:407-470, contracted with the eigenstrain
// before any tensor is formed: field_contract.cuh), and the order-1 rows are the same
// combination of the gradient g_ijk = d r_ij / d x_k.
//
// In units of the source's radius (a = 1), with E the order-0 and F the order-1 coefficients as
// tensors symmetric in their first two indices, V_n and J_m the sphere's radial potentials,
// Ps = V_0 - V_1 and Q = V_1 - V_2 and a number the rung of their ladder of derivatives in
// u = |x|^2 / 2 (V_n^(k) = -J_{n+1}^(k-1), J_m' = -(2m+3) J_{m+1} outside, 0 inside), t = 1 - nu0:
//   L, S, w, v: sums of F, formed once per source (contract_num.cuh)
//   Ep_ij = F_ijl x_l,  N_ik = L_ikl x_l,  n = N x,  k = N x / 2 + N' x
//   Z  = 2 t (Ph2 E x + V1_2 n / 2 + V1_1 v),            Zu the same one rung up
//   dB = 2 Ps3 E x + Q3 k + 2 Q2 v + b2 w,  W = dB - Z   (b_k = Q_k - 2 nu V1_{k-1})
//   dA = 2 Ps4 E x + Q4 k + 2 Q3 v + b3 w,  Wu = dA - Zu
//   A, Au, B: scalars of x.E.x, tr E, x.n, w.x and v.x
//   r_ij  = p_i x_j + p_j x_i + C0 E_ij - 2 Q2 Ep_ij + C2 (N_ij + N_ji) + d_ij B,   p = A x / 2 + W
//   R_ij  = C0u E_ij - 2 Q3 Ep_ij + C2u (N_ij + N_ji) + d_ij A
//   Y_ik  = cE E_ik - 2 Q3 Ep_ik + 2 Q3 N_ki + C2u N_ik + dA_k x_i / 2 + (Au x_i / 2 + Wu_i) x_k + d_ik A
//   g_ijk = R_ij x_k + Y_ik x_j + Y_jk x_i + C1 F_ijk + C2 S_ijk + d_ij dB_k + d_ik W_j + d_jk W_i
// About 430 multiply-adds per pair (1,140 additions and multiplications, most of them not
// fusable, when r and the tensors of g were expanded term by term from E and F; ~6,000 for the
// generated block and its 576 multiply-adds).  The products that use it are bound by the
// arithmetic pipe of their type (FP64, double-float and FP32), so their time is this count.
#pragma once
#include "contract_num.cuh"

namespace ibem {

// y += a b, rounded as an addition to y (for double-float numbers the sum is normalised)
template <class R>
IBEM_HD IBEM_INLINE void mf_acc(R& y, R a, R b) {
  Sum<R> s(y);
  s.add(a, b);
  y = s.val();
}

// The raw contraction for the target at offset x in units of the source's radius: r_t is added to
// y[t], row_scale * g_tk to y[6 + 3 t + k] (t over the pairs above).  The caller applies the
// kmu / klam map once after the sum over sources (sph_pair_map24: the map is linear and the
// same for every source of a target).  f = 2 (1 - nu0), rec the source's record (16-byte
// aligned on the device).
template <class R>
IBEM_HD IBEM_INLINE void sph_pair_raw24(R x0, R x1, R x2, R f, const R* __restrict__ rec, R row_scale, R (&y)[24]) {
  constexpr int pi[6] = {0, 0, 0, 1, 1, 2}, pj[6] = {0, 1, 2, 1, 2, 2};
  constexpr int at[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
  const R x[3] = {x0, x1, x2};
  const R r2 = dot3_t(x0, x0, x1, x1, x2, x2);
  const bool outside = r2 > R(1);
  // rho^2 = 1 + lambda: |x|^2 outside, 1 inside (lambda = 0, integratorElastic3DHelper.cpp:51-54)
  const R ir = rsqrt_t(outside ? r2 : R(1));
  const R i2 = ir * ir;
  const R p1 = R(4.0 * IBEM_PI) * (ir * i2), p2 = p1 * i2, p3 = p2 * i2;
  // rungs above the first vanish inside
  const R e2 = outside ? p2 : R(0), e3 = outside ? p3 : R(0);
  const R e4 = e3 * i2, e5 = e4 * i2, e6 = e5 * i2;
  const R q1 = R(1.0 / 3.0) * p1, q2 = R(1.0 / 5.0) * p2, q3 = R(1.0 / 7.0) * p3;   // J_1, J_2, J_3
  const R f1 = f * q1, f2 = f * q2, fe2 = f * e2, fe3 = f * e3, fe4 = f * e4;
  const R e3x5 = mulc_t(5.f, e3), e4x7 = mulc_t(7.f, e4);
  const R Q2 = q3 - q2, Q3 = e3 - e4, Q4 = mulc_t(9.f, e5) - e4x7;
  const R Ps3 = e2 - e3, Ps4 = e4x7 - e3x5, Q3x2 = pow2_t(2.f, Q3), Q2x2 = pow2_t(2.f, Q2);
  const R a3 = fe2 - (e2 + e3);
  const R b2 = (q2 + q3) - f2, b3 = fe3 - (e3 + e4);
  const R C2 = Q2x2 + f2, C2u = Q3x2 - fe3;
  const R Ps3x2 = pow2_t(2.f, Ps3), cE = Ps3x2 - fe2;

  R Ex[3], n[3], k[3], v[3], w[3], Ep[6], N[3][3];
  R q, tE;
  R Z[3];
  {
    R L[20];
    mf_ld(rec + kRecL, L);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j)
        N[i][j] = dot3_t(L[6 * i + at[j][0]], x0, L[6 * i + at[j][1]], x1, L[6 * i + at[j][2]], x2);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      n[i] = dot3_t(N[i][0], x0, N[i][1], x1, N[i][2], x2);
      Sum<R> s(pow2_t(0.5f, n[i]));
      s.add(N[0][i], x0);
      s.add(N[1][i], x1);
      s.add(N[2][i], x2);
      k[i] = s.val();
    }
  }
  R E[8];
  mf_ld(rec + kRecE, E);
  tE = E[6];
#pragma unroll
  for (int i = 0; i < 3; ++i) Ex[i] = dot3_t(E[at[i][0]], x0, E[at[i][1]], x1, E[at[i][2]], x2);
  q = dot3_t(Ex[0], x0, Ex[1], x1, Ex[2], x2);
  {
    R wv[8];
    mf_ld(rec + kRecW, wv);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      w[i] = wv[i];
      v[i] = wv[3 + i];
    }
  }
  R A, Au, B, W[3], dB[3], hA[3], m[3];
  {
    const R nx = pow2_t(0.5f, dot3_t(n[0], x0, n[1], x1, n[2], x2));
    const R wx = dot3_t(w[0], x0, w[1], x1, w[2], x2);
    const R vx = dot3_t(v[0], x0, v[1], x1, v[2], x2);
    const R Q4x2 = pow2_t(2.f, Q4);
    Sum<R> s(Ps4, q);
    s.add(a3, tE);
    s.add(Q4, nx);
    s.add(b3, wx);
    s.add(Q3x2, vx);
    A = s.val();
    Sum<R> su(mulc_t(35.f, e4) - mulc_t(63.f, e5), q);
    su.add((e3x5 + e4x7) - mulc_t(5.f, fe3), tE);
    su.add(mulc_t(63.f, e5) - mulc_t(99.f, e6), nx);
    su.add((e4x7 + mulc_t(9.f, e5)) - mulc_t(7.f, fe4), wx);
    su.add(Q4x2, vx);
    Au = pow2_t(0.5f, su.val());
    Sum<R> sb(Ps3, q);
    sb.add((q1 + q2) - f1, tE);
    sb.add(Q3, nx);
    sb.add(b2, wx);
    sb.add(Q2x2, vx);
    B = sb.val();
    const R Ps4x2 = pow2_t(2.f, Ps4);
    const R z1 = pow2_t(0.5f, fe3), z1u = mulc_t(-3.5f, fe4), z0u = mulc_t(-5.f, fe3);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      Sum<R> z(fe2, Ex[i]);
      z.add(z1, n[i]);
      z.add(-f2, v[i]);
      Sum<R> zu(z0u, Ex[i]);
      zu.add(z1u, n[i]);
      zu.add(fe3, v[i]);
      Sum<R> b(Ps3x2, Ex[i]);
      b.add(Q3, k[i]);
      b.add(Q2x2, v[i]);
      b.add(b2, w[i]);
      dB[i] = b.val();
      W[i] = dB[i] - z.val();
      Sum<R> a(Ps4x2, Ex[i]);
      a.add(Q4, k[i]);
      a.add(Q3x2, v[i]);
      a.add(b3, w[i]);
      const R dA = a.val();
      hA[i] = pow2_t(0.5f, dA);
      Sum<R> mm(dA - zu.val());
      mm.add(Au, x[i]);
      m[i] = mm.val();
    }
  }
  R F[20];
  mf_ld(rec + kRecF, F);
#pragma unroll
  for (int t = 0; t < 6; ++t) Ep[t] = dot3_t(F[3 * t], x0, F[3 * t + 1], x1, F[3 * t + 2], x2);
  // order 0
  const R Q2m = -Q2x2;
  {
    const R hAs = pow2_t(0.5f, A);
    const R C0 = pow2_t(2.f, (q2 - q1) + f1), C2x2 = pow2_t(2.f, C2);
    R p[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      Sum<R> s(W[i]);
      s.add(hAs, x[i]);
      p[i] = s.val();
    }
#pragma unroll
    for (int t = 0; t < 6; ++t) {
      const int i = pi[t], j = pj[t];
      Sum<R> s(i == j ? B : p[j] * x[i]);
      s.add(i == j ? pow2_t(2.f, p[i]) : p[i], x[j]);
      s.add(C0, E[t]);
      s.add(Q2m, Ep[t]);
      if (i == j) s.add(C2x2, N[i][i]);
      else s.add(C2, N[i][j] + N[j][i]);
      y[t] += s.val();
    }
  }
  // order 1
  R Rr[6], Y[3][3];
  {
    const R C0u = pow2_t(2.f, Ps3 - fe2), C2ux2 = pow2_t(2.f, C2u), Q3m = -Q3x2;
#pragma unroll
    for (int t = 0; t < 6; ++t) {
      const int i = pi[t], j = pj[t];
      R X;
      if (i == j) {
        Sum<R> s(A);
        s.add(Q3m, Ep[t]);
        X = s.val();
      } else {
        X = Q3m * Ep[t];
      }
      Sum<R> s(X);
      s.add(C0u, E[t]);
      if (i == j) s.add(C2ux2, N[i][i]);
      else s.add(C2u, N[i][j] + N[j][i]);
      Rr[t] = s.val();
      Sum<R> d(X);
      d.add(cE, E[t]);
      Y[i][j] = Y[j][i] = d.val();
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        Sum<R> s(Y[i][j]);
        s.add(Q3x2, N[j][i]);
        s.add(C2u, N[i][j]);
        s.add(hA[j], x[i]);
        s.add(m[i], x[j]);
        Y[i][j] = s.val();
      }
  }
  R S[20];
  mf_ld(rec + kRecS, S);
  const R C1 = C2 + f2;
  const R xx[3] = {pow2_t(2.f, x0), pow2_t(2.f, x1), pow2_t(2.f, x2)};
#pragma unroll
  for (int t = 0; t < 6; ++t) {
    const int i = pi[t], j = pj[t];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      R g;
      if (i == j) {
        Sum<R> s(i == c ? dB[c] + pow2_t(2.f, W[c]) : dB[c]);
        s.add(Y[i][c], xx[i]);
        s.add(Rr[t], x[c]);
        s.add(C1, F[3 * t + c]);
        s.add(C2, S[3 * t + c]);
        g = s.val();
      } else {
        Sum<R> s(i == c ? W[j] : (j == c ? W[i] : Rr[t] * x[c]));
        if (i == c || j == c) s.add(Rr[t], x[c]);
        s.add(Y[i][c], x[j]);
        s.add(Y[j][c], x[i]);
        s.add(C1, F[3 * t + c]);
        s.add(C2, S[3 * t + c]);
        g = s.val();
      }
      mf_acc(y[6 + 3 * t + c], row_scale, g);
    }
  }
}

// y = the kmu / klam map of a raw accumulation
template <class R>
IBEM_HD IBEM_INLINE void sph_pair_map24(const R (&acc)[24], R kmu, R klam, R (&y)[24]) {
  const R tr = acc[0] + acc[3] + acc[5];
  R dtr[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) dtr[k] = acc[6 + k] + acc[6 + 9 + k] + acc[6 + 15 + k];
#pragma unroll
  for (int t = 0; t < 6; ++t) {
    const bool d = (t == 0 || t == 3 || t == 5);
    y[t] = d ? kmu * acc[t] + klam * tr : kmu * acc[t];
#pragma unroll
    for (int k = 0; k < 3; ++k) y[6 + 3 * t + k] = d ? kmu * acc[6 + 3 * t + k] + klam * dtr[k] : kmu * acc[6 + 3 * t + k];
  }
}

// y[24] += the pair block (target at offset x from a source of radius a) times Eu[24];
// kmu, klam, tn1 = 1 - nu0, tn2 = 2 nu0 as in SphMat; row_scale multiplies the order-1 rows.  For single
// pairs: the contraction in units of the radius, where the order-1 coefficients take a factor a
// and the gradient 1 / a.
template <class R>
IBEM_HD IBEM_INLINE void sph_pair_apply24(R x0, R x1, R x2, R a, R kmu, R klam, R /*tn1*/, R tn2,
                                          const R* __restrict__ Eu, R row_scale, R (&y)[24]) {
  const R ia = R(1) / a;
  constexpr MfRecTab tab = mf_rec_tab();
  R c[25];
#pragma unroll
  for (int i = 0; i < 24; ++i) c[i] = i < 6 ? Eu[i] : a * Eu[i];
  c[24] = R(0);
  alignas(16) R rec[kRecLen];
#pragma unroll
  for (int e = 0; e < kRecLen; ++e) rec[e] = mf_rec_entry(tab.v[e], c);
  R raw[24], b[24];
#pragma unroll
  for (int i = 0; i < 24; ++i) raw[i] = R(0);
  sph_pair_raw24<R>(x0 * ia, x1 * ia, x2 * ia, R(2) - tn2, rec, row_scale * ia, raw);
  sph_pair_map24<R>(raw, kmu, klam, b);
#pragma unroll
  for (int i = 0; i < 24; ++i) y[i] += b[i];
}

}  // namespace ibem
