// Strain at a field point from one sphere with a linear Taylor eigenstrain (24 unknowns),
// contracted with the eigenstrain before any tensor is formed.
//
// postProcessorElastic3D.cpp:407-470 forms e_ij = sum_cols D_ijmn(..)·map·E_col with the
// Eshelby-type tensors of integratorElastic3DHelper.cpp:2394-2442 (D_40, D_50).  Writing
// E_mn (order 0) and F_mnp (order 1) as full tensors symmetric in (m, n) absorbs map[m][n],
// and every derivative of the sphere potentials is a radial pattern:
//   d_ij F = F2 x_i x_j + F1 d_ij,   d_ijk F = F3 x_i x_j x_k + F2 (d_ij x_k + 2 more),
//   d_ijkl F = F4 xxxx + F3 (6 d xx) + F2 (3 d d),   Fk = k-th derivative of F in u = |x|^2/2.
// With psi = Psi0, phi = V0, psi_p = a^2 x_p Q, phi_p = a^2 x_p V1 the contraction gives
//   e_ij = c { T(Psi, E)_ij - 2 nu trE phi_,ij - 2 (1-nu) [M_ij + M_ji]
//            + a^2 [ T(Q, E')_ij + 2 (Q3 (v.x) x_i x_j + Q2 (v_i x_j + v_j x_i + d_ij v.x))
//                    + Q3 (s_i x_j + s_j x_i) + Q2 (g_i x_j + g_j x_i + 2 (G^j x)_i + 2 (G^i x)_j) ]
//            - 2 nu a^2 [ (w.x)(V1'' x_i x_j + V1' d_ij) + V1' (w_i x_j + w_j x_i) ]
//            - 2 (1-nu) a^2 [ P_ij + P_ji ] },   c = 1 / (8 pi (1 - nu))
// with T(G, E)_ij = G4 q x_i x_j + G3 (d_ij q + 2 (Ex)_i x_j + 2 x_i (Ex)_j + trE x_i x_j)
//                   + G2 (d_ij trE + 2 E_ij),  q = x.E.x,
//      M_ij = Phi2 (Ex)_i x_j + Phi1 E_ij,  E'_mn = sum_p F_mnp x_p,  v_n = sum_m F_mnm,
//      w_p = sum_m F_mmp,  G^i_mn = F_mni,  s_i = x.G^i.x,  g_i = tr G^i,
//      P_ij = V1'' (E'x)_i x_j + V1' (E'_ij + v_i x_j + (G^j x)_i).
// Collecting like terms, per (point, sphere) pair:
//   e_ij / c = A x_i x_j + B d_ij + W_i x_j + W_j x_i + C0 E_ij + C1 E'_ij + C2 ((G^i x)_j + (G^j x)_i)
// with scalar A, B, C0..C2 and vector W computed once.  In units of the sphere's radius (x / a,
// a = 1, the order-1 eigenstrain scaled to a F: the strain depends on x / a only, and the sums run
// on numbers of the order of 1, inside the FP32 exponent range for any sphere size) and with the
// source sums of contract_num.cuh, H_ij = S_ijl x_l = (G^i x)_j + (G^j x)_i:
//   e_ij / c = p_i x_j + p_j x_i + C0 E_ij + C1 E'_ij + C2 H_ij + d_ij B,   p = A x / 2 + W,
//   W = cE E x + (Q3 - 2 (1 - nu) V1'') E' x + Q3 H x + C2 v + b2 w
// in about 180 multiply-adds per pair (260 operations in the form above).
// Inside the sphere (lambda = 0) the u-derivatives of J vanish, exactly as the reference.
#pragma once
#include "contract_num.cuh"
#include "gen_sphere_common.cuh"

namespace ibem {

// Radial coefficients of the contraction at ir = |x|^-1 outside and 1 inside; f = 2 (1 - nu0).
template <class R>
struct FieldCoef {
  R aq, aE, aqp, aw, av;    // A = aq q + aE tr E + aqp x.E'x + aw w.x + av v.x
  R bq, bE, bqp, bw, bv;    // B
  R cE, cEp, cH, cv, cw;    // W
  R C0, C1, C2;
};
template <class R>
IBEM_HD IBEM_INLINE FieldCoef<R> sph_field_coef(R p0, R ir, bool outside, R f) {
  const R i2 = ir * ir;
  const R p1 = p0 * (ir * i2), p2 = p1 * i2, p3 = p2 * i2;
  // rungs above the first vanish inside
  const R e2 = outside ? p2 : R(0), e3 = outside ? p3 : R(0);
  const R e4 = e3 * i2, e5 = e4 * i2;
  const R q1 = R(1.0 / 3.0) * p1, q2 = R(1.0 / 5.0) * p2, q3 = R(1.0 / 7.0) * p3;   // J_1, J_2, J_3
  const R f1 = f * q1, f2 = f * q2, fe2 = f * e2, fe3 = f * e3;
  const R e4x7 = mulc_t(7.f, e4);
  const R Q2 = q3 - q2, Q3 = e3 - e4, Q2x2 = pow2_t(2.f, Q2), Ps3 = e2 - e3, C2 = Q2x2 + f2;
  FieldCoef<R> c;
  c.aq = e4x7 - mulc_t(5.f, e3);
  c.aE = fe2 - (e2 + e3);
  c.aqp = mulc_t(9.f, e5) - e4x7;
  c.aw = fe3 - (e3 + e4);
  c.av = pow2_t(2.f, Q3);
  c.bq = Ps3;
  c.bE = (q1 + q2) - f1;
  c.bqp = c.cH = Q3;
  c.bw = c.cw = (q2 + q3) - f2;
  c.bv = Q2x2;
  c.cE = pow2_t(2.f, Ps3) - fe2;
  c.cEp = Q3 - fe3;
  c.cv = c.C2 = C2;
  c.C0 = pow2_t(2.f, (q2 - q1) + f1);
  c.C1 = C2 + f2;
  return c;
}

// Strain / c at offset x (in units of the radius) of the source with record rec: the
// components' sums continue e (CHAIN) or replace it.
template <class R, bool CHAIN>
IBEM_HD IBEM_INLINE void sph_field24_raw(const R (&x)[3], const FieldCoef<R>& k, const R* __restrict__ rec,
                                         Sum<R> (&e)[6]) {
  constexpr int pi[6] = {0, 0, 0, 1, 1, 2}, pj[6] = {0, 1, 2, 1, 2, 2};
  constexpr int at[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
  R Ex[3], Epx[3], Hx[3], Ep[6], H[6], w[3], v[3], W[3];
  R E[8], F[20], S[20], wv[8];
  mf_ld(rec + kRecF, F);
#pragma unroll
  for (int t = 0; t < 6; ++t) Ep[t] = dot3_t(F[3 * t], x[0], F[3 * t + 1], x[1], F[3 * t + 2], x[2]);
  mf_ld(rec + kRecS, S);
#pragma unroll
  for (int t = 0; t < 6; ++t) H[t] = dot3_t(S[3 * t], x[0], S[3 * t + 1], x[1], S[3 * t + 2], x[2]);
  mf_ld(rec + kRecE, E);
  mf_ld(rec + kRecW, wv);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    Ex[i] = dot3_t(E[at[i][0]], x[0], E[at[i][1]], x[1], E[at[i][2]], x[2]);
    Epx[i] = dot3_t(Ep[at[i][0]], x[0], Ep[at[i][1]], x[1], Ep[at[i][2]], x[2]);
    Hx[i] = dot3_t(H[at[i][0]], x[0], H[at[i][1]], x[1], H[at[i][2]], x[2]);
    w[i] = wv[i];
    v[i] = wv[3 + i];
  }
  const R tE = E[6];
  const R q = dot3_t(Ex[0], x[0], Ex[1], x[1], Ex[2], x[2]);
  const R qp = dot3_t(Epx[0], x[0], Epx[1], x[1], Epx[2], x[2]);
  const R wx = dot3_t(w[0], x[0], w[1], x[1], w[2], x[2]);
  const R vx = dot3_t(v[0], x[0], v[1], x[1], v[2], x[2]);
  Sum<R> sa(k.aq, q);
  sa.add(k.aE, tE);
  sa.add(k.aqp, qp);
  sa.add(k.aw, wx);
  sa.add(k.av, vx);
  const R hA = pow2_t(0.5f, sa.val());
  Sum<R> sb(k.bq, q);
  sb.add(k.bE, tE);
  sb.add(k.bqp, qp);
  sb.add(k.bw, wx);
  sb.add(k.bv, vx);
  const R B = sb.val();
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    Sum<R> s(k.cE, Ex[i]);
    s.add(k.cEp, Epx[i]);
    s.add(k.cH, Hx[i]);
    s.add(k.cv, v[i]);
    s.add(k.cw, w[i]);
    s.add(hA, x[i]);
    W[i] = s.val();   // p
  }
#pragma unroll
  for (int t = 0; t < 6; ++t) {
    const int i = pi[t], j = pj[t];
    Sum<R> s;
    if (CHAIN) {
      s = e[t];
      if (i == j) s.add(B);
      else s.add(W[j], x[i]);
    } else {
      s = i == j ? Sum<R>(B) : Sum<R>(W[j], x[i]);
    }
    s.add(i == j ? pow2_t(2.f, W[i]) : W[i], x[j]);
    s.add(k.C0, E[t]);
    s.add(k.C1, Ep[t]);
    s.add(k.C2, H[t]);
    e[t] = s;
  }
}

}  // namespace ibem

// e[6] += the strain at offset x from a sphere of radius a with coefficients Eu (FP64).  For
// single pairs; the stress sums keep the sphere's record.
IBEM_HD IBEM_INLINE void sph_field24_contracted(const double x0, const double x1, const double x2, const double a,
                                                const SphMat& mc, const double* __restrict__ Eu,
                                                double* __restrict__ e) {
  constexpr ibem::MfRecTab tab = ibem::mf_rec_tab();
  double c[25];
  for (int i = 0; i < 24; ++i) c[i] = i < 6 ? Eu[i] : a * Eu[i];
  c[24] = 0.0;
  alignas(16) double rec[ibem::kRecField];
  for (int i = 0; i < ibem::kRecField; ++i) rec[i] = ibem::mf_rec_entry(tab.v[i], c);
  const double ia = 1.0 / a;
  const double x[3] = {x0 * ia, x1 * ia, x2 * ia};
  const double r2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
  const bool outside = r2 > 1.0;
  ibem::Sum<double> r[6];
  ibem::sph_field24_raw<double, false>(
      x, ibem::sph_field_coef<double>(4.0 * IBEM_PI, ibem::rsqrt_t(outside ? r2 : 1.0), outside, 2.0 * mc.tn1), rec, r);
  for (int t = 0; t < 6; ++t) e[t] += mc.kd * r[t].val();
}

// ----------------------------------------------------------------------------------------
// The double-float and FP32 forms of the mixed stress sums.
namespace ibem {

// per-sphere constants of the double-float sum (scaled coordinates)
struct SphDF {
  dfloat c[3];   // centre
  dfloat ia;     // 1 / a
  DF rec[kRecField];   // of E and a F
};
static_assert(sizeof(SphDF) % 16 == 0, "records are loaded 16 bytes at a time");
// and of the FP32 sum
struct SphF {
  float hi[3], ia, lo[3], pad;
  float rec[kRecField];
};
static_assert(sizeof(SphF) % 16 == 0, "records are loaded 16 bytes at a time");

IBEM_HD inline SphDF sph_df_make(const double* cen, double a, const double* Eu) {
  constexpr MfRecTab tab = mf_rec_tab();
  SphDF s;
  const double ia = 1.0 / a;
  for (int i = 0; i < 3; ++i) s.c[i] = df_make(cen[i]);
  s.ia = df_make(ia);
  double c[25];
  for (int i = 0; i < 24; ++i) c[i] = i < 6 ? Eu[i] : a * Eu[i];
  c[24] = 0.0;
  for (int i = 0; i < kRecField; ++i) s.rec[i] = DF(mf_rec_entry(tab.v[i], c));
  return s;
}
IBEM_HD inline SphF sph_f_make(const SphDF& d) {
  SphF s;
  for (int i = 0; i < 3; ++i) {
    s.hi[i] = d.c[i].hi;
    s.lo[i] = d.c[i].lo;
  }
  s.ia = d.ia.hi;
  s.pad = 0.f;
  for (int i = 0; i < kRecField; ++i) s.rec[i] = d.rec[i].v.hi;
  return s;
}

// e[6] += strain / c at the point p (double-float, point already converted), each e[t] a
// compensated sum over the spheres; returns whether the point lies inside or on the sphere.
// The caller multiplies by c = 1 / (8 pi (1 - nu)) once, after the sum.
IBEM_HD IBEM_INLINE bool sph_field24_df(const dfloat* p, const SphDF& sp, dfloat tn1, dfloat /*tn2*/, dacc* e) {
  DF x[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) x[i] = DF((p[i] - sp.c[i]) * sp.ia);
  const DF r2 = dot3_t(x[0], x[0], x[1], x[1], x[2], x[2]);
  const bool ext = r2 > DF(1.0);
  Sum<DF> s[6];
#pragma unroll
  for (int t = 0; t < 6; ++t) s[t].s = e[t];
  sph_field24_raw<DF, true>(
      x, sph_field_coef<DF>(DF(4.0 * IBEM_PI), rsqrt_t(ext ? r2 : DF(1.0)), ext, pow2_t(2.f, DF(tn1))), sp.rec, s);
#pragma unroll
  for (int t = 0; t < 6; ++t) e[t] = s[t].s;
  return !ext;
}

// The same contraction in FP32 for far pairs of the mixed form's split sum: a sphere whose
// centre lies beyond kFarRadii of its radius from every point of a warp contributes at most
// (1/kFarRadii)^3 of a near sphere, so its FP32 rounding (a few 1e-7 of the contribution,
// unbiased) stays near 1e-9 of the strain when summed over all far spheres.  The random-sign
// errors add in squares, so the nearest far shell dominates and the summed error grows as
// kFarRadii^-1.5: stresses of the 2,000-sphere, 64^3-point workload from its solution, against
// FP64 sums, 3.2e-9 at 14 radii, 4.2e-9 at 12, 5.5e-9 at 10 (the solution target is 1e-8).
// The sphere's constants are the high parts of its SphDF.
constexpr float kFarRadii = 12.0f;

// Written out term by term: the roundings of its coefficients are the same for every sphere, and
// those of a regrouped sum (sph_field24_raw) moved the summed stresses by 1.6e-9 to 5e-9 for 2,000
// spheres, as much as their error, for 6% of the pass.
IBEM_HD IBEM_INLINE void sph_field24_f32(const dfloat* p, const SphF& sp, float tn1, float tn2, float* e) {
  float x[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) x[i] = ((p[i].hi - sp.hi[i]) + (p[i].lo - sp.lo[i])) * sp.ia;
  const float r2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
  // outside by construction (far pair): rho^2 = |x|^2
  float ir;
#ifdef __CUDA_ARCH__
  ir = rsqrtf(r2);
#else
  ir = 1.0f / std::sqrt(r2);
#endif
  ir = ir * (1.5f - 0.5f * r2 * ir * ir);  // one Newton step
  const float irho2 = ir * ir;
  const float p1 = 4.0f * 3.14159265358979f * ir * irho2, p2 = p1 * irho2, p3 = p2 * irho2, p4 = p3 * irho2,
              p5 = p4 * irho2;
  const float J1 = p1 * (1.0f / 3.0f), J2 = p2 * 0.2f, J3 = p3 * (1.0f / 7.0f), J4 = p4 * (1.0f / 9.0f),
              J5 = p5 * (1.0f / 11.0f);
  const float V0_1 = -J1, V0_2 = 5.0f * J2, V0_3 = -35.0f * J3;
  const float V1_1 = -J2, V1_2 = 7.0f * J3, V1_3 = -63.0f * J4;
  const float V2_1 = -J3, V2_2 = 9.0f * J4, V2_3 = -99.0f * J5;
  const float Ps2 = V0_1 - V1_1, Ps3 = V0_2 - V1_2, Ps4 = V0_3 - V1_3;
  const float Q2 = V1_1 - V2_1, Q3 = V1_2 - V2_2, Q4 = V1_3 - V2_3;
  const float Ph1 = V0_1, Ph2 = V0_2;
  const int ti[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
  float E[8], wv[8], F[20];
  mf_ld(sp.rec + kRecE, E);
  mf_ld(sp.rec + kRecW, wv);
  mf_ld(sp.rec + kRecF, F);
  const float *w0 = wv, *v0 = wv + 3;
  float Ex[3], Ep[6], Epx[3], Gx[3][3], s[3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
    Ex[i] = E[ti[i][0]] * x[0] + E[ti[i][1]] * x[1] + E[ti[i][2]] * x[2];
#pragma unroll
  for (int t = 0; t < 6; ++t) Ep[t] = F[3 * t] * x[0] + F[3 * t + 1] * x[1] + F[3 * t + 2] * x[2];
#pragma unroll
  for (int n = 0; n < 3; ++n) Epx[n] = Ep[ti[n][0]] * x[0] + Ep[ti[n][1]] * x[1] + Ep[ti[n][2]] * x[2];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
#pragma unroll
    for (int j = 0; j < 3; ++j)
      Gx[i][j] = F[3 * ti[j][0] + i] * x[0] + F[3 * ti[j][1] + i] * x[1] + F[3 * ti[j][2] + i] * x[2];
    s[i] = Gx[i][0] * x[0] + Gx[i][1] * x[1] + Gx[i][2] * x[2];
  }
  const float q = Ex[0] * x[0] + Ex[1] * x[1] + Ex[2] * x[2];
  const float qp = Epx[0] * x[0] + Epx[1] * x[1] + Epx[2] * x[2];
  const float tEp = Ep[0] + Ep[3] + Ep[5];
  const float vx = v0[0] * x[0] + v0[1] * x[1] + v0[2] * x[2];
  const float wx = w0[0] * x[0] + w0[1] * x[1] + w0[2] * x[2];
  const float tE = E[6];
  const float tv = tEp + 2.0f * vx;
  const float A = Ps4 * q + Ps3 * tE - tE * Ph2 * tn2 + (Q4 * qp + Q3 * tv - wx * V1_2 * tn2);
  const float B = Ps3 * q + Ps2 * tE - tE * Ph1 * tn2 + (Q3 * qp + Q2 * tv - wx * V1_1 * tn2);
  const float cE = 2.0f * Ps3 - 2.0f * tn1 * Ph2;
  const float cEp = 2.0f * Q3 - 2.0f * tn1 * V1_2, cv = 2.0f * Q2 - 2.0f * tn1 * V1_1;
  const float cs = Q3, cgw = Q2 - tn2 * V1_1;
  float W[3];
#pragma unroll
  for (int i = 0; i < 3; ++i)
    W[i] = cE * Ex[i] + cEp * Epx[i] + cv * v0[i] + cs * s[i] + cgw * w0[i];
  const float C0 = 2.0f * Ps2 - 4.0f * tn1 * Ph1;
  const float C1 = 2.0f * Q2 - 4.0f * tn1 * V1_1;
  const float C2 = 2.0f * Q2 - 2.0f * tn1 * V1_1;
  const int pi[6] = {0, 0, 0, 1, 1, 2}, pj[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
  for (int t = 0; t < 6; ++t) {
    const int i = pi[t], j = pj[t];
    float r = A * x[i] * x[j] + W[i] * x[j] + W[j] * x[i] + C0 * E[t] + C1 * Ep[t] + C2 * (Gx[i][j] + Gx[j][i]);
    if (i == j) r += B;
    e[t] = r;
  }
}

IBEM_HD IBEM_INLINE void sph_field24_f32(const dfloat* p, const SphDF& sp, float tn1, float tn2, float* e) {
  sph_field24_f32(p, sph_f_make(sp), tn1, tn2, e);
}

// a += b (double-float plus FP32, error-free sum of the high parts)
IBEM_HD IBEM_INLINE void df_add_f(dfloat& a, float b) {
  const dfloat s = df_two_sum(a.hi, b);
  a = df_fast_two_sum(s.hi, s.lo + a.lo);
}

}  // namespace ibem
