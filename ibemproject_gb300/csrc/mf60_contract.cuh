// Product of one 60 x 60 sphere pair block (orders 0 to 2 on both sides) with the source's
// coefficients, for a target outside the source, in the frame of the offset, where the block
// is sparse (gen_mf60.cuh, derived in codegen_mf60.py).  Everything in coordinates scaled by
// the source's radius.
//
// Operations per pair (multiply-adds): frame 60, rotation of the coefficients 566, radial
// coefficients about 1,200 (they depend on the pair's distance and on nu), sparse block 520,
// rotation back 580; the dense generated block costs about 25,000 and 3,600 more to apply.
#pragma once
#include "gen_sphere_common.cuh"

#include "gen_mf60.cuh"

namespace ibem {

IBEM_HD IBEM_INLINE float mf60_rcp(float v) { return 1.0f / v; }
IBEM_HD IBEM_INLINE double mf60_rcp(double v) { return 1.0 / v; }

// Components of a symmetric tensor: 0 trace, 1 zz, 2 xx - yy, 3 xy, 4 xz, 5 yz of the frame
// (e[0], e[1], e[2]) = (x, y, z); g[a - 1] holds component a's matrix at (i, j), i <= j.
template <class R>
struct Mf60Frame {
  R e[3][3];
  R g[5][6];
};

template <class R>
IBEM_HD IBEM_INLINE void mf60_frame(R n0, R n1, R n2, Mf60Frame<R>& f) {
  // orthonormal frame of the unit vector n without a branch or a square root (Duff et al. 2017)
  const R sg = n2 < R(0) ? R(-1) : R(1);
  const R a = -mf60_rcp(sg + n2), b = n0 * n1 * a;
  f.e[0][0] = R(1) + sg * n0 * n0 * a;
  f.e[0][1] = sg * b;
  f.e[0][2] = -sg * n0;
  f.e[1][0] = b;
  f.e[1][1] = sg + n1 * n1 * a;
  f.e[1][2] = -n1;
  f.e[2][0] = n0;
  f.e[2][1] = n1;
  f.e[2][2] = n2;
  const int pi[6] = {0, 0, 0, 1, 1, 2}, pj[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
  for (int t = 0; t < 6; ++t) {
    const int i = pi[t], j = pj[t];
    const R xi = f.e[0][i], xj = f.e[0][j], yi = f.e[1][i], yj = f.e[1][j], zi = f.e[2][i], zj = f.e[2][j];
    f.g[0][t] = zi * zj;
    f.g[1][t] = xi * xj - yi * yj;
    f.g[2][t] = xi * yj + yi * xj;
    f.g[3][t] = xi * zj + zi * xj;
    f.g[4][t] = yi * zj + zi * yj;
  }
}

// v: a symmetric tensor (xx, 2 xy, 2 xz, yy, 2 yz, zz) -> its six components
template <class R>
IBEM_HD IBEM_INLINE void mf60_to_frame(const Mf60Frame<R>& f, const R (&v)[6], R (&c)[6]) {
  c[0] = v[0] + v[3] + v[5];
#pragma unroll
  for (int a = 0; a < 5; ++a) {
    R s = f.g[a][0] * v[0];
#pragma unroll
    for (int t = 1; t < 6; ++t) s += f.g[a][t] * v[t];
    c[a + 1] = s;
  }
}
// and back: v (xx, xy, xz, yy, yz, zz) += sum over the components
template <class R>
IBEM_HD IBEM_INLINE void mf60_from_frame(const Mf60Frame<R>& f, const R (&c)[6], R (&v)[6]) {
#pragma unroll
  for (int t = 0; t < 6; ++t) {
    R s = v[t];
#pragma unroll
    for (int a = 0; a < 5; ++a) s += f.g[a][t] * c[a + 1];
    v[t] = (t == 0 || t == 3 || t == 5) ? s + c[0] : s;
  }
}

// The source's coefficients in the frame.  e: its 60 coefficients (layout 60) times 2 for
// each off-diagonal index pair (i < j, and p < q of the order-2 ones): mf60_weight.
IBEM_HD IBEM_INLINE int mf60_off(int t) { return t == 1 || t == 2 || t == 4; }
IBEM_HD IBEM_INLINE float mf60_weight(int i) {
  const int t = i < 6 ? i : (i < 24 ? (i - 6) / 3 : (i - 24) / 6);
  return (float)((1 + mf60_off(t)) * (i < 24 ? 1 : 1 + mf60_off((i - 24) % 6)));
}
template <class R>
IBEM_HD IBEM_INLINE void mf60_source(const Mf60Frame<R>& f, const R* __restrict__ e, R (&A0)[6], R (&A1)[6][3],
                                     R (&A2)[6][6]) {
  R v[6], c[6];
#pragma unroll
  for (int t = 0; t < 6; ++t) v[t] = e[t];
  mf60_to_frame(f, v, A0);
#pragma unroll
  for (int p = 0; p < 3; ++p) {
#pragma unroll
    for (int t = 0; t < 6; ++t)
      v[t] = f.e[p][0] * e[6 + 3 * t] + f.e[p][1] * e[7 + 3 * t] + f.e[p][2] * e[8 + 3 * t];
    mf60_to_frame(f, v, c);
#pragma unroll
    for (int a = 0; a < 6; ++a) A1[a][p] = c[a];
  }
  R T[6][6];   // [component of the order-2 index pair][tensor index]
#pragma unroll
  for (int t = 0; t < 6; ++t) {
#pragma unroll
    for (int s = 0; s < 6; ++s) v[s] = e[24 + 6 * t + s];
    mf60_to_frame(f, v, c);
#pragma unroll
    for (int b = 0; b < 6; ++b) T[b][t] = c[b];
  }
#pragma unroll
  for (int b = 0; b < 6; ++b) {
    mf60_to_frame(f, T[b], c);
#pragma unroll
    for (int a = 0; a < 6; ++a) A2[a][b] = c[a];
  }
}

// powers r^-3 .. r^-9 times `scale`
template <class R>
IBEM_HD IBEM_INLINE void mf60_powers(R ir, R scale, R (&q)[7]) {
  q[0] = ir * ir * ir * scale;
#pragma unroll
  for (int n = 1; n < 7; ++n) q[n] = q[n - 1] * ir;
}

// Rows of order RO, before the material map: acc += scale * (strain derivatives of order RO)
template <int RO, class R>
IBEM_HD IBEM_INLINE void mf60_rows(const Mf60Frame<R>& f, const R (&A0)[6], const R (&A1)[6][3], const R (&A2)[6][6], R ir,
                                   R scale, R nu, R* acc) {
  R q[7];
  mf60_powers(ir, scale, q);
  if constexpr (RO == 0) {
    R W[6], v[6];
    mf60_sparse_r0(A0, A1, A2, q, nu, W);
#pragma unroll
    for (int t = 0; t < 6; ++t) v[t] = acc[t];
    mf60_from_frame(f, W, v);
#pragma unroll
    for (int t = 0; t < 6; ++t) acc[t] = v[t];
  } else if constexpr (RO == 1) {
    R W[6][3];
    mf60_sparse_r1(A0, A1, A2, q, nu, W);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      R c[6], v[6];
#pragma unroll
      for (int a = 0; a < 6; ++a) c[a] = f.e[0][k] * W[a][0] + f.e[1][k] * W[a][1] + f.e[2][k] * W[a][2];
#pragma unroll
      for (int t = 0; t < 6; ++t) v[t] = acc[3 * t + k];
      mf60_from_frame(f, c, v);
#pragma unroll
      for (int t = 0; t < 6; ++t) acc[3 * t + k] = v[t];
    }
  } else {
    R W[6][6], T[6][6];
    mf60_sparse_r2(A0, A1, A2, q, nu, W);
#pragma unroll
    for (int a = 0; a < 6; ++a) {
      R v[6] = {R(0), R(0), R(0), R(0), R(0), R(0)};
      mf60_from_frame(f, W[a], v);
#pragma unroll
      for (int s = 0; s < 6; ++s) T[s][a] = v[s];
    }
#pragma unroll
    for (int s = 0; s < 6; ++s) {
      R v[6];
#pragma unroll
      for (int t = 0; t < 6; ++t) v[t] = acc[6 * t + s];
      mf60_from_frame(f, T[s], v);
#pragma unroll
      for (int t = 0; t < 6; ++t) acc[6 * t + s] = v[t];
    }
  }
}

// The rows of the system from the summed strain derivatives: (C0 - C1) applied to the tensor
// indices (kmu and klam as in SphMat), V = 4 pi / 3, and the 1/2 of the order-2 rows.
template <int RO, class R>
IBEM_HD IBEM_INLINE void mf60_map(R kmu, R klam, R* acc) {
  constexpr int n = RO == 0 ? 1 : (RO == 1 ? 3 : 6);   // derivatives
  const R v = R(4.0 * IBEM_PI / 3.0) * (RO == 2 ? R(0.5) : R(1));
#pragma unroll
  for (int k = 0; k < n; ++k) {
    const R tr = acc[k] + acc[3 * n + k] + acc[5 * n + k];
#pragma unroll
    for (int t = 0; t < 6; ++t) {
      const R m = kmu * acc[n * t + k];
      acc[n * t + k] = v * ((t == 0 || t == 3 || t == 5) ? m + klam * tr : m);
    }
  }
}

}  // namespace ibem
