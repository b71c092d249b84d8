// Numbers, sums of products and source records of the layout-24 contractions (field_contract.cuh,
// mf_contract.cuh), each a template over float, double and double-float (DF).
#pragma once
#include "gen_sphere_common.cuh"   // first: IBEM_HD and IBEM_INLINE

#include "dfnum.cuh"
#include "fp64_math.cuh"

namespace ibem {

IBEM_HD IBEM_INLINE float rsqrt_t(float x) {
#ifdef __CUDA_ARCH__
  return rsqrtf(x);
#else
  return 1.0f / sqrtf(x);
#endif
}
IBEM_HD IBEM_INLINE double rsqrt_t(double x) { return rsqrt_h3(x); }

// A sum of products: plain for float and double, compensated (dfloat.cuh: 12 instead of 18
// FP32 instructions a term) for double-float numbers.
template <class R>
struct Sum {
  R s;
  Sum() = default;
  IBEM_HD IBEM_INLINE explicit Sum(R a) : s(a) {}
  IBEM_HD IBEM_INLINE Sum(R a, R b) : s(a * b) {}
  IBEM_HD IBEM_INLINE void add(R a, R b) { s = s + a * b; }
  IBEM_HD IBEM_INLINE void add(R a) { s = s + a; }
  IBEM_HD IBEM_INLINE R val() const { return s; }
};
template <>
struct Sum<DF> {
  dacc s;
  Sum() = default;
  IBEM_HD IBEM_INLINE explicit Sum(DF a) : s(dacc_of(a.v)) {}
  IBEM_HD IBEM_INLINE Sum(DF a, DF b) : s(dacc_prod(a.v, b.v)) {}
  IBEM_HD IBEM_INLINE void add(DF a, DF b) { dacc_fma(s, a.v, b.v); }
  IBEM_HD IBEM_INLINE void add(DF a) { dacc_add(s, a.v); }
  IBEM_HD IBEM_INLINE DF val() const { return DF(dacc_val(s)); }
};
// times a power of two (exact) or another FP32 constant
IBEM_HD IBEM_INLINE float pow2_t(float c, float x) { return c * x; }
IBEM_HD IBEM_INLINE double pow2_t(float c, double x) { return (double)c * x; }
IBEM_HD IBEM_INLINE DF pow2_t(float c, DF x) { return DF(dfloat{c * x.v.hi, c * x.v.lo}); }
IBEM_HD IBEM_INLINE float mulc_t(float c, float x) { return c * x; }
IBEM_HD IBEM_INLINE double mulc_t(float c, double x) { return (double)c * x; }
IBEM_HD IBEM_INLINE DF mulc_t(float c, DF x) { return DF(x.v * c); }
template <class R>
IBEM_HD IBEM_INLINE R dot3_t(R a0, R b0, R a1, R b1, R a2, R b2) {
  Sum<R> s(a0, b0);
  s.add(a1, b1);
  s.add(a2, b2);
  return s.val();
}

// ---- record of a source's coefficients E (order 0) and F (order 1), tensors symmetric in their
// first two indices, with the sums that the contractions take:
//   L_ikl = F_ikl + F_ilk,  S_ijk = F_ikj + F_jki,  w_n = F_mmn,  v_n = F_mnm
// [E (6), tr E, -] [w (3), v (3), -, -] [F (18), -, -] [S (18), -, -] [L (18), -, -];
// F, S: 3 (ij) + k, L: 6 i + (kl), pairs in the order 00 01 02 11 12 22.  The strain alone does
// without L.
constexpr int kRecE = 0, kRecW = 8, kRecF = 16, kRecS = 36, kRecField = 56, kRecL = 56, kRecLen = 76;
// Every entry of the record is a sum of at most three coefficients: their indices, a byte each
// (24: none).
struct MfRecTab {
  unsigned v[kRecLen];
};
constexpr MfRecTab mf_rec_tab() {
  MfRecTab t{};
  const int pi[6] = {0, 0, 0, 1, 1, 2}, pj[6] = {0, 1, 2, 1, 2, 2};
  const int at[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
  struct F {
    static constexpr unsigned pack(int a, int b = 24, int c = 24, int d = 24) {
      return (unsigned)a | (unsigned)b << 8 | (unsigned)c << 16 | (unsigned)d << 24;
    }
  };
  for (int e = 0; e < kRecLen; ++e) t.v[e] = F::pack(24);
  for (int i = 0; i < 6; ++i) t.v[kRecE + i] = F::pack(i);
  t.v[kRecE + 6] = F::pack(0, 3, 5);
  for (int n = 0; n < 3; ++n) {
    t.v[kRecW + n] = F::pack(6 + n, 6 + 9 + n, 6 + 15 + n);
    t.v[kRecW + 3 + n] = F::pack(6 + 3 * at[0][n], 6 + 3 * at[1][n] + 1, 6 + 3 * at[2][n] + 2);
  }
  for (int i = 0; i < 18; ++i) t.v[kRecF + i] = F::pack(6 + i);
  for (int i = 0; i < 3; ++i)
    for (int q = 0; q < 6; ++q) {
      const int k = pi[q], l = pj[q];
      t.v[kRecL + 6 * i + q] = F::pack(6 + 3 * at[i][k] + l, 6 + 3 * at[i][l] + k);
    }
  for (int q = 0; q < 6; ++q)
    for (int k = 0; k < 3; ++k) {
      const int i = pi[q], j = pj[q];
      t.v[kRecS + 3 * q + k] = F::pack(6 + 3 * at[i][k] + j, 6 + 3 * at[j][k] + i);
    }
  return t;
}
// entry of a record from its packed indices and the coefficients (c[24] = 0)
template <class R>
IBEM_HD IBEM_INLINE R mf_rec_entry(unsigned q, const R* c) {
  return (c[q & 31u] + c[(q >> 8) & 31u]) + (c[(q >> 16) & 31u] + c[q >> 24]);
}

// loads of N consecutive numbers from a 16-byte boundary
template <int N>
IBEM_HD IBEM_INLINE void mf_ld(const float* p, float (&o)[N]) {
#ifdef __CUDA_ARCH__
#pragma unroll
  for (int i = 0; i < N; i += 4) {
    const float4 q = *reinterpret_cast<const float4*>(p + i);
    o[i] = q.x;
    o[i + 1] = q.y;
    o[i + 2] = q.z;
    o[i + 3] = q.w;
  }
#else
  for (int i = 0; i < N; ++i) o[i] = p[i];
#endif
}
template <int N>
IBEM_HD IBEM_INLINE void mf_ld(const double* p, double (&o)[N]) {
#ifdef __CUDA_ARCH__
#pragma unroll
  for (int i = 0; i < N; i += 2) {
    const double2 q = *reinterpret_cast<const double2*>(p + i);
    o[i] = q.x;
    o[i + 1] = q.y;
  }
#else
  for (int i = 0; i < N; ++i) o[i] = p[i];
#endif
}
template <int N>
IBEM_HD IBEM_INLINE void mf_ld(const DF* p, DF (&o)[N]) {
#ifdef __CUDA_ARCH__
#pragma unroll
  for (int i = 0; i < N; i += 2) {
    const float4 q = *reinterpret_cast<const float4*>(p + i);
    o[i].v = dfloat{q.x, q.y};
    o[i + 1].v = dfloat{q.z, q.w};
  }
#else
  for (int i = 0; i < N; ++i) o[i] = p[i];
#endif
}

}  // namespace ibem
