// GENERATED by ibemproject_gb300/codegen.py -- do not edit by hand.
// FP32 materials and own (C0) term of the matrix-free layout-24 products, which work in
// coordinates scaled by the source radius (a = 1), so that every intermediate is O(1) in
// single precision.  Same derivation as gen_sphere24.cuh.
#pragma once
#include "gen_sphere_common.cuh"

// Dimensionless material constants of the FP32 products (sph_matf_init: SphMat / mu0).
struct SphMatF {
  float kmu, klam, tn1, tn2;  // as SphMat, contrast terms divided by mu0
  float lam0, mu0;            // C0 / mu0 (self term): lam0 / mu0 and 1
};

IBEM_HD inline SphMatF sph_matf_init(const SphMat& m) {
  SphMatF f;
  const double s = 1.0 / m.mu0;
  f.kmu = (float)(m.kmu * s);
  f.klam = (float)(m.klam * s);
  f.tn1 = (float)m.tn1;
  f.tn2 = (float)m.tn2;
  f.lam0 = (float)(m.lam0 * s);
  f.mu0 = 1.0f;
  return f;
}


template <class Sink>
IBEM_HD IBEM_INLINE void sph_self24f(const SphMatF& mc, Sink& sink) {
  sink(0, 0, 1.0f * (mc.lam0 + 2.0f * mc.mu0));
  sink(0, 3, 1.0f * (mc.lam0));
  sink(0, 5, 1.0f * (mc.lam0));
  sink(1, 1, 2.0f * (1.0f * mc.mu0));
  sink(2, 2, 2.0f * (1.0f * mc.mu0));
  sink(3, 0, 1.0f * (mc.lam0));
  sink(3, 3, 1.0f * (mc.lam0 + 2.0f * mc.mu0));
  sink(3, 5, 1.0f * (mc.lam0));
  sink(4, 4, 2.0f * (1.0f * mc.mu0));
  sink(5, 0, 1.0f * (mc.lam0));
  sink(5, 3, 1.0f * (mc.lam0));
  sink(5, 5, 1.0f * (mc.lam0 + 2.0f * mc.mu0));
  sink(6, 6, 1.0f * (mc.lam0 + 2.0f * mc.mu0));
  sink(6, 15, 1.0f * (mc.lam0));
  sink(6, 21, 1.0f * (mc.lam0));
  sink(7, 7, 1.0f * (mc.lam0 + 2.0f * mc.mu0));
  sink(7, 16, 1.0f * (mc.lam0));
  sink(7, 22, 1.0f * (mc.lam0));
  sink(8, 8, 1.0f * (mc.lam0 + 2.0f * mc.mu0));
  sink(8, 17, 1.0f * (mc.lam0));
  sink(8, 23, 1.0f * (mc.lam0));
  sink(9, 9, 2.0f * (1.0f * mc.mu0));
  sink(10, 10, 2.0f * (1.0f * mc.mu0));
  sink(11, 11, 2.0f * (1.0f * mc.mu0));
  sink(12, 12, 2.0f * (1.0f * mc.mu0));
  sink(13, 13, 2.0f * (1.0f * mc.mu0));
  sink(14, 14, 2.0f * (1.0f * mc.mu0));
  sink(15, 6, 1.0f * (mc.lam0));
  sink(15, 15, 1.0f * (mc.lam0 + 2.0f * mc.mu0));
  sink(15, 21, 1.0f * (mc.lam0));
  sink(16, 7, 1.0f * (mc.lam0));
  sink(16, 16, 1.0f * (mc.lam0 + 2.0f * mc.mu0));
  sink(16, 22, 1.0f * (mc.lam0));
  sink(17, 8, 1.0f * (mc.lam0));
  sink(17, 17, 1.0f * (mc.lam0 + 2.0f * mc.mu0));
  sink(17, 23, 1.0f * (mc.lam0));
  sink(18, 18, 2.0f * (1.0f * mc.mu0));
  sink(19, 19, 2.0f * (1.0f * mc.mu0));
  sink(20, 20, 2.0f * (1.0f * mc.mu0));
  sink(21, 6, 1.0f * (mc.lam0));
  sink(21, 15, 1.0f * (mc.lam0));
  sink(21, 21, 1.0f * (mc.lam0 + 2.0f * mc.mu0));
  sink(22, 7, 1.0f * (mc.lam0));
  sink(22, 16, 1.0f * (mc.lam0));
  sink(22, 22, 1.0f * (mc.lam0 + 2.0f * mc.mu0));
  sink(23, 8, 1.0f * (mc.lam0));
  sink(23, 17, 1.0f * (mc.lam0));
  sink(23, 23, 1.0f * (mc.lam0 + 2.0f * mc.mu0));
}
