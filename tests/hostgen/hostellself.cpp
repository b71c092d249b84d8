// Host build of an ellipsoid's own block by the two routes (ellipsoid.cuh, ellipsoid_ext.cuh).
#include "ellipsoid.cuh"

using namespace ibem::ell;

extern "C" int he_self24(const double* quat, const double* a, double nu0, double* general, double* ext) {
  const double d[3] = {0.0, 0.0, 0.0};
  double Q[9], M[kRotSize];
  quat_to_rot(quat, Q);
  rot_matrices(Q, M);
  const SphMat mc = sph_mat_init(70e9, nu0, 400e9, 0.2);
  ell_block24_any<double>(d, Q, a, mc, true, general);
  if (!ell_block24_ext<double>(d, Q, a, M, mc, ext)) return 0;
  ell_self_add(mc, ext);
  return 1;
}
