// Host build of the two routes of the ellipsoid pair block (ellipsoid.cuh, ellipsoid_ext.cuh).
#include "ellipsoid.cuh"

using namespace ibem::ell;

extern "C" int hx_block24(const double* d, const double* quat, const double* a, double nu0, double* general, double* ext) {
  double Q[9], M[kRotSize];
  quat_to_rot(quat, Q);
  rot_matrices(Q, M);
  const SphMat mc = sph_mat_init(70e9, nu0, 400e9, 0.2);
  ell_block24_any<double>(d, Q, a, mc, false, general);
  return ell_block24_ext<double>(d, Q, a, M, mc, ext) ? 1 : 0;
}

// the integrals I_k by quadrature (kappa_max given) and by Carlson's algorithm
extern "C" void hx_ik(const double* x, double kmax, double* quad, double* carlson) {
  EllSeries<double> S;
  ell_series<double>(x, kmax, S);
  for (int i = 0; i < 20; ++i) quad[i] = S.c[i][0];
  carlson_ik<double>(x, carlson);
}
