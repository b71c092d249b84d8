// Host build of the boundary kernels' pair functions (bem_moments.cuh, bem_contract.cuh) beside
// the generated stress kernels.
#include "bem_contract.cuh"
#include "bem_moments.cuh"
#include "gen_bem.cuh"

struct Mom {
  const double* M;
  double operator()(int c, int i) const { return M[4 * i + c]; }
};

// one Gauss point of weight 1 at offset x with normal nv: rows of order 0 (6), 1 (6 + 3 t + w)
// and 2 (24 + 6 t + pair), three dofs each
extern "C" void hb_entries(const double* x, const double* nv, double E0, double nu0, double E1, double nu1, double* su,
                           double* st) {
  const BemMat bm = bem_mat_init(E0, nu0, E1, nu1);
  double M[74 * 4];
  const double ir = 1.0 / sqrt(x[0] * x[0] + x[1] * x[1] + x[2] * x[2]);
  ibem::bmo_derivatives<6>(x[0], x[1], x[2], ir, [&](int i, double v) {
    M[4 * i] = v;
    for (int m = 0; m < 3; ++m) M[4 * i + 1 + m] = v * nv[m];
  });
  const ibem::BmoEntries<Mom> en{Mom{M}, bm.kA, bm.kB, bm.lam0, bm.mu0, bm.dlam, bm.dmu};
  const int pi[6] = {0, 0, 0, 1, 1, 2}, pj[6] = {0, 1, 2, 1, 2, 2};
  for (int t = 0; t < 6; ++t)
    for (int n = 0; n < 3; ++n) {
      en.entry(pi[t], pj[t], 0, 0, n, st[3 * t + n], su[3 * t + n]);
      for (int w = 0; w < 3; ++w) {
        const int r = 3 * (6 + 3 * t + w) + n;
        en.entry(pi[t], pj[t], 1, ibem::bmo_e(w), n, st[r], su[r]);
      }
      for (int q = 0; q < 6; ++q) {
        const int r = 3 * (24 + 6 * t + q) + n;
        en.entry(pi[t], pj[t], 2, ibem::bmo_e(pi[q]) + ibem::bmo_e(pj[q]), n, st[r], su[r]);
      }
    }
}

// stress at p of one Gauss point (record r of 13): per-pair form times the weight, and the summed form
extern "C" void hb_post(const double* p, const double* r, double E0, double nu0, double E1, double nu1, double* pair,
                        double* summed) {
  const BemPostCoef c = bem_post_coef(bem_mat_init(E0, nu0, E1, nu1));
  bem_post_contracted(r[0] - p[0], r[1] - p[1], r[2] - p[2], r[3], r[4], r[5], r[7], r[8], r[9], r[10], r[11], r[12], c, pair);
  double acc[6] = {0, 0, 0, 0, 0, 0};
  bem_post_add(p[0], p[1], p[2], bem_post_rec(r, c), c, acc);
  for (int q = 0; q < 6; ++q) {
    pair[q] *= r[6];
    summed[q] = bem_post_value(acc, q);
  }
}
