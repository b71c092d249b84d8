// Host build of the layout-60 pair product (mf60_contract.cuh) beside the generated dense block.
#include "gen_sphere60.cuh"
#include "mf60_contract.cuh"

struct Put {
  double* M;
  void operator()(int r, int c, double v) const { M[r * 60 + c] += v; }
};

template <class R>
static void apply(const double* x, double as, double ah, const SphMat& mc, const double* e, double* y) {
  R ew[60], a[60];
  for (int i = 0; i < 60; ++i) {
    ew[i] = (R)e[i] * (R)ibem::mf60_weight(i);
    a[i] = R(0);
  }
  const R ia = R(1) / (R)ah, x0 = (R)x[0] * ia, x1 = (R)x[1] * ia, x2 = (R)x[2] * ia;
  const R ir = R(1) / (R)sqrt((double)(x0 * x0 + x1 * x1 + x2 * x2)), nu = R(0.5) * (R)mc.tn2;
  ibem::Mf60Frame<R> f;
  ibem::mf60_frame<R>(x0 * ir, x1 * ir, x2 * ir, f);
  R A0[6], A1[6][3], A2[6][6];
  ibem::mf60_source<R>(f, ew, A0, A1, A2);
  ibem::mf60_rows<0, R>(f, A0, A1, A2, ir, R(1), nu, a);
  ibem::mf60_rows<1, R>(f, A0, A1, A2, ir, ia, nu, a + 6);
  ibem::mf60_rows<2, R>(f, A0, A1, A2, ir, ia * ia, nu, a + 24);
  ibem::mf60_map<0, R>((R)mc.kmu, (R)mc.klam, a);
  ibem::mf60_map<1, R>((R)mc.kmu, (R)mc.klam, a + 6);
  ibem::mf60_map<2, R>((R)mc.kmu, (R)mc.klam, a + 24);
  for (int i = 0; i < 60; ++i) y[i] = (double)(a[i] * (i < 6 ? R(1) : i < 24 ? (R)as : (R)(as * as)));
}

// scaled product of the pair (target radius as, source radius ah, offset x): dense block, and the
// contraction in FP64 and FP32
extern "C" void hg_mf60(const double* x, double as, double ah, double E0, double nu0, double E1, double nu1, const double* e,
                        double* dense, double* y64, double* y32) {
  SphMat mc = sph_mat_init(E0, nu0, E1, nu1);
  mc.kmu /= mc.mu0;
  mc.klam /= mc.mu0;
  double M[3600] = {0};
  Put p{M};
  const double u[3] = {x[0] / ah, x[1] / ah, x[2] / ah};
  sph_block60_c0_r0(u[0], u[1], u[2], 1.0, mc, p);
  sph_block60_c1_r0(u[0], u[1], u[2], 1.0, mc, p);
  sph_block60_c2_r0(u[0], u[1], u[2], 1.0, mc, p);
  sph_block60_c0_r1(u[0], u[1], u[2], 1.0, mc, p);
  sph_block60_c1_r1(u[0], u[1], u[2], 1.0, mc, p);
  sph_block60_c2_r1(u[0], u[1], u[2], 1.0, mc, p);
  sph_block60_c0_r2(u[0], u[1], u[2], 1.0, mc, p);
  sph_block60_c1_r2(u[0], u[1], u[2], 1.0, mc, p);
  sph_block60_c2_r2(u[0], u[1], u[2], 1.0, mc, p);
  for (int r = 0; r < 60; ++r) {
    const double f = r < 6 ? 1.0 : r < 24 ? as / ah : as * as / (ah * ah);
    dense[r] = 0.0;
    for (int c = 0; c < 60; ++c) dense[r] += f * M[r * 60 + c] * e[c];
  }
  apply<double>(x, as, ah, mc, e, y64);
  apply<float>(x, as, ah, mc, e, y32);
}
