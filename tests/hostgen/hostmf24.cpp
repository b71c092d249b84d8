// Host build of the layout-24 raw pair contraction (mf_contract.cuh) in double-float numbers.
#include "mf_contract.cuh"

extern "C" void hm_raw24(int df, const double* x, double f, const double* coef, double row_scale, double* y) {
  constexpr ibem::MfRecTab tab = ibem::mf_rec_tab();
  if (df) {
    using ibem::DF;
    DF c[25], a[24];
    alignas(16) DF rec[ibem::kRecLen];
    for (int i = 0; i < 24; ++i) c[i] = DF(coef[i]);
    for (int e = 0; e < ibem::kRecLen; ++e) rec[e] = ibem::mf_rec_entry(tab.v[e], c);
    ibem::sph_pair_raw24<DF>(DF(x[0]), DF(x[1]), DF(x[2]), DF(f), rec, DF(row_scale), a);
    for (int i = 0; i < 24; ++i) y[i] = ibem::df_value(a[i]);
  } else {
    double c[25] = {}, a[24] = {};
    alignas(16) double rec[ibem::kRecLen];
    for (int i = 0; i < 24; ++i) c[i] = coef[i];
    for (int e = 0; e < ibem::kRecLen; ++e) rec[e] = ibem::mf_rec_entry(tab.v[e], c);
    ibem::sph_pair_raw24<double>(x[0], x[1], x[2], f, rec, row_scale, a);
    for (int i = 0; i < 24; ++i) y[i] = a[i];
  }
}
