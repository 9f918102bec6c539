// Host build of bem_gmsh_gb300/csrc/fast64.cuh for tests/test_fast64_cpu.py.
#include "../../bem_gmsh_gb300/csrc/bem_crmath.cuh"

extern "C" {
void h_log(const double* x, int n, double* o) { for (int i = 0; i < n; ++i) o[i] = bem::f64::log(x[i]); }
void h_div(const double* a, const double* b, int n, double* o) { for (int i = 0; i < n; ++i) o[i] = bem::f64::div(a[i], b[i]); }
void h_sqrt(const double* x, int n, double* o) { for (int i = 0; i < n; ++i) o[i] = bem::f64::sqrt(x[i]); }
void h_rcp(const double* x, int n, double* o) { for (int i = 0; i < n; ++i) o[i] = bem::f64::rcp(x[i]); }
void h_tan(const double* x, int n, double* o) { for (int i = 0; i < n; ++i) o[i] = bem::crm::cr_tan(x[i]); }
void h_tan_full(const double* x, int n, double* o) { for (int i = 0; i < n; ++i) o[i] = bem::crm::cr_tan_full(x[i]); }
void h_table(double* o) {
  for (int i = 0; i < 129; ++i)
    for (int k = 0; k < 3; ++k) o[3 * i + k] = bem::f64::kLogTab[i][k];
  o[387] = BEM_LN2_HI;
  o[388] = BEM_LN2_LO;
}
}
