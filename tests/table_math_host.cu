// Test harness: the FP64 table-driven exponential and logarithm, compiled for the host,
// for tests/test_table_math_host.py.  Not part of the library.
#include "../braincell_gb300/csrc/bc_mech.cuh"

extern "C" void bc_test_exp2_256(const double* y, int n, double* out) {
  for (int i = 0; i < n; ++i) out[i] = bc::exp2_256(y[i]);
}
extern "C" void bc_test_ln(const double* x, int n, double* out) {
  for (int i = 0; i < n; ++i) out[i] = bc::ln_pos(x[i]);
}
extern "C" void bc_test_line(const double* v, int n, double* out) {
  constexpr bc::ExpLine e(-1.0, -59.0, 6.2);
  for (int i = 0; i < n; ++i) out[i] = bc::lin_exp(v[i], e);
}
extern "C" void bc_test_bell(const double* v, int n, double* out) {
  constexpr bc::ExpLine e(-1.0, 0.0, 9.5);
  for (int i = 0; i < n; ++i) out[i] = bc::exp_neg_abs(v[i], e);
}
