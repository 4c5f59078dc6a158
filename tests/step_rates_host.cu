// Test harness: the FP64 step forms of the main mix's gates and the decay series,
// compiled for the host, for tests/test_step_rates_host.py.  Not part of the library.
#include "../braincell_gb300/csrc/bc_mech.cuh"

using namespace bc;

// Step form `which` at n voltages: out[4 i ..] = its steady state and exponent with
// k = -1, then the rate structure's steady state and -1 / tau.
extern "C" int bc_test_step_rates(int which, const double* v, int n, double* out) {
  for (int i = 0; i < n; ++i) {
    const double x = v[i];
    GateStep<double> g{};
    double inf = 0.0, tau = 1.0;
    const CaLRates<double> l(x, 0.0);
    const CaTRates<double> t(x, 0.0);
    const HcnRates<double> h(x);
    switch (which) {
      case 0: g = cal_p_step(x, -1.0); inf = l.pinf; tau = l.ptau; break;
      case 1: g = cal_q_step(x, -1.0); inf = l.qinf; tau = l.qtau; break;
      case 2: g = cat_p_step(x, -1.0); inf = t.pinf; tau = t.ptau; break;
      case 3: g = cat_q_step(x, -1.0); inf = t.qinf; tau = t.qtau; break;
      case 4: g = hcn_step(x, -1.0); inf = h.pinf; tau = h.ptau; break;
      default: return -1;
    }
    out[4 * i] = g.inf;
    out[4 * i + 1] = g.x;
    out[4 * i + 2] = inf;
    out[4 * i + 3] = -1.0 / tau;
  }
  return 0;
}

extern "C" void bc_test_decay(const double* x, int n, double* out) {
  for (int i = 0; i < n; ++i) out[i] = decay_em1(x[i]);
}
