// The conversions of csrc/pair_arith.cuh on the host.
#include "../pynfam_gb300/csrc/pair_arith.cuh"

using namespace pnfam;

extern "C" void pair_host_check(int n, const double* x, const float* y, int s, float* hi, float* lo, float* f, double* d,
                                int* scale) {
  for (int i = 0; i < n; ++i) {
    const float2 p = pair_split(x[i], s);
    hi[i] = p.x;
    lo[i] = p.y;
    f[i] = f32_of(x[i]);
    d[i] = f64_of(y[i], s);
    scale[i] = pair_scale(x[i] < 0 ? -x[i] : x[i]);
  }
}
extern "C" unsigned long long pair_host_max(int n, const double* x) {
  unsigned long long m = 0;
  for (int i = 0; i < n; ++i) m = abs_max(m, x[i]);
  return m;
}
