// The layout of the unit sums (csrc/separable.cuh) on the host.
#include "../pynfam_gb300/csrc/separable.cuh"

// places: gpair[0], gpair[1], values of a point, values of an F unit
extern "C" void sep_layout_check(long long ngl, const long long* nu, long long* places) {
  long long gpair[2];
  places[2] = pnfam::sep_sums(ngl, nu, gpair);
  places[0] = gpair[0];
  places[1] = gpair[1];
  places[3] = 2 * pnfam::SH_N;
}
