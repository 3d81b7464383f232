// Test harness (CPU): the FP32 log map of pcm_filter.cuh, one pose at a time.
// Loaded by tests/test_pair_filter_logmap_cpu.py.
#include <cmath>

#include "pcm_filter.cuh"

extern "C" {

// n poses (R row-major, t): the log maps xi[6 n], the bounds of their rotation
// and translation entries e[2 n], and whether each is certain
void pair_logmap(int n, const double* pose, float* xi, float* e, unsigned char* ok) {
  using namespace rpgo::pf;
  for (int k = 0; k < n; ++k) {
    Pose p;
    for (int i = 0; i < 9; ++i) p.R[i] = split(pose[12 * k + i]);
    for (int i = 0; i < 3; ++i) p.t[i] = split(pose[12 * k + 9 + i]);
    float x[6];
    ok[k] = logmap(p, x, e[2 * k], e[2 * k + 1]);
    for (int i = 0; i < 6; ++i) xi[6 * k + i] = x[i];
  }
}
}
