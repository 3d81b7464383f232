// Test harness (CPU): the FP32 pair filter of pcm_filter.cuh over all pairs
// of a group of closures. Loaded by tests/test_pair_filter_cpu.py.
#include <cmath>
#include <vector>

#include "pcm_filter.cuh"

extern "C" {

// out[j * n + i], i < j: 0 inconsistent, 1 consistent, 2 unsure
void pair_filter(int n, const int32_t* sa, const int32_t* sb, const uint8_t* flip, const double* zp,
                 const double* zc, const double* tp, const double* tc, const uint8_t* rot, double th, uint8_t* out) {
  using namespace rpgo::pf;
  std::vector<D2> df((size_t)kPairs * n);
  std::vector<float> f((size_t)kFloats * n);
  std::vector<uint8_t> ok(n);
  for (int k = 0; k < n; ++k) {
    const double *pa = tp + 12 * sa[k], *pb = tp + 12 * sb[k], *ca = tc + 36 * sa[k], *cb = tc + 36 * sb[k];
    const double *z = zp + 12 * k, *c = zc + 36 * k;
    for (int v = 0; v < kPairs; ++v) df[(size_t)v * n + k] = pack_pair(v, pa, ca, pb, cb, z);
    for (int v = 0; v < kFloats; ++v) f[(size_t)v * n + k] = pack_float(v, pa, ca, pb, cb, z, c);
    ok[k] = rot[sa[k]] && rot[sb[k]] && cov_premise(ca, true) && cov_premise(cb, true) && cov_premise(c, false) &&
            pose_premise(pa) && pose_premise(pb) && pose_premise(z);
  }
  const Group g{df.data(), f.data(), ok.data(), n};
  for (int j = 0; j < n; ++j)
    for (int i = 0; i < j; ++i) out[(size_t)j * n + i] = (uint8_t)verdict(g, i, j, flip[i] != flip[j], (float)(th * th));
}
}
