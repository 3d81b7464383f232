// Test harness (CPU): the FP32 pair filter of pcm_filter.cuh over all pairs
// of a group of closures, packed as the kernel packs them: positions from the
// group's origins. Loaded by tests/test_pair_filter_origin_cpu.py.
#include <cmath>
#include <vector>

#include "pcm_filter.cuh"

namespace {

template <int DIM>
void run(int n, const int32_t* sa, const int32_t* sb, const uint8_t* flip, const double* zp, const double* zc,
         const double* tp, const double* tc, const uint8_t* rot, double th, uint8_t* out) {
  using namespace rpgo::pf;
  using F = Filter<DIM>;
  constexpr int st = DIM == 3 ? 12 : 4, dd = DIM == 3 ? 36 : 9;
  std::vector<D2> df((size_t)F::pairs * n);
  std::vector<float> f((size_t)F::floats * n);
  std::vector<uint8_t> ok(n);
  for (int k = 0; k < n; ++k) {
    const double *pa = tp + st * sa[k], *pb = tp + st * sb[k], *ca = tc + dd * sa[k], *cb = tc + dd * sb[k];
    const double *z = zp + st * k, *c = zc + dd * k;
    const Origin o = origin(tp + st * sa[0], tp + st * sb[0], flip[k] != flip[0]);
    for (int v = 0; v < F::pairs; ++v) df[(size_t)v * n + k] = F::pair(v, pa, ca, pb, cb, z, o);
    for (int v = 0; v < F::floats; ++v) f[(size_t)v * n + k] = F::single(v, pa, ca, pb, cb, z, c, o);
    ok[k] = rot[sa[k]] && rot[sb[k]] && F::premise(pa, ca, pb, cb, z, c);
  }
  const Group g{df.data(), f.data(), ok.data(), n};
  for (int j = 0; j < n; ++j)
    for (int i = 0; i < j; ++i) out[(size_t)j * n + i] = (uint8_t)F::test(g, i, j, flip[i] != flip[j], (float)(th * th));
}

}  // namespace

extern "C" {

// out[j * n + i], i < j: 0 inconsistent, 1 consistent, 2 unsure
void pair_filter(int dim, int n, const int32_t* sa, const int32_t* sb, const uint8_t* flip, const double* zp,
                 const double* zc, const double* tp, const double* tc, const uint8_t* rot, double th, uint8_t* out) {
  if (dim == 3) run<3>(n, sa, sb, flip, zp, zc, tp, tc, rot, th, out);
  else run<2>(n, sa, sb, flip, zp, zc, tp, tc, rot, th, out);
}
}

extern "C" {

// the verdict from the sums of a pair (pcm_filter.cuh, decide)
int pair_decide(float d2, float yx, float yCy, float py, float ey, float ph, float eh, float eta, float th2) {
  return rpgo::pf::decide(d2, yx, yCy, py, ey, ph, eh, eta, th2);
}
}
