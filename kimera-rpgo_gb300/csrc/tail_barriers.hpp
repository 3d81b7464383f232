// Order of the named barriers in the one-CTA factorisation of the dense tail
// (df_tail in chol_kernels.cu), apart from the arithmetic, so that a CPU model
// can run it in every order of the warps (tests/native/tail_barriers.cpp).
//
// The lead warp scales column c and publishes it: it arrives at published(c),
// where the other warps wait. They subtract column c from the columns behind
// it and arrive at subtracted(c), where the lead waits one column later.
// A barrier's phase takes one arrival of each warp, so no warp may come to a
// barrier again before all the others have come to the phase before. Each of
// the two has two barriers, taken in turn:
//  * the lead comes to published(c + 2) after its wait at subtracted(c), and
//    every other warp came there after it had left published(c);
//  * another warp comes to subtracted(c + 2) after published(c + 2), and the
//    lead came there after it had left subtracted(c).
// With one barrier for all published columns the lead could arrive for column
// c + 1 while a late warp had yet to come for column c: the phase would be
// complete without that warp, which then waits for an arrival that cannot come.
// A warp has to be converged at each.
#pragma once

#ifdef __CUDACC__
#define RPGO_TAIL_FN __device__ __forceinline__
#else
#define RPGO_TAIL_FN inline
#endif

namespace rpgo {

RPGO_TAIL_FN constexpr int tail_published(int c) { return (c & 1) ? 6 : 3; }
RPGO_TAIL_FN constexpr int tail_subtracted(int c) { return (c & 1) ? 5 : 4; }

// the lead: scale(c), then, with every column before c subtracted, next(c)
template <class Barriers, class Scale, class Next>
RPGO_TAIL_FN void tail_lead(int n, Barriers& b, Scale scale, Next next) {
  for (int c = 0; c < n; ++c) {
    scale(c);
    b.arrive(tail_published(c));
    if (c > 0) b.wait(tail_subtracted(c - 1));
    next(c);
  }
  b.wait(tail_subtracted(n - 1));
}
// every other warp
template <class Barriers, class Subtract>
RPGO_TAIL_FN void tail_follow(int n, Barriers& b, Subtract subtract) {
  for (int c = 0; c < n; ++c) {
    b.wait(tail_published(c));
    subtract(c);
    b.arrive(tail_subtracted(c));
  }
}

}  // namespace rpgo
