// Decides most pairwise consistency tests of uncertain poses (3D, 2D)
// (Pcm::areLoopsConsistent, include/KimeraRPGO/outlier/Pcm.h:670-718) in FP32
// arithmetic, with a bound on its own error; the rest is left to the exact
// FP64 test of pcm_kernels.cu. Host and device code: the tests run it on the
// CPU against the exact verdicts.
//
// What the exact test computes is d = |Logmap(loop)| in the metric of the
// loop's covariance, compared with a threshold. Its operations only matter
// through their rounding errors, so the verdict is known as soon as d, known
// to within E, is further than E from the threshold. Some things are decided
// on the way: which of its two formulas each `between` takes (a positive
// definiteness test, GeometryUtils.h:143-170), which formula the logarithm
// takes, and the sign of the axis of a rotation by nearly pi. Where any of them
// is not certain, or a bound's premise fails (NaN, an asymmetric trajectory
// covariance, a correlation beyond 1, no rotation information, values near the
// limits of FP32, a loop covariance not certain to be positive definite), the
// pair is unsure.
//
// Precision. Covariances along the odometry grow with the square of the
// distance travelled, and `between` subtracts two of them, so `between` and
// the pose chain run in pairs of FP32 (high + low, about 2^-46): their error
// is at most kDf q_i q_j in entry (i, j), q from the magnitudes of what was
// subtracted. All later covariances are sums of congruences without
// cancellation and run in FP32: their error in entry (i, j) is at most
// eps p_i p_j, with p the vector of magnitudes carried through |Ad|. With the
// final covariance C, x the loop's log map (error e_i) and any y,
//   d^2 >= 2 y.x - y^T C y - eps (sum p_i |y_i|)^2 - 2 sum e_i |y_i|,
// taken at C y = x, where it is close to d^2; both with C's error relative to C
// itself, kap = eps (sum p_i sqrt(C^-1_ii))^2, below 1 (else unsure), and
//   d <= (computed d + sum e_i sqrt(C^-1_ii)) / sqrt(1 - kap),
// or, for kap <= 1/8, the lower bound's terms 1.5 times above the computed d^2.
#pragma once
#include <cmath>
#include <cstdint>

#ifdef __CUDACC__
#define RPGO_HD __host__ __device__ __forceinline__
#else
#define RPGO_HD inline
#endif

namespace rpgo {
namespace pf {

// ------------------------------------------------------------------ FP32 operations, never contracted
RPGO_HD float fadd(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fadd_rn(a, b);
#else
  return a + b;
#endif
}
RPGO_HD float fsub(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fsub_rn(a, b);
#else
  return a - b;
#endif
}
RPGO_HD float fmulf(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fmul_rn(a, b);
#else
  return a * b;
#endif
}
RPGO_HD float ffma(float a, float b, float c) {
#ifdef __CUDA_ARCH__
  return __fmaf_rn(a, b, c);
#else
  return std::fmaf(a, b, c);
#endif
}
RPGO_HD float fdvd(float a, float b) {
#ifdef __CUDA_ARCH__
  return __fdiv_rn(a, b);
#else
  return a / b;
#endif
}
RPGO_HD float fsqr(float a) {
#ifdef __CUDA_ARCH__
  return __fsqrt_rn(a);
#else
  return std::sqrt(a);
#endif
}
RPGO_HD float fabsv(float a) { return a < 0.f ? -a : a; }  // (NaN stays NaN)

constexpr float kU = 5.9604644775390625e-8f;      // 2^-24
// 2^-38: 2.4 times what about 420 roundings of 2^-48, the longest way into an
// entry of a `between`, add up to if each is as bad as can be. Worst of 400,000
// random ones against 64-bit significands: 0.006 of the bound.
constexpr float kDf = 3.637978807091713e-12f;
// A difference of two positions has an error of at most kDt (|t_a| + |t_c|)
// (1-norms): 2^-48 of each from its pair, 2^-46 from the subtraction in pairs.
// It moves the covariances through their lever arms: by kDt (|t_a| + |t_c|)
// times what the lever's length multiplies. With the lever's magnitude written as
// u + kLever (|t_a| + |t_c|), u the difference itself, half of kDf q_i q_j covers
// it (kDf's own roundings take 1 / 2.4); in compositions in FP32, 4 of the 64
// units of decide(), of which the roundings take 58.
constexpr float kDt = 2.842170943040401e-14f;         // 2^-45
constexpr float kLever = 0.015625f;                   // 2 kDt / kDf
constexpr float kLeverFp32 = 1.1920928955078125e-7f;  // 2^22 kDt

// ------------------------------------------------------------------ FP32 pairs
struct alignas(8) D2 {
  float h, l;
};
RPGO_HD D2 split(double x) {
  const float h = (float)x;
  return D2{h, (float)(x - (double)h)};
}
RPGO_HD D2 neg(D2 a) { return D2{-a.h, -a.l}; }
// running sum of products: s + c with the low parts collected in c
struct Acc {
  float s, c;
};
RPGO_HD Acc acc_mul(D2 a, D2 b) {
  const float p = fmulf(a.h, b.h);
  float e = ffma(a.h, b.h, -p);
  e = ffma(a.h, b.l, e);
  e = ffma(a.l, b.h, e);
  return Acc{p, e};
}
RPGO_HD void acc_two_sum(Acc& x, float p, float e) {
  const float s = fadd(x.s, p);
  const float b = fsub(s, x.s);
  const float err = fadd(fsub(x.s, fsub(s, b)), fsub(p, b));
  x.c = fadd(x.c, fadd(err, e));
  x.s = s;
}
RPGO_HD void acc_fma(Acc& x, D2 a, D2 b) {
  const Acc m = acc_mul(a, b);
  acc_two_sum(x, m.s, m.c);
}
RPGO_HD void acc_add(Acc& x, D2 a) { acc_two_sum(x, a.h, a.l); }
RPGO_HD D2 norm(const Acc& x) {
  const float h = fadd(x.s, x.c);
  return D2{h, fsub(x.c, fsub(h, x.s))};
}
// the same names for the two number types of the congruence below
RPGO_HD D2 dot3(D2 a0, D2 a1, D2 a2, D2 b0, D2 b1, D2 b2) {
  Acc x = acc_mul(a0, b0);
  acc_fma(x, a1, b1);
  acc_fma(x, a2, b2);
  return norm(x);
}
// v + a b - c d
RPGO_HD D2 cross1(D2 v, D2 a, D2 b, D2 c, D2 d) {
  Acc x{v.h, v.l};
  acc_fma(x, a, b);
  acc_fma(x, neg(c), d);
  return norm(x);
}
RPGO_HD D2 sub(D2 a, D2 b) {
  Acc x{a.h, a.l};
  acc_add(x, neg(b));
  return norm(x);
}
RPGO_HD float dot3(float a0, float a1, float a2, float b0, float b1, float b2) {
  return ffma(a2, b2, ffma(a1, b1, fmulf(a0, b0)));
}
RPGO_HD float cross1(float v, float a, float b, float c, float d) { return ffma(-c, d, ffma(a, b, v)); }
RPGO_HD float lo(D2 a) { return a.h; }

// ------------------------------------------------------------------ per-closure data
// One closure's trajectory entries and measurement, structure of arrays over
// the closures of a group: value v of closure k is at [v * n + k].
constexpr int kPairs = 78;   // FP32 pairs: pose a (R, t), cov a (lower), pose b, cov b, measured pose
constexpr int kFloats = 44;  // FP32: inverse measurement's t (3), its covariance (21), sqrt of its diagonal (6),
                             // sqrt of the diagonals of cov a and cov b (6 each), |t_a|, |t_b| (1-norms, from the
                             // group's origins)
constexpr int kPoseA = 0, kCovA = 12, kPoseB = 33, kCovB = 45, kPoseZ = 66;
constexpr int kZt = 0, kZc = 3, kZg = 24, kGA = 30, kGB = 36, kTA = 42, kTB1 = 43;
RPGO_HD constexpr int tri(int i, int j) { return i * (i + 1) / 2 + j; }  // j <= i
RPGO_HD int tri_full(int e) {  // lower-triangle entry e as an index of the full 6 x 6
  int i = 0;
  while (e > i) e -= ++i;
  return 6 * i + e;
}

struct Group {
  const D2* df;
  const float* f;
  const uint8_t* ok;
  int n;
};
struct Item {
  const D2* df;
  const float* f;
  int n;
  RPGO_HD D2 d(int v) const { return df[(size_t)v * n]; }
  RPGO_HD float g(int v) const { return f[(size_t)v * n]; }
};
RPGO_HD Item item(const Group& g, int k) { return Item{g.df + k, g.f + k, g.n}; }

// Where a group's poses are measured from. A verdict depends on differences
// of positions only, so the bounds need not grow with the distance of the map
// from its frame's origin (a new robot's first pose can be anywhere, in metres
// of a map grid for instance). A pair compares entries of one side of closure 0
// with each other: the side of a closure that lies on side a (b) of closure 0
// is measured from that endpoint of closure 0, flipped closures the other way
// round. The subtraction is the one rounding that this adds, 2^-53 of the
// result.
struct Origin {
  const double *a, *b;  // the poses whose positions endpoints a and b are measured from; null: the frame's
};
RPGO_HD double from_origin(double x, const double* origin, int at) {
  if (!origin) return x;
  const double o = origin[at];
  return std::fabs(o) < 1e12 ? x - o : x;  // (NaN: as it is)
}
// value v of a closure from its trajectory entries (pose 12, covariance 36)
// and measurement (pose 12)
RPGO_HD D2 pack_pair(int v, const double* pa, const double* ca, const double* pb, const double* cb,
                     const double* zp, Origin o = {nullptr, nullptr}) {
  if (v < kCovA) return split(v < 9 ? pa[v] : from_origin(pa[v], o.a, v));
  if (v < kPoseB) return split(ca[tri_full(v - kCovA)]);
  if (v < kCovB) return split(v < kPoseB + 9 ? pb[v - kPoseB] : from_origin(pb[v - kPoseB], o.b, v - kPoseB));
  if (v < kPoseZ) return split(cb[tri_full(v - kCovB)]);
  return split(zp[v - kPoseZ]);
}
RPGO_HD float pack_float(int v, const double* pa, const double* ca, const double* pb, const double* cb,
                         const double* zp, const double* zc, Origin o = {nullptr, nullptr}) {
  if (v < kZc) return (float)-(zp[v] * zp[9] + zp[3 + v] * zp[10] + zp[6 + v] * zp[11]);
  if (v < kZg) return (float)zc[tri_full(v - kZc)];
  if (v < kGA) return fsqr((float)zc[7 * (v - kZg)]);
  if (v < kGB) return fsqr((float)ca[7 * (v - kGA)]);
  if (v < kTA) return fsqr((float)cb[7 * (v - kGB)]);
  const double *p = v == kTA ? pa : pb, *q = v == kTA ? o.a : o.b;
  return (float)(std::fabs(from_origin(p[9], q, 9)) + std::fabs(from_origin(p[10], q, 10)) +
                 std::fabs(from_origin(p[11], q, 11)));
}
// the premises of the bounds on one covariance: symmetric (the exact test
// reads all of a trajectory covariance), |S_kl| <= sqrt(S_kk S_ll), inside
// the range of FP32
RPGO_HD bool cov_premise(const double* c, bool whole) {
  bool ok = true;
  for (int i = 0; i < 6; ++i)
    for (int j = 0; j <= i; ++j) {
      const double x = c[6 * i + j], b = c[7 * i] * c[7 * j];
      ok = ok && x * x <= 1.0001 * b && (!whole || c[6 * j + i] == x) && c[7 * i] >= 0.0 && c[7 * i] < 1e15;
    }
  return ok;
}
RPGO_HD bool pose_premise(const double* p) {
  bool ok = true;
  for (int e = 0; e < 9; ++e) ok = ok && std::fabs(p[e]) <= 1.00001;
  for (int e = 9; e < 12; ++e) ok = ok && std::fabs(p[e]) < 1e12;
  return ok;
}

// ------------------------------------------------------------------ covariances
// A symmetric 6 x 6 covariance as blocks: rr (lower 6), tr (9), tt (lower 6).
template <class T>
struct Cov {
  T rr[6], tr[9], tt[6];
};
// R B R^T of a symmetric block (lower triangles)
template <class T>
RPGO_HD void rot_sym(const T* R, const T* B, T* C) {
  T M[9];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    M[3 * i] = dot3(R[3 * i], R[3 * i + 1], R[3 * i + 2], B[0], B[1], B[3]);
    M[3 * i + 1] = dot3(R[3 * i], R[3 * i + 1], R[3 * i + 2], B[1], B[2], B[4]);
    M[3 * i + 2] = dot3(R[3 * i], R[3 * i + 1], R[3 * i + 2], B[3], B[4], B[5]);
  }
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j <= i; ++j)
      C[tri(i, j)] = dot3(M[3 * i], M[3 * i + 1], M[3 * i + 2], R[3 * j], R[3 * j + 1], R[3 * j + 2]);
}
template <class T>
RPGO_HD void rot_full(const T* R, const T* B, T* C) {
  T M[9];
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      M[3 * i + j] = dot3(R[3 * i], R[3 * i + 1], R[3 * i + 2], B[j], B[3 + j], B[6 + j]);
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      C[3 * i + j] = dot3(M[3 * i], M[3 * i + 1], M[3 * i + 2], R[3 * j], R[3 * j + 1], R[3 * j + 2]);
}
RPGO_HD constexpr int sym(int i, int j) { return i >= j ? tri(i, j) : tri(j, i); }
// Ad S Ad^T for Ad = [[R, 0], [[t]x R, R]]: both blocks rotated, then sheared
// by t (186 products instead of the 261 of the two 6 x 6 products)
template <class T>
RPGO_HD void congruence(const T* R, const T* t, const Cov<T>& S, Cov<T>& C) {
  rot_sym(R, S.rr, C.rr);
  T tr[9], tt[6];
  rot_full(R, S.tr, tr);
  rot_sym(R, S.tt, tt);
  // C_tr = tr + [t]x rr
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    C.tr[j] = cross1(tr[j], t[1], C.rr[sym(2, j)], t[2], C.rr[sym(1, j)]);
    C.tr[3 + j] = cross1(tr[3 + j], t[2], C.rr[sym(0, j)], t[0], C.rr[sym(2, j)]);
    C.tr[6 + j] = cross1(tr[6 + j], t[0], C.rr[sym(1, j)], t[1], C.rr[sym(0, j)]);
  }
  // C_tt = tt + [t]x tr^T + C_tr [t]x^T
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j <= i; ++j) {
      const int a = (i + 1) % 3, b = (i + 2) % 3, p = (j + 1) % 3, q = (j + 2) % 3;
      const T v = cross1(tt[tri(i, j)], t[a], tr[3 * j + b], t[b], tr[3 * j + a]);
      C.tt[tri(i, j)] = cross1(v, t[p], C.tr[3 * i + q], t[q], C.tr[3 * i + p]);
    }
}
// entry (i, j), j <= i, of a covariance
template <class T>
RPGO_HD T entry(const Cov<T>& S, int i, int j) {
  return i < 3 ? S.rr[tri(i, j)] : (j < 3 ? S.tr[3 * (i - 3) + j] : S.tt[tri(i - 3, j - 3)]);
}

// LDL^T of a covariance in FP32: L and L^-1 (unit lower, below the diagonal,
// row by row) in L and W, reciprocal pivots in iD, the diagonal of C^-1 in h;
// false when a pivot is not positive
RPGO_HD bool factor(const Cov<float>& S, float (&L)[15], float (&W)[15], float (&iD)[6], float (&h)[6]) {
  bool ok = true;
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    float e[6];
#pragma unroll
    for (int j = 0; j < i; ++j) {
      float acc = entry(S, i, j);
#pragma unroll
      for (int k = 0; k < j; ++k) acc = ffma(-e[k], L[j * (j - 1) / 2 + k], acc);
      e[j] = acc;
      L[i * (i - 1) / 2 + j] = fmulf(acc, iD[j]);
    }
    float acc = entry(S, i, i);
#pragma unroll
    for (int k = 0; k < i; ++k) acc = ffma(-e[k], L[i * (i - 1) / 2 + k], acc);
    ok = ok && acc > 0.f;
    iD[i] = fdvd(1.f, acc);
  }
#pragma unroll
  for (int i = 1; i < 6; ++i)
#pragma unroll
    for (int j = i - 1; j >= 0; --j) {
      float acc = -L[i * (i - 1) / 2 + j];
#pragma unroll
      for (int k = j + 1; k < i; ++k) acc = ffma(-L[i * (i - 1) / 2 + k], W[k * (k - 1) / 2 + j], acc);
      W[i * (i - 1) / 2 + j] = acc;
    }
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    h[i] = iD[i];
#pragma unroll
    for (int k = i + 1; k < 6; ++k) {
      const float w = W[k * (k - 1) / 2 + i];
      h[i] = ffma(fmulf(w, w), iD[k], h[i]);
    }
  }
  return ok;
}

// ------------------------------------------------------------------ poses
struct Pose {
  D2 R[9], t[3];
};
RPGO_HD void load_pose(const Item& x, int v, Pose& p) {
#pragma unroll
  for (int e = 0; e < 9; ++e) p.R[e] = x.d(v + e);
#pragma unroll
  for (int e = 0; e < 3; ++e) p.t[e] = x.d(v + 9 + e);
}
RPGO_HD void compose(const Pose& A, const Pose& B, Pose& C) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
#pragma unroll
    for (int j = 0; j < 3; ++j)
      C.R[3 * i + j] = dot3(A.R[3 * i], A.R[3 * i + 1], A.R[3 * i + 2], B.R[j], B.R[3 + j], B.R[6 + j]);
    Acc x{A.t[i].h, A.t[i].l};
    acc_fma(x, A.R[3 * i], B.t[0]);
    acc_fma(x, A.R[3 * i + 1], B.t[1]);
    acc_fma(x, A.R[3 * i + 2], B.t[2]);
    C.t[i] = norm(x);
  }
}
// -R^T t
RPGO_HD void inverse_t(const D2* R, const D2* t, D2* o) {
#pragma unroll
  for (int i = 0; i < 3; ++i) o[i] = neg(dot3(R[i], R[3 + i], R[6 + i], t[0], t[1], t[2]));
}

// The covariance of `between` of two trajectory entries (endpoint va / ga /
// ta of item x, endpoint vc / gc / tc of item y; v*: pose's first value), its
// error eta (relative to s_i s_j) and the square roots s of its diagonal;
// pose = x^-1 y. False when the formula that the exact test takes, or the
// bound, is not certain.
RPGO_HD bool between(const Item& x, int va, int ga, int ta, const Item& y, int vc, int gc, int tc, Pose& pose,
                     Cov<float>& S, float (&s)[6], float& eta) {
  Pose A, B;
  load_pose(x, va, A);
  load_pose(y, vc, B);
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j)
      pose.R[3 * i + j] = dot3(A.R[i], A.R[3 + i], A.R[6 + i], B.R[j], B.R[3 + j], B.R[6 + j]);
  D2 dt[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) dt[i] = sub(B.t[i], A.t[i]);
#pragma unroll
  for (int i = 0; i < 3; ++i) pose.t[i] = dot3(A.R[i], A.R[3 + i], A.R[6 + i], dt[0], dt[1], dt[2]);
  // the main formula's first pivot: cov_y(0, 0) - r^T cov_x,rr r with r the
  // first column of pose.R; the test fails at once when it is negative
  float gr = 0.f, gt = 0.f, hr = 0.f, ht = 0.f;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    gr = fadd(gr, x.g(ga + i));
    gt = fadd(gt, x.g(ga + 3 + i));
    hr = fadd(hr, y.g(gc + i));
    ht = fadd(ht, y.g(gc + 3 + i));
  }
  const float qr = fadd(gr, hr);
  bool main, known;
  {
    D2 c[6];
#pragma unroll
    for (int e = 0; e < 6; ++e) c[e] = x.d(va + 12 + e);
    const D2 r0 = pose.R[0], r1 = pose.R[3], r2 = pose.R[6];
    const D2 m0 = dot3(r0, r1, r2, c[0], c[1], c[3]), m1 = dot3(r0, r1, r2, c[1], c[2], c[4]),
             m2 = dot3(r0, r1, r2, c[3], c[4], c[5]);
    const D2 piv = sub(y.d(vc + 12), dot3(m0, m1, m2, r0, r1, r2));
    const float e = fmulf(kDf, fmulf(qr, qr));
    main = piv.h > e;
    known = main || piv.h < -e;
  }
  // X -> Y: cov_Y - Ad cov_X Ad^T with Ad of (X^-1 Y)^-1; main: X = x
  const Item& X = main ? x : y;
  const Item& Y = main ? y : x;
  const int vX = main ? va : vc, vY = main ? vc : va;
  D2 R[9], t[3];
  {
    D2 tr[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const D2 b = dot3(B.R[i], B.R[3 + i], B.R[6 + i], neg(dt[0]), neg(dt[1]), neg(dt[2]));
      tr[i] = main ? pose.t[i] : b;
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) R[3 * i + j] = main ? pose.R[3 * j + i] : pose.R[3 * i + j];
#pragma unroll
    for (int i = 0; i < 3; ++i) t[i] = neg(dot3(R[3 * i], R[3 * i + 1], R[3 * i + 2], tr[0], tr[1], tr[2]));
  }
  Cov<D2> C;
  {
    Cov<D2> SX;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j <= i; ++j) {
        SX.rr[tri(i, j)] = X.d(vX + 12 + tri(i, j));
        SX.tt[tri(i, j)] = X.d(vX + 12 + tri(i + 3, j + 3));
      }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) SX.tr[3 * i + j] = X.d(vX + 12 + tri(i + 3, j));
    congruence(R, t, SX, C);
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
#pragma unroll
    for (int j = 0; j <= i; ++j) {
      S.rr[tri(i, j)] = lo(sub(Y.d(vY + 12 + tri(i, j)), C.rr[tri(i, j)]));
      S.tt[tri(i, j)] = lo(sub(Y.d(vY + 12 + tri(i + 3, j + 3)), C.tt[tri(i, j)]));
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) S.tr[3 * i + j] = lo(sub(Y.d(vY + 12 + tri(i + 3, j)), C.tr[3 * i + j]));
  }
  // the magnitudes that were subtracted, |R| taken as all ones (kLever: the
  // error of the difference of the positions)
  const float lever =
      fadd(fadd(fabsv(t[0].h), fabsv(t[1].h)), ffma(kLever, fadd(x.g(ta), y.g(tc)), fabsv(t[2].h)));
  const float qt = ffma(lever, qr, fadd(gt, ht));
  float L[15], W[15], iD[6], h[6];
  bool ok = factor(S, L, W, iD, h) && known;
  float vr = entry(S, 0, 0), vt = entry(S, 3, 3), sum = 0.f;
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    const float v = entry(S, i, i);
    ok = ok && v > 1e-24f;
    s[i] = fsqr(v);
    if (i < 3) vr = v < vr ? v : vr;
    else vt = v < vt ? v : vt;
    sum = fadd(sum, fsqr(fmulf(v, h[i])));
  }
  const float er = fdvd(fmulf(qr, qr), vr), et = fdvd(fmulf(qt, qt), vt);
  eta = ffma(kDf, er > et ? er : et, 16.f * kU);
  // every matrix within eta is positive definite: the formula is certain, and
  // |S_ij| <= s_i s_j to within the same
  return ok && fmulf(eta, fmulf(sum, sum)) < 0.5f;
}

// what the callers of verdict() do between its phases: nothing, or a barrier
// of the block, so that its warps fetch the code of a phase together
struct NoSync {
  RPGO_HD void operator()() const {}
};

// covariance and magnitudes of a composition: S <- Ad S Ad^T + Z, p <- |Ad| p + g;
// dt: what the translation's own error adds to its magnitude
RPGO_HD void compose_cov(const float* R, const float* t, Cov<float>& S, float (&p)[6], const float* zrr,
                         const float* ztr, const float* ztt, const float* g, float dt) {
  Cov<float> C;
  congruence(R, t, S, C);
#pragma unroll
  for (int e = 0; e < 6; ++e) {
    S.rr[e] = fadd(C.rr[e], zrr[e]);
    S.tt[e] = fadd(C.tt[e], ztt[e]);
  }
#pragma unroll
  for (int e = 0; e < 9; ++e) S.tr[e] = fadd(C.tr[e], ztr[e]);
  float w[3], v[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const float a = fabsv(R[3 * i]), b = fabsv(R[3 * i + 1]), c = fabsv(R[3 * i + 2]);
    w[i] = dot3(a, b, c, p[0], p[1], p[2]);
    v[i] = dot3(a, b, c, p[3], p[4], p[5]);
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int a = (i + 1) % 3, b = (i + 2) % 3;
    p[i] = fadd(w[i], g[i]);
    p[3 + i] = fadd(ffma(fadd(fabsv(t[a]), dt), w[b], ffma(fadd(fabsv(t[b]), dt), w[a], v[i])), g[3 + i]);
  }
}
RPGO_HD void compose_cov_z(const Item& z, Cov<float>& S, float (&p)[6]) {
  float R[9], t[3], rr[6], tr[9], tt[6], g[6];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      R[3 * i + j] = z.d(kPoseZ + 3 * j + i).h;
      tr[3 * i + j] = z.g(kZc + tri(i + 3, j));
    }
#pragma unroll
    for (int j = 0; j <= i; ++j) {
      rr[tri(i, j)] = z.g(kZc + tri(i, j));
      tt[tri(i, j)] = z.g(kZc + tri(i + 3, j + 3));
    }
    t[i] = z.g(kZt + i);
    g[i] = z.g(kZg + i);
    g[3 + i] = z.g(kZg + 3 + i);
  }
  compose_cov(R, t, S, p, rr, tr, tt, g, 0.f);
}

// log map of a pose in FP32 with the bounds ew (each rotation entry) and et
// (each translation entry); false where the axis' sign, the formula that the
// exact test takes or the rotation itself is not certain. For a matrix that is
// not quite a rotation (a long chain of rounded ones) the formulas on the two
// sides of the angle's line differ, and so do those of two diagonal entries as
// large as each other (the check of the rotation sees neither a symmetric part
// that is off nor less than 1e-6), so both sides have to come to the same one:
// cs has an error of at most 10 kU here, a difference of diagonal entries 2 kU.
// The bounds are 12 times what the formulas give (worst of 4e6 rotations of all
// angles, axes along the coordinates and pairs of them: 11 kU, and 8 kU of the
// translation's 1-norm).
RPGO_HD bool logmap(const Pose& T, float (&xi)[6], float& ew, float& et) {
  float R[9];
#pragma unroll
  for (int e = 0; e < 9; ++e) R[e] = T.R[e].h;
  const float cs = fsub(fadd(fadd(R[0], R[4]), R[8]), 1.f);
  const float vx = fsub(R[7], R[5]), vy = fsub(R[2], R[6]), vz = fsub(R[3], R[1]);
  const float sn2 = dot3(vx, vy, vz, vx, vy, vz);
  const float sn = fsqr(sn2);
  bool ok = fabsv(fsub(ffma(cs, cs, sn2), 4.f)) < 1e-5f;  // a rotation matrix
  const float th = atan2f(sn, cs);
  const float t2 = fmulf(th, th);
  float w0, w1, w2;
  ok = ok && fabsv(fadd(cs, 1.6f)) > 32.f * kU;
  if (cs > -1.6f) {
    const float k = th < 0.01f ? ffma(t2, 1.f / 12.f, 0.5f) : fdvd(th, sn);
    w0 = fmulf(k, vx);
    w1 = fmulf(k, vy);
    w2 = fmulf(k, vz);
  } else {
    const float c = fmulf(cs, 0.5f), omc = fsub(1.f, c);
    // the largest diagonal entry's axis component first
    const float s10 = fadd(R[1], R[3]), s20 = fadd(R[2], R[6]), s21 = fadd(R[5], R[7]);
    const bool i1 = R[4] > R[0], i2 = R[8] > (i1 ? R[4] : R[0]);
    ok = ok && fabsv(fsub(R[8], i1 ? R[4] : R[0])) > 8.f * kU && (i2 || fabsv(fsub(R[4], R[0])) > 8.f * kU);
    const float dg = i2 ? R[8] : (i1 ? R[4] : R[0]);
    const float ni = fsqr(fdvd(fsub(dg, c), omc));
    const float den = fmulf(fmulf(2.f, omc), ni);
    const float n0 = i2 ? fdvd(s20, den) : (i1 ? fdvd(s10, den) : ni);
    const float n1 = i2 ? fdvd(s21, den) : (i1 ? ni : fdvd(s10, den));
    const float n2 = i2 ? ni : (i1 ? fdvd(s21, den) : fdvd(s20, den));
    const float sg = dot3(n0, n1, n2, vx, vy, vz);
    ok = ok && fabsv(sg) > 64.f * kU;
    const float f = sg < 0.f ? -th : th;
    w0 = fmulf(f, n0);
    w1 = fmulf(f, n1);
    w2 = fmulf(f, n2);
  }
  const float s = fmulf(sn, 0.5f), c = fmulf(cs, 0.5f);
  const float a = T.t[0].h, b = T.t[1].h, d = T.t[2].h;
  const float W0 = cross1(0.f, w1, d, w2, b), W1 = cross1(0.f, w2, a, w0, d), W2 = cross1(0.f, w0, b, w1, a);
  const float V0 = cross1(0.f, w1, W2, w2, W1), V1 = cross1(0.f, w2, W0, w0, W2),
              V2 = cross1(0.f, w0, W1, w1, W0);
  float beta;
  if (th < 0.01f) {
    beta = ffma(t2, 1.f / 720.f, 1.f / 12.f);
  } else {
    const float omc = fsub(1.f, c);
    beta = fdvd(fsub(1.f, fdvd(fmulf(th, s), ffma(s, s, fmulf(omc, omc)))), t2);
  }
  xi[0] = w0;
  xi[1] = w1;
  xi[2] = w2;
  xi[3] = ffma(beta, V0, ffma(-0.5f, W0, a));
  xi[4] = ffma(beta, V1, ffma(-0.5f, W1, b));
  xi[5] = ffma(beta, V2, ffma(-0.5f, W2, d));
  ew = 128.f * kU;
  et = 256.f * kU * fadd(fadd(fabsv(a), fabsv(b)), fabsv(d));
  return ok;
}

// The verdict from the computed d^2, y.x and y^T C y, the sums p.|y|, e.|y|,
// p.sqrt(C^-1_ii), e.sqrt(C^-1_ii) and the error eta of the two `between`.
RPGO_HD int decide(float d2, float yx, float yCy, float py, float ey, float ph, float eh, float eta, float th2) {
  // the covariances of the two `between` (eta), 16 roundings in each of three
  // compositions, 10 in the factorisation and in y^T C y; what was computed
  // from them with a margin of 1.1
  const float eps = fmulf(1.1f, fadd(eta, 64.f * kU));
  const float low = fsub(fsub(fmulf(2.f, yx), yCy), ffma(eps, fmulf(py, py), fmulf(2.2f, ey)));
  // kap < 1: whatever is within eps of the computed C is positive definite,
  // which every bound here is for. The measurements' covariances are not known
  // to be (their premise looks at pairs of variables only), and where the exact
  // test's C is not, it takes an elimination whose result no bound here is for.
  const float kap = fmulf(eps, fmulf(ph, ph));
  if (!(kap < 1.f)) return 2;
  if (low > fmulf(th2, 1.f + 16.f * kU)) return 0;
  const float d = fadd(fmulf(fsqr(d2), 1.f + 64.f * kU), fmulf(1.1f, eh));
  const float top = fmulf(th2, 1.f - 16.f * kU);
  if (kap < 0.9f && fmulf(d, d) < fmulf(top, fsub(1.f, kap))) return 1;
  // nearer to the threshold: the lower bound's terms, to first order in kap
  const float up = ffma(1.5f, ffma(eps, fmulf(py, py), ffma(2.f, ey, fmulf(eh, eh))), fmulf(d2, 1.f + 64.f * kU));
  return kap < 0.125f && up < top ? 1 : 2;
}

// The translations that the pose chain goes through (1-norms); the loop's
// translation has at most kPoseErr of their sum as error from the chain (about
// 40 roundings of 2^-48, and a margin of 6; worst of 400,000 random chains against
// 64-bit significands: 0.013 of the bound).
constexpr float kPoseErr = 9.094947017729282e-13f;  // 2^-40
template <int D>
RPGO_HD float chain_length(const Item& I, const Item& J, int ta, int tb, int zt) {
  float s = fadd(fadd(I.g(ta), I.g(tb)), fadd(J.g(ta), J.g(tb)));
  for (int a = 0; a < D; ++a) s = fadd(s, fadd(fabsv(I.g(zt + a)), fabsv(J.g(zt + a))));
  return s;
}

// The verdict on closures i and j (flip: the group stores them in opposite
// directions, so j's endpoints change places) against the threshold's square:
// 0 inconsistent, 1 consistent, 2 unsure. No early returns: every thread of a
// block passes every phase.
template <class Sync = NoSync>
RPGO_HD int verdict(const Group& g, int i, int j, bool flip, float th2, Sync sync = Sync()) {
  bool ok = g.ok[i] && g.ok[j];
  const Item I = item(g, i), J = item(g, j);
  // Loops that are not unrolled: the code of one `between` is about 60 KB, and
  // straight through the whole test the warps wait for instructions most of
  // the time.
  Pose Q, P;
  Cov<float> S;
  float p[6], eta = 0.f;
#pragma unroll 1
  for (int side = 0; side < 2; ++side) {
    const bool jb = flip != (side == 1);  // j's second endpoint
    Cov<float> SB;
    float sb[6], e;
    sync();
    ok &= between(I, side ? kPoseB : kPoseA, side ? kGB : kGA, side ? kTB1 : kTA, J, jb ? kPoseB : kPoseA,
                  jb ? kGB : kGA, jb ? kTB1 : kTA, P, SB, sb, e);
    sync();
    eta = e > eta ? e : eta;
    if (side == 0) {
      // (A o Z_j)^-1 o Z_i
      S = SB;
#pragma unroll
      for (int a = 0; a < 6; ++a) p[a] = sb[a];
#pragma unroll 1
      for (int k = 0; k < 2; ++k) {
        const Item& z = k ? I : J;
        Pose Z, T;
        load_pose(z, kPoseZ, Z);
        compose(P, Z, T);
        compose_cov_z(z, S, p);
        if (k) {
          Q = T;
        } else {
#pragma unroll
          for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) P.R[3 * a + b] = T.R[3 * b + a];
          inverse_t(T.R, T.t, P.t);
        }
      }
    } else {
      // loop = Q o B
      float R[9], t[3];
      D2 ti[3];
      inverse_t(P.R, P.t, ti);
#pragma unroll
      for (int a = 0; a < 3; ++a) {
#pragma unroll
        for (int b = 0; b < 3; ++b) R[3 * a + b] = P.R[3 * b + a].h;
        t[a] = ti[a].h;
      }
      compose_cov(R, t, S, p, SB.rr, SB.tr, SB.tt, sb,
                  fmulf(kLeverFp32, fadd(I.g(kTB1), J.g(jb ? kTB1 : kTA))));
    }
  }
  Pose L;
  compose(Q, P, L);
  float xi[6], ew, et;
  ok &= logmap(L, xi, ew, et);
  et = ffma(kPoseErr, chain_length<3>(I, J, kTA, kTB1, kZt), et);
  // d^2 = x^T C^-1 x: L z = x, y = L^-T D^-1 z
  float F[15], W[15], iD[6], h[6];
  ok &= factor(S, F, W, iD, h);
  float z[6], y[6], d2 = 0.f;
#pragma unroll
  for (int a = 0; a < 6; ++a) {
    float acc = xi[a];
#pragma unroll
    for (int k = 0; k < a; ++k) acc = ffma(-F[a * (a - 1) / 2 + k], z[k], acc);
    z[a] = acc;
    y[a] = fmulf(acc, iD[a]);
    d2 = ffma(y[a], acc, d2);
  }
#pragma unroll
  for (int a = 4; a >= 0; --a)
#pragma unroll
    for (int k = a + 1; k < 6; ++k) y[a] = ffma(-F[k * (k - 1) / 2 + a], y[k], y[a]);
  // Bounds. Below, for any y: d^2 >= 2 y.x - y^T C y. Above, with kap >= the
  // relative error of C in its own metric: d^2 <= (d + eh)^2 / (1 - kap).
  float py = 0.f, ey = 0.f, ph = 0.f, eh = 0.f, yx = 0.f, yCy = 0.f;
#pragma unroll
  for (int a = 0; a < 6; ++a) {
    const float e = a < 3 ? ew : et, sh = fsqr(h[a]), ay = fabsv(y[a]);
    py = ffma(p[a], ay, py);
    ey = ffma(e, ay, ey);
    ph = ffma(p[a], sh, ph);
    eh = ffma(e, sh, eh);
    ok = ok && entry(S, a, a) > 1e-24f && p[a] < 1e15f;
    yx = ffma(y[a], xi[a], yx);
    float c = fmulf(0.5f * entry(S, a, a), y[a]);
#pragma unroll
    for (int k = 0; k < a; ++k) c = ffma(entry(S, a, k), y[k], c);
    yCy = ffma(2.f * c, y[a], yCy);
  }
  if (!ok) return 2;
  return decide(d2, yx, yCy, py, ey, ph, eh, eta, th2);
}

// ------------------------------------------------------------------ 2D
// The same test for Pose2: tangent (v_x, v_y, omega), Ad = [[R, (y, -x)], [0, 1]].
// Bounds as in 3D, with fewer terms; a covariance as its lower triangle
// (xx, yx, yy, wx, wy, ww).
constexpr int kPairs2 = 24;   // pose a (c, s, x, y), cov a, pose b, cov b, measured pose
constexpr int kFloats2 = 19;  // inverse measurement's (x, y), its covariance (6), sqrt of its diagonal (3), sqrt of
                              // the diagonals of cov a and cov b (3 each), |t_a|, |t_b|
constexpr int kCov2 = 4, kPoseB2 = 10, kPoseZ2 = 20;
constexpr int kZt2 = 0, kZc2 = 2, kZg2 = 8, kGA2 = 11, kGB2 = 14, kTA2 = 17, kTB2 = 18;

RPGO_HD int tri_full2(int e) {
  int i = 0;
  while (e > i) e -= ++i;
  return 3 * i + e;
}
RPGO_HD D2 pack_pair2(int v, const double* pa, const double* ca, const double* pb, const double* cb,
                      const double* zp, Origin o = {nullptr, nullptr}) {
  if (v < kCov2) return split(v < 2 ? pa[v] : from_origin(pa[v], o.a, v));
  if (v < kPoseB2) return split(ca[tri_full2(v - kCov2)]);
  if (v < kPoseB2 + kCov2)
    return split(v < kPoseB2 + 2 ? pb[v - kPoseB2] : from_origin(pb[v - kPoseB2], o.b, v - kPoseB2));
  if (v < kPoseZ2) return split(cb[tri_full2(v - kPoseB2 - kCov2)]);
  return split(zp[v - kPoseZ2]);
}
RPGO_HD float pack_float2(int v, const double* pa, const double* ca, const double* pb, const double* cb,
                          const double* zp, const double* zc, Origin o = {nullptr, nullptr}) {
  if (v == 0) return (float)-(zp[0] * zp[2] + zp[1] * zp[3]);
  if (v == 1) return (float)-(zp[0] * zp[3] - zp[1] * zp[2]);
  if (v < kZg2) return (float)zc[tri_full2(v - kZc2)];
  if (v < kGA2) return fsqr((float)zc[4 * (v - kZg2)]);
  if (v < kGB2) return fsqr((float)ca[4 * (v - kGA2)]);
  if (v < kTA2) return fsqr((float)cb[4 * (v - kGB2)]);
  const double *p = v == kTA2 ? pa : pb, *q = v == kTA2 ? o.a : o.b;
  return (float)(std::fabs(from_origin(p[2], q, 2)) + std::fabs(from_origin(p[3], q, 3)));
}
RPGO_HD bool cov_premise2(const double* c, bool whole) {
  bool ok = true;
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j <= i; ++j) {
      const double x = c[3 * i + j], b = c[4 * i] * c[4 * j];
      ok = ok && x * x <= 1.0001 * b && (!whole || c[3 * j + i] == x) && c[4 * i] >= 0.0 && c[4 * i] < 1e15;
    }
  return ok;
}
RPGO_HD bool pose_premise2(const double* p) {
  return std::fabs(p[0] * p[0] + p[1] * p[1] - 1.0) < 1e-7 && std::fabs(p[2]) < 1e12 && std::fabs(p[3]) < 1e12;
}

RPGO_HD D2 dot2(D2 a0, D2 a1, D2 b0, D2 b1) {
  Acc x = acc_mul(a0, b0);
  acc_fma(x, a1, b1);
  return norm(x);
}
RPGO_HD D2 fma2(D2 a, D2 b, D2 v) {
  Acc x{v.h, v.l};
  acc_fma(x, a, b);
  return norm(x);
}
RPGO_HD float dot2(float a0, float a1, float b0, float b1) { return ffma(a1, b1, fmulf(a0, b0)); }
RPGO_HD float fma2(float a, float b, float v) { return ffma(a, b, v); }
RPGO_HD float neg(float a) { return -a; }

// Ad S Ad^T for rotation (c, s) and r = (y, -x) (lower triangles)
template <class T>
RPGO_HD void congruence2(T c, T s, T r0, T r1, const T* S, T* C) {
  const T m00 = dot2(c, neg(s), S[0], S[1]), m01 = dot2(c, neg(s), S[1], S[2]);
  const T m10 = dot2(s, c, S[0], S[1]), m11 = dot2(s, c, S[1], S[2]);
  const T b0 = dot2(c, neg(s), S[3], S[4]), b1 = dot2(s, c, S[3], S[4]);
  C[5] = S[5];
  C[3] = fma2(r0, S[5], b0);
  C[4] = fma2(r1, S[5], b1);
  C[0] = fma2(b0, r0, fma2(r0, C[3], dot2(m00, m01, c, neg(s))));
  C[1] = fma2(b1, r0, fma2(r1, C[3], dot2(m10, m11, c, neg(s))));
  C[2] = fma2(b1, r1, fma2(r1, C[4], dot2(m10, m11, s, c)));
}

struct Pose2D {
  D2 c, s, x, y;
};
RPGO_HD Pose2D load_pose2(const Item& i, int v) { return Pose2D{i.d(v), i.d(v + 1), i.d(v + 2), i.d(v + 3)}; }
RPGO_HD Pose2D compose2(const Pose2D& A, const Pose2D& B) {
  Acc x{A.x.h, A.x.l}, y{A.y.h, A.y.l};
  acc_fma(x, A.c, B.x);
  acc_fma(x, neg(A.s), B.y);
  acc_fma(y, A.s, B.x);
  acc_fma(y, A.c, B.y);
  return Pose2D{dot2(A.c, neg(A.s), B.c, B.s), dot2(A.s, A.c, B.c, B.s), norm(x), norm(y)};
}
RPGO_HD Pose2D inverse2(const Pose2D& A) {
  return Pose2D{A.c, neg(A.s), neg(dot2(A.c, A.s, A.x, A.y)), neg(dot2(A.c, neg(A.s), A.y, A.x))};
}
RPGO_HD Pose2D between2(const Pose2D& A, const Pose2D& B) {
  const D2 dx = sub(B.x, A.x), dy = sub(B.y, A.y);
  return Pose2D{dot2(A.c, A.s, B.c, B.s), dot2(A.c, neg(A.s), B.s, B.c), dot2(A.c, A.s, dx, dy),
                dot2(A.c, neg(A.s), dy, dx)};
}

// LDL^T (see factor): L and L^-1 as (10, 20, 21)
RPGO_HD bool factor2(const float* S, float (&L)[3], float (&W)[3], float (&iD)[3], float (&h)[3]) {
  iD[0] = fdvd(1.f, S[0]);
  L[0] = fmulf(S[1], iD[0]);
  const float d1 = ffma(-S[1], L[0], S[2]);
  iD[1] = fdvd(1.f, d1);
  L[1] = fmulf(S[3], iD[0]);
  const float e = ffma(-S[3], L[0], S[4]);
  L[2] = fmulf(e, iD[1]);
  const float d2 = ffma(-e, L[2], ffma(-S[3], L[1], S[5]));
  iD[2] = fdvd(1.f, d2);
  W[0] = -L[0];
  W[2] = -L[2];
  W[1] = ffma(-L[2], W[0], -L[1]);
  h[0] = ffma(fmulf(W[1], W[1]), iD[2], ffma(fmulf(W[0], W[0]), iD[1], iD[0]));
  h[1] = ffma(fmulf(W[2], W[2]), iD[2], iD[1]);
  h[2] = iD[2];
  return S[0] > 0.f && d1 > 0.f && d2 > 0.f;
}

RPGO_HD bool between_cov2(const Item& x, int va, int ga, int ta, const Item& y, int vc, int gc, int tc, Pose2D& pose,
                          float (&S)[6], float (&s)[3], float& eta) {
  const Pose2D A = load_pose2(x, va), B = load_pose2(y, vc);
  pose = between2(A, B);
  const float gv = fadd(x.g(ga), x.g(ga + 1)), hv = fadd(y.g(gc), y.g(gc + 1));
  const float qw = fadd(x.g(ga + 2), y.g(gc + 2));
  // (kLever: the error of the difference of the positions)
  const float lever = ffma(kLever, fadd(x.g(ta), y.g(tc)), fadd(fabsv(pose.x.h), fabsv(pose.y.h)));
  const float qv = ffma(lever, qw, fadd(gv, hv));
  // Ad of the inverse: rotation (c, -s), r = (y', -x') of the inverse's
  // translation; first for the main formula's first pivot, cov(v_x, v_x)
  const Pose2D im = inverse2(pose);
  bool main, known;
  {
    D2 Sx[6];
#pragma unroll
    for (int e = 0; e < 6; ++e) Sx[e] = x.d(va + kCov2 + e);
    const D2 c = im.c, ns = neg(im.s), r0 = im.y;
    const D2 m0 = dot2(c, ns, Sx[0], Sx[1]), m1 = dot2(c, ns, Sx[1], Sx[2]), b0 = dot2(c, ns, Sx[3], Sx[4]);
    const D2 c3 = fma2(r0, Sx[5], b0);
    const D2 piv = sub(y.d(vc + kCov2), fma2(b0, r0, fma2(r0, c3, dot2(m0, m1, c, ns))));
    const float e = fmulf(kDf, fmulf(qv, qv));
    main = piv.h > e;
    known = main || piv.h < -e;
  }
  const Item& X = main ? x : y;
  const Item& Y = main ? y : x;
  const int vX = main ? va : vc, vY = main ? vc : va;
  const Pose2D ib = inverse2(between2(B, A));
  const D2 c = main ? im.c : ib.c, sn = main ? im.s : ib.s, r0 = main ? im.y : ib.y, r1 = neg(main ? im.x : ib.x);
  D2 SX[6], C[6];
#pragma unroll
  for (int e = 0; e < 6; ++e) SX[e] = X.d(vX + kCov2 + e);
  congruence2(c, sn, r0, r1, SX, C);
#pragma unroll
  for (int e = 0; e < 6; ++e) S[e] = lo(sub(Y.d(vY + kCov2 + e), C[e]));
  float L[3], W[3], iD[3], h[3];
  bool ok = factor2(S, L, W, iD, h) && known;
  const float dg[3] = {S[0], S[2], S[5]};
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    ok = ok && dg[i] > 1e-24f;
    s[i] = fsqr(dg[i]);
    sum = fadd(sum, fsqr(fmulf(dg[i], h[i])));
  }
  const float ev = fdvd(fmulf(qv, qv), dg[0] < dg[1] ? dg[0] : dg[1]), ew = fdvd(fmulf(qw, qw), dg[2]);
  eta = ffma(kDf, ev > ew ? ev : ew, 16.f * kU);
  return ok && fmulf(eta, fmulf(sum, sum)) < 0.5f;
}

RPGO_HD void compose_cov2(float c, float sn, float r0, float r1, float (&S)[6], float (&p)[3], const float* Z,
                          const float* g, float dt) {
  float C[6];
  congruence2(c, sn, r0, r1, S, C);
#pragma unroll
  for (int e = 0; e < 6; ++e) S[e] = fadd(C[e], Z[e]);
  const float ac = fabsv(c), as = fabsv(sn), v0 = p[0], v1 = p[1];
  p[0] = fadd(ffma(fadd(fabsv(r0), dt), p[2], ffma(as, v1, fmulf(ac, v0))), g[0]);
  p[1] = fadd(ffma(fadd(fabsv(r1), dt), p[2], ffma(ac, v1, fmulf(as, v0))), g[1]);
  p[2] = fadd(p[2], g[2]);
}

template <class Sync = NoSync>
RPGO_HD int verdict2(const Group& g, int i, int j, bool flip, float th2, Sync sync = Sync()) {
  bool ok = g.ok[i] && g.ok[j];
  const Item I = item(g, i), J = item(g, j);
  Pose2D Q, P;
  float S[6], p[3], eta = 0.f;
#pragma unroll 1
  for (int side = 0; side < 2; ++side) {
    const bool jb = flip != (side == 1);  // j's second endpoint
    float SB[6], sb[3], e;
    sync();
    ok &= between_cov2(I, side ? kPoseB2 : 0, side ? kGB2 : kGA2, side ? kTB2 : kTA2, J, jb ? kPoseB2 : 0,
                       jb ? kGB2 : kGA2, jb ? kTB2 : kTA2, P, SB, sb, e);
    eta = e > eta ? e : eta;
    if (side == 0) {
      // (A o Z_j)^-1 o Z_i
#pragma unroll
      for (int a = 0; a < 6; ++a) S[a] = SB[a];
#pragma unroll
      for (int a = 0; a < 3; ++a) p[a] = sb[a];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const Item& z = k ? I : J;
        const Pose2D Z = load_pose2(z, kPoseZ2), T = compose2(P, Z);
        float zc[6], zg[3];
#pragma unroll
        for (int a = 0; a < 6; ++a) zc[a] = z.g(kZc2 + a);
#pragma unroll
        for (int a = 0; a < 3; ++a) zg[a] = z.g(kZg2 + a);
        compose_cov2(Z.c.h, -Z.s.h, z.g(kZt2 + 1), -z.g(kZt2), S, p, zc, zg, 0.f);
        if (k) Q = T;
        else P = inverse2(T);
      }
    } else {
      const Pose2D ib = inverse2(P);  // loop = Q o B
      compose_cov2(ib.c.h, ib.s.h, ib.y.h, -ib.x.h, S, p, SB, sb,
                   fmulf(kLeverFp32, fadd(I.g(kTB2), J.g(jb ? kTB2 : kTA2))));
    }
  }
  const Pose2D T = compose2(Q, P);
  // Log map. 1 - c comes from the pair, so that it keeps its digits for small
  // angles; its error of about 2^-43 counts by 1 / angle. Below 1e-10 the
  // exact test takes the translation itself; up to 1e-8 the pair is unsure.
  const float c = T.c.h, s = T.s.h, x = T.x.h, y = T.y.h;
  const float th = atan2f(s, c), at = fabsv(th), omc = fsub(fsub(1.f, c), T.c.l);
  const bool none = at < 0.9e-10f;
  ok = ok && fabsv(fsub(ffma(c, c, fmulf(s, s)), 1.f)) < 1e-6f && (c > 0.f || fabsv(s) > 64.f * kU) &&
       (none || at > 1e-8f);
  const float k = fdvd(th, ffma(s, s, fmulf(omc, omc)));
  const float a = none ? 1.f : fmulf(k, s), b = none ? 0.f : fmulf(k, omc);
  const float xi[3] = {ffma(b, y, fmulf(a, x)), ffma(-b, x, fmulf(a, y)), th};
  const float et = ffma(kPoseErr, chain_length<2>(I, J, kTA2, kTB2, kZt2),
                        fmulf(fadd(64.f * kU, none ? 0.f : fdvd(kPoseErr, at)), fadd(fabsv(x), fabsv(y))));
  const float ew = ffma(16.f * kU, at, 1e-10f);
  float L[3], W[3], iD[3], h[3];
  ok &= factor2(S, L, W, iD, h);
  const float z0 = xi[0], z1 = ffma(-L[0], z0, xi[1]), z2 = ffma(-L[2], z1, ffma(-L[1], z0, xi[2]));
  const float d0 = fmulf(z0, iD[0]), d1 = fmulf(z1, iD[1]), d2y = fmulf(z2, iD[2]);
  const float d2 = ffma(d2y, z2, ffma(d1, z1, fmulf(d0, z0)));
  const float y2 = d2y, y1 = ffma(-L[2], y2, d1), y0 = ffma(-L[1], y2, ffma(-L[0], y1, d0));
  const float yv[3] = {y0, y1, y2}, dg[3] = {S[0], S[2], S[5]};
  float py = 0.f, ey = 0.f, ph = 0.f, eh = 0.f, yx = 0.f;
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const float e = q < 2 ? et : ew, sh = fsqr(h[q]), ay = fabsv(yv[q]);
    py = ffma(p[q], ay, py);
    ey = ffma(e, ay, ey);
    ph = ffma(p[q], sh, ph);
    eh = ffma(e, sh, eh);
    ok = ok && dg[q] > 1e-24f && p[q] < 1e15f;
    yx = ffma(yv[q], xi[q], yx);
  }
  // C y
  const float s0 = ffma(S[3], y2, ffma(S[1], y1, fmulf(S[0], y0)));
  const float s1 = ffma(S[4], y2, ffma(S[2], y1, fmulf(S[1], y0)));
  const float s2 = ffma(S[5], y2, ffma(S[4], y1, fmulf(S[3], y0)));
  const float yCy = ffma(y2, s2, ffma(y1, s1, fmulf(y0, s0)));
  if (!ok) return 2;
  return decide(d2, yx, yCy, py, ey, ph, eh, eta, th2);
}

// ------------------------------------------------------------------ both
// closure k's origins in a group: a0, b0 are the poses of closure 0's endpoints
RPGO_HD Origin origin(const double* a0, const double* b0, bool flipped) {
  return flipped ? Origin{b0, a0} : Origin{a0, b0};
}
template <int DIM>
struct Filter;
template <>
struct Filter<3> {
  static constexpr int pairs = kPairs, floats = kFloats;
  RPGO_HD static D2 pair(int v, const double* pa, const double* ca, const double* pb, const double* cb,
                         const double* z, Origin o = {nullptr, nullptr}) {
    return pack_pair(v, pa, ca, pb, cb, z, o);
  }
  RPGO_HD static float single(int v, const double* pa, const double* ca, const double* pb, const double* cb,
                              const double* z, const double* c, Origin o = {nullptr, nullptr}) {
    return pack_float(v, pa, ca, pb, cb, z, c, o);
  }
  RPGO_HD static bool premise(const double* pa, const double* ca, const double* pb, const double* cb,
                              const double* z, const double* c) {
    return cov_premise(ca, true) && cov_premise(cb, true) && cov_premise(c, false) && pose_premise(pa) &&
           pose_premise(pb) && pose_premise(z);
  }
  template <class Sync = NoSync>
  RPGO_HD static int test(const Group& g, int i, int j, bool flip, float th2, Sync sync = Sync()) {
    return verdict(g, i, j, flip, th2, sync);
  }
};
template <>
struct Filter<2> {
  static constexpr int pairs = kPairs2, floats = kFloats2;
  RPGO_HD static D2 pair(int v, const double* pa, const double* ca, const double* pb, const double* cb,
                         const double* z, Origin o = {nullptr, nullptr}) {
    return pack_pair2(v, pa, ca, pb, cb, z, o);
  }
  RPGO_HD static float single(int v, const double* pa, const double* ca, const double* pb, const double* cb,
                              const double* z, const double* c, Origin o = {nullptr, nullptr}) {
    return pack_float2(v, pa, ca, pb, cb, z, c, o);
  }
  RPGO_HD static bool premise(const double* pa, const double* ca, const double* pb, const double* cb,
                              const double* z, const double* c) {
    return cov_premise2(ca, true) && cov_premise2(cb, true) && cov_premise2(c, false) && pose_premise2(pa) &&
           pose_premise2(pb) && pose_premise2(z);
  }
  template <class Sync = NoSync>
  RPGO_HD static int test(const Group& g, int i, int j, bool flip, float th2, Sync sync = Sync()) {
    return verdict2(g, i, j, flip, th2, sync);
  }
};

}  // namespace pf
}  // namespace rpgo
