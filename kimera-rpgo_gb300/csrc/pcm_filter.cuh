// Decides most pairwise consistency tests of 3D uncertain poses
// (Pcm::areLoopsConsistent, include/KimeraRPGO/outlier/Pcm.h:670-718) in FP32
// arithmetic, with a bound on its own error; the rest is left to the exact
// FP64 test of pcm_kernels.cu. Host and device code: the tests run it on the
// CPU against the exact verdicts.
//
// What the exact test computes is d = |Logmap(loop)| in the metric of the
// loop's covariance, compared with a threshold. Its operations only matter
// through their rounding errors, so the verdict is known as soon as d, known
// to within E, is further than E from the threshold. Two things are decided
// on the way: which of its two formulas each `between` takes (a positive
// definiteness test, GeometryUtils.h:143-170) and the sign of the axis of a
// rotation by nearly pi. Where any of them is not certain, or a bound's
// premise fails (NaN, an asymmetric or indefinite input covariance, no
// rotation information, values near the limits of FP32), the pair is unsure.
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
// taken at C y = x, where it is close to d^2; and with C's error relative to C
// itself, kap = eps (sum p_i sqrt(C^-1_ii))^2 < 1,
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
constexpr float kDf = 3.637978807091713e-12f;     // 2^-38: about 2.4 times the worst case of a `between`
                                                  // (about 420 roundings of 2^-48)

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
                             // sqrt of the diagonals of cov a and cov b (6 each), |t_a|, |t_b| (1-norms)
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

// value v of a closure from its trajectory entries (pose 12, covariance 36)
// and measurement (pose 12)
RPGO_HD D2 pack_pair(int v, const double* pa, const double* ca, const double* pb, const double* cb,
                     const double* zp) {
  if (v < kCovA) return split(pa[v]);
  if (v < kPoseB) return split(ca[tri_full(v - kCovA)]);
  if (v < kCovB) return split(pb[v - kPoseB]);
  if (v < kPoseZ) return split(cb[tri_full(v - kCovB)]);
  return split(zp[v - kPoseZ]);
}
RPGO_HD float pack_float(int v, const double* pa, const double* ca, const double* pb, const double* cb,
                         const double* zp, const double* zc) {
  if (v < kZc) return (float)-(zp[v] * zp[9] + zp[3 + v] * zp[10] + zp[6 + v] * zp[11]);
  if (v < kZg) return (float)zc[tri_full(v - kZc)];
  if (v < kGA) return fsqr((float)zc[7 * (v - kZg)]);
  if (v < kGB) return fsqr((float)ca[7 * (v - kGA)]);
  if (v < kTA) return fsqr((float)cb[7 * (v - kGB)]);
  const double* t = (v == kTA ? pa : pb) + 9;
  return (float)(std::fabs(t[0]) + std::fabs(t[1]) + std::fabs(t[2]));
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
  // the magnitudes that were subtracted, |R| taken as all ones
  const float lever = fadd(fadd(fabsv(t[0].h), fabsv(t[1].h)), fadd(fabsv(t[2].h), fadd(x.g(ta), y.g(tc))));
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

// covariance and magnitudes of a composition: S <- Ad S Ad^T + Z, p <- |Ad| p + g
RPGO_HD void compose_cov(const float* R, const float* t, Cov<float>& S, float (&p)[6], const float* zrr,
                         const float* ztr, const float* ztt, const float* g) {
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
    p[3 + i] = fadd(ffma(fabsv(t[a]), w[b], ffma(fabsv(t[b]), w[a], v[i])), g[3 + i]);
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
  compose_cov(R, t, S, p, rr, tr, tt, g);
}

// log map of a pose in FP32 with the bounds ew (each rotation entry) and et
// (each translation entry); false where the axis' sign or the rotation itself
// is not certain
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
      compose_cov(R, t, S, p, SB.rr, SB.tr, SB.tt, sb);
    }
  }
  Pose L;
  compose(Q, P, L);
  float xi[6], ew, et;
  ok &= logmap(L, xi, ew, et);
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
  // the covariances of the two `between` (eta), 16 roundings in each of three
  // compositions, 10 in the factorisation and in y^T C y; what was computed
  // from them with a margin of 1.1
  const float eps = fmulf(1.1f, fadd(eta, 64.f * kU));
  const float low = fsub(fsub(fmulf(2.f, yx), yCy), ffma(eps, fmulf(py, py), fmulf(2.2f, ey)));
  if (low > fmulf(th2, 1.f + 16.f * kU)) return 0;
  const float kap = fmulf(eps, fmulf(ph, ph));
  const float d = fadd(fmulf(fsqr(d2), 1.f + 64.f * kU), fmulf(1.1f, eh));
  const float top = fmulf(th2, 1.f - 16.f * kU);
  if (kap < 0.9f && fmulf(d, d) < fmulf(top, fsub(1.f, kap))) return 1;
  // nearer to the threshold: the lower bound's terms, to first order in kap
  const float up = ffma(1.5f, ffma(eps, fmulf(py, py), ffma(2.f, ey, fmulf(eh, eh))), fmulf(d2, 1.f + 64.f * kU));
  return kap < 0.125f && up < top ? 1 : 2;
}

}  // namespace pf
}  // namespace rpgo
