// PCM outlier-rejection kernels (sm_103a).
//
//  K0 trajectory scan   Pcm::updateOdom (Pcm.h:516-557): the odometry chain
//                       T_k = T_{k-1} o Delta_k with the covariance
//                       Ad(Delta^-1) S Ad(Delta^-1)^T + S_Delta, sequential in
//                       factor order (one warp per block of the covariance).
//  K1 odometry check    Pcm::isOdomConsistent / checkOdomConsistent
//                       (Pcm.h:564-629), one thread per loop closure.
//  K2 pairwise check    Pcm::areLoopsConsistent / checkLoopConsistent /
//                       incrementAdjMatrix (Pcm.h:638-768): one thread per
//                       closure pair (i < j), 32 consecutive i per warp, the
//                       verdicts packed into 32-bit adjacency words with one
//                       warp ballot; a last kernel mirrors the lower
//                       triangle into the upper one with warp bit transposes.
// All arithmetic is the exact FP64 sequence of pcm_math.cuh, but for groups of
// 65,536 pairs of uncertain poses and more: there an FP32 test with a bound on
// its error decides the pairs that it can (pcm_filter.cuh), and the exact
// sequence the others, so that every verdict is the exact one.
#include <algorithm>
#include <type_traits>

#include "pcm_filter.cuh"
#include "pcm_kernels.hpp"
#include "pcm_math.cuh"

namespace rpgo {
namespace {

using namespace pm;

// ------------------------------------------------------------------ uncertain poses
template <int DIM>
struct Lie;
template <>
struct Lie<3> {
  using Pose = P3;
  static constexpr int d = 6, rd = 3, td = 3, stride = 12;
  __device__ static void load(const double* s, Pose& p) { p3_load(s, p); }
  __device__ static void store(const Pose& p, double* s) { p3_store(p, s); }
  __device__ static void compose(const Pose& a, const Pose& b, Pose& c) { p3_compose(a, b, c); }
  __device__ static void inverse(const Pose& a, Pose& c) { p3_inverse(a, c); }
  __device__ static void between(const Pose& a, const Pose& b, Pose& c) { p3_between(a, b, c); }
  __device__ static void congruence(const Pose& T, const double* S, double* C) { p3_congruence(T, S, C); }
  __device__ static void logmap(const Pose& T, double* xi) { p3_logmap(T, xi); }
  __device__ static double rot_trace(const double* c) { return add(add(c[0], c[7]), c[14]); }
};
template <>
struct Lie<2> {
  using Pose = P2;
  static constexpr int d = 3, rd = 1, td = 2, stride = 4;
  __device__ static void load(const double* s, Pose& p) { p2_load(s, p); }
  __device__ static void store(const Pose& p, double* s) { p2_store(p, s); }
  __device__ static void compose(const Pose& a, const Pose& b, Pose& c) { p2_compose(a, b, c); }
  __device__ static void inverse(const Pose& a, Pose& c) { p2_inverse(a, c); }
  __device__ static void between(const Pose& a, const Pose& b, Pose& c) { p2_between(a, b, c); }
  __device__ static void congruence(const Pose& T, const double* S, double* C) { p2_congruence(T, S, C); }
  __device__ static void logmap(const Pose& T, double* xi) { p2_logmap(T, xi); }
  __device__ static double rot_trace(const double* c) { return c[0]; }
};

// PoseWithCovariance (GeometryUtils.h:56-187)
template <int DIM>
struct PWC {
  using L = Lie<DIM>;
  static constexpr int d = L::d;
  typename L::Pose pose;
  double cov[d * d];
  bool rot;

  __device__ void from_factor(const double* zp, const double* zc) {
    L::load(zp, pose);
    rot = !isnan(L::rot_trace(zc));
#pragma unroll
    for (int i = 0; i < d; ++i)
#pragma unroll
      for (int j = 0; j < d; ++j) cov[d * i + j] = (rot || (i >= L::rd && j >= L::rd)) ? zc[d * i + j] : 0.0;
  }
  __device__ void from_traj(const TrajView& t, int s) {
    L::load(t.pose + (size_t)s * L::stride, pose);
#pragma unroll
    for (int i = 0; i < d * d; ++i) cov[i] = t.cov[(size_t)s * d * d + i];
    rot = t.rot[s] != 0;
  }
  // this o other (GeometryUtils.h:119-129)
  __device__ void compose(const PWC& other, PWC& out) const {
    typename L::Pose inv;
    L::compose(pose, other.pose, out.pose);
    L::inverse(other.pose, inv);
    double C[d * d];
    L::congruence(inv, cov, C);
#pragma unroll
    for (int i = 0; i < d; ++i)
#pragma unroll
      for (int j = 0; j <= i; ++j) {
        const double v = add(C[d * i + j], other.cov[d * i + j]);
        out.cov[d * i + j] = v;
        out.cov[d * j + i] = v;
      }
    out.rot = rot && other.rot;
  }
  // the same composition with the inverse of other's pose given as its
  // rotation and the K block of its adjoint (per-closure constants, 3D)
  __device__ void compose_pre(const PWC& other, const double* pre, PWC& out) const {
    L::compose(pose, other.pose, out.pose);
    double C[d * d];
    pm::p3_congruence_RK(pre, pre + 9, cov, C);
#pragma unroll
    for (int i = 0; i < d; ++i)
#pragma unroll
      for (int j = 0; j <= i; ++j) {
        const double v = add(C[d * i + j], other.cov[d * i + j]);
        out.cov[d * i + j] = v;
        out.cov[d * j + i] = v;
      }
    out.rot = rot && other.rot;
  }
  // GeometryUtils.h:133-139
  __device__ void inverse_inplace() {
    typename L::Pose p;
    L::inverse(pose, p);
    pose = p;
  }
  // this^-1 o other with the LLT fallback (GeometryUtils.h:143-170)
  __device__ void between(const PWC& other, PWC& out) const {
    typename L::Pose res, inv;
    L::between(pose, other.pose, res);
    L::inverse(res, inv);
    double C[d * d];
    L::congruence(inv, cov, C);
#pragma unroll
    for (int i = 0; i < d; ++i)
#pragma unroll
      for (int j = 0; j <= i; ++j) {
        const double v = sub(other.cov[d * i + j], C[d * i + j]);
        out.cov[d * i + j] = v;
        out.cov[d * j + i] = v;
      }
    if (!chol_ok<d>(out.cov)) {
      typename L::Pose res2, inv2;
      L::between(other.pose, pose, res2);
      L::inverse(res2, inv2);
      L::congruence(inv2, other.cov, C);
#pragma unroll
      for (int i = 0; i < d; ++i)
#pragma unroll
        for (int j = 0; j <= i; ++j) {
          const double v = sub(cov[d * i + j], C[d * i + j]);
          out.cov[d * i + j] = v;
          out.cov[d * j + i] = v;
        }
    }
    out.pose = res;
    out.rot = rot && other.rot;
  }
  __device__ double mahalanobis() const {
    double xi[d];
    L::logmap(pose, xi);
    if (!rot) {
      constexpr int m = L::td, r = L::rd;
      double B[m * m];
#pragma unroll
      for (int i = 0; i < m; ++i)
#pragma unroll
        for (int j = 0; j < m; ++j) B[m * i + j] = cov[d * (r + i) + (r + j)];
      return sqrtd(quad_inv<m>(B, xi + r));
    }
    return sqrtd(quad_inv<d>(cov, xi));
  }
};

// PoseWithNode (GeometryUtils.h:193-289)
template <int DIM>
struct PWN {
  using L = Lie<DIM>;
  static constexpr int d = L::d;
  typename L::Pose pose;
  int node;
  bool rot;
  __device__ void from_factor(const double* zp, const double* zc) {
    L::load(zp, pose);
    rot = !isnan(L::rot_trace(zc));
    node = 1;
  }
  __device__ void from_traj(const TrajView& t, int s) {
    L::load(t.pose + (size_t)s * L::stride, pose);
    node = t.node[s];
    rot = t.rot[s] != 0;
  }
  __device__ void compose(const PWN& o, PWN& out) const {
    L::compose(pose, o.pose, out.pose);
    out.node = node + o.node;
    out.rot = rot && o.rot;
  }
  __device__ void inverse_inplace() {
    typename L::Pose p;
    L::inverse(pose, p);
    pose = p;
  }
  __device__ void between(const PWN& o, PWN& out) const {
    L::between(pose, o.pose, out.pose);
    out.node = abs(o.node - node);
    out.rot = rot && o.rot;
  }
  __device__ static double norm_slice(const double* v, int m) {
    double acc = mul(v[0], v[0]);
    for (int i = 1; i < m; ++i) acc = fmad(v[i], v[i], acc);
    return sqrtd(acc);
  }
  __device__ void norms(double& trans, double& rotn) const {
    double xi[d];
    L::logmap(pose, xi);
    trans = dvd(norm_slice(xi + L::rd, L::td), (double)node);
    rotn = rot ? dvd(norm_slice(xi, L::rd), (double)node) : 0.0;
  }
};

template <class U>
__device__ __forceinline__ bool check_mahal(const U& u, double th0, double) {
  return u.mahalanobis() < th0;
}
template <int DIM>
__device__ __forceinline__ bool check_u(const PWC<DIM>& u, double th0, double) {
  return u.mahalanobis() < th0;
}
template <int DIM>
__device__ __forceinline__ bool check_u(const PWN<DIM>& u, double th0, double th1) {
  double t, r;
  u.norms(t, r);
  return t < th0 && r < th1;
}

// ------------------------------------------------------------------ K0
// Per-odometry-factor constants of the covariance walk, one record per step:
// Ad(Delta^-1) (3D: its blocks R and K, 9 each; 2D: 9) and the lower triangle
// of the measurement's covariance as an uncertain pose (GeometryUtils.h:91-115).
template <int DIM>
struct ScanRec {
  static constexpr int ad = DIM == 3 ? 18 : 9, d = DIM == 3 ? 6 : 3, n = ad + d * (d + 1) / 2;
};
template <int DIM>
__global__ void k_odom_prep(int64_t count, const double* __restrict__ dpose, const double* __restrict__ dcov,
                            double* __restrict__ rec, uint8_t* __restrict__ rot_out) {
  using L = Lie<DIM>;
  using C = ScanRec<DIM>;
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= count) return;
  PWC<DIM> z;
  z.from_factor(dpose + k * L::stride, dcov + k * L::d * L::d);
  rot_out[k] = z.rot ? 1 : 0;
  double* r = rec + k * C::n;
  typename L::Pose inv;
  L::inverse(z.pose, inv);
  if constexpr (DIM == 3) {
    double K[9];
    p3_adjoint_K(inv, K);
    for (int i = 0; i < 9; ++i) r[i] = inv.R[i];
    for (int i = 0; i < 9; ++i) r[9 + i] = K[i];
  } else {
    double A[9];
    p2_adjoint(inv, A);
    for (int i = 0; i < 9; ++i) r[i] = A[i];
  }
  for (int i = 0, e = C::ad; i < C::d; ++i)
    for (int j = 0; j <= i; ++j, ++e) r[e] = z.cov[C::d * i + j];
}

// The walk: S_k = A S_{k-1} A^T + Sigma_Delta with A = Ad(Delta^-1) known for
// every step beforehand, and the poses. An FP64 instruction takes 64 cycles of
// its warp whether or not the next one waits for it, so a step costs what its
// longest chain of dependent FMAs takes, and the chains are cut to what has to
// be sequential. In blocks (r: rotation, t: translation; A = [[R, 0], [K, R]]),
// with the term order of M_elem and C_elem (pcm_math.cuh) kept,
//   rr' = (R rr) R^T + Q,   tr' = (K rr + R tr) R^T + Q,
//   tt' = (K rr + R tr) K^T + (K rt + R tt) R^T + Q,
// so rr needs only rr, tr only rr and tr, and each block's own loop is seven
// instructions (three products, three products, the sum with Q): one warp per
// block, each a chunk of steps behind the one before, which hands it its
// partial sums (K rr; then K rt and the first three terms of tt') through
// shared memory. The columns M_rt of the first product are never read. The
// poses are a chain of their own on another SM.
// Bound by the latency of a step: seven FP64 instructions (448 cycles alone,
// about 530 with three warps on the SM's FP64 pipe) and the exchange of the
// block between its lanes twice; 812 cycles in all. 20,000 steps: 3D 17.9 ->
// 7.85 ms (before: two warps, 13 instructions and two block barriers a step),
// 2D 20.5 -> 6.5 ms (one warp).
constexpr int kScanChunk = 16;  // steps per chunk

template <int DIM>
struct ScanCov {
  double cst[4][kScanChunk * ScanRec<DIM>::n];
  double rr[2][kScanChunk][9];   // K rr
  double tr[2][kScanChunk][18];  // K rt, then the first three terms of tt'
  int32_t src[4][kScanChunk], dst[4][kScanChunk];
};
template <int DIM>
struct ScanPose {
  double dp[2][kScanChunk][Lie<DIM>::stride];
  int32_t src[2][kScanChunk], dst[2][kScanChunk];
  uint8_t rot[2][kScanChunk];
};

__device__ __forceinline__ double shfl_d(double v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }

// The covariance block of `role` (0 rr or the whole 2D covariance, 1 tr, 2 tt)
// over the steps [0, n) of chunk c. Lane 3 i + j < 9 holds entry (i, j) of the
// block (mirrored where it is symmetric: the entry of the lower triangle),
// lanes 9-17 the second job that shares its instructions; role 1: entry (i, j)
// of rt. last: the slot written by the step before.
template <int DIM, int role>
__device__ __forceinline__ void scan_chunk(int c, int n, ScanCov<DIM>& s, double* __restrict__ cov,
                                           double& S, int32_t& last, int lane) {
  constexpr int d = ScanRec<DIM>::d, dd = d * d, ad = ScanRec<DIM>::ad;
  const bool second = lane >= 9 && lane < 18;
  const int e = lane < 18 ? lane % 9 : 0, i = e / 3, j = e % 3;
  // the products' left rows (R or K, row i) and right rows (row b)
  const int left = (second && DIM == 3 ? 9 : 0) + 3 * i;
  const bool tri = !(role == 1 && !second);  // a symmetric result: its lower entry (a, b)
  const int a = tri ? max(i, j) : i, b = tri ? min(i, j) : j;
  const int right = (role == 1 && second ? 9 : 0) + 3 * b;
  const int qi = (role ? 3 : 0) + a, qj = (role == 2 ? 3 : 0) + b;
  const int q = ad + qi * (qi + 1) / 2 + qj;
  // the entry's place in the covariance
  const int row = role == 1 ? (second ? i : 3 + i) : (role ? 3 : 0) + i;
  const int col = role == 1 ? (second ? 3 + j : j) : (role ? 3 : 0) + j;
  const bool out = lane < 9 || (role == 1 && second);
  // step k's operands; those of step k + 1 are read while step k computes
  struct Step {
    double l0, l1, l2, r0, r1, r2, Q, m0, c0;
    int32_t from, to;
  };
  auto load = [&](int k) {
    const double* cst = s.cst[c & 3] + k * ScanRec<DIM>::n;
    Step x{cst[left], cst[left + 1], cst[left + 2], cst[right], cst[right + 1], cst[right + 2], cst[q], -0.0, -0.0,
           s.src[c & 3][k], s.dst[c & 3][k]};
    // what the products are added to (-0 + x = x)
    if (role == 1) {
      const double v = s.rr[c & 1][k][e];
      x.m0 = second ? -0.0 : v;
    }
    if (role == 2) {
      x.m0 = s.tr[c & 1][k][e];
      x.c0 = s.tr[c & 1][k][9 + 3 * a + b];
    }
    return x;
  };
  double* const place = cov + d * row + col;
  Step cur = load(0);
  bool again = cur.from != last;
  for (int k = 0; k < n; ++k) {
    if (again) {  // the chain continues from an older pose: read it back
      __syncwarp();
      S = out ? place[(size_t)cur.from * dd] : 0.0;
    }
    // M: left row times column j of the block (lanes 9-17 of role 1: of rt)
    const int at = (role == 1 && second ? 9 : 0) + j;
    const double s0 = shfl_d(S, at), s1 = shfl_d(S, at + 3), s2 = shfl_d(S, at + 6);
    double M = fmad(cur.l0, s0, cur.m0);
    const Step nxt = load(min(k + 1, n - 1));
    M = fmad(cur.l1, s1, M);
    M = fmad(cur.l2, s2, M);
    const double t0 = shfl_d(M, 3 * a), t1 = shfl_d(M, 3 * a + 1), t2 = shfl_d(M, 3 * a + 2);
    // C: row a of M times the right row
    double C = fmad(t0, cur.r0, cur.c0);
    if (second && role == 0 && DIM == 3) s.rr[c & 1][k][e] = M;
    if (second && role == 1) s.tr[c & 1][k][e] = M;
    C = fmad(t1, cur.r1, C);
    C = fmad(t2, cur.r2, C);
    S = add(C, cur.Q);
    if (second && role == 1) s.tr[c & 1][k][9 + e] = C;
    again = nxt.from != cur.to;
    double* const o = place + (size_t)cur.to * dd;
    cur = nxt;
    if (role == 1) {
      const double x = shfl_d(S, 3 * j + i);  // rt = tr^T
      if (second) S = x;
    }
    if (out) *o = S;
  }
  last = s.dst[c & 3][n - 1];
}

// chunk c's constants, by one warp (it has the time of a chunk for it: a copy
// that gathered the record's parts from two arrays took longer than that)
template <int DIM>
__device__ __forceinline__ void scan_load(int c, int n, ScanCov<DIM>& s, const int32_t* __restrict__ src,
                                          const int32_t* __restrict__ dst, const double* __restrict__ rec, int lane) {
  constexpr int nc = ScanRec<DIM>::n;
  const int64_t k0 = (int64_t)c * kScanChunk;
  const double* from = rec + k0 * nc;
  double* to = s.cst[c & 3];
#pragma unroll 10
  for (int x = lane; x < n * nc; x += 32) to[x] = from[x];
  if (lane < n) {
    s.src[c & 3][lane] = src[k0 + lane];
    s.dst[c & 3][lane] = dst[k0 + lane];
  }
}

template <int DIM>
__device__ void scan_cov(int64_t count, const int32_t* __restrict__ src, const int32_t* __restrict__ dst,
                         const double* __restrict__ rec, TrajView tr, ScanCov<DIM>& s) {
  constexpr int roles = DIM == 3 ? 3 : 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int chunks = (int)((count + kScanChunk - 1) / kScanChunk);
  double S = 0.0;
  int32_t last = -1;
  // warp w < roles works on chunk it - 1 - w, the last warp loads chunk it
  for (int it = 0; it < chunks + roles; ++it) {
    const int c = warp < roles ? it - 1 - warp : it;
    if (c >= 0 && c < chunks) {
      const int n = (int)min((int64_t)kScanChunk, count - (int64_t)c * kScanChunk);
      if (warp == 0) scan_chunk<DIM, 0>(c, n, s, tr.cov, S, last, lane);
      else if (DIM == 3 && warp == 1) scan_chunk<DIM, DIM == 3 ? 1 : 0>(c, n, s, tr.cov, S, last, lane);
      else if (DIM == 3 && warp == 2) scan_chunk<DIM, DIM == 3 ? 2 : 0>(c, n, s, tr.cov, S, last, lane);
      else if (warp == 3) scan_load<DIM>(c, n, s, src, dst, rec, lane);
    }
    __syncthreads();
  }
}

// The poses (and node counts): lane e computes entry e of the new pose, the
// operations of p3_compose / p2_compose (one instruction stream for all
// entries: diverging lanes would issue theirs one after another).
template <int DIM, int MODE>
__device__ void scan_pose(int64_t count, const int32_t* __restrict__ src, const int32_t* __restrict__ dst,
                          const double* __restrict__ dpose, const uint8_t* __restrict__ drot, TrajView tr,
                          ScanPose<DIM>& s) {
  constexpr int st = Lie<DIM>::stride;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int chunks = (int)((count + kScanChunk - 1) / kScanChunk);
  double P = 0.0;
  int32_t last = -1, node = 0;
  uint8_t rot = 0;
  const int e = lane < st ? lane : 0;
  const int i = e < 9 ? e / 3 : e - 9, j = e < 9 ? e % 3 : 0;
  for (int it = 0; it <= chunks; ++it) {
    const int c = warp == 0 ? it - 1 : it;
    const int64_t k0 = (int64_t)c * kScanChunk;
    const int n = c >= 0 && c < chunks ? (int)min((int64_t)kScanChunk, count - k0) : 0;
    if (warp == 3) {
      for (int x = lane; x < n * st; x += 32) s.dp[c & 1][x / st][x % st] = dpose[k0 * st + x];
      if (lane < n) {
        s.src[c & 1][lane] = src[k0 + lane];
        s.dst[c & 1][lane] = dst[k0 + lane];
        s.rot[c & 1][lane] = drot[k0 + lane];
      }
    } else if (warp == 0) {
      for (int k = 0; k < n; ++k) {
        const double* D = s.dp[c & 1][k];
        const int32_t from = s.src[c & 1][k], to = s.dst[c & 1][k];
        if (from != last) {  // the chain continues from an older pose: read it back
          __syncwarp();
          P = tr.pose[(size_t)from * st + e];
          rot = tr.rot[from];
          if (MODE == 1) node = tr.node[from];
        }
        if constexpr (DIM == 3) {
          const bool t = e >= 9;
          const double x0 = t ? D[9] : D[j], x1 = t ? D[10] : D[3 + j], x2 = t ? D[11] : D[6 + j];
          double acc = fmad(shfl_d(P, 3 * i), x0, t ? P : -0.0);
          acc = fmad(shfl_d(P, 3 * i + 1), x1, acc);
          P = fmad(shfl_d(P, 3 * i + 2), x2, acc);
        } else {
          // (c, s, x, y): u and w are the two products of the entry's formula
          const double ac = shfl_d(P, 0), as = shfl_d(P, 1);
          const double u = mul(e & 1 ? ac : as, e < 2 ? D[1] : D[3]);
          const double w = fmad(e & 1 ? as : ac, e < 2 ? D[0] : D[2], e & 1 ? u : -u);
          const double x = add(P, w);
          P = e < 2 ? w : x;
        }
        rot = rot && s.rot[c & 1][k] ? 1 : 0;
        ++node;
        if (lane < st) tr.pose[(size_t)to * st + lane] = P;
        if (lane == 0) {
          tr.rot[to] = rot;
          if (MODE == 1) tr.node[to] = node;
        }
        last = to;
      }
    }
    __syncthreads();
  }
}

// block 0: the covariances (MODE 0), the other one: the poses
template <int DIM, int MODE>
__global__ void __launch_bounds__(128) k_traj_scan(int64_t count, const int32_t* __restrict__ src,
                                                   const int32_t* __restrict__ dst,
                                                   const double* __restrict__ dpose,
                                                   const double* __restrict__ rec,
                                                   const uint8_t* __restrict__ drot, TrajView tr) {
  __shared__ __align__(8) unsigned char raw[sizeof(ScanCov<DIM>) > sizeof(ScanPose<DIM>) ? sizeof(ScanCov<DIM>)
                                                                                       : sizeof(ScanPose<DIM>)];
  if (MODE == 0 && blockIdx.x == 0)
    scan_cov<DIM>(count, src, dst, rec, tr, *reinterpret_cast<ScanCov<DIM>*>(raw));
  else
    scan_pose<DIM, MODE>(count, src, dst, dpose, drot, tr, *reinterpret_cast<ScanPose<DIM>*>(raw));
}

// ------------------------------------------------------------------ K1
template <int DIM, class U>
__global__ void k_odom_check(int64_t count, const int32_t* __restrict__ si, const int32_t* __restrict__ sj,
                             const double* __restrict__ zp, const double* __restrict__ zc, TrajView tr, double th0,
                             double th1, uint8_t* __restrict__ ok) {
  using L = Lie<DIM>;
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= count) return;
  U a, b, pij, z, res;
  a.from_traj(tr, si[k]);
  b.from_traj(tr, sj[k]);
  a.between(b, pij);
  z.from_factor(zp + k * L::stride, zc + k * L::d * L::d);
  z.inverse_inplace();
  pij.compose(z, res);
  ok[k] = check_u<DIM>(res, th0, th1) ? 1 : 0;
}

// ------------------------------------------------------------------ K2
// Per-closure constants of the 3D PoseWithCovariance test: the rotation of
// the inverse of each measured pose and the K block of that inverse's adjoint
// (what each composition with the closure computes first), 18 doubles per
// closure. The pairwise test uses them instead of recomputing them per pair:
// the same operations, so the same bits.
constexpr int kClosurePre = 18;
__global__ void k_closure_pre3(int n, const double* __restrict__ zp, double* __restrict__ pre) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  pm::P3 Z, inv;
  pm::p3_load(zp + (size_t)k * 12, Z);
  pm::p3_inverse(Z, inv);
  double* o = pre + (size_t)k * kClosurePre;
#pragma unroll
  for (int e = 0; e < 9; ++e) o[e] = inv.R[e];
  pm::p3_adjoint_K(inv, o + 9);
}

template <int DIM, class U>
__device__ __forceinline__ bool pair_consistent(int i, int j, const int32_t* __restrict__ sa,
                                                const int32_t* __restrict__ sb, const uint8_t* __restrict__ flip,
                                                const double* __restrict__ zp, const double* __restrict__ zc,
                                                const TrajView& tr, double th0, double th1,
                                                const double* __restrict__ pre) {
  using L = Lie<DIM>;
  int a = sa[i], b = sb[i], c = sa[j], dd = sb[j];
  if (flip[i] != flip[j]) {
    const int t = c;
    c = dd;
    dd = t;
  }
  U A, B, Ta, Tc, Zj, Zi, P, Q, loop;
  Ta.from_traj(tr, a);
  Tc.from_traj(tr, c);
  Ta.between(Tc, A);
  Ta.from_traj(tr, b);
  Tc.from_traj(tr, dd);
  Ta.between(Tc, B);
  Zj.from_factor(zp + (size_t)j * L::stride, zc + (size_t)j * L::d * L::d);
  Zi.from_factor(zp + (size_t)i * L::stride, zc + (size_t)i * L::d * L::d);
  if constexpr (std::is_same<U, PWC<3>>::value) {
    A.compose_pre(Zj, pre + (size_t)j * kClosurePre, P);
    P.inverse_inplace();
    P.compose_pre(Zi, pre + (size_t)i * kClosurePre, Q);
  } else {
    A.compose(Zj, P);
    P.inverse_inplace();
    P.compose(Zi, Q);
  }
  Q.compose(B, loop);
  return check_u<DIM>(loop, th0, th1);
}

// Landmark pair (Pcm.h:775-844): observations i, j (pose -> landmark) of one
// landmark. i_odom_j = getBetween(pose_i, pose_j) of pose_i's trajectory
// (GraphUtils.h:37-58): slots (s.x, s.y) for one robot; for two robots
// (s.x, s.y, s.z, s.w) = (root a0, pose_i, root b0, pose_j) as looked up in
// pose_i's trajectory. loop = (i_odom_j o Z_j)^-1 o Z_i.
template <int DIM, class U>
__global__ void k_landmark_pairs(int count, const int4* __restrict__ desc, const int2* __restrict__ ij,
                                 const double* __restrict__ zp, const double* __restrict__ zc, TrajView tr,
                                 double th0, double th1, uint32_t* __restrict__ adj, int words) {
  using L = Lie<DIM>;
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= count) return;
  const int4 s = desc[k];
  const int i = ij[k].x, j = ij[k].y;
  U iodomj, X, Y;
  if (s.z < 0) {
    X.from_traj(tr, s.x);
    Y.from_traj(tr, s.y);
    X.between(Y, iodomj);
  } else {
    U pa, pb, pab, t;
    X.from_traj(tr, s.x);
    Y.from_traj(tr, s.y);
    X.between(Y, pa);
    U B0, Kb;
    B0.from_traj(tr, s.z);
    Kb.from_traj(tr, s.w);
    B0.between(Kb, pb);
    X.between(B0, pab);
    pa.inverse_inplace();
    pa.compose(pab, t);
    t.compose(pb, iodomj);
  }
  U zj, zi, path, loop;
  zj.from_factor(zp + (size_t)j * L::stride, zc + (size_t)j * L::d * L::d);
  iodomj.compose(zj, path);
  path.inverse_inplace();
  zi.from_factor(zp + (size_t)i * L::stride, zc + (size_t)i * L::d * L::d);
  path.compose(zi, loop);
  if (check_u<DIM>(loop, th0, th1)) {
    atomicOr(adj + (size_t)i * words + (j >> 5), 1u << (j & 31));
    atomicOr(adj + (size_t)j * words + (i >> 5), 1u << (i & 31));
  }
}

// block (32, ROWS): lane -> column i = 32*bx + lane, row j = row_begin + ROWS*by + ty.
// lower[(j - row_begin) * words + bx] receives bits i < j.
template <int DIM, class U, int ROWS>
__global__ void __launch_bounds__(32 * ROWS) k_pairwise(int n, int row_begin, const int32_t* __restrict__ sa,
                                                        const int32_t* __restrict__ sb,
                                                        const uint8_t* __restrict__ flip,
                                                        const double* __restrict__ zp,
                                                        const double* __restrict__ zc, TrajView tr, double th0,
                                                        double th1, uint32_t* __restrict__ lower, int words,
                                                        const double* __restrict__ pre) {
  const int lane = threadIdx.x;
  const int j = row_begin + ROWS * blockIdx.y + threadIdx.y;
  const int i0 = 32 * blockIdx.x;
  if (j >= n || i0 >= j) return;  // whole warp: tile above the diagonal or past the end
  const int i = i0 + lane;
  bool ok = false;
  if (i < j) ok = pair_consistent<DIM, U>(i, j, sa, sb, flip, zp, zc, tr, th0, th1, pre);
  const unsigned bits = __ballot_sync(0xffffffffu, ok);
  if (lane == 0) lower[(size_t)(j - row_begin) * words + blockIdx.x] = bits;
}

// The PoseWithCovariance test of many pairs: FP32 with an error bound
// decides more than 99 % of them (pcm_filter.cuh; on the walks of 2,000 and
// 12,000 poses 99.92 and 99.5 %, wherever the map lies in its frame), the exact
// FP64 test the rest.
// The FP64 pipe issues a warp instruction in 64 cycles, FP32 in one, and a
// `between` in pairs of FP32 costs about 12 FP32 instructions per FP64 FMA:
// 10,900 instructions per 32 pairs where the exact test takes 165,000 cycles.
// 3D, 4,001 closures: 35.0 -> 3.6 ms; 16,000: 556 -> 55 ms. 2D, 3,000 closures:
// 5.3 -> 0.6 ms; 12,000: 80.7 -> 7.7 ms. Bound by FP32 issue (0.67 of its
// slots). The code is larger than the first-level instruction cache, so the
// phases' loops are rolled (16,000 closures in 3D, when the exact test still
// took 6 ms more of it: 115 -> 63 ms) and the 12 warps of a block go through the
// phases together (-> 60 ms; with 4, 8 and 16 warps 64, 66 and 72 ms).
// k_pair_filter leaves its verdicts in `lower` and its unsure pairs as bits in
// `unsure` (both one word per 32 x 1 tile); k_pair_exact gathers those bits
// into full warps and adds the consistent ones to `lower`.

// per-closure data of the filter: a thread per value, the last one the closure's premises
template <int DIM>
__global__ void k_filter_pack(int n, const int32_t* __restrict__ sa, const int32_t* __restrict__ sb,
                              const uint8_t* __restrict__ flip, const double* __restrict__ zp,
                              const double* __restrict__ zc, TrajView tr,
                              pf::D2* __restrict__ df, float* __restrict__ f, uint8_t* __restrict__ ok) {
  using F = pf::Filter<DIM>;
  constexpr int st = Lie<DIM>::stride, dd = Lie<DIM>::d * Lie<DIM>::d;
  const int k = blockIdx.x * blockDim.x + threadIdx.x, v = blockIdx.y;
  if (k >= n) return;
  const size_t a = sa[k], b = sb[k];
  const double *pa = tr.pose + a * st, *pb = tr.pose + b * st, *ca = tr.cov + a * dd, *cb = tr.cov + b * dd;
  const double *z = zp + (size_t)k * st, *c = zc + (size_t)k * dd;
  const pf::Origin o =
      pf::origin(tr.pose + (size_t)sa[0] * st, tr.pose + (size_t)sb[0] * st, flip[k] != flip[0]);
  if (v < F::pairs)
    df[(size_t)v * n + k] = F::pair(v, pa, ca, pb, cb, z, o);
  else if (v < F::pairs + F::floats)
    f[(size_t)(v - F::pairs) * n + k] = F::single(v - F::pairs, pa, ca, pb, cb, z, c, o);
  else
    ok[k] = tr.rot[a] && tr.rot[b] && F::premise(pa, ca, pb, cb, z, c);
}

struct BlockSync {
  __device__ void operator()() const { __syncthreads(); }
};
template <int DIM, int ROWS>
__global__ void __launch_bounds__(32 * ROWS) k_pair_filter(int n, int row_begin, const uint8_t* __restrict__ flip,
                                                           pf::Group g, float th2, uint32_t* __restrict__ lower,
                                                           uint32_t* __restrict__ unsure, int words) {
  const int lane = threadIdx.x;
  const int j0 = row_begin + ROWS * blockIdx.y, i0 = 32 * blockIdx.x;
  if (i0 >= min(j0 + ROWS, n) - 1) return;  // whole block: tiles above the diagonal
  const int j = min(j0 + (int)threadIdx.y, n - 1), i = min(i0 + lane, n - 1);
  const int r = pf::Filter<DIM>::test(g, i, j, flip[i] != flip[j], th2, BlockSync());
  const bool pair = j0 + (int)threadIdx.y < n && i0 + lane < j;
  const unsigned yes = __ballot_sync(0xffffffffu, pair && r == 1), open = __ballot_sync(0xffffffffu, pair && r == 2);
  if (lane == 0 && j0 + (int)threadIdx.y < n && i0 < j) {
    const size_t w = (size_t)(j - row_begin) * words + blockIdx.x;
    lower[w] = yes;
    unsure[w] = open;
  }
}

constexpr int kExactThreads = 128;
// each block takes `chunk` consecutive words of the rows x nb tiles: their set
// bits go to a list in shared memory, which the block works off a full block at a time
template <int DIM>
__global__ void __launch_bounds__(kExactThreads) k_pair_exact(
    int n, int row_begin, int nb, int64_t chunk, const int32_t* __restrict__ sa, const int32_t* __restrict__ sb,
    const uint8_t* __restrict__ flip, const double* __restrict__ zp, const double* __restrict__ zc, TrajView tr,
    double th0, const uint32_t* __restrict__ unsure, uint32_t* __restrict__ lower, int words,
    const double* __restrict__ pre) {
  __shared__ int2 list[33 * kExactThreads];
  __shared__ int count;
  const int64_t total = (int64_t)(n - row_begin) * nb;
  const int64_t t0 = blockIdx.x * chunk, t1 = min(total, t0 + chunk);
  if (threadIdx.x == 0) count = 0;
  __syncthreads();
  for (int64_t t = t0; t < t1 || count > 0; t += kExactThreads) {
    const int64_t u = t + threadIdx.x;
    if (u < t1) {
      const int row = (int)(u / nb), bx = (int)(u % nb), j = row_begin + row;
      uint32_t m = 32 * bx < j ? unsure[(size_t)row * words + bx] : 0u;
      if (m) {
        int at = atomicAdd(&count, __popc(m));
        for (; m; m &= m - 1) list[at++] = make_int2(32 * bx + __ffs(m) - 1, j);
      }
    }
    __syncthreads();
    const bool last = t + kExactThreads >= t1;
    // (count is read by all before it changes: the barrier below)
    int left = count;
    while (left >= kExactThreads || (last && left > 0)) {
      const int take = min(left, kExactThreads);
      left -= take;
      if ((int)threadIdx.x < take) {
        const int2 p = list[left + threadIdx.x];
        if (pair_consistent<DIM, PWC<DIM>>(p.x, p.y, sa, sb, flip, zp, zc, tr, th0, 0.0, pre))
          atomicOr(lower + (size_t)(p.y - row_begin) * words + (p.x >> 5), 1u << (p.x & 31));
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) count = left;
    __syncthreads();
  }
}

// Mirror: adj[r][c] for c < r from lower rows (r >= row_begin) or the old
// matrix (r < row_begin); for c > r from lower[c][r] (c >= row_begin) or the
// old matrix. One warp per 32x32 block, lane = row within the block.
__global__ void k_symmetrize(int n, int row_begin, const uint32_t* __restrict__ lower, uint32_t* __restrict__ adj,
                             int words) {
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nb = (n + 31) / 32;
  if (warp >= nb * nb) return;
  const int bi = warp / nb, bj = warp % nb;
  const int r = 32 * bi + lane;
  // transpose source: word (rows c = 32*bj + lane) column block bi of lower
  const int c_src = 32 * bj + lane;
  uint32_t src = 0;
  if (c_src < n && c_src >= row_begin) src = lower[(size_t)(c_src - row_begin) * words + bi];
  uint32_t tr_word = 0;
#pragma unroll 4
  for (int b = 0; b < 32; ++b) {
    const uint32_t col = __ballot_sync(0xffffffffu, (src >> b) & 1u);
    if (b == lane) tr_word = col;  // bits over c of row 32*bi + b
  }
  if (r >= n) return;
  const uint32_t old = (r < row_begin) ? adj[(size_t)r * words + bj] : 0u;
  uint32_t out = 0;
  // column mask helpers within block bj
  const int c0 = 32 * bj;
  uint32_t lt = 0, gt = 0, valid = 0;
  for (int b = 0; b < 32; ++b) {
    const int c = c0 + b;
    if (c >= n) break;
    valid |= 1u << b;
    if (c < r) lt |= 1u << b;
    if (c > r) gt |= 1u << b;
  }
  // lower part
  if (r >= row_begin) out |= lower[(size_t)(r - row_begin) * words + bj] & lt;
  else out |= old & lt;
  // upper part: new columns from the transpose, old columns from the old matrix
  uint32_t newcols = 0;
  for (int b = 0; b < 32; ++b)
    if (c0 + b >= row_begin && c0 + b < n) newcols |= 1u << b;
  out |= tr_word & gt & newcols;
  out |= old & gt & ~newcols;
  adj[(size_t)r * words + bj] = out & valid;
}

}  // namespace

// ------------------------------------------------------------------ launchers
void launch_traj_scan(int dim, int mode, int64_t count, const int32_t* src, const int32_t* dst,
                      const double* dpose, const double* dcov, TrajView tr, DeviceBuffer<double>& scratch_rec,
                      DeviceBuffer<uint8_t>& scratch_rot, cudaStream_t st) {
  if (count <= 0) return;
  scratch_rec.resize((size_t)count * (dim == 3 ? ScanRec<3>::n : ScanRec<2>::n));
  scratch_rot.resize((size_t)count);
  const int tb = 128;
  if (dim == 3)
    k_odom_prep<3><<<div_up(count, tb), tb, 0, st>>>(count, dpose, dcov, scratch_rec.get(), scratch_rot.get());
  else
    k_odom_prep<2><<<div_up(count, tb), tb, 0, st>>>(count, dpose, dcov, scratch_rec.get(), scratch_rot.get());
  RPGO_LAUNCHED();
  const int blocks = mode == 0 ? 2 : 1;
  auto scan = [&](auto kernel) {
    kernel<<<blocks, 128, 0, st>>>(count, src, dst, dpose, scratch_rec.get(), scratch_rot.get(), tr);
  };
  if (dim == 3) {
    if (mode == 0) scan(k_traj_scan<3, 0>);
    else scan(k_traj_scan<3, 1>);
  } else {
    if (mode == 0) scan(k_traj_scan<2, 0>);
    else scan(k_traj_scan<2, 1>);
  }
  RPGO_LAUNCHED();
}

void launch_odom_check(int dim, int mode, int64_t count, const int32_t* si, const int32_t* sj, const double* zp,
                       const double* zc, TrajView tr, double th0, double th1, uint8_t* ok, cudaStream_t st) {
  if (count <= 0) return;
  const int tb = 64;
  const int g = div_up(count, tb);
  if (dim == 3) {
    if (mode == 0) k_odom_check<3, PWC<3>><<<g, tb, 0, st>>>(count, si, sj, zp, zc, tr, th0, th1, ok);
    else k_odom_check<3, PWN<3>><<<g, tb, 0, st>>>(count, si, sj, zp, zc, tr, th0, th1, ok);
  } else {
    if (mode == 0) k_odom_check<2, PWC<2>><<<g, tb, 0, st>>>(count, si, sj, zp, zc, tr, th0, th1, ok);
    else k_odom_check<2, PWN<2>><<<g, tb, 0, st>>>(count, si, sj, zp, zc, tr, th0, th1, ok);
  }
  RPGO_LAUNCHED();
}

namespace {
// The filter's memory, held for the call: 801 bytes per closure in 3D, 269 in
// 2D, and the unsure pairs, a bit each, as many words as the new rows of the
// adjacency (50 MB at 20,000 closures, 1.25 GB at 100,000).
struct PairFilter {
  DeviceBuffer<pf::D2> df;
  DeviceBuffer<float> f;
  DeviceBuffer<uint8_t> ok;
  DeviceBuffer<uint32_t> unsure;
  void resize(int dim, int n, size_t tiles) {
    df.resize((size_t)(dim == 3 ? pf::Filter<3>::pairs : pf::Filter<2>::pairs) * n);
    f.resize((size_t)(dim == 3 ? pf::Filter<3>::floats : pf::Filter<2>::floats) * n);
    ok.resize(n);
    unsure.resize(tiles);
  }
};

template <int DIM>
void pair_filter(PairFilter& p, int n, int row_begin, const int32_t* sa, const int32_t* sb, const uint8_t* flip,
                 const double* zp, const double* zc, TrajView tr, double th, uint32_t* lower, int words,
                 const double* pre, cudaStream_t st) {
  using F = pf::Filter<DIM>;
  constexpr int FR = 12;
  const int rows = n - row_begin;
  k_filter_pack<DIM><<<dim3(div_up(n, 128), F::pairs + F::floats + 1), 128, 0, st>>>(
      n, sa, sb, flip, zp, zc, tr, p.df.get(), p.f.get(), p.ok.get());
  RPGO_LAUNCHED();
  const pf::Group g{p.df.get(), p.f.get(), p.ok.get(), n};
  k_pair_filter<DIM, FR><<<dim3(div_up(n, 32), div_up(rows, FR)), dim3(32, FR), 0, st>>>(
      n, row_begin, flip, g, (float)(th * th), lower, p.unsure.get(), words);
  RPGO_LAUNCHED();
  const int nb = div_up(n, 32), blocks = 4 * device_sm_count();
  const int64_t chunk = std::max<int64_t>(kExactThreads, ((int64_t)rows * nb + blocks - 1) / blocks);
  k_pair_exact<DIM><<<div_up((int64_t)rows * nb, chunk), kExactThreads, 0, st>>>(
      n, row_begin, nb, chunk, sa, sb, flip, zp, zc, tr, th, p.unsure.get(), lower, words, pre);
}
}  // namespace

void launch_pairwise(int dim, int mode, int n, int row_begin, const int32_t* sa, const int32_t* sb,
                     const uint8_t* flip, const double* zp, const double* zc, TrajView tr, double th0, double th1,
                     uint32_t* adj, int words, uint32_t* lower_scratch, cudaStream_t st) {
  if (n <= 0 || row_begin >= n) return;
  constexpr int ROWS = 4;
  const int rows = n - row_begin;
  dim3 block(32, ROWS), grid(div_up(n, 32), div_up(rows, ROWS));
  if (n > 1) {
    DeviceBuffer<double> pre;
    if (dim == 3 && mode == 0) {
      pre.resize((size_t)n * kClosurePre);
      k_closure_pre3<<<div_up(n, 128), 128, 0, st>>>(n, zp, pre.get());
      RPGO_LAUNCHED();
    }
    // The filter and the exact test of what it leaves take two launches, and
    // the second lasts at least one exact test (90 us) where it has any pair:
    // below 65,536 pairs, which the exact test alone takes in three waves,
    // they are not faster. (2D, exact alone and with the filter: 363 closures,
    // 65,703 pairs, 0.30 and 0.28 ms with the transfers; 1,000: 0.79 and 0.35.)
    const double pairs = 0.5 * n * (n - 1.0) - 0.5 * row_begin * (row_begin - 1.0);
    const bool filter = mode == 0 && pairs >= 65536.0 && th0 > 0.0 && th0 < 1e15;
    PairFilter pack;
    if (filter) pack.resize(dim, n, (size_t)rows * words);
    EventTimer timer(st);
    if (filter && dim == 3) {
      pair_filter<3>(pack, n, row_begin, sa, sb, flip, zp, zc, tr, th0, lower_scratch, words, pre.get(), st);
    } else if (filter) {
      pair_filter<2>(pack, n, row_begin, sa, sb, flip, zp, zc, tr, th0, lower_scratch, words, nullptr, st);
    } else if (dim == 3) {
      if (mode == 0)
        k_pairwise<3, PWC<3>, ROWS><<<grid, block, 0, st>>>(n, row_begin, sa, sb, flip, zp, zc, tr, th0, th1,
                                                            lower_scratch, words, pre.get());
      else
        k_pairwise<3, PWN<3>, ROWS><<<grid, block, 0, st>>>(n, row_begin, sa, sb, flip, zp, zc, tr, th0, th1,
                                                            lower_scratch, words, nullptr);
    } else {
      if (mode == 0)
        k_pairwise<2, PWC<2>, ROWS><<<grid, block, 0, st>>>(n, row_begin, sa, sb, flip, zp, zc, tr, th0, th1,
                                                            lower_scratch, words, nullptr);
      else
        k_pairwise<2, PWN<2>, ROWS><<<grid, block, 0, st>>>(n, row_begin, sa, sb, flip, zp, zc, tr, th0, th1,
                                                            lower_scratch, words, nullptr);
    }
    RPGO_LAUNCHED();
    kernel_times().pair_ms += timer.elapsed_ms();
    kernel_times().pair_launches += 1;
  }
  // rows whose tiles were all skipped (j < 32*bx) keep stale words; the
  // ballot writes only tiles with i0 < j, so clear the rest first: the
  // mirror kernel reads only words bx <= j/32, all of which were written
  // except word j/32 when 32*(j/32) >= j, i.e. j a multiple of 32 -> handled
  // by masking with c < r in the mirror.
  const int nb = div_up(n, 32);
  const int warps = nb * nb;
  k_symmetrize<<<div_up((int64_t)warps * 32, 256), 256, 0, st>>>(n, row_begin, lower_scratch, adj, words);
  RPGO_LAUNCHED();
}

void launch_landmark_pairs(int dim, int mode, int count, const int4* desc, const int2* ij, const double* zp,
                           const double* zc, TrajView tr, double th0, double th1, uint32_t* adj, int words,
                           cudaStream_t st) {
  if (count <= 0) return;
  const int tb = 128, nb = div_up(count, tb);
  if (dim == 3) {
    if (mode == 0) k_landmark_pairs<3, PWC<3>><<<nb, tb, 0, st>>>(count, desc, ij, zp, zc, tr, th0, th1, adj, words);
    else k_landmark_pairs<3, PWN<3>><<<nb, tb, 0, st>>>(count, desc, ij, zp, zc, tr, th0, th1, adj, words);
  } else {
    if (mode == 0) k_landmark_pairs<2, PWC<2>><<<nb, tb, 0, st>>>(count, desc, ij, zp, zc, tr, th0, th1, adj, words);
    else k_landmark_pairs<2, PWN<2>><<<nb, tb, 0, st>>>(count, desc, ij, zp, zc, tr, th0, th1, adj, words);
  }
  RPGO_LAUNCHED();
}

namespace {
// rows [0, rows): clear every bit of columns >= from
__global__ void k_clear_columns(uint32_t* __restrict__ adj, int words, int rows, int from) {
  const int w0 = from >> 5;
  const int per_row = words - w0;
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (per_row <= 0 || t >= (int64_t)rows * per_row) return;
  const int r = (int)(t / per_row), w = w0 + (int)(t % per_row);
  uint32_t* word = adj + (size_t)r * words + w;
  *word = (w == w0) ? (*word & ((1u << (from & 31)) - 1u)) : 0u;
}
}  // namespace

void launch_clear_columns(uint32_t* adj, int words, int rows, int from, cudaStream_t st) {
  const int per_row = words - (from >> 5);
  if (rows <= 0 || per_row <= 0) return;
  const int64_t n = (int64_t)rows * per_row;
  k_clear_columns<<<div_up(n, 256), 256, 0, st>>>(adj, words, rows, from);
  RPGO_LAUNCHED();
}

std::atomic<int64_t>& launch_counter() {
  static std::atomic<int64_t> c{0};
  return c;
}
std::atomic<int64_t>& alloc_counter() {
  static std::atomic<int64_t> c{0};
  return c;
}
int64_t& thread_launch_counter() {
  thread_local int64_t c = 0;
  return c;
}
KernelTimes& kernel_times() {
  thread_local KernelTimes t;
  return t;
}
cudaStream_t& alloc_stream() {
  thread_local cudaStream_t st = nullptr;
  return st;
}

}  // namespace rpgo
