// Learned GNC warm start kernels: closure features, the closure network's
// forward pass, and its training step (forward + backward + Adam).
//
// The network is tiny (5,313 trainable parameters) and its batches are a few
// thousand closures: one thread per closure for inference with the whole
// parameter set in shared memory (weights rounded to BF16 once per block, FP32
// FMAs), and a training step in two kernels (below). Every sum runs in a fixed
// order, so a training step is reproducible bit for bit.
#include <cuda_bf16.h>

#include "solver_kernels.hpp"
#include "solver_math.cuh"
#include "warm.hpp"

namespace rpgo {
namespace {

using namespace sm;

// ------------------------------------------------------------------ features
template <int DIM>
__global__ void k_closure_features(int nlc, int n_known, const int32_t* __restrict__ kind,
                                   const int32_t* __restrict__ vi, const int32_t* __restrict__ vj,
                                   const double* __restrict__ z, const double* __restrict__ R,
                                   const double* __restrict__ x0, const float* __restrict__ aux,
                                   float* __restrict__ out) {
  using L = SLie<DIM>;
  constexpr int d = L::d, st = L::stride;
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= nlc) return;
  const int f = n_known + q;
  float* o = out + (size_t)q * kFeat;
  if (kind[f] != 0) {
    for (int k = 0; k < kFeat; ++k) o[k] = 0.f;
    return;
  }
  typename L::Pose Xi, Xj, Z, h, rel;
  L::load(x0 + (size_t)vi[f] * st, Xi);
  L::load(x0 + (size_t)vj[f] * st, Xj);
  L::load(z + (size_t)f * st, Z);
  L::between(Xi, Xj, h);
  L::between(Z, h, rel);
  double e[d], ez[d];
  L::logmap(rel, e);
  L::logmap(Z, ez);
  const double* Rf = R + (size_t)f * d * d;
  double c = 0.0;
#pragma unroll
  for (int i = 0; i < 6; ++i) {
    double r = 0.0;
    if (i < d) {
#pragma unroll
      for (int k = 0; k < d; ++k) r += Rf[d * i + k] * e[k];
      c += r * r;
    }
    o[i] = (float)log1p(fabs(r));
  }
  double rot, tr, zrot, ztr;
  if (DIM == 3) {
    rot = sqrt(e[0] * e[0] + e[1] * e[1] + e[2] * e[2]);
    tr = sqrt(e[3] * e[3] + e[4] * e[4] + e[5] * e[5]);
    zrot = sqrt(ez[0] * ez[0] + ez[1] * ez[1] + ez[2] * ez[2]);
    const double* zt = z + (size_t)f * st + 9;
    ztr = sqrt(zt[0] * zt[0] + zt[1] * zt[1] + zt[2] * zt[2]);
  } else {
    rot = fabs(e[d - 1]);
    tr = sqrt(e[0] * e[0] + e[1] * e[1]);
    zrot = fabs(ez[d - 1]);
    const double* zt = z + (size_t)f * st + 2;
    ztr = sqrt(zt[0] * zt[0] + zt[1] * zt[1]);
  }
  const float* a = aux + (size_t)q * 4;
  const double gap = a[0];
  o[6] = (float)log1p(c);
  o[7] = (float)rot;
  o[8] = (float)log1p(tr);
  o[9] = (float)log1p(gap);
  o[10] = (float)log1p(c / fmax(1.0, gap));
  o[11] = a[1];
  o[12] = a[2];
  o[13] = a[3];
  o[14] = (float)log1p(ztr);
  o[15] = (float)zrot;
}

// one warp per listed row: popcount of the row and of the row AND mask
__global__ void k_row_stats(int n, const uint32_t* __restrict__ adj, int words, const uint32_t* __restrict__ mask,
                            const int32_t* __restrict__ rows, int count, int32_t* __restrict__ deg,
                            int32_t* __restrict__ support) {
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= count) return;
  const uint32_t* row = adj + (size_t)rows[w] * words;
  const int nw = (n + 31) / 32;
  int a = 0, b = 0;
  for (int k = lane; k < nw; k += 32) {
    const uint32_t x = row[k];
    a += __popc(x);
    b += __popc(x & mask[k]);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  if (lane == 0) {
    deg[w] = a;
    support[w] = b;
  }
}

// ------------------------------------------------------------------ network
constexpr int kTpb = 128;

__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// parameters into shared memory, weights rounded to BF16
__device__ __forceinline__ void load_params(const float* __restrict__ params, float* sp) {
  for (int k = threadIdx.x; k < kMlpParams; k += blockDim.x) {
    const float v = params[k];
    const bool weight = (k >= kOffW1 && k < kOffB1) || (k >= kOffW2 && k < kOffB2) || (k >= kOffW3 && k < kOffB3);
    sp[k] = weight ? bf16_round(v) : v;
  }
  __syncthreads();
}

__device__ __forceinline__ void normalise(const float* sp, const float* __restrict__ x, float* xn) {
#pragma unroll
  for (int i = 0; i < kFeat; ++i) xn[i] = (x[i] - sp[kOffMu + i]) * sp[kOffIsd + i];
}

__device__ __forceinline__ void layer1(const float* sp, const float* xn, float* h1) {
#pragma unroll
  for (int j = 0; j < kHid; ++j) {
    float acc = sp[kOffB1 + j];
#pragma unroll
    for (int i = 0; i < kFeat; ++i) acc = fmaf(sp[kOffW1 + j * kFeat + i], xn[i], acc);
    h1[j] = fmaxf(acc, 0.f);
  }
}

__device__ __forceinline__ float hidden2(const float* sp, const float* h1, int j) {
  float acc = sp[kOffB2 + j];
#pragma unroll
  for (int i = 0; i < kHid; ++i) acc = fmaf(sp[kOffW2 + j * kHid + i], h1[i], acc);
  return fmaxf(acc, 0.f);
}

__global__ void __launch_bounds__(kTpb) k_mlp_forward(int64_t n, const float* __restrict__ params,
                                                      const float* __restrict__ X, float* __restrict__ prob) {
  __shared__ float sp[kMlpParams];
  load_params(params, sp);
  const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  float xn[kFeat], h1[kHid];
  normalise(sp, X + s * kFeat, xn);
  layer1(sp, xn, h1);
  float logit = sp[kOffB3];
  for (int j = 0; j < kHid; ++j) logit = fmaf(sp[kOffW3 + j], hidden2(sp, h1, j), logit);
  prob[s] = 1.f / (1.f + expf(-logit));
}

// ------------------------------------------------------------------ training step
// One block takes kTS samples through the forward and the backward pass and
// sums their gradients, everything in shared memory: activations and errors as
// [unit][sample] rows, four samples by four units per thread in the layers,
// four by four parameters per thread in the gradient sums. The blocks' sums
// are added in block order by k_mlp_reduce, which also takes the Adam step.
// Bound by FP32 issue and shared-memory reads (4 float4 loads per 64 FMAs in the
// gradients, 2 per 16 in the layers). 8,192 samples: 1,120 us -> 50 us a call
// (before: one thread per parameter walked the whole batch through L2, 5,313
// threads on 42 blocks, with six arrays of activations written and read back).
constexpr int kTS = 64, kTSP = kTS + 4;  // samples per block; row stride (16-byte aligned, rows on different banks)
constexpr int kStepThreads = 256;

struct StepSmem {
  float xn[kFeat][kTSP], h1[kHid][kTSP], h2[kHid][kTSP], d1[kHid][kTSP];  // h2: then its errors
  float w1t[kFeat][kTSP], w2t[kHid][kTSP], w2[kHid][kHid];  // BF16-rounded; w1t, w2t: [input][unit]
  float b1[kHid], b2[kHid], w3[kHid], b3, dl[kTS];
  double loss[kTS / 32];
};

__device__ __forceinline__ void fma16(const float4& a, const float4& b, float (&acc)[4][4]) {
  const float x[4] = {a.x, a.y, a.z, a.w}, y[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int s = 0; s < 4; ++s) acc[u][s] = fmaf(x[u], y[s], acc[u][s]);
}
__device__ __forceinline__ float4 at4(const float* p) { return *reinterpret_cast<const float4*>(p); }

__global__ void __launch_bounds__(kStepThreads, 2) k_mlp_step(int64_t n, const float* __restrict__ params,
                                                              const float* __restrict__ X,
                                                              const float* __restrict__ Y, float inv_n,
                                                              float* __restrict__ part, double* __restrict__ loss) {
  extern __shared__ __align__(16) unsigned char raw[];
  StepSmem& s = *reinterpret_cast<StepSmem*>(raw);
  const int t = threadIdx.x;
  const int64_t s0 = (int64_t)blockIdx.x * kTS;
  for (int k = t; k < kHid * kFeat; k += kStepThreads)
    s.w1t[k % kFeat][k / kFeat] = bf16_round(params[kOffW1 + k]);
  for (int k = t; k < kHid * kHid; k += kStepThreads) {
    const float w = bf16_round(params[kOffW2 + k]);
    s.w2[k / kHid][k % kHid] = w;
    s.w2t[k % kHid][k / kHid] = w;
  }
  if (t < kHid) {
    s.b1[t] = params[kOffB1 + t];
    s.b2[t] = params[kOffB2 + t];
    s.w3[t] = bf16_round(params[kOffW3 + t]);
    if (t == 0) s.b3 = params[kOffB3];
  }
  for (int k = t; k < kTS * kFeat; k += kStepThreads) {
    const int i = k % kFeat, q = k / kFeat;
    s.xn[i][q] = s0 + q < n ? (X[(s0 + q) * kFeat + i] - params[kOffMu + i]) * params[kOffIsd + i] : 0.f;
  }
  __syncthreads();
  // ---- forward: units 4 y .. 4 y + 3 of samples 4 x .. 4 x + 3
  const int x = 4 * (t & 15), y = 4 * (t >> 4);
  float acc[4][4];
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[u][q] = s.b1[y + u];
#pragma unroll
  for (int i = 0; i < kFeat; ++i) fma16(at4(&s.w1t[i][y]), at4(&s.xn[i][x]), acc);
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int q = 0; q < 4; ++q) s.h1[y + u][x + q] = fmaxf(acc[u][q], 0.f);
  __syncthreads();
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[u][q] = s.b2[y + u];
#pragma unroll 8
  for (int i = 0; i < kHid; ++i) fma16(at4(&s.w2t[i][y]), at4(&s.h1[i][x]), acc);
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int q = 0; q < 4; ++q) s.h2[y + u][x + q] = fmaxf(acc[u][q], 0.f);
  __syncthreads();
  if (t < kTS) {
    float logit = s.b3;
#pragma unroll 16
    for (int j = 0; j < kHid; ++j) logit = fmaf(s.w3[j], s.h2[j][t], logit);
    const bool on = s0 + t < n;
    const float lab = on ? Y[s0 + t] : 0.f;
    const float p = 1.f / (1.f + expf(-logit));
    double l = on ? (double)(fmaxf(logit, 0.f) - logit * lab + log1pf(expf(-fabsf(logit)))) : 0.0;
#pragma unroll
    for (int o = 16; o; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if ((t & 31) == 0) s.loss[t >> 5] = l;
    s.dl[t] = on ? (p - lab) * inv_n : 0.f;
  }
  __syncthreads();
  float* const out = part + (size_t)blockIdx.x * kMlpTrainable - kOffW1;
  if (t == 0) loss[blockIdx.x] = s.loss[0] + s.loss[1];
  if (t <= kHid) {  // the last layer's gradients (thread kHid: its bias)
    float g = 0.f;
    for (int q = 0; q < kTS; ++q) g = fmaf(s.dl[q], t < kHid ? s.h2[t < kHid ? t : 0][q] : 1.f, g);
    out[t < kHid ? kOffW3 + t : kOffB3] = g;
  }
  __syncthreads();
  // ---- backward: errors of the second layer over its activations
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int q = 0; q < 4; ++q)
      s.h2[y + u][x + q] = acc[u][q] > 0.f ? s.dl[x + q] * s.w3[y + u] : 0.f;
  __syncthreads();
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[u][q] = 0.f;
#pragma unroll 8
  for (int j = 0; j < kHid; ++j) fma16(at4(&s.w2[j][y]), at4(&s.h2[j][x]), acc);
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int q = 0; q < 4; ++q) s.d1[y + u][x + q] = s.h1[y + u][x + q] > 0.f ? acc[u][q] : 0.f;
  __syncthreads();
  // ---- gradients: inputs i = c + 16 k of units j = r + 16 k, over the samples in order
  const int c = t & 15, r = t >> 4;
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[u][q] = 0.f;
  float a1[4] = {0.f, 0.f, 0.f, 0.f};
  for (int q = 0; q < kTS; q += 4) {
    float4 d2[4], d1[4], h[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      d2[k] = at4(&s.h2[r + 16 * k][q]);
      d1[k] = at4(&s.d1[r + 16 * k][q]);
      h[k] = at4(&s.h1[c + 16 * k][q]);
    }
    const float4 xn = at4(&s.xn[c][q]);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        float v = acc[u][k];
        v = fmaf(d2[u].x, h[k].x, v);
        v = fmaf(d2[u].y, h[k].y, v);
        v = fmaf(d2[u].z, h[k].z, v);
        acc[u][k] = fmaf(d2[u].w, h[k].w, v);
      }
      a1[u] = fmaf(d1[u].w, xn.w, fmaf(d1[u].z, xn.z, fmaf(d1[u].y, xn.y, fmaf(d1[u].x, xn.x, a1[u]))));
    }
  }
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    const int j = r + 16 * u;
#pragma unroll
    for (int k = 0; k < 4; ++k) out[kOffW2 + j * kHid + c + 16 * k] = acc[u][k];
    out[kOffW1 + j * kFeat + c] = a1[u];
  }
  if (t < 2 * kHid) {
    const float* e = t < kHid ? s.d1[t] : s.h2[t - kHid];
    float g = 0.f;
    for (int q = 0; q < kTS; ++q) g += e[q];
    out[t < kHid ? kOffB1 + t : kOffB2 + t - kHid] = g;
  }
}

// The gradients (the blocks' sums in block order, eight interleaved chains per
// parameter) and, with lr > 0, the Adam step; the last block adds the losses.
__global__ void __launch_bounds__(256) k_mlp_reduce(int blocks, const float* __restrict__ part,
                                                    const double* __restrict__ loss, float* __restrict__ grad,
                                                    float* __restrict__ params, float* __restrict__ m,
                                                    float* __restrict__ v, float lr, float c1, float c2,
                                                    double* __restrict__ total) {
  __shared__ float sh[8][33];
  __shared__ double shl[256];
  if (blockIdx.x == gridDim.x - 1) {
    double a = 0.0;
    for (int b = threadIdx.x; b < blocks; b += 256) a += loss[b];
    shl[threadIdx.x] = a;
    __syncthreads();
    for (int o = 128; o; o >>= 1) {
      if ((int)threadIdx.x < o) shl[threadIdx.x] += shl[threadIdx.x + o];
      __syncthreads();
    }
    if (threadIdx.x == 0) *total = shl[0];
    if (threadIdx.x < kOffW1) grad[threadIdx.x] = 0.f;
    return;
  }
  const int l = threadIdx.x & 31, w = threadIdx.x >> 5, q = blockIdx.x * 32 + l;
  float a = 0.f;
  if (q < kMlpTrainable)
    for (int b = w; b < blocks; b += 8) a += part[(size_t)b * kMlpTrainable + q];
  sh[w][l] = a;
  __syncthreads();
  if (w != 0 || q >= kMlpTrainable) return;
  float g = sh[0][l];
#pragma unroll
  for (int k = 1; k < 8; ++k) g += sh[k][l];
  const int k = q + kOffW1;
  grad[k] = g;
  if (!(lr > 0.f)) return;
  constexpr float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  const float mk = b1 * m[k] + (1.f - b1) * g;
  const float vk = b2 * v[k] + (1.f - b2) * g * g;
  m[k] = mk;
  v[k] = vk;
  params[k] -= lr * (mk / c1) / (sqrtf(vk / c2) + eps);
}

}  // namespace

void closure_features(const SolverDev& s, int n_known, const float* aux_dev, float* out_dev, cudaStream_t st) {
  const int nlc = s.F - n_known;
  if (nlc <= 0) return;
  const int tb = 128;
  if (s.dim == 3)
    k_closure_features<3><<<div_up(nlc, tb), tb, 0, st>>>(nlc, n_known, s.kind.get(), s.vi.get(), s.vj.get(),
                                                          s.z.get(), s.sqrt_info.get(), s.x0.get(), aux_dev, out_dev);
  else
    k_closure_features<2><<<div_up(nlc, tb), tb, 0, st>>>(nlc, n_known, s.kind.get(), s.vi.get(), s.vj.get(),
                                                          s.z.get(), s.sqrt_info.get(), s.x0.get(), aux_dev, out_dev);
  RPGO_LAUNCHED();
}

void launch_row_stats(int n, const uint32_t* adj, int words, const uint32_t* mask, const int32_t* rows, int count,
                      int32_t* deg, int32_t* support, cudaStream_t st) {
  if (count <= 0) return;
  const int tb = 256;
  k_row_stats<<<div_up((int64_t)count * 32, tb), tb, 0, st>>>(n, adj, words, mask, rows, count, deg, support);
  RPGO_LAUNCHED();
}

void mlp_forward(const float* params, int64_t n, const float* features, float* prob, cudaStream_t st) {
  if (n <= 0) return;
  k_mlp_forward<<<div_up(n, kTpb), kTpb, 0, st>>>(n, params, features, prob);
  RPGO_LAUNCHED();
}

double mlp_train_step(float* params, float* m, float* v, int64_t step, float lr, int64_t n, const float* features,
                      const float* labels, float* grad, cudaStream_t st) {
  if (n <= 0) {
    RPGO_CUDA(cudaMemsetAsync(grad, 0, sizeof(float) * kMlpParams, st));
    return 0.0;
  }
  const int blocks = div_up(n, kTS);
  DeviceBuffer<float> part((size_t)blocks * kMlpTrainable);
  DeviceBuffer<double> loss((size_t)blocks + 1);
  // (per device and cheap; the limit is above the default 48 KB)
  RPGO_CUDA(cudaFuncSetAttribute(k_mlp_step, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(StepSmem)));
  k_mlp_step<<<blocks, kStepThreads, sizeof(StepSmem), st>>>(n, params, features, labels, 1.f / (float)n, part.get(),
                                                            loss.get());
  RPGO_LAUNCHED();
  const bool adam = lr > 0.f && step >= 1;
  const float c1 = 1.f - powf(0.9f, (float)step), c2 = 1.f - powf(0.999f, (float)step);
  k_mlp_reduce<<<div_up(kMlpTrainable, 32) + 1, 256, 0, st>>>(blocks, part.get(), loss.get(), grad, params, m, v,
                                                             adam ? lr : 0.f, c1, c2, loss.get() + blocks);
  RPGO_LAUNCHED();
  double total = 0.0;
  RPGO_CUDA(cudaMemcpyAsync(&total, loss.get() + blocks, sizeof(double), cudaMemcpyDeviceToHost, st));
  RPGO_CUDA(cudaStreamSynchronize(st));
  return total / (double)n;
}

}  // namespace rpgo
