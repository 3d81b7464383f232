// Test harness (GPU): one damped step of the direct solve, with the limits of
// its dataflow part set by the caller; alone and as a joint batch of two
// copies. Links librpgo_gb300.so. Loaded by tests/test_gpu_solve_steps.py.
#include <cstdio>
#include <vector>

#include "chol.hpp"
#include "solver_kernels.hpp"

using namespace rpgo;

namespace {

struct System {
  int dim, n, f, stride, d;
  std::vector<int32_t> kind, vi, vj;
  std::vector<double> z, R, x;
};

void load(SolverDev& s, const System& y, int copies, cudaStream_t st) {
  std::vector<double> z, R, x;
  for (int c = 0; c < copies; ++c) {
    z.insert(z.end(), y.z.begin(), y.z.end());
    R.insert(R.end(), y.R.begin(), y.R.end());
    x.insert(x.end(), y.x.begin(), y.x.end());
  }
  s.z.upload(z, st);
  s.sqrt_info.upload(R, st);
  s.x0.upload(x, st);
  s.x.upload(x, st);
  s.weights.upload(std::vector<double>((size_t)copies * y.f, 1.0), st);
  cudaStreamSynchronize(st);
  solver_error(s, false, st);
  solver_linearize(s, true, st);
}

}  // namespace

extern "C" {

// The step (n * d doubles; joint: of two copies) for each of `runs` entries of
// coop, cols, polls: coop_ctas, df_cols, df_polls. All runs of one coop and
// cols go one after another through the same buffers. status[k]: 0, 1 a failed
// pivot, 2 a wait ran out. info: sparse levels, tail blocks, df_tail and first
// dataflow level of the last plan. Returns 0, or 1 for any other error.
int solve_steps(int dim, int n, int f, const int32_t* kind, const int32_t* vi, const int32_t* vj, const double* z,
                const double* R, const double* x, double lambda, int joint, int runs, const int32_t* coop,
                const int32_t* cols, const int32_t* polls, double* step, double* change, int32_t* status,
                int32_t* info) try {
  System y{dim, n, f, dim == 3 ? 12 : 4, dim == 3 ? 6 : 3, {kind, kind + f}, {vi, vi + f}, {vj, vj + f}, {}, {}, {}};
  y.z.assign(z, z + (size_t)f * y.stride);
  y.R.assign(R, R + (size_t)f * y.d * y.d);
  y.x.assign(x, x + (size_t)n * y.stride);
  const cudaStream_t st = nullptr;
  const int copies = joint ? 2 : 1;
  const size_t len = (size_t)copies * n * y.d;
  for (int k = 0; k < runs;) {
    SolverDev s;
    s.coop_ctas = coop[k];
    s.df_cols = cols[k];
    BatchDev b;
    if (joint) {
      std::vector<CholPlan> plans(2);
      for (auto& p : plans) p = make_chol_plan(n, y.d, y.kind, y.vi, y.vj, false);
      CholPlan merged = merge_chol_plans(plans, {0, f, 2 * f});
      std::vector<int32_t> k2 = y.kind, i2 = y.vi, j2 = y.vj, sys(n, 0);
      k2.insert(k2.end(), y.kind.begin(), y.kind.end());
      for (int e = 0; e < f; ++e) {
        i2.push_back(y.vi[e] + n);
        j2.push_back(y.vj[e] + n);
      }
      sys.resize(2 * n, 1);
      solver_upload(s, dim, k2, i2, j2, 2 * n, st, true, &merged);
      b.G = 2;
      b.vsys.upload(sys, st);
      b.voff.upload({0, n, 2 * n}, st);
      b.ctl.upload({kBatchActive, kBatchActive}, st);
      b.lam.upload({lambda, lambda}, st);
      b.status.resize(2);
      b.out.resize(4);
      b.term.resize((size_t)4 * n);
      cudaStreamSynchronize(st);
    } else {
      solver_upload(s, dim, y.kind, y.vi, y.vj, n, st, true);
    }
    load(s, y, copies, st);
    const CholPlan& p = s.chol->plan;
    info[0] = p.levels(), info[1] = p.T, info[2] = p.df_tail, info[3] = p.df_level;
    for (const int k0 = k; k < runs && coop[k] == coop[k0] && cols[k] == cols[k0]; ++k) {
      s.df_polls = polls[k];
      status[k] = 0;
      try {
        if (joint) {
          chol_enqueue_batch(s, *s.chol, b, st);
          double out[4];
          b.out.download(out, 4, st);
          cudaStreamSynchronize(st);
          for (int g = 0; g < 2; ++g) {
            chol_check_status(out[2 * g + 1]);
            if (out[2 * g + 1] != 0.0) status[k] = 1;
          }
          change[k] = out[0];
        } else {
          const SolveOut o = chol_solve(s, *s.chol, lambda, st);
          if (!o.ok) status[k] = 1;
          change[k] = o.lin_change;
        }
      } catch (const CudaError&) {
        if (cudaGetLastError() != cudaSuccess) throw;
        status[k] = 2;
      }
      s.delta.download(step + (size_t)k * len, len, st);
      if (cudaStreamSynchronize(st) != cudaSuccess) return 1;
    }
  }
  return 0;
} catch (const std::exception& e) {
  std::fprintf(stderr, "solve_steps: %s\n", e.what());
  return 1;
}
}
