// Direct solve of the damped normal equations (H + lambda D) delta = -g:
// sparse block Cholesky over the plan of chol_plan.hpp, in FP64, as one
// cooperative kernel per solve (factorisation, forward and backward
// substitution, model change).
#pragma once
#include <cuda_runtime.h>

#include "chol_plan.hpp"
#include "common.cuh"
#include "solver_kernels.hpp"

namespace rpgo {

struct CholDev {
  CholPlan plan;
  int levels = 0;
  DeviceBuffer<int32_t> diag_blk;  // per variable: its diagonal block of L, -1 in the dense tail
  DeviceBuffer<int32_t> perm, col_ptr, blk_row, blk_col, lvl_col_ptr, lvl_cols, lvl_task_ptr, tasks, btask, ftask;
  DeviceBuffer<int32_t> upd_ptr, upd_src, tupd_ptr, tupd_src, a_ptr, a_src, ta_ptr, ta_src;
  DeviceBuffer<int32_t> row_ptr, row_blk, trow_ptr, trow_blk, ttasks, ttask_ptr;
  DeviceBuffer<double> L;     // sparse blocks of L (off-diagonal; the diagonal slots are unused)
  DeviceBuffer<double> Ldiag; // factors of the sparse diagonal blocks (reciprocal pivots on the diagonal)
  DeviceBuffer<double> M;     // dense tail, column-major, padded to whole tiles
  DeviceBuffer<double> Ldd;   // factors of the tail's diagonal tiles (reciprocal pivots on the diagonal)
  DeviceBuffer<double> y;     // right-hand side / solution in elimination order
  DeviceBuffer<double> part;  // per-CTA partial sums
  DeviceBuffer<double> Spart; // level-task partial sums (D x D per task)
  DeviceBuffer<double> Tpart; // tail row task sums (D per task)
  DeviceBuffer<double> out;   // model change, status (chol_solve)
  DeviceBuffer<double> Hs;    // H in the block layout of L (per linearisation)
  DeviceBuffer<double> dampS; // damping diagonal of the diagonal blocks, same layout
  DeviceBuffer<int32_t> status;  // pivot failure; a wait of the dataflow part ran out; CTAs done
  // dataflow part (chol_plan.hpp) and the words its columns hand on: update
  // products, forward and backward solutions
  DeviceBuffer<int32_t> df_col, df_blk, df_dst, df_pre, df_row, df_trow;
  DeviceBuffer<double> prod, ys, xs;
  cudaEvent_t ev[2] = {nullptr, nullptr};  // around each launch (kernel time)
  ~CholDev();
  void upload(CholPlan&& p, cudaStream_t st);
};

// CTAs of the solver's direct solve, and the widest level that its dataflow
// part takes
int chol_grid(const SolverDev& s);
int chol_dataflow_cols(const SolverDev& s);
// Assembles the linearised system (fH64, fg): the diagonal blocks, the
// gradient and the damping diagonal per variable, and H and the damping
// diagonal in the block layout of L; enqueued after every linearisation.
// mask: a joint batch's variable control words (bit 0: graph in this round)
void chol_assemble(SolverDev& s, CholDev& c, bool diagonal_damping, cudaStream_t st, const uint8_t* mask = nullptr);
// Solve with the factorisation of (H + lambda D); fills s.delta.
SolveOut chol_solve(SolverDev& s, CholDev& c, double lambda, cudaStream_t st);
// Enqueue the same solve without waiting: the kernel writes the model change
// and the status to host[0] and host[1] (page-locked); call chol_finish after
// the stream reached that point.
void chol_enqueue(SolverDev& s, CholDev& c, double lambda, cudaStream_t st, double* host);
SolveOut chol_finish(SolverDev& s, CholDev& c, const double* host);
// throws when a solve's status word (0 solved, 1 a failed pivot, 2 a wait
// between columns ran out) says that its kernel gave up
void chol_check_status(double status);
// Joint batch: enqueue one launch that solves every active system of the
// batch b with its own damping; per-system model change and status land in
// b.out (2 per system), the steps in s.delta.
void chol_enqueue_batch(SolverDev& s, CholDev& c, const BatchDev& b, cudaStream_t st);
// Joint batch: compact the plan's level lists to the graphs whose control
// word (already on the device) has kBatchActive; later chol_enqueue_batch
// launches use the compacted lists.
void chol_batch_compact(CholDev& c, BatchDev& b, cudaStream_t st);
// kernel time of the last enqueued launch (after the stream passed it)
float chol_last_ms(CholDev& c);

}  // namespace rpgo
