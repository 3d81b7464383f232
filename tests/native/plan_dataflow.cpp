// Test harness (CPU): the dataflow part of a solve plan (add_dataflow)
// against the update, Hessian and row lists of the level form, which it must
// restate entry by entry: the same operands for the same sums in the same
// order. Loaded by tests/test_plan_dataflow_cpu.py.
#include <algorithm>
#include <cstdint>
#include <vector>

#include "chol_plan.hpp"

using rpgo::CholPlan;

namespace {

struct Product {
  int a = -1, b = -1, code = -1, seen = 0;
};

// 0, or the number of the first rule that the plan breaks
int check(const CholPlan& p, int max_cols) {
  const int L = p.levels(), ns = p.n_sparse, l0 = p.df_level;
  if (l0 < 0 || l0 > L) return 1;
  const int w0 = L >= 0 && l0 < L ? p.lvl_col_ptr[l0] : ns, nc = (int)p.df_col.size() / rpgo::kDfColInts;
  if (nc != (l0 < L ? ns - w0 : 0)) return 2;
  if (l0 == L) return p.df_col.empty() && p.df_dst.empty() && p.df_pre.empty() ? 0 : 3;
  for (int l = l0; l < L; ++l)
    if (p.lvl_col_ptr[l + 1] - p.lvl_col_ptr[l] > max_cols) return 4;
  std::vector<uint8_t> in_df(ns, 0);
  for (int w = w0; w < ns; ++w) in_df[p.lvl_cols[w]] = 1;
  // every product and who makes it
  std::vector<Product> prod(p.df_products);
  auto put = [&](int k, int a, int b, int code) {
    if (k < 0 || k >= p.df_products) return false;
    prod[k].a = a, prod[k].b = b, prod[k].code = code, ++prod[k].seen;
    return true;
  };
  for (int w = 0; w < nc; ++w) {
    const int32_t* r = &p.df_col[(size_t)w * rpgo::kDfColInts];
    const int j = r[0], p0 = r[1], m = r[2];
    if (j != p.lvl_cols[w0 + w] || p0 != p.col_ptr[j] || m != p.col_ptr[j + 1] - p0 - 1) return 5;
    if (m > rpgo::kDfMaxBlocks) return 6;
    const int32_t* d = p.df_dst.data() + (size_t)4 * r[4];
    for (int a = 0; a < m; ++a)
      for (int b = a; b < m; ++b, d += 4) {
        if (d[2] != a || d[3] != b) return 7;
        if (d[0] >= 0 && !put(d[0], p0 + 1 + b, p0 + 1 + a, d[1])) return 8;
        if (d[0] < 0 && p.blk_row[p0 + 1 + a] < ns) return 9;  // only tail targets may have none
      }
    // the row list
    if (r[6] != p.row_ptr[j + 1] - p.row_ptr[j]) return 10;
    for (int u = 0; u < r[6]; ++u) {
      const int q = p.row_blk[2 * (p.row_ptr[j] + u)], k = p.row_blk[2 * (p.row_ptr[j] + u) + 1];
      if (p.df_row[2 * (r[5] + u)] != q || p.df_row[2 * (r[5] + u) + 1] != (k << 1 | in_df[k])) return 11;
    }
  }
  for (size_t k = 0; k < p.df_pre.size(); k += 4) {
    if (in_df[p.blk_col[p.df_pre[k + 1]]]) return 12;
    if (!put(p.df_pre[k], p.df_pre[k + 1], p.df_pre[k + 2], p.df_pre[k + 3])) return 13;
  }
  // every block's products are its update pairs, in order
  auto block = [&](int entry, const std::vector<int32_t>& src, int u0, int u1, int code) {
    const int first = p.df_blk[2 * entry];
    if (p.df_blk[2 * entry + 1] != u1 - u0) return false;
    for (int u = u0; u < u1; ++u) {
      const Product& x = prod[first + u - u0];
      const int c = code < 0 ? 0 : code | (u == u0 ? 1 : 0);
      if (x.seen != 1 || x.a != src[2 * u] || x.b != src[2 * u + 1] || x.code != c) return false;
    }
    return true;
  };
  int np = 0;
  for (int w = 0; w < nc; ++w) {
    const int32_t* r = &p.df_col[(size_t)w * rpgo::kDfColInts];
    for (int b = 0; b <= r[2]; ++b) {
      const int q = r[1] + b;
      if (!block(r[3] + b, p.upd_src, p.upd_ptr[q], p.upd_ptr[q + 1], q << 2 | (b == 0 ? 2 : 0))) return 14;
      np += p.upd_ptr[q + 1] - p.upd_ptr[q];
    }
  }
  bool tail = rpgo::tail_fits(p.T, p.d);
  for (int t = 0; t < p.n_tail_blocks(); ++t)
    tail = tail && p.tupd_ptr[t + 1] - p.tupd_ptr[t] <= rpgo::tail_slots(p.d);
  if ((p.df_tail != 0) != tail) return 15;
  if (tail) {
    for (int t = 0; t < p.n_tail_blocks(); ++t) {
      if (!block(p.df_tail_blk + t, p.tupd_src, p.tupd_ptr[t], p.tupd_ptr[t + 1], -1)) return 16;
      np += p.tupd_ptr[t + 1] - p.tupd_ptr[t];
    }
    for (int t = 0; t < p.T; ++t) {
      const int r0 = p.df_trow[2 * t];
      if (p.df_trow[2 * t + 1] != p.trow_ptr[t + 1] - p.trow_ptr[t]) return 17;
      for (int u = p.trow_ptr[t]; u < p.trow_ptr[t + 1]; ++u) {
        const int e = r0 + u - p.trow_ptr[t], k = p.trow_blk[2 * u + 1];
        if (p.df_row[2 * e] != p.trow_blk[2 * u] || p.df_row[2 * e + 1] != (k << 1 | in_df[k])) return 18;
      }
    }
  }
  return np == p.df_products ? 0 : 19;
}

}  // namespace

extern "C" {

// One system; info: levels, first dataflow level, columns, products from
// earlier columns, tail blocks, df_tail.
int dataflow_check(int n, int d, int f, const int32_t* kind, const int32_t* vi, const int32_t* vj, int max_cols,
                   int32_t* info) {
  CholPlan p = rpgo::make_chol_plan(n, d, {kind, kind + f}, {vi, vi + f}, {vj, vj + f});
  rpgo::add_dataflow(p, max_cols);
  const int32_t v[6] = {p.levels(), p.df_level, (int32_t)p.df_col.size() / rpgo::kDfColInts,
                        (int32_t)p.df_pre.size() / 4, p.T, p.df_tail};
  std::copy(v, v + 6, info);
  return check(p, max_cols);
}

// The same system twice, merged (a joint batch's plan).
int dataflow_check_joint(int n, int d, int f, const int32_t* kind, const int32_t* vi, const int32_t* vj,
                         int max_cols) {
  std::vector<CholPlan> plans(2);
  for (auto& p : plans) p = rpgo::make_chol_plan(n, d, {kind, kind + f}, {vi, vi + f}, {vj, vj + f}, false);
  CholPlan u = rpgo::merge_chol_plans(plans, {0, f, 2 * f});
  rpgo::add_dataflow(u, max_cols);
  return check(u, max_cols);
}
}
