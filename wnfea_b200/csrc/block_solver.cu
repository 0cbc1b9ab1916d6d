// Multi-right-hand-side solve: load cases in batches, each of the narrowest width that holds it.
//
// A batch of kBatch columns (8, 16 or 32; block_batch.cuh) moves kBatch values per gathered DOF
// whatever the number of live cases, so five cases in a 32-wide batch pay for 32: on a 71,000-DOF bar
// in FP64 a batch takes 8.8 ms 8 wide, 10.9 ms 16 wide and 18.3 ms 32 wide.  Every width runs
// the same sums in the same order per case, so a case's solution does not depend on the batch it
// is solved in.
#include <algorithm>

#include "amg.h"
#include "block.h"
#include "common.cuh"
#include "solid.h"
#include "solver.h"

namespace wn {
namespace {

// The row of the fine level at each position of a row kernel of `grid` CTAs: pass k of CTA b covers
// rows 32 (k grid + b) ..., eight warps of four, and takes them by length.  A warp pads its four rows
// to the longest: on the I-beam the rows name 10 to 65 blocks (vertex and mid-edge nodes alternate),
// 25 on average, and 63 % of the padded work was work in the mesh's numbering against 90 % by
// length.  The quads go to the warps by the work the warps have had so far, the longest to the
// least, so that a CTA's warps end together.
std::vector<int32_t> batch_order(const std::vector<int32_t>& rp, int64_t n, int64_t grid) {
  constexpr int kRows = 32, kQuads = 8;
  const int64_t passes = (n + kRows - 1) / kRows;
  std::vector<int32_t> order(passes * kRows, (int32_t)n);
  auto len = [&](int32_t r) { return r < n ? rp[r + 1] - rp[r] : 0; };
  for (int64_t b = 0; b < std::min(grid, passes); ++b) {
    int64_t load[kQuads] = {};
    for (int64_t p = b; p < passes; p += grid) {
      int32_t rows[kRows];
      for (int k = 0; k < kRows; ++k) rows[k] = (int32_t)std::min<int64_t>(n, p * kRows + k);
      std::stable_sort(rows, rows + kRows, [&](int32_t x, int32_t y) { return len(x) > len(y); });
      int warp[kQuads];
      for (int q = 0; q < kQuads; ++q) warp[q] = q;
      std::stable_sort(warp, warp + kQuads, [&](int x, int y) { return load[x] < load[y]; });
      for (int q = 0; q < kQuads; ++q) {
        std::copy(rows + 4 * q, rows + 4 * q + 4, order.begin() + p * kRows + 4 * warp[q]);
        load[warp[q]] += 2 + (len(rows[4 * q]) + 3) / 4;
      }
    }
  }
  return order;
}

int ensure_block_set(Solid* s) {
  if (s->batch) return 0;
  auto B = std::make_unique<BlockSet>();
  std::vector<int32_t> order[2];
  for (int k = 0; k < 2; ++k) {
    order[k] = batch_order(s->h_row_ptr, s->n_nodes, (int64_t)kNumSMs * (k + 2));
    WN_CHECK(B->order[k].upload(order[k]));
  }
  WN_CUDA(cudaEventCreate(&B->ev0));
  WN_CUDA(cudaEventCreate(&B->ev1));
  WN_CUDA(cudaStreamSynchronize(0));  // the uploads' host buffers end here
  s->batch = std::move(B);
  return 0;
}

}  // namespace

int solver_solve_multi(Solid* s, int n_rhs, const double* F, double* U, const wn_solve_params& prm,
                       wn_solve_stats* stats, int* case_iters, double* case_rel, cudaStream_t st) {
  WN_REQUIRE(s->assembled, WN_ESTATE, "multi-RHS solve: matrix not assembled");
  WN_REQUIRE(s->bs == 3, WN_ESTATE, "multi-RHS solve: not a C3D10 system");
  WN_REQUIRE(n_rhs >= 0, WN_EINVAL, "multi-RHS solve: n_rhs >= 0 required");
  WN_REQUIRE(prm.precond >= 0 && prm.precond <= 2, WN_EINVAL, "multi-RHS solve: precond in {0, 1, 2}");
  WN_REQUIRE(prm.precision == 0 || prm.precision == 1, WN_EINVAL,
             "multi-RHS solve: precision must be 0 (fp64) or 1 (fp32 V-cycle in fp64 PCG)");
  WN_REQUIRE(prm.max_iter > 0 && prm.rtol > 0.0, WN_EINVAL, "multi-RHS solve: max_iter > 0 and rtol > 0 required");
  if (prm.precond == 2 && !s->amg) WN_CHECK(solver_setup(s, amg_default_params()));
  WN_CHECK(ensure_block_set(s));
  BlockSet& B = *s->batch;
  if (st == 0) {
    if (!B.own) WN_CUDA(cudaStreamCreate(&B.own));
    st = B.own;
  }
  // the streamed and staged fine levels are built for the widest batch
  const bool widest = s->stream_batched || s->batch_stage_x;
  WN_CUDA(cudaEventRecord(B.ev0, st));
  int64_t launches = 0;
  int total_iters = 0, total_outer = 0, status = 0;
  double worst = 0.0;
  for (int j0 = 0; j0 < n_rhs; j0 += kMaxBatch) {
    const int m = std::min(kMaxBatch, n_rhs - j0);
    BatchResult res;
    auto* solve = widest || m > 16 ? solve_batch<32> : m > 8 ? solve_batch<16> : solve_batch<8>;
    WN_CHECK(solve(s, F, U, n_rhs, j0, m, prm, res, st));
    launches += res.launches;
    total_iters += res.iterations;
    total_outer += res.outer;
    if (res.status == WN_EBREAKDOWN || (res.status != 0 && status == 0)) status = res.status;
    for (int j = 0; j < m; ++j) {
      if (case_iters) case_iters[j0 + j] = res.case_iters[j];
      if (case_rel) case_rel[j0 + j] = res.case_rel[j];
      worst = std::max(worst, res.case_rel[j]);
    }
  }
  WN_CUDA(cudaEventRecord(B.ev1, st));
  WN_CUDA(cudaEventSynchronize(B.ev1));
  float ms = 0.f;
  WN_CUDA(cudaEventElapsedTime(&ms, B.ev0, B.ev1));
  if (stats) {
    stats->iterations = total_iters;
    stats->outer_iterations = total_outer;
    stats->status = status;
    stats->rel_res = worst;
    stats->solve_seconds = ms * 1e-3;
    stats->kernel_launches = launches;
    stats->algorithmic_bytes = 0.0;  // not counted for the batched solve
    stats->setup_seconds = s->amg ? s->amg->setup_seconds : 0.0;
    stats->n_levels = s->amg ? (int)s->amg->levels.size() + 1 : 0;
  }
  return 0;
}

}  // namespace wn
