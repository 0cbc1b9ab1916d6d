// Multi-right-hand-side (batched) PCG workspace: up to kBatch (8, 16 or 32) load cases solved
// together against one assembled matrix and one AMG hierarchy.
//
// Layout: a batched vector of n scalar DOFs is n x kBatch, DOF-major with the kBatch load
// cases of one DOF contiguous (element (i, j) at i * kBatch + j).  A block row of the matrix is
// handled by 8 lanes, each owning kBatch / 8 load cases, so every matrix block is read once per
// product for all kBatch cases.
#pragma once

#include <cuda_runtime.h>

#include <memory>
#include <vector>

#include "amg.h"
#include "device_array.h"
#include "wnfea_cuda.h"

namespace wn {

struct Solid;  // solid.h

constexpr int kMaxBatch = 32;

// per-load-case PCG state (device)
template <int kBatch>
struct BlockScalarsT {
  double rz[kBatch];      // r . z of the current iteration
  double alpha[kBatch];   // step of the current iteration (0 for finished cases)
  double beta[kBatch];    // p = z + beta p of the next iteration (0 for finished cases)
  double bnorm2[kBatch];  // ||b_j||^2
  double tol2[kBatch];    // (rtol_j ||b_j||)^2
  double rr[kBatch];      // ||r_j||^2 of the last check
  int col_done[kBatch];
  int col_iters[kBatch];
  int col_status[kBatch];
  int done;      // every case finished (or the iteration limit reached)
  int iters;     // iterations of the batch
  int status;
  int max_iter;
};

// The device vectors of the batched solves of one handle, shared by the batch widths: one batch runs
// at a time and leaves nothing in them for the next, so each vector is kept once, as long as the widest
// batch so far needs it, and a narrower one uses its beginning.  (A workspace per width held 56
// columns after a load book of 32, one of 16 and one of 5 cases.)
struct BatchStore {
  std::vector<DArray<unsigned char>> vecs;
  uint64_t epoch = 0;         // changes whenever a vector moves: captured graphs hold the addresses
  uint64_t hierarchy_id = 0;  // the AmgHierarchy that the level vectors were sized for
  int at_least(int id, int64_t bytes) {
    if ((size_t)id >= vecs.size()) vecs.resize(id + 1);
    if (vecs[id].n >= bytes) return 0;
    ++epoch;
    return vecs[id].alloc(bytes);
  }
  void release_from(int id) {
    ++epoch;
    if ((size_t)id < vecs.size()) vecs.resize(id);
  }
};
enum BatchVecId {
  kVecPartA, kVecPartB, kVecPartC, kVecF, kVecU, kVecUlo, kVecR, kVecX, kVecRes, kVecP0, kVecP1, kVecQ, kVecDinv64,
  kVecDinv32, kVecZ32, kVecR32, kVecD32, kVecZ64, kVecD64,
  kVecHierarchy,  // from here on sized for the hierarchy: the coarsest level's four, then 7 per level and precision
  kVecCb32 = kVecHierarchy, kVecCx32, kVecCb64, kVecCx64, kVecLevels
};
template <typename T>
struct BatchVec {
  T* p = nullptr;
  int take(BatchStore& M, int id, int64_t n) {
    p = nullptr;
    WN_CHECK(M.at_least(id, n * (int64_t)sizeof(T)));
    p = reinterpret_cast<T*>(M.vecs[id].p);
    return 0;
  }
};

// Vectors of a V-cycle level.  The finest level's right-hand side and result are the PCG's, and r, d
// and d2 belong to Chebyshev steps beyond the first: left out where nothing reads them (at 32 cases
// a fine vector of a million DOFs is 130 MB in FP32).
template <typename T>
struct BatchLevelVecs {
  BatchVec<T> b, x, x2, r, d, d2, res;
  int take(BatchStore& M, int level, int64_t n, int degree) {
    const int id = kVecLevels + 7 * (2 * level + (sizeof(T) == 8));
    if (level > 0) {
      WN_CHECK(b.take(M, id, n));
      WN_CHECK(x2.take(M, id + 1, n));
    }
    WN_CHECK(x.take(M, id + 2, n));
    WN_CHECK(res.take(M, id + 3, n));
    if (degree > 1) {
      WN_CHECK(r.take(M, id + 4, n));
      WN_CHECK(d.take(M, id + 5, n));
      WN_CHECK(d2.take(M, id + 6, n));
    }
    return 0;
  }
};

template <int kBatch>
struct BlockWorkT {
  int64_t n = 0;  // scalar DOFs of the fine level
  static constexpr int kMaxParts = 148 * 16;
  int npA = 0, npB = 0, npC = 0;
  uint64_t epoch = 0;  // the store's when the graphs were captured
  BatchVec<double> partA, partB, partC;  // kMaxParts x kBatch
  DArray<BlockScalarsT<kBatch>> scal;    // [0] inner PCG, [1] outer column norms
  DArray<double> rtol_cols;              // kBatch inner targets
  std::vector<double> h_rtol;
  // outer refinement: F, U = U + Ulo (double-double), R = F - K U
  BatchVec<double> F, U, Ulo, R;
  // Krylov vectors (FP64)
  BatchVec<double> x, r, p0, p1, q;
  // 1 / diag of the fine matrix (refreshed per solve)
  BatchVec<double> dinv64;
  BatchVec<float> dinv32;
  // preconditioner input / output in the V-cycle precision
  BatchVec<float> z32, r32;
  BatchVec<double> z64;
  // the fine V-cycle's first smoothing input dinv r / theta, written by the PCG update
  BatchVec<float> d0_32;
  BatchVec<double> d0_64;
  // V-cycle vectors per level and the coarsest right-hand side / solution
  std::vector<BatchLevelVecs<float>> lv32;
  std::vector<BatchLevelVecs<double>> lv64;
  BatchVec<float> cb32, cx32;
  BatchVec<double> cb64, cx64;
  // x-tiles of the fine level (block_batch.cuh build_x_tiles): runs of rows whose blocks name at
  // most 256 columns; per tile its sorted columns, per block its column's index among them
  DArray<int32_t> xt_rows, xt_col_ptr, xt_cols;
  DArray<uint8_t> xt_lcol;
  int xt_n = 0;         // tiles (0: no plan)
  bool xt_tried = false;
  GraphCache graphs[2][3];          // [V-cycle precision 0 fp64 / 1 fp32][preconditioner]
  int64_t launches = 0;
  ~BlockWorkT() {
    for (auto& a : graphs)
      for (auto& g : a) g.reset();
  }
};

// the batched solver of one handle
struct BlockSet {
  // the fine level's rows as the row kernels of 2 and 3 CTAs per SM take them (batch_order)
  DArray<int32_t> order[2];
  BatchStore store;
  std::unique_ptr<BlockWorkT<8>> w8;
  std::unique_ptr<BlockWorkT<16>> w16;
  std::unique_ptr<BlockWorkT<32>> w32;
  template <int W>
  std::unique_ptr<BlockWorkT<W>>& width() {
    if constexpr (W == 8)
      return w8;
    else if constexpr (W == 16)
      return w16;
    else
      return w32;
  }
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  cudaStream_t own = nullptr;
  ~BlockSet() {
    w8.reset();
    w16.reset();
    w32.reset();
    if (ev0) cudaEventDestroy(ev0);
    if (ev1) cudaEventDestroy(ev1);
    if (own) cudaStreamDestroy(own);
  }
};

struct BatchResult {
  int iterations = 0, outer = 0, status = 0;
  int case_iters[kMaxBatch] = {};
  int case_status[kMaxBatch] = {};
  double case_rel[kMaxBatch] = {};
  int64_t launches = 0;
};

// load cases j0 .. j0 + m - 1 (m <= W) of the row-major n x n_rhs F into U (block_batch.cuh)
template <int W>
int solve_batch(Solid* s, const double* F, double* U, int n_rhs, int j0, int m, const wn_solve_params& prm,
                BatchResult& res, cudaStream_t st);
template <>
int solve_batch<8>(Solid*, const double*, double*, int, int, int, const wn_solve_params&, BatchResult&, cudaStream_t);
template <>
int solve_batch<16>(Solid*, const double*, double*, int, int, int, const wn_solve_params&, BatchResult&, cudaStream_t);
template <>
int solve_batch<32>(Solid*, const double*, double*, int, int, int, const wn_solve_params&, BatchResult&, cudaStream_t);

}  // namespace wn
