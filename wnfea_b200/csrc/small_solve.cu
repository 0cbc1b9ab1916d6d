// PCG of a small system in one kernel: a cluster of 16 CTAs runs every iteration.
//
// A system of a few thousand nodes gives each of an iteration's kernels (five with point Jacobi, nine
// with a two-level V-cycle) a microsecond of work and three to five of launch, ramp-up and
// dependence, whatever the matrix (small_system has the figures).
// Here the stages of an iteration are the phases of one persistent kernel, separated by the
// hardware barrier of a thread-block cluster (16 CTAs on 16 SMs of one GPC: co-scheduled by the
// launch, no spinning).  What bounds it is the chain of phases, so nothing on it goes through L2
// that need not:
//   * every CTA holds a copy of the gathered vectors in its shared memory; a CTA computes its run of
//     rows and stores the result into all 16 copies before the barrier.  (Gathering through L2
//     instead, two round trips per phase, took 11 and 35 us per iteration at 1,025 nodes.)
//   * p = z + beta p is formed by every CTA for itself, so only z travels;
//   * x, r and q of the CTA's own DOFs stay in its registers or shared memory, as do its matrix
//     blocks when they fit; otherwise the blocks are read from L2, which does not depend on any
//     phase;
//   * dot products: one partial per warp, stored into every CTA before the barrier; each warp adds
//     the partials in the same order, so all threads take the same alpha, beta and decisions.
// Two kernels: k_small_diag for no, point-Jacobi or block-Jacobi preconditioning, and k_small_amg
// for a hierarchy of at most one level above its dense one.
// The arithmetic is that of the launched kernels (solver.cu): FP64 Krylov vectors, matrix and dots;
// the preconditioner in TM.  k_small_diag also adds its dot products in the launched kernels'
// order: an unpreconditioned or Jacobi solve that stops at its iteration limit hundreds of
// iterations from convergence (a slender bar) has an iterate that depends on that order in its third
// digit, and a call's result must not depend on which kernels ran it.
#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>

#include "amg.h"
#include "common.cuh"
#include "small_solve.h"
#include "solid.h"
#include "spmv.cuh"
#include "stream.cuh"
#include "wnfea_cuda.h"

namespace cg = cooperative_groups;

namespace wn {
namespace {

constexpr int kCtas = 16, kThreads = 512, kWarps = kThreads / 32;
constexpr int kLanes = 8;                   // lanes per block row
constexpr int kGroups = kThreads / kLanes;  // rows of a CTA side by side
constexpr int kTeam = 4, kTeams = kWarps / kTeam;  // warps per row of the restriction
constexpr int64_t kMaxNodes = 2048;         // (small_system)
// Iterations of one launch (8 to 26 ms; 4 ms with AMG, whose solves take some 40): the caller's max_iter
// bounds a solve, not the length of a kernel.  The next launch goes on from x, r, p and the scalars in
// global memory, with the same bits.
constexpr int kDiagSteps = 2048, kAmgSteps = 128;
constexpr size_t kSmemLimit = 214 * 1024;   // dynamic shared memory (5 KB are static)

__host__ __device__ constexpr size_t pad16(size_t bytes) { return (bytes + 15) & ~size_t(15); }

// the run [i0, i1) of a vector, complete in this CTA's copy, into the other CTAs' copies (visible
// after the next cluster barrier); i0 sizeof(T) is a multiple of 16
template <int THREADS, typename T>
__device__ __forceinline__ void publish_run(const cg::cluster_group& c, int rank, T* v, int64_t i0, int64_t i1) {
  __syncthreads();  // the run is complete
  const int64_t u0 = i0 * sizeof(T) / 16, u1 = (i1 * sizeof(T) + 15) / 16;
  const int n = (int)(u1 - u0);
  uint4* own = reinterpret_cast<uint4*>(v) + u0;
  for (int k = threadIdx.x; k < n * (kCtas - 1); k += THREADS) {
    const int peer = k / n, at = k - peer * n;
    uint4* there = c.map_shared_rank(own, peer + (peer >= rank));
    there[at] = own[at];
  }
}

// ---------------------------------------------------------------------------------------
// no, point-Jacobi or block-Jacobi preconditioning
// ---------------------------------------------------------------------------------------
// The dot products in the launched kernels' order:
//   p . q   a tile of the streamed fine matrix is a CTA of eight consumer warps there, warp w taking the
//           rows 4 w .. 4 w + 3 of every 32; such a warp's rows are a unit here, and the units are shared
//           out evenly over the 16 CTAs.  A tile's eight sums are added as block_sum adds them,
//           then the tiles' as reduce_parts does.
//   r . r, r . z   a warp there takes 32 consecutive DOFs (block Jacobi, r . z: nodes) and a CTA eight
//           such warps; so a CTA here owns whole runs of 32 nodes (96 DOFs) of x, r and z.
// q = A p is stored by the warp that computes it into the shared memory of its owner.
// Bound by the chain of phases: two cluster barriers with their sums, the row products and the copies of
// z.  1,025 nodes 7.0 us per iteration (about as much as with sums in the cheapest order, 7.4 with an
// earlier split of the rows); the part of the matrix that shared memory cannot hold is read from L2 by the
// first units of a CTA, 2,025 nodes 12.7 us.
constexpr int kDiagThreads = 512, kDiagWarps = kDiagThreads / 32;
constexpr int kMaxTiles = 128;                  // (as many as one CTA of the update reduces in four warps)
constexpr size_t kDiagSmemLimit = 226 * 1024;   // dynamic shared memory (no static)
static_assert(kMaxNodes / kCtas * 3 <= kDiagThreads, "one owned DOF per thread");

template <typename TM>
struct DiagArgs {
  int64_t n_nodes, nnzb;
  const int32_t *rp, *ci;
  const double* k64;
  const TM* dinv;  // 1 / diag
  const TM* binv;  // block Jacobi
  int precond;
  const double* b;
  double *x, *r, *p;  // r, p: the state between launches
  int first;          // from x = 0, or on from the state
  const int4* plan;  // kCtas runs (first unit, end, first row, end), then the units (small_plan)
  int slots;         // tiles rounded up to 32
  int own_max, rows_max, units_max;
  int slice_blocks;  // the last blocks of a CTA's run, in shared memory; those before are read from L2
  double rtol;
  int max_iter;
  PcgScalars* S;
};

// first run of 32 nodes that CTA k owns
__host__ __device__ __forceinline__ int64_t own_begin(int64_t n_nodes, int k) {
  return (n_nodes + 31) / 32 * k / kCtas;
}

// dynamic shared memory of a CTA, in this order
template <typename TM>
struct DiagLayout {
  size_t p, z, pq, rr, rz, q, units, kv, ci, rp, end;
  __host__ __device__ DiagLayout(int64_t n_nodes, int slots, int own, int rows, int n_units, int slice) {
    const size_t n = 3 * (size_t)n_nodes, bl = (size_t)slice;
    p = 0;
    z = p + pad16(n * 8);
    pq = z + pad16(n * sizeof(TM));
    rr = pq + 8 * (size_t)slots * 8;
    rz = rr + 8 * 32 * 8;
    q = rz + 8 * 32 * 8;
    units = q + pad16(3 * (size_t)own * 8);
    kv = units + 16 * (size_t)n_units;
    ci = kv + pad16(9 * bl * 8);
    rp = ci + pad16(bl * 4);
    end = rp + pad16(4 * (size_t)(rows + 1));
  }
};

// the sum of eight warps as block_sum adds them (its butterfly over lanes 0 .. 7), v[k * stride]
__device__ __forceinline__ double sum8(const double* v, int stride) {
  return ((v[0] + v[4 * stride]) + (v[2 * stride] + v[6 * stride])) +
         ((v[stride] + v[5 * stride]) + (v[3 * stride] + v[7 * stride]));
}

// kWhole: every CTA's matrix blocks are in its shared memory
template <typename TM, bool kWhole>
__global__ void __cluster_dims__(kCtas, 1, 1) __launch_bounds__(kDiagThreads, 1)
    k_small_diag(const __grid_constant__ DiagArgs<TM> A) {
  extern __shared__ __align__(16) unsigned char smem[];
  const cg::cluster_group c = cg::this_cluster();
  const int rank = (int)c.block_rank(), tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t n = 3 * A.n_nodes, n_runs = (A.n_nodes + 31) / 32;
  const DiagLayout<TM> lay(A.n_nodes, A.slots, A.own_max, A.rows_max, A.units_max,
                           A.slice_blocks);
  double* const p = reinterpret_cast<double*>(smem + lay.p);    // search direction, all DOFs
  TM* const z = reinterpret_cast<TM*>(smem + lay.z);            // M^-1 r, all DOFs
  double* const pq = reinterpret_cast<double*>(smem + lay.pq);  // [warp of a tile][tile]
  double* const srr = reinterpret_cast<double*>(smem + lay.rr);  // [warp of a CTA][CTA] of the launched update
  double* const srz = reinterpret_cast<double*>(smem + lay.rz);  // ... of the launched preconditioner
  double* const q = reinterpret_cast<double*>(smem + lay.q);    // the owned DOFs of A p
  // the owned DOFs, one per thread
  const int64_t i0 = 96 * own_begin(A.n_nodes, rank), i1 = min(n, 96 * own_begin(A.n_nodes, rank + 1));
  const int n_own = (int)(i1 - i0);
  const bool own = tid < n_own;
  const int64_t mine = i0 + tid;

  // the matrix rows of the CTA's units
  const int4 run = __ldg(A.plan + rank);
  const int64_t c0 = run.z, c1 = run.w;
  const int32_t q0 = __ldg(A.rp + c0);
  const int cnt = __ldg(A.rp + c1) - q0;
  int32_t* const rp = reinterpret_cast<int32_t*>(smem + lay.rp);
  for (int64_t k = tid; k <= c1 - c0; k += kDiagThreads) rp[k] = __ldg(A.rp + c0 + k) - q0;
  int4* const units = reinterpret_cast<int4*>(smem + lay.units);
  for (int k = tid; k < run.y - run.x; k += kDiagThreads) units[k] = __ldg(A.plan + kCtas + run.x + k);
  double* const sk = reinterpret_cast<double*>(smem + lay.kv);
  int32_t* const sc = reinterpret_cast<int32_t*>(smem + lay.ci);
  const int far = max(0, cnt - A.slice_blocks);  // blocks read from L2
  for (int b = tid; b < cnt - far; b += kDiagThreads) {
    sc[b] = __ldg(A.ci + q0 + far + b);
#pragma unroll
    for (int k = 0; k < 9; ++k) sk[k * A.slice_blocks + b] = __ldg(A.k64 + k * A.nnzb + q0 + far + b);
  }
  const TM di = A.precond == 1 && own ? __ldg(A.dinv + mine) : TM(1);
  for (int64_t i = tid; i < n; i += kDiagThreads) p[i] = A.first ? 0.0 : A.p[i];
  for (int i = tid; i < 8 * A.slots; i += kDiagThreads) pq[i] = 0.0;  // units and warps without rows add zero
  for (int i = tid; i < 8 * 32; i += kDiagThreads) srr[i] = srz[i] = 0.0;

  // a warp's sum into place j of every CTA's partials
  auto put = [&](double* part, int j, double v) {
    const double s = warp_sum(v);
    if (lane < kCtas) c.map_shared_rank(part, lane)[(j & 7) * 32 + (j >> 3)] = s;
  };
  // r . r (the thread's share in `rr`) and z = M^-1 r of the owned r with r . z; both sums
  auto precondition = [&](double r, double rr, double& sum_rr, double& sum_rz) {
    const int j0 = (int)(i0 / 32);  // the first launched warp of the owned DOFs
    if (warp * 32 < n_own) put(srr, j0 + warp, rr);
    if (A.precond == 3) {
      if (own) q[tid] = r;  // (q is used up)
      __syncthreads();
      if (warp * 96 < n_own) {  // a node per thread
        double dot = 0.0;
        if (tid * 3 < n_own) {
          TM rv[3];
#pragma unroll
          for (int j = 0; j < 3; ++j) rv[j] = (TM)q[tid * 3 + j];
          const TM* b = A.binv + (mine - tid) * 3 + (int64_t)tid * 9;
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            TM zk = TM(0);
#pragma unroll
            for (int j = 0; j < 3; ++j) zk = fma(__ldg(b + k * 3 + j), rv[j], zk);
            z[i0 + tid * 3 + k] = zk;
            dot = fma((double)rv[k], (double)zk, dot);
          }
        }
        put(srz, (int)(i0 / 96) + warp, dot);
      }
    } else {
      const TM ri = (TM)r;
      const TM zi = di * ri;
      if (own) z[mine] = zi;
      if (warp * 32 < n_own) put(srz, j0 + warp, (double)ri * (double)zi);
    }
    publish_run<kDiagThreads>(c, rank, z, i0, i1);
    c.sync();
    sum_rr = warp_sum(sum8(srr + lane, 32));
    sum_rz = warp_sum(sum8(srz + lane, 32));
  };
  // q = A p of the CTA's units; p . q
  auto product = [&]() {
    const int grp = lane / kLanes, gl = lane % kLanes;
    const int my_r = gl >> 1;  // (group_sum_transposed: row DOF r in the lanes 2 r, 2 r + 1)
    const bool owner = (gl & 1) == 0 && my_r < 3;
    // (to and fro over the warps: those with two units from L2 are not those with three)
    for (int u0 = 0, turn = 0; u0 < run.y - run.x; u0 += kDiagWarps, turn ^= 1) {
      const int u = u0 + (!kWhole && turn ? kDiagWarps - 1 - warp : warp);
      if (u >= run.y - run.x) continue;
      const int4 unit = units[u];  // first row, end of the tile, place of its sum
      double dot = 0.0;
      for (int base = unit.x; base < unit.y; base += 32) {
        const int row = base + grp;
        const bool active = row < unit.y;
        double acc[3] = {0.0, 0.0, 0.0};
        int b = 0, e = 0;
        if (active) {
          b = rp[row - c0] + gl;
          e = rp[row - c0 + 1];
        }
        const int at = (16 * (row >> 5) + 15) / (int)n_runs;  // the CTA that owns the row's DOFs
        // component k of block b at v[k * stride + b]; two blocks in flight, added in order
        auto blocks = [&](const double* v, const int32_t* ci, int64_t stride) {
          for (; b < e; b += 2 * kLanes) {
            const bool two = b + kLanes < e;
            const int b2 = two ? b + kLanes : b;
            const double* xa = p + ci[b] * 3;
            const double* xb = p + ci[b2] * 3;
            double va[9], vb[9];
#pragma unroll
            for (int k = 0; k < 9; ++k) {
              va[k] = v[k * stride + b];
              vb[k] = v[k * stride + b2];
            }
#pragma unroll
            for (int r = 0; r < 3; ++r)
#pragma unroll
              for (int j = 0; j < 3; ++j) acc[r] = fma(va[r * 3 + j], xa[j], acc[r]);
            if (two)
#pragma unroll
              for (int r = 0; r < 3; ++r)
#pragma unroll
                for (int j = 0; j < 3; ++j) acc[r] = fma(vb[r * 3 + j], xb[j], acc[r]);
          }
        };
        if (kWhole || __all_sync(0xffffffffu, !active || b - gl >= far))
          blocks(sk - far, sc - far, A.slice_blocks);
        else
          blocks(A.k64 + q0, A.ci + q0, A.nnzb);
        const double t = group_sum_transposed<3, kLanes>(acc, gl);
        if (active && owner) {
          const int64_t i = (int64_t)row * 3 + my_r;
          c.map_shared_rank(q, at)[i - 96 * own_begin(A.n_nodes, at)] = t;
          dot = fma(p[i], t, dot);
        }
      }
      const double s = warp_sum(dot);
      if (lane < kCtas) c.map_shared_rank(pq, lane)[unit.z] = s;
    }
    c.sync();
    double w[kMaxTiles / 32];
#pragma unroll
    for (int g = 0; g < kMaxTiles / 32; ++g) w[g] = g * 32 < A.slots ? warp_sum(sum8(pq + g * 32 + lane, A.slots)) : 0.0;
    return (w[0] + w[2]) + (w[1] + w[3]);
  };

  c.sync();  // every CTA of the cluster has started; its zeros are in place
  double x = own && !A.first ? A.x[mine] : 0.0, r = own ? (A.first ? A.b[mine] : A.r[mine]) : 0.0, rr, rz;
  precondition(r, r * r, rr, rz);
  const double bb = A.first ? rr : A.S->bnorm2, tol2 = A.rtol * A.rtol * bb;
  double rz_prev = A.first ? 0.0 : A.S->rz[1], alpha = 0.0;
  const int it0 = A.first ? 0 : A.S->iters;
  int it = it0, status = 0;
  bool done = false, running = false;
  if (bb == 0.0 || !isfinite(bb)) {
    done = true;
    status = isfinite(bb) ? 0 : WN_EBREAKDOWN;
  }
  while (!done) {
    const double beta = it == 0 ? 0.0 : rz / rz_prev;
    for (int64_t i = tid; i < n; i += kDiagThreads) p[i] = fma(beta, p[i], (double)z[i]);
    __syncthreads();
    const double gamma = product();
    alpha = rz / gamma;
    if (!(gamma > 0.0) || !isfinite(alpha)) {
      status = WN_EBREAKDOWN;
      break;
    }
    if (own) {
      x = fma(alpha, p[mine], x);
      r = fma(-alpha, q[tid], r);
    }
    rz_prev = rz;
    precondition(r, r * r, rr, rz);
    ++it;
    if (!isfinite(rr)) {
      status = WN_EBREAKDOWN;
      break;
    }
    if (rr <= tol2) break;
    if (it >= A.max_iter) {
      status = WN_ENOCONV;
      break;
    }
    if (it - it0 >= kDiagSteps) {
      running = true;
      break;
    }
  }
  if (own) A.x[mine] = x;
  if (own && running) {
    A.r[mine] = r;
    A.p[mine] = p[mine];
  }
  if (rank == 0 && tid == 0) {
    PcgScalars* S = A.S;
    S->rz[0] = rz;
    S->rz[1] = rz_prev;
    S->bnorm2 = bb;
    S->tol2 = tol2;
    S->rr = rr;
    S->alpha = alpha;
    S->iters = it;
    S->status = status;
    S->max_iter = A.max_iter;
    S->done = !running;
  }
  c.sync();  // no CTA leaves while another may still store into its shared memory
}

// The plan of k_small_diag from the row pointer: the row tiles of the streamed fine matrix (a row over
// a tile's capacity, which the streamed kernels leave alone, by itself) in units, shared out evenly.
struct SmallPlan {
  std::vector<int4> table;
  int tiles = 0, rows_max = 0, blocks_max = 0, units_max = 0;
};
SmallPlan small_plan(const int32_t* rp, int64_t n_nodes) {
  SmallPlan P;
  std::vector<int4> units;
  for (int64_t r = 0; r < n_nodes; ++P.tiles) {
    const int64_t r0 = r++;
    while (r < n_nodes && r - r0 < kStreamRowCap && rp[r + 1] - rp[r0] <= kStreamCap) ++r;
    for (int w = 0; w < 8 && r0 + 4 * w < r; ++w) units.push_back({(int)(r0 + 4 * w), (int)r, w, P.tiles});
  }
  const int slots = (P.tiles + 31) / 32 * 32;
  const int64_t n = (int64_t)units.size();
  for (int k = 0; k < kCtas; ++k) {
    const int u0 = (int)(n * k / kCtas), u1 = (int)(n * (k + 1) / kCtas);
    int lo = 0, hi = 0;
    for (int u = u0; u < u1; ++u) {
      const int4& t = units[u];
      if (u == u0) lo = t.x;
      hi = std::max(hi, std::min(t.y, t.x + 4));
      if (t.y > t.x + 32) hi = t.y;  // rows of a further pass over the tile
    }
    P.table.push_back({u0, u1, lo, hi});
    P.rows_max = std::max(P.rows_max, hi - lo);
    P.blocks_max = std::max(P.blocks_max, rp[hi] - rp[lo]);
    P.units_max = std::max(P.units_max, u1 - u0);
  }
  for (int4& u : units) u = {u.x, u.y, u.z * slots + u.w, 0};
  P.table.insert(P.table.end(), units.begin(), units.end());
  return P;
}

// ---------------------------------------------------------------------------------------
// AMG with at most one level above the dense one
// ---------------------------------------------------------------------------------------
// first row of CTA k: multiples of 4 nodes, so that a run starts on 16 bytes in every vector
__host__ __device__ __forceinline__ int64_t run_begin(int64_t n, int k) {
  return k >= kCtas ? n : (n * k / kCtas) & ~int64_t(3);
}

template <typename TM>
struct AmgArgs {
  int64_t n_nodes, nnzb;
  const int32_t *rp, *ci;
  const double* k64;
  const TM* km;    // the matrix in the preconditioner's precision
  const TM* dinv;  // 1 / diag
  int n_levels;    // 0 (the hierarchy is its dense level) or 1
  TM it;                  // 1 / theta of the fine level
  const int32_t *r_rp, *r_ci, *p_rp, *p_ci;
  const TM *rv, *pv;
  int64_t n_coarse;
  const double* coarse_inv;
  const double* b;
  double *x, *r, *p;  // r, p: the state between launches
  int first;          // from x = 0, or on from the state
  int slice_blocks;  // blocks of the longest run in shared memory, 0: read from L2
  int rows_max;
  double rtol;
  int max_iter;
  PcgScalars* S;
};

// dynamic shared memory of a CTA, in this order
template <typename TM>
struct AmgLayout {
  size_t p, z, w, x, r, q, d0, cb, cx, kv, mv, ci, rp, end;
  __host__ __device__ AmgLayout(int64_t n_nodes, int rows, int64_t n_coarse, int n_levels, int slice) {
    const size_t n = 3 * (size_t)n_nodes, own = 3 * (size_t)rows, bl = (size_t)slice;
    const bool two = n_levels > 0;
    p = 0;
    z = p + pad16(n * 8);
    w = z + pad16(n * sizeof(TM));
    x = w + (two ? pad16(n * sizeof(TM)) : 0);
    r = x + pad16(own * 8);
    q = r + pad16(own * 8);
    d0 = q + pad16(own * 8);
    cb = d0 + (two ? pad16(own * sizeof(TM)) : 0);
    cx = cb + pad16((size_t)n_coarse * sizeof(TM));
    kv = cx + (two ? pad16((size_t)n_coarse * sizeof(TM)) : 0);
    mv = kv + pad16(9 * bl * 8);
    ci = mv + (two && sizeof(TM) != 8 ? pad16(9 * bl * sizeof(TM)) : 0);
    rp = ci + pad16(bl * 4);
    end = rp + pad16(4 * (size_t)(rows + 1));
  }
};

struct Shared {
  double part[2][kCtas * kWarps];  // [turn]: every warp's partial
};

struct Cluster {
  cg::cluster_group c;
  Shared* sh;
  int rank, warp, lane;
  int turn = 0;
  // the sum of this thread's contributions to a dot product over the cluster, past its barrier
  __device__ __forceinline__ double dot(double d) {
    const double w = warp_sum(d);
    if (lane < kCtas) c.map_shared_rank(sh, lane)->part[turn][rank * kWarps + warp] = w;
    c.sync();
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < kCtas * kWarps / 32; ++i) s += sh->part[turn][i * 32 + lane];
    turn ^= 1;  // the next partials go elsewhere: a slow warp may still be adding these
    return warp_sum(s);
  }
  template <typename T>
  __device__ __forceinline__ void publish(T* v, int64_t i0, int64_t i1) const {
    publish_run<kThreads>(c, rank, v, i0, i1);
  }
};

// the CTA's run of the fine matrix: rows c0 .. c1, component k of its block b at v[k * stride + b]
template <typename T>
struct Slice {
  const T* v;
  const int32_t *ci, *rp;
  int64_t stride;
  int64_t c0, c1;
};
// its rows against the vector x (shared memory), 8 lanes each, two blocks in flight per lane;
// epi(i, value) by the lane that owns DOF i
template <typename T, typename EPI>
__device__ __forceinline__ void fine_rows(const Slice<T>& M, const T* x, const EPI& epi) {
  const int gl = threadIdx.x % kLanes;
  for (int64_t base = M.c0; base < M.c1; base += kGroups) {
    const int64_t row = base + threadIdx.x / kLanes;
    const bool active = row < M.c1;
    T acc[3] = {T(0), T(0), T(0)};
    int s = 0, e = 0;
    if (active) {
      s = M.rp[row - M.c0] + gl;
      e = M.rp[row - M.c0 + 1];
    }
    for (int b = s; b < e; b += 2 * kLanes) {
      const bool two = b + kLanes < e;
      const int b2 = two ? b + kLanes : b;
      const T* xa = x + M.ci[b] * 3;
      const T* xb = x + M.ci[b2] * 3;
      T va[9], vb[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        va[k] = M.v[k * M.stride + b];
        vb[k] = M.v[k * M.stride + b2];
      }
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[r] = fma(va[r * 3 + c], xa[c], acc[r]);
      if (two)
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
          for (int c = 0; c < 3; ++c) acc[r] = fma(vb[r * 3 + c], xb[c], acc[r]);
    }
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
      for (int o = kLanes / 2; o > 0; o >>= 1) acc[r] += __shfl_xor_sync(0xffffffffu, acc[r], o);
    if (active && gl < 3) epi(row * 3 + gl, gl == 0 ? acc[0] : gl == 1 ? acc[1] : acc[2]);
  }
}

template <typename TM, bool kSlice>
__global__ void __cluster_dims__(kCtas, 1, 1) __launch_bounds__(kThreads, 1)
    k_small_amg(const __grid_constant__ AmgArgs<TM> A) {
  constexpr bool kSame = std::is_same<TM, double>::value;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ Shared sh;
  __shared__ TM team_sum[kWarps][6];
  Cluster C{cg::this_cluster(), &sh, 0, (int)threadIdx.x >> 5, (int)threadIdx.x & 31};
  C.rank = (int)C.c.block_rank();
  const int64_t c0 = run_begin(A.n_nodes, C.rank), c1 = run_begin(A.n_nodes, C.rank + 1);
  const int64_t i0 = 3 * c0, i1 = 3 * c1, n = 3 * A.n_nodes;
  const AmgLayout<TM> lay(A.n_nodes, A.rows_max, A.n_coarse, A.n_levels, kSlice ? A.slice_blocks : 0);
  auto at = [&](size_t off, auto tag) { return reinterpret_cast<decltype(tag)>(smem + off); };
  double* const p = at(lay.p, (double*)nullptr);   // search direction, all DOFs
  TM* const z = at(lay.z, (TM*)nullptr);           // M^-1 r, all DOFs (two-level: the residual before)
  TM* const w = at(lay.w, (TM*)nullptr);           // two-level: smoothing input and iterate, all DOFs
  double* const x = at(lay.x, (double*)nullptr) - i0;  // the CTA's own rows, indexed globally
  double* const r = at(lay.r, (double*)nullptr) - i0;
  double* const q = at(lay.q, (double*)nullptr) - i0;
  TM* const d0 = at(lay.d0, (TM*)nullptr) - i0;
  TM* const cb = at(lay.cb, (TM*)nullptr);
  TM* const cx = at(lay.cx, (TM*)nullptr);
  const bool two_level = A.n_levels > 0;
  const int gl = threadIdx.x % kLanes;

  // the CTA's run of the fine matrix
  const int32_t q0 = A.rp[c0];
  const int cnt = A.rp[c1] - q0;
  int32_t* const sr = at(lay.rp, (int32_t*)nullptr);
  for (int64_t k = threadIdx.x; k <= c1 - c0; k += kThreads) sr[k] = __ldg(A.rp + c0 + k) - q0;
  Slice<double> K{A.k64 + q0, A.ci + q0, sr, A.nnzb, c0, c1};
  Slice<TM> M{A.km + q0, A.ci + q0, sr, A.nnzb, c0, c1};
  if constexpr (kSlice) {
    double* sk = at(lay.kv, (double*)nullptr);
    TM* sm = at(lay.mv, (TM*)nullptr);
    int32_t* sc = at(lay.ci, (int32_t*)nullptr);
    for (int b = threadIdx.x; b < cnt; b += kThreads) {
      sc[b] = __ldg(A.ci + q0 + b);
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        sk[k * A.slice_blocks + b] = __ldg(A.k64 + k * A.nnzb + q0 + b);
        if (!kSame && two_level) sm[k * A.slice_blocks + b] = __ldg(A.km + k * A.nnzb + q0 + b);
      }
    }
    K = {sk, sc, sr, A.slice_blocks, c0, c1};
    if constexpr (kSame)
      M = {sk, sc, sr, A.slice_blocks, c0, c1};
    else
      M = {sm, sc, sr, A.slice_blocks, c0, c1};
  }
  for (int64_t i = threadIdx.x; i < n; i += kThreads) p[i] = A.first ? 0.0 : A.p[i];

  // f(i) for the DOFs of the CTA's rows, by the lanes that own them in fine_rows
  auto own_dofs = [&](auto f) {
    for (int64_t row = c0 + threadIdx.x / kLanes; row < c1; row += kGroups)
      if (gl < 3) f(row * 3 + gl);
  };
  // the V-cycle's input of the own rows: the first smoothing step's x, or r itself
  auto vcycle_input = [&]() {
    if (two_level) {
      own_dofs([&](int64_t i) { w[i] = d0[i] = __ldg(A.dinv + i) * (TM)r[i] * A.it; });
      C.publish(w, i0, i1);
    } else {
      own_dofs([&](int64_t i) { cb[i] = (TM)r[i]; });
      C.publish(cb, i0, i1);
    }
  };
  // dense rows of the coarsest inverse, a warp each: out(row, value)
  constexpr int kAhead = 12;
  auto coarse = [&](auto out) {
    for (int64_t row = C.rank * kWarps + C.warp; row < A.n_coarse; row += kCtas * kWarps) {
      const double* a = A.coarse_inv + row * A.n_coarse;
      double s[2] = {0.0, 0.0};
      for (int64_t j0 = C.lane; j0 < A.n_coarse; j0 += 32 * kAhead) {  // kAhead loads in flight
        double v[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) v[u] = j0 + 32 * u < A.n_coarse ? __ldg(a + j0 + 32 * u) : 0.0;
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
          if (j0 + 32 * u < A.n_coarse) s[u & 1] = fma(v[u], (double)cb[j0 + 32 * u], s[u & 1]);
      }
      out(row, (TM)warp_sum(s[0] + s[1]));
    }
  };
  // z = V(r) after a barrier that has made the input visible; this thread's part of r . z
  auto vcycle = [&](double& dot) {
    if (!two_level) {  // (the rows of z are those of the dense level, in any CTA)
      coarse([&](int64_t row, TM v) {
        if (C.lane < kCtas) C.c.map_shared_rank(z, C.lane)[row] = v;
        if (C.lane == 0) dot += (double)cb[row] * (double)v;
      });
      return;
    }
    fine_rows<TM>(M, w, [&](int64_t i, TM t) { z[i] = (TM)r[i] - t; });  // the residual
    C.publish(z, i0, i1);
    C.c.sync();
    // restriction: kTeam warps per coarse node (its rows are the longest of the cycle, up to some
    // hundred blocks, and there are fewer of them than warps)
    for (int64_t row0 = (int64_t)C.rank * kTeams; row0 * 6 < A.n_coarse; row0 += kCtas * kTeams) {
      const int team = C.warp / kTeam, tl = (C.warp % kTeam) * 32 + C.lane;
      const int64_t row = row0 + team;
      TM acc[6] = {};
      if (row * 6 < A.n_coarse) {
        const int32_t e = __ldg(A.r_rp + row + 1);
        for (int32_t b = __ldg(A.r_rp + row) + tl; b < e; b += 32 * kTeam) {
          const TM* xb = z + __ldg(A.r_ci + b) * 3;
          TM v[18];
          BlockLoad<TM, 18>::load(A.rv + (int64_t)b * 18, v);
#pragma unroll
          for (int k = 0; k < 6; ++k)
#pragma unroll
            for (int c = 0; c < 3; ++c) acc[k] = fma(v[k * 3 + c], xb[c], acc[k]);
        }
      }
#pragma unroll
      for (int k = 0; k < 6; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
        if (C.lane == k) team_sum[C.warp][k] = acc[k];
      }
      __syncthreads();
      // thread (target CTA, team, DOF) of the CTA's kTeams x 6 sums
      for (int k = threadIdx.x; k < kCtas * kTeams * 6; k += kThreads) {
        const int peer = k % kCtas, dof = k / kCtas % 6, t = k / (kCtas * 6);
        if ((row0 + t) * 6 < A.n_coarse) {
          TM sum = team_sum[t * kTeam][dof];
#pragma unroll
          for (int m = 1; m < kTeam; ++m) sum += team_sum[t * kTeam + m][dof];
          C.c.map_shared_rank(cb, peer)[(row0 + t) * 6 + dof] = sum;
        }
      }
      __syncthreads();
    }
    C.c.sync();
    coarse([&](int64_t row, TM v) {
      if (C.lane < kCtas) C.c.map_shared_rank(cx, C.lane)[row] = v;
    });
    C.c.sync();
    // prolongation of the own rows: x = d0 + P xc
    for (int64_t base = c0; base < c1; base += kGroups) {
      const int64_t row = base + threadIdx.x / kLanes;
      TM acc[3];
      group_block_row<3, 6, kLanes, kAoS, TM, TM>(A.p_rp, A.p_ci, A.pv, 0, row, row < c1, XLoad<TM, TM>{cx}, acc, gl);
      if (row < c1 && gl < 3) {
        const int64_t i = row * 3 + gl;
        w[i] = d0[i] + (gl == 0 ? acc[0] : gl == 1 ? acc[1] : acc[2]);
      }
    }
    C.publish(w, i0, i1);
    C.c.sync();
    fine_rows<TM>(M, w, [&](int64_t i, TM t) {
      const TM bi = (TM)r[i];
      const TM r0 = __ldg(A.dinv + i) * (bi - t);
      const TM zi = fma(r0, A.it, w[i]);
      z[i] = zi;
      dot += (double)bi * (double)zi;
    });
    C.publish(z, i0, i1);
  };

  C.c.sync();  // every CTA of the cluster has started; the run and p are in place
  // x = 0, r = b, ||b||
  double d = 0.0;
  own_dofs([&](int64_t i) {
    const double ri = A.first ? A.b[i] : A.r[i];
    x[i] = A.first ? 0.0 : A.x[i];
    r[i] = ri;
    d += ri * ri;
  });
  __syncthreads();
  vcycle_input();
  double rr = C.dot(d);
  const double bb = A.first ? rr : A.S->bnorm2, tol2 = A.rtol * A.rtol * bb;
  double rz = A.first ? 0.0 : A.S->rz[0], rz_prev = 0.0, alpha = 0.0;
  const int it0 = A.first ? 0 : A.S->iters;
  int it = it0, status = 0;
  bool done = false, running = false;
  if (bb == 0.0 || !isfinite(bb)) {
    done = true;
    status = isfinite(bb) ? 0 : WN_EBREAKDOWN;
  }
  while (!done) {
    d = 0.0;
    vcycle(d);
    rz_prev = rz;
    rz = C.dot(d);
    const double beta = it == 0 ? 0.0 : rz / rz_prev;
    for (int64_t i = threadIdx.x; i < n; i += kThreads) p[i] = fma(beta, p[i], (double)z[i]);
    __syncthreads();
    d = 0.0;
    fine_rows<double>(K, p, [&](int64_t i, double t) {
      q[i] = t;
      d += p[i] * t;
    });
    const double gamma = C.dot(d);
    alpha = rz / gamma;
    if (!(gamma > 0.0) || !isfinite(alpha)) {
      status = WN_EBREAKDOWN;
      break;
    }
    d = 0.0;
    own_dofs([&](int64_t i) {
      x[i] = fma(alpha, p[i], x[i]);
      const double ri = fma(-alpha, q[i], r[i]);
      r[i] = ri;
      d += ri * ri;
    });
    __syncwarp();
    vcycle_input();
    rr = C.dot(d);
    ++it;
    if (!isfinite(rr)) {
      status = WN_EBREAKDOWN;
      break;
    }
    if (rr <= tol2) break;
    if (it >= A.max_iter) {
      status = WN_ENOCONV;
      break;
    }
    if (it - it0 >= kAmgSteps) {
      running = true;
      break;
    }
  }
  own_dofs([&](int64_t i) {
    A.x[i] = x[i];
    if (running) {
      A.r[i] = r[i];
      A.p[i] = p[i];
    }
  });
  if (C.rank == 0 && threadIdx.x == 0) {
    PcgScalars* S = A.S;
    S->rz[0] = rz;
    S->rz[1] = rz_prev;
    S->bnorm2 = bb;
    S->tol2 = tol2;
    S->rr = rr;
    S->alpha = alpha;
    S->iters = it;
    S->status = status;
    S->max_iter = A.max_iter;
    S->done = !running;
  }
  C.c.sync();  // no CTA leaves while another may still store into its shared memory
}

double mat_bytes(const DevBsr& M, int value) {
  return (double)M.nnzb * (M.br * M.bc * value + 4) + 4.0 * (double)(M.n_rows + 1);
}

}  // namespace

// The sizes at which the cluster wins (launched kernels -> cluster, us per iteration, FP64):
//   point Jacobi   153 nodes 13.2 -> 3.9, 1,025 14.2 -> 7.0, 1,325 14.4 -> 7.6, 2,025 15.6 -> 12.7 (block Jacobi
//   0.4 more, none the same); beyond, a thread has more than one DOF, and at 2,597 nodes an earlier
//   form was level with the launched kernels;
//   two-level V-cycle   625 nodes 34 -> 20, 1,025 34 -> 27.5 with the matrix blocks in shared memory, 1,325
//   35 -> 39 without, so there only while they fit; a dense level alone (153 nodes) 250 -> 87 us per
//   solve.
static bool small_system(const Solid* s, const SolverWork& W, int precond) {
  if (s->bs != 3 || s->n_nodes > kMaxNodes || W.profile || W.half) return false;
  // (the failure hook and shortened waits of the streamed kernels are theirs to report)
  if (s->fine.ctl.withhold >= 0 || s->fine.ctl.wait_ns != kStreamWaitLimitNs) return false;
  return precond != 2 || s->amg->levels.empty() || (s->amg->degree == 1 && s->amg->levels.size() == 1);
}

// a kernel of one cluster (an error where 16 SMs of a GPC are not to be had)
template <typename ARGS>
static cudaError_t launch_cluster(void (*kern)(ARGS), const ARGS& A, int threads, size_t smem, size_t limit,
                                  cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit);
  if (e != cudaSuccess) return e;
  kern<<<kCtas, threads, smem, st>>>(A);
  return cudaGetLastError();
}

// none / Jacobi / block Jacobi: 0 with the kernel under way, 1 for the launched kernels
template <typename TM>
static int start_diag(Solid* s, SolverWork& W, const double* b, double rtol, int max_iter, int precond, bool first,
                      PcgScalars* S, cudaStream_t st) {
  if (W.small_tiles == 0) {  // the pattern's plan, kept with the workspace
    const SmallPlan P = small_plan(s->h_row_ptr.data(), s->n_nodes);
    WN_CHECK(W.small_plan.upload(P.table));
    WN_CUDA(cudaStreamSynchronize(0));
    W.small_tiles = P.tiles;
    W.small_rows = P.rows_max;
    W.small_blocks = P.blocks_max;
    W.small_units = P.units_max;
  }
  if (W.small_tiles > kMaxTiles) return 1;
  DiagArgs<TM> A{};
  A.n_nodes = s->n_nodes;
  A.nnzb = s->nnzb;
  A.rp = s->row_ptr.p;
  A.ci = s->col_idx.p;
  A.k64 = s->k64.p;
  if constexpr (std::is_same<TM, double>::value) {
    A.dinv = W.dinv64.p;
    A.binv = W.binv64.p;
  } else {
    A.dinv = W.dinv32.p;
    A.binv = W.binv32.p;
  }
  A.precond = precond;
  A.b = b;
  A.x = W.p64.x.p;
  A.r = W.p64.r.p;
  A.p = W.p64.p0.p;
  A.first = first;
  A.plan = W.small_plan.p;
  A.slots = (W.small_tiles + 31) / 32 * 32;
  for (int k = 0; k < kCtas; ++k)
    A.own_max = std::max(A.own_max, 32 * (int)(own_begin(s->n_nodes, k + 1) - own_begin(s->n_nodes, k)));
  A.rows_max = W.small_rows;
  A.units_max = W.small_units;
  A.rtol = rtol;
  A.max_iter = max_iter;
  A.S = S;
  auto bytes = [&](int held) { return DiagLayout<TM>(A.n_nodes, A.slots, A.own_max, A.rows_max, A.units_max, held).end; };
  constexpr int kBlockBytes = 9 * 8 + 4;
  if (bytes(0) + 32 > kDiagSmemLimit) return 1;  // (two roundings to 16 bytes)
  A.slice_blocks = std::min<int>(W.small_blocks, (int)((kDiagSmemLimit - 32 - bytes(0)) / kBlockBytes));
  const size_t smem = bytes(A.slice_blocks);
  const cudaError_t e =
      A.slice_blocks == W.small_blocks
          ? launch_cluster(k_small_diag<TM, true>, A, kDiagThreads, smem, kDiagSmemLimit, st)
          : launch_cluster(k_small_diag<TM, false>, A, kDiagThreads, smem, kDiagSmemLimit, st);
  return e == cudaSuccess ? 0 : 1;
}

// AMG with at most one level above the dense one: 0 with the kernel under way, 1 for the launched kernels
template <typename TM>
static int start_amg(Solid* s, SolverWork& W, const double* b, double rtol, int max_iter, bool first,
                     PcgScalars* S, cudaStream_t st) {
  constexpr bool kSame = std::is_same<TM, double>::value;
  AmgHierarchy& H = *s->amg;
  AmgArgs<TM> A{};
  A.n_nodes = s->n_nodes;
  A.nnzb = s->nnzb;
  A.rp = s->row_ptr.p;
  A.ci = s->col_idx.p;
  A.k64 = s->k64.p;
  A.b = b;
  A.x = W.p64.x.p;
  A.r = W.p64.r.p;
  A.p = W.p64.p0.p;
  A.first = first;
  if constexpr (kSame) {
    A.km = s->k64.p;
    A.dinv = W.dinv64.p;
  } else {
    A.km = s->k32.p;
    A.dinv = W.dinv32.p;
  }
  A.n_levels = (int)H.levels.size();
  A.n_coarse = H.n_coarse;
  A.coarse_inv = H.coarse_inv.p;
  if (A.n_levels > 0) {
    DevLevel& L = H.levels[0];
    A.it = (TM)L.inv_theta;
    A.r_rp = L.R.rp.p;
    A.r_ci = L.R.ci.p;
    A.p_rp = L.P.rp.p;
    A.p_ci = L.P.ci.p;
    if constexpr (kSame) {
      A.rv = L.R.v64.p;
      A.pv = L.P.v64.p;
    } else {
      A.rv = L.R.v32.p;
      A.pv = L.P.v32.p;
    }
  }
  A.rtol = rtol;
  A.max_iter = max_iter;
  A.S = S;
  int64_t blocks = 0, rows = 0;
  for (int k = 0; k < kCtas; ++k) {
    const int64_t c0 = run_begin(s->n_nodes, k), c1 = run_begin(s->n_nodes, k + 1);
    blocks = std::max<int64_t>(blocks, s->h_row_ptr[c1] - s->h_row_ptr[c0]);
    rows = std::max(rows, c1 - c0);
  }
  A.rows_max = (int)rows;
  A.slice_blocks = (int)blocks;
  auto bytes = [&](int slice) { return AmgLayout<TM>(A.n_nodes, A.rows_max, A.n_coarse, A.n_levels, slice).end; };
  const bool slice = bytes(A.slice_blocks) <= kSmemLimit;
  if (!slice && A.n_levels > 0) return 1;
  const size_t smem = bytes(slice ? A.slice_blocks : 0);
  if (smem > kSmemLimit) return 1;
  const cudaError_t e = slice ? launch_cluster(k_small_amg<TM, true>, A, kThreads, smem, kSmemLimit, st)
                              : launch_cluster(k_small_amg<TM, false>, A, kThreads, smem, kSmemLimit, st);
  return e == cudaSuccess ? 0 : 1;
}

template <typename TM>
int small_pcg(Solid* s, SolverWork& W, const double* b, double rtol, int max_iter, int precond, PcgScalars* S,
              cudaStream_t st, PcgScalars* hS) {
  if (!small_system(s, W, precond)) return 1;
  hS->done = 0;
  for (bool first = true; !hS->done; first = false) {
    const int rc = precond == 2 ? start_amg<TM>(s, W, b, rtol, max_iter, first, S, st)
                                : start_diag<TM>(s, W, b, rtol, max_iter, precond, first, S, st);
    if (rc != 0) {
      cudaGetLastError();
      return rc;  // 1: too many tiles, or no room for a cluster of 16 here
    }
    W.launches++;
    WN_CUDA(cudaMemcpyAsync(hS, S, sizeof(PcgScalars), cudaMemcpyDeviceToHost, st));
    WN_CUDA(cudaStreamSynchronize(st));
  }
  // algorithmic bytes as the launched kernels count them: I products and updates, I preconditioner
  // applies (the first before the iterations, none after the last)
  const double n = (double)W.n, nK = 8.0 * n, nM = n * sizeof(TM);
  const double rows = 4.0 * (double)(s->n_nodes + 1);
  double prec_bytes = (precond == 1 ? 3.0 : precond == 3 ? 5.0 : 2.0) * nM;
  if (precond == 2) {
    const AmgHierarchy& H = *s->amg;
    const double nc = (double)H.n_coarse;
    prec_bytes = 8.0 * nc * nc + 2.0 * nc * sizeof(TM);
    if (!H.levels.empty())
      prec_bytes += 2.0 * ((double)s->nnzb * (9 * sizeof(TM) + 4) + rows) + mat_bytes(H.levels[0].P, sizeof(TM)) +
                    mat_bytes(H.levels[0].R, sizeof(TM)) + 11.0 * nM;
  }
  const double fine64 = (double)s->nnzb * 76.0 + rows;
  W.bytes += 3.0 * nK + hS->iters * (fine64 + nM + 9.0 * nK) + std::max(1, hS->iters) * prec_bytes;
  return 0;
}
template int small_pcg<double>(Solid*, SolverWork&, const double*, double, int, int, PcgScalars*, cudaStream_t,
                               PcgScalars*);
template int small_pcg<float>(Solid*, SolverWork&, const double*, double, int, int, PcgScalars*, cudaStream_t,
                              PcgScalars*);

}  // namespace wn
