// PCG of a small system in one kernel: a cluster of 16 CTAs runs every iteration.
//
// A system of a few thousand nodes gives each of an iteration's kernels (five with point Jacobi, nine
// with a two-level V-cycle) a microsecond of work and three to five of launch, ramp-up and
// dependence: 15.8 us per point-Jacobi and 35 us per AMG iteration at 1,025 nodes, whatever the matrix.
// Here the stages of an iteration are the phases of one persistent kernel, separated by the
// hardware barrier of a thread-block cluster (16 CTAs on 16 SMs of one GPC: co-scheduled by the
// launch, no spinning).  What bounds it is the chain of phases, so nothing on it goes through L2
// that need not:
//   * every CTA holds a copy of the gathered vectors in its shared memory; a CTA computes its run of
//     rows and stores the result into all 16 copies before the barrier.  (Gathering through L2
//     instead, two round trips per phase, took 11 and 35 us per iteration.)
//   * p = z + beta p is formed by every CTA for itself, so only z travels;
//   * x, r and q of the CTA's own rows stay in its shared memory, as do their matrix blocks when they
//     fit (about 2,000 FP64 blocks per CTA); otherwise the blocks are read from L2, which does not
//     depend on any phase;
//   * dot products: one partial per warp, stored into every CTA before the barrier; each warp adds
//     the 256 partials in the same order, so all threads take the same alpha, beta and decisions.
// The arithmetic is that of the launched kernels (solver.cu): FP64 Krylov vectors, matrix and dots;
// the preconditioner in TM.  Sums run in another order.
#include <cooperative_groups.h>

#include <algorithm>
#include <type_traits>

#include "amg.h"
#include "common.cuh"
#include "small_solve.h"
#include "solid.h"
#include "spmv.cuh"
#include "wnfea_cuda.h"

namespace cg = cooperative_groups;

namespace wn {
namespace {

constexpr int kCtas = 16, kThreads = 512, kWarps = kThreads / 32;
constexpr int kLanes = 8;                   // lanes per block row
constexpr int kGroups = kThreads / kLanes;  // rows of a CTA side by side
constexpr int kTeam = 4, kTeams = kWarps / kTeam;  // warps per row of the restriction
constexpr int64_t kMaxNodes = 2048;         // (small_system)
constexpr size_t kSmemLimit = 214 * 1024;   // dynamic shared memory (11 KB are static)

// first row of CTA k: multiples of 4 nodes, so that a run starts on 16 bytes in every vector
__host__ __device__ __forceinline__ int64_t run_begin(int64_t n, int k) {
  return k >= kCtas ? n : (n * k / kCtas) & ~int64_t(3);
}
__host__ __device__ constexpr size_t pad16(size_t bytes) { return (bytes + 15) & ~size_t(15); }

template <typename TM>
struct SmallArgs {
  int64_t n_nodes, nnzb;
  const int32_t *rp, *ci;
  const double* k64;
  const TM* km;    // the matrix in the preconditioner's precision
  const TM* dinv;  // 1 / diag
  const TM* binv;  // block Jacobi
  int precond, n_levels;  // n_levels: 0 (the hierarchy is its dense level) or 1
  TM it;                  // 1 / theta of the fine level
  const int32_t *r_rp, *r_ci, *p_rp, *p_ci;
  const TM *rv, *pv;
  int64_t n_coarse;
  const double* coarse_inv;
  const double* b;
  double* x;
  int slice_blocks;  // blocks of the longest run in shared memory, 0: read from L2
  int rows_max;
  double rtol;
  int max_iter;
  PcgScalars* S;
};

// dynamic shared memory of a CTA, in this order
template <typename TM>
struct Layout16 {
  size_t p, z, w, x, r, q, d0, cb, cx, kv, mv, ci, rp, end;
  __host__ __device__ Layout16(int64_t n_nodes, int rows, int64_t n_coarse, int precond, int n_levels, int slice) {
    const size_t n = 3 * (size_t)n_nodes, own = 3 * (size_t)rows, bl = (size_t)slice;
    const bool amg = precond == 2, two = amg && n_levels > 0;
    p = 0;
    z = p + pad16(n * 8);
    w = z + pad16(n * sizeof(TM));
    x = w + (two ? pad16(n * sizeof(TM)) : 0);
    r = x + pad16(own * 8);
    q = r + pad16(own * 8);
    d0 = q + pad16(own * 8);
    cb = d0 + (two ? pad16(own * sizeof(TM)) : 0);
    cx = cb + (amg ? pad16((size_t)n_coarse * sizeof(TM)) : 0);
    kv = cx + (two ? pad16((size_t)n_coarse * sizeof(TM)) : 0);
    mv = kv + pad16(9 * bl * 8);
    ci = mv + (two && sizeof(TM) != 8 ? pad16(9 * bl * sizeof(TM)) : 0);
    rp = ci + pad16(bl * 4);
    end = rp + pad16(4 * (size_t)(rows + 1));
  }
};

struct Shared {
  double part[2][2][kCtas * kWarps];  // [dot][turn]: every warp's partial
};

struct Cluster {
  cg::cluster_group c;
  Shared* sh;
  int rank, warp, lane;
  int turn = 0;
  // this thread's contributions to N dot products, then the cluster barrier; the sums
  template <int N>
  __device__ __forceinline__ void dots(double (&d)[N]) {
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const double s = warp_sum(d[k]);
      if (lane < kCtas) c.map_shared_rank(sh, lane)->part[k][turn][rank * kWarps + warp] = s;
    }
    c.sync();
#pragma unroll
    for (int k = 0; k < N; ++k) {
      double s = 0.0;
#pragma unroll
      for (int i = 0; i < kCtas * kWarps / 32; ++i) s += sh->part[k][turn][i * 32 + lane];
      d[k] = warp_sum(s);
    }
    turn ^= 1;  // the next partials go elsewhere: a slow warp may still be adding these
  }
  // the CTA's own run [i0, i1) of a vector into the other CTAs' copies (visible after the next barrier)
  template <typename T>
  __device__ __forceinline__ void publish(T* v, int64_t i0, int64_t i1) const {
    __syncthreads();  // the run is complete
    const int64_t u0 = i0 * sizeof(T) / 16, u1 = (i1 * sizeof(T) + 15) / 16;
    const int n = (int)(u1 - u0);
    uint4* own = reinterpret_cast<uint4*>(v) + u0;
    for (int k = threadIdx.x; k < n * (kCtas - 1); k += kThreads) {
      const int peer = k / n, at = k - peer * n;
      uint4* there = c.map_shared_rank(own, peer + (peer >= rank));
      there[at] = own[at];
    }
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
    k_small_pcg(const __grid_constant__ SmallArgs<TM> A) {
  constexpr bool kSame = std::is_same<TM, double>::value;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ Shared sh;
  __shared__ TM team_sum[kWarps][6];
  Cluster C{cg::this_cluster(), &sh, 0, (int)threadIdx.x >> 5, (int)threadIdx.x & 31};
  C.rank = (int)C.c.block_rank();
  const int64_t c0 = run_begin(A.n_nodes, C.rank), c1 = run_begin(A.n_nodes, C.rank + 1);
  const int64_t i0 = 3 * c0, i1 = 3 * c1, n = 3 * A.n_nodes;
  const Layout16<TM> lay(A.n_nodes, A.rows_max, A.n_coarse, A.precond, A.n_levels, kSlice ? A.slice_blocks : 0);
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
  const bool two_level = A.precond == 2 && A.n_levels > 0;
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
  for (int64_t i = threadIdx.x; i < n; i += kThreads) p[i] = 0.0;

  // f(i) for the DOFs of the CTA's rows, by the lanes that own them in fine_rows
  auto own_dofs = [&](auto f) {
    for (int64_t row = c0 + threadIdx.x / kLanes; row < c1; row += kGroups)
      if (gl < 3) f(row * 3 + gl);
  };
  // point / block Jacobi or none: z of the own rows, with this thread's part of r . z
  auto diagonal = [&](double& dot) {
    for (int64_t base = c0; base < c1; base += kGroups) {  // uniform: the shuffles need the warp
      const int64_t row = base + threadIdx.x / kLanes;
      const bool own = row < c1 && gl < 3;
      const int64_t i = row * 3 + gl;
      const TM ri = own ? (TM)r[i] : TM(0);
      TM zi = ri;
      if (A.precond == 3) {
        zi = TM(0);
#pragma unroll
        for (int j = 0; j < 3; ++j) {
          const TM rj = __shfl_sync(0xffffffffu, ri, j, kLanes);
          if (own) zi = fma(__ldg(A.binv + row * 9 + gl * 3 + j), rj, zi);
        }
      } else if (A.precond == 1 && own) {
        zi = __ldg(A.dinv + i) * ri;
      }
      if (own) {
        z[i] = zi;
        dot += (double)ri * (double)zi;
      }
    }
    C.publish(z, i0, i1);
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
  // x = 0, r = b, ||b||, z = M^-1 r
  double d2[2] = {0.0, 0.0};
  own_dofs([&](int64_t i) {
    const double bi = __ldg(A.b + i);
    x[i] = 0.0;
    r[i] = bi;
    d2[0] += bi * bi;
  });
  __syncthreads();
  if (A.precond == 2)
    vcycle_input();
  else
    diagonal(d2[1]);
  C.dots(d2);
  const double bb = d2[0], tol2 = A.rtol * A.rtol * bb;
  double rr = bb, rz = d2[1], rz_prev = 0.0, alpha = 0.0;
  int it = 0, status = 0;
  bool done = false;
  if (bb == 0.0 || !isfinite(bb)) {
    done = true;
    status = isfinite(bb) ? 0 : WN_EBREAKDOWN;
  }
  while (!done) {
    if (A.precond == 2) {
      double d[1] = {0.0};
      vcycle(d[0]);
      C.dots(d);
      rz_prev = rz;
      rz = d[0];
    }
    const double beta = it == 0 ? 0.0 : rz / rz_prev;
    for (int64_t i = threadIdx.x; i < n; i += kThreads) p[i] = fma(beta, p[i], (double)z[i]);
    __syncthreads();
    double d[1] = {0.0};
    fine_rows<double>(K, p, [&](int64_t i, double t) {
      q[i] = t;
      d[0] += p[i] * t;
    });
    C.dots(d);
    const double gamma = d[0];
    alpha = rz / gamma;
    if (!(gamma > 0.0) || !isfinite(alpha)) {
      status = WN_EBREAKDOWN;
      break;
    }
    d2[0] = d2[1] = 0.0;
    own_dofs([&](int64_t i) {
      x[i] = fma(alpha, p[i], x[i]);
      const double ri = fma(-alpha, q[i], r[i]);
      r[i] = ri;
      d2[0] += ri * ri;
    });
    __syncwarp();
    if (A.precond == 2)
      vcycle_input();
    else
      diagonal(d2[1]);
    C.dots(d2);
    rr = d2[0];
    if (A.precond != 2) {
      rz_prev = rz;
      rz = d2[1];
    }
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
  }
  own_dofs([&](int64_t i) { A.x[i] = x[i]; });
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
    S->done = 1;
  }
  C.c.sync();  // no CTA leaves while another may still store into its shared memory
}

double mat_bytes(const DevBsr& M, int value) {
  return (double)M.nnzb * (M.br * M.bc * value + 4) + 4.0 * (double)(M.n_rows + 1);
}

}  // namespace

// The sizes at which the cluster wins (launched kernels -> cluster, us per iteration, FP64):
//   none / point / block Jacobi   153 nodes 14.7 -> 4.8, 1,025 14.6 -> 7.4, 2,009 15.8 -> 12.5, 2,597 15.8 -> 15.9;
//   two-level V-cycle   625 nodes 34 -> 23, 1,025 34 -> 29 with the matrix blocks in shared memory, 1,325
//   35 -> 39 without, so there only while they fit; a dense level alone (500 nodes at most) 260 -> 90
//   us per solve.
static bool small_system(const Solid* s, const SolverWork& W, int precond) {
  if (s->bs != 3 || s->n_nodes > kMaxNodes || W.profile || W.half) return false;
  // (the failure hook and shortened waits of the streamed kernels are theirs to report)
  if (s->fine.ctl.withhold >= 0 || s->fine.ctl.wait_ns != kStreamWaitLimitNs) return false;
  return precond != 2 || s->amg->levels.empty() || (s->amg->degree == 1 && s->amg->levels.size() == 1);
}

template <typename TM>
int small_pcg(Solid* s, SolverWork& W, const double* b, double rtol, int max_iter, int precond, PcgScalars* S,
              cudaStream_t st, PcgScalars* hS) {
  if (!small_system(s, W, precond)) return 1;
  constexpr bool kSame = std::is_same<TM, double>::value;
  SmallArgs<TM> A{};
  A.n_nodes = s->n_nodes;
  A.nnzb = s->nnzb;
  A.rp = s->row_ptr.p;
  A.ci = s->col_idx.p;
  A.k64 = s->k64.p;
  A.b = b;
  A.x = W.p64.x.p;
  if constexpr (kSame) {
    A.km = s->k64.p;
    A.dinv = W.dinv64.p;
    A.binv = W.binv64.p;
  } else {
    A.km = s->k32.p;
    A.dinv = W.dinv32.p;
    A.binv = W.binv32.p;
  }
  A.precond = precond;
  const double n = (double)W.n, nK = 8.0 * n, nM = n * sizeof(TM);
  double prec_bytes = (precond == 1 ? 3.0 : precond == 3 ? 5.0 : 2.0) * nM;
  if (precond == 2) {
    AmgHierarchy& H = *s->amg;
    A.n_levels = (int)H.levels.size();
    A.n_coarse = H.n_coarse;
    A.coarse_inv = H.coarse_inv.p;
    prec_bytes = 8.0 * (double)H.n_coarse * (double)H.n_coarse + 2.0 * (double)H.n_coarse * sizeof(TM);
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
      const double fine = (double)s->nnzb * (9 * sizeof(TM) + 4) + 4.0 * (double)(s->n_nodes + 1);
      prec_bytes += 2.0 * fine + mat_bytes(L.P, sizeof(TM)) + mat_bytes(L.R, sizeof(TM)) + 11.0 * nM;
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
  auto bytes = [&](int slice) {
    return Layout16<TM>(A.n_nodes, A.rows_max, A.n_coarse, precond, A.n_levels, slice).end;
  };
  const bool slice = bytes(A.slice_blocks) <= kSmemLimit;
  if (!slice && A.n_levels > 0) return 1;
  const size_t smem = bytes(slice ? A.slice_blocks : 0);
  if (smem > kSmemLimit) return 1;
  auto launch = [&](auto kern) -> cudaError_t {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit);
    if (e != cudaSuccess) return e;
    kern<<<kCtas, kThreads, smem, st>>>(A);
    return cudaGetLastError();
  };
  if ((slice ? launch(k_small_pcg<TM, true>) : launch(k_small_pcg<TM, false>)) != cudaSuccess) {
    cudaGetLastError();
    return 1;  // no room for a cluster of 16 here: the launched kernels
  }
  W.launches++;
  WN_CUDA(cudaMemcpyAsync(hS, S, sizeof(PcgScalars), cudaMemcpyDeviceToHost, st));
  WN_CUDA(cudaStreamSynchronize(st));
  // Out of iterations, hundreds from convergence: such an iterate depends on the order of the dot
  // products, so it is left to the launched kernels, whose order does not depend on this rule.
  if (hS->status == WN_ENOCONV && precond != 2) return 1;
  // algorithmic bytes as the launched kernels count them: I products and updates, I preconditioner
  // applies (the first before the iterations, none after the last)
  const double fine64 = (double)s->nnzb * 76.0 + 4.0 * (double)(s->n_nodes + 1);
  W.bytes += 3.0 * nK + hS->iters * (fine64 + nM + 9.0 * nK) + std::max(1, hS->iters) * prec_bytes;
  return 0;
}
template int small_pcg<double>(Solid*, SolverWork&, const double*, double, int, int, PcgScalars*, cudaStream_t,
                               PcgScalars*);
template int small_pcg<float>(Solid*, SolverWork&, const double*, double, int, int, PcgScalars*, cudaStream_t,
                              PcgScalars*);

}  // namespace wn
