// Co-rotational beam frames on sm_100a: internal force, consistent tangent assembled into a
// 6x6-block BSR matrix through an atomic-free element -> block gather, Dirichlet rows, and a
// block-Jacobi BiCGStab for the (in general nonsymmetric) tangent.
//
// The reference evaluates only the internal force (fast_kernels.py:451-537,
// kernels.cpp:19-204, hip_kernels.cpp:53-241) and obtains tangent actions by finite
// differences of the residual (jfnk_operator.py:98-134).  Here the tangent is the exact
// derivative of the same force code (forward-mode dual numbers, beam.cuh), one thread per
// (element, seed direction), so K_t v agrees with the JFNK directional derivative up to its
// truncation error and Newton converges quadratically.
#include <algorithm>
#include <cstring>
#include <vector>

#include "beam.cuh"
#include "common.cuh"
#include "device_array.h"
#include "kernels.h"
#include "wnfea_cuda.h"

namespace wn {

__device__ __forceinline__ void load_element(int64_t e, const double* __restrict__ nodes,
                                             const int32_t* __restrict__ el, const double* __restrict__ props,
                                             const double* __restrict__ eref, const double* __restrict__ L0,
                                             double x1[3], double x2[3], double ev[9], double p[6], double& l0,
                                             int64_t& n1, int64_t& n2) {
  n1 = el[e * 2];
  n2 = el[e * 2 + 1];
  for (int k = 0; k < 3; ++k) {
    x1[k] = nodes[n1 * 3 + k];
    x2[k] = nodes[n2 * 3 + k];
  }
  for (int k = 0; k < 9; ++k) ev[k] = eref[e * 9 + k];
  for (int k = 0; k < 6; ++k) p[k] = props[e * 6 + k];
  l0 = L0[e];
}

// f_e (n_el x 12), one thread per element (FP64)
__global__ void beam_force_kernel(int64_t n_el, const double* __restrict__ nodes, const int32_t* __restrict__ el,
                                  const double* __restrict__ props, const double* __restrict__ eref,
                                  const double* __restrict__ L0, const double* __restrict__ U,
                                  double* __restrict__ fe) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n_el; e += (int64_t)gridDim.x * blockDim.x) {
    double x1[3], x2[3], ev[9], p[6], l0;
    int64_t n1, n2;
    load_element(e, nodes, el, props, eref, L0, x1, x2, ev, p, l0, n1, n2);
    double u1[3], t1[3], u2[3], t2[3], f[12];
    for (int k = 0; k < 3; ++k) {
      u1[k] = U[n1 * 6 + k];
      t1[k] = U[n1 * 6 + 3 + k];
      u2[k] = U[n2 * 6 + k];
      t2[k] = U[n2 * 6 + 3 + k];
    }
    beam_internal_force<double>(x1, x2, ev, l0, p, u1, t1, u2, t2, f);
    for (int k = 0; k < 12; ++k) fe[e * 12 + k] = f[k];
  }
}

// K_e column j = d f_e / d u_e[j]: one thread per (element, j), dual numbers seeded with
// e_j.  ke is n_el x 12 x 12 row-major (ke[e][i][j] = d f_i / d u_j).
__global__ void beam_tangent_kernel(int64_t n_el, const double* __restrict__ nodes, const int32_t* __restrict__ el,
                                    const double* __restrict__ props, const double* __restrict__ eref,
                                    const double* __restrict__ L0, const double* __restrict__ U,
                                    double* __restrict__ ke) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n_el * 12;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t e = t / 12;
    const int j = (int)(t - e * 12);
    double x1[3], x2[3], ev[9], p[6], l0;
    int64_t n1, n2;
    load_element(e, nodes, el, props, eref, L0, x1, x2, ev, p, l0, n1, n2);
    Dual u1[3], t1[3], u2[3], t2[3], f[12];
    for (int k = 0; k < 3; ++k) {
      u1[k] = Dual(U[n1 * 6 + k], j == k ? 1.0 : 0.0);
      t1[k] = Dual(U[n1 * 6 + 3 + k], j == 3 + k ? 1.0 : 0.0);
      u2[k] = Dual(U[n2 * 6 + k], j == 6 + k ? 1.0 : 0.0);
      t2[k] = Dual(U[n2 * 6 + 3 + k], j == 9 + k ? 1.0 : 0.0);
    }
    beam_internal_force<Dual>(x1, x2, ev, l0, p, u1, t1, u2, t2, f);
    for (int i = 0; i < 12; ++i) ke[e * 144 + i * 12 + j] = f[i].d;
  }
}

// F (6 n) = sum over each node's incident (element, end) pairs, in element order
__global__ void beam_node_gather_kernel(int64_t n_nodes, const int64_t* __restrict__ inc_ptr,
                                        const int32_t* __restrict__ inc_ea, const double* __restrict__ fe,
                                        int accumulate, double* __restrict__ F) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n_nodes * 6;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t n = t / 6;
    const int c = (int)(t - n * 6);
    double s = 0.0;
    for (int64_t q = inc_ptr[n]; q < inc_ptr[n + 1]; ++q) s += fe[(int64_t)inc_ea[q] * 6 + c];
    F[t] = accumulate ? F[t] + s : s;
  }
}

// BSR6 values: block b = sum of its element blocks (gather list src = e * 4 + 2 a + b,
// element order), Dirichlet rows/columns -> identity.  Block-contiguous (AoS) output.
__global__ void beam_gather_kernel(int64_t nnzb, const int32_t* __restrict__ gptr, const int32_t* __restrict__ gsrc,
                                   const double* __restrict__ ke, const int32_t* __restrict__ block_row,
                                   const int32_t* __restrict__ col_idx, const uint8_t* __restrict__ fixed,
                                   double* __restrict__ K) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < nnzb * 36;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = t / 36;
    const int k = (int)(t - b * 36);
    const int i = k / 6, j = k - (k / 6) * 6;
    double acc = 0.0;
    for (int32_t q = gptr[b]; q < gptr[b + 1]; ++q) {
      const int32_t src = gsrc[q];
      const int64_t e = src >> 2;
      const int a = (src >> 1) & 1, c = src & 1;
      acc += ke[e * 144 + (a * 6 + i) * 12 + c * 6 + j];
    }
    if (fixed) {
      const int64_t rd = (int64_t)block_row[b] * 6 + i, cd = (int64_t)col_idx[b] * 6 + j;
      if (fixed[rd] | fixed[cd]) acc = (rd == cd) ? 1.0 : 0.0;
    }
    K[t] = acc;
  }
}

// Inverse of each 6x6 diagonal block (Gauss-Jordan, partial pivoting); a singular block
// falls back to the inverse of its diagonal.
__global__ void beam_block_inverse_kernel(int64_t n_nodes, const int32_t* __restrict__ diag_block,
                                          const double* __restrict__ K, double* __restrict__ inv) {
  for (int64_t n = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; n < n_nodes; n += (int64_t)gridDim.x * blockDim.x) {
    double a[6][12];
    const double* blk = K + (int64_t)diag_block[n] * 36;
    for (int i = 0; i < 6; ++i)
      for (int j = 0; j < 12; ++j) a[i][j] = j < 6 ? blk[i * 6 + j] : (j - 6 == i ? 1.0 : 0.0);
    bool ok = true;
    for (int c = 0; c < 6 && ok; ++c) {
      int piv = c;
      for (int r = c + 1; r < 6; ++r)
        if (fabs(a[r][c]) > fabs(a[piv][c])) piv = r;
      if (!(fabs(a[piv][c]) > 0.0)) {
        ok = false;
        break;
      }
      if (piv != c)
        for (int j = 0; j < 12; ++j) {
          const double tmp = a[c][j];
          a[c][j] = a[piv][j];
          a[piv][j] = tmp;
        }
      const double d = 1.0 / a[c][c];
      for (int j = 0; j < 12; ++j) a[c][j] *= d;
      for (int r = 0; r < 6; ++r)
        if (r != c) {
          const double f = a[r][c];
          for (int j = 0; j < 12; ++j) a[r][j] -= f * a[c][j];
        }
    }
    double* out = inv + n * 36;
    for (int i = 0; i < 6; ++i)
      for (int j = 0; j < 6; ++j) {
        const double dg = blk[i * 6 + i];
        out[i * 6 + j] = ok ? a[i][j + 6] : (i == j ? (dg != 0.0 ? 1.0 / dg : 1.0) : 0.0);
      }
  }
}

// y_n = inv_n x_n (6x6 per node)
__global__ void beam_block_apply_kernel(int64_t n_nodes, const double* __restrict__ inv, const double* __restrict__ x,
                                        double* __restrict__ y) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n_nodes * 6;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t n = t / 6;
    const int i = (int)(t - n * 6);
    double s = 0.0;
    for (int j = 0; j < 6; ++j) s += inv[n * 36 + i * 6 + j] * x[n * 6 + j];
    y[t] = s;
  }
}

// partial dots of (a, b) pairs into part[cta * 2 + k]; second stage sums in fixed order
__global__ void beam_dot2_kernel(int64_t n, const double* __restrict__ a0, const double* __restrict__ b0,
                                 const double* __restrict__ a1, const double* __restrict__ b1,
                                 double* __restrict__ part) {
  __shared__ double sh[8];
  double s0 = 0.0, s1 = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    s0 += a0[i] * b0[i];
    if (a1) s1 += a1[i] * b1[i];
  }
  s0 = block_sum(s0, sh);
  s1 = block_sum(s1, sh);
  if (threadIdx.x == 0) {
    part[blockIdx.x * 2] = s0;
    part[blockIdx.x * 2 + 1] = s1;
  }
}

// y = a x + b y + c z   (z may be null)
__global__ void beam_lincomb_kernel(int64_t n, double a, const double* __restrict__ x, double b, double* __restrict__ y,
                                    double c, const double* __restrict__ z) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    y[i] = a * x[i] + (b != 0.0 ? b * y[i] : 0.0) + (z ? c * z[i] : 0.0);  // b == 0 ignores y
}


// Dense copy (row-major n x n, n = 6 n_nodes) of the BSR6 matrix; A must be zeroed first.
__global__ void beam_dense_kernel(int64_t n_nodes, const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
                                  const double* __restrict__ K, double* __restrict__ A) {
  const int64_t n = n_nodes * 6;
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n_nodes * 6;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = t / 6;
    const int i = (int)(t - row * 6);
    for (int32_t q = rp[row]; q < rp[row + 1]; ++q)
      for (int j = 0; j < 6; ++j) A[t * n + (int64_t)ci[q] * 6 + j] = K[(int64_t)q * 36 + i * 6 + j];
  }
}

// Blocked right-looking LU with partial pivoting and the solve of A x = b (x overwrites b),
// in panels of NB columns, limited to the band of the matrix: with half bandwidth kb (the largest
// |i - j| of a nonzero) column k of the factors ends at row k + kb and, with row exchanges, row k
// at column k + 2 kb; outside, every operation of the dense algorithm has a zero operand and
// changes nothing.  Per panel
//   beam_lu_panel_kernel    (one CTA)   pivots, row swaps, multipliers and rank-1 updates inside
//                                       the panel's columns, and the forward elimination of b;
//   beam_lu_trailing_kernel (a CTA per 32 trailing columns) the panel's row swaps, then
//                                       U12 = L11^-1 A12, and with few rows below the panel also
//                                       A22 -= L21 U12;
//   beam_lu_update_kernel   (32 x 32 tiles) A22 -= L21 U12 where the rows are many;
// then beam_lu_backsub_kernel (one CTA).  Every element sees the unblocked dense algorithm's
// operations in its order (fused multiply-adds), so the factors and x depend neither on the panel
// width nor on the band.  The multipliers of earlier panels are never read again (b is
// eliminated as the panels go), so row swaps touch the panel, the trailing columns and b only.
// status: 0 ok, 1 singular (a zero pivot column; the later kernels then see status != 0 and
// return).  Every loop is bounded by n.
//
// What bounds it: the serial chain of pivots.  A panel's rows stay in the registers of one CTA
// (RPT rows of NB columns per thread), so a column costs one barrier, two three-step warp
// reductions, a division and its multiply-adds instead of several passes over global memory;
// NB x RPT is chosen so that the rows that the band leaves fit (dense_lu).  Measured on the
// 10 x 10 frame (600 DOFs, kb = 65) against the same algorithm over all n rows and columns from
// global memory: panel 165 -> 28 us, trailing columns 56 -> 11 us per panel, back substitution
// 300 -> 48 us per solve, bit for bit the same x; ten load steps 95.7 -> 21.8 ms.
constexpr int kLuThreads = 512;   // most threads of a panel
constexpr int kLuMaxPanel = 32;   // widest panel
constexpr int kLuFuseRows = 256;  // up to so many rows below the panel are updated by the trailing kernel

// the panel's row exchanges, as one permutation: src[k] = the row that moves to panel row k; moved
// pairs (dest, src) for the rows below the panel
struct LuSwaps {
  int src[kLuMaxPanel];
  int n_moved;
  int dest[kLuMaxPanel];
  int from[kLuMaxPanel];
};

// argmax of (key, pos), ties to the smaller pos, over a warp; all lanes get the result.  One lane
// usually has the largest high word alone.
__device__ __forceinline__ void lu_warp_argmax(unsigned long long& key, int& pos, int& winner) {
  const unsigned hi = (unsigned)(key >> 32), lo = (unsigned)key;
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  unsigned best = __ballot_sync(0xffffffffu, hi == mh);
  if (best & (best - 1)) {
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
    const bool top = hi == mh && lo == ml;
    const unsigned mp = __reduce_min_sync(0xffffffffu, top ? (unsigned)pos : 0x7fffffffu);
    best = __ballot_sync(0xffffffffu, top && (unsigned)pos == mp);
  }
  winner = __ffs(best) - 1;
  key = __shfl_sync(0xffffffffu, key, winner);
  pos = __shfl_sync(0xffffffffu, pos, winner);
}

// rows k0 .. rend - 1 (at most RPT * blockDim), columns k0 .. k0 + NB - 1.
//   * A row stays with its thread; an exchange changes only the positions that the two threads
//     hold (moving the rows cost 600 of 2,100 cycles per column).
//   * Every warp publishes its best candidate's row before the column's one barrier; after it,
//     all threads pick the pivot among the warps' and read its row.
//   * The rows rotate by one column per step -- the current column is always a[.][0], a finished
//     one (a multiplier below the pivot, an entry of U above) goes to the end -- so the loop over
//     the columns stays rolled.
template <int NB, int RPT>
__global__ void __launch_bounds__(kLuThreads) beam_lu_panel_kernel(int n, int k0, int rend, double* __restrict__ A,
                                                                   double* __restrict__ b,
                                                                   LuSwaps* __restrict__ swaps,
                                                                   int* __restrict__ status) {
  constexpr int kWarps = kLuThreads / 32;
  // per warp, in turns: its best candidate (zeros for the finished columns), the row's b, |value|
  // as bits (ordered as |value| is; 0 also for NaN) and position
  __shared__ __align__(16) double s_u[2][kWarps][NB];
  __shared__ double s_rhs[2][kWarps];
  __shared__ unsigned long long s_key[2][kWarps];
  __shared__ int s_pos[2][kWarps];
  __shared__ int s_moved;
  if (status[0] != 0) return;
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  const int m = rend - k0, w = min(NB, n - k0);
  double a[RPT][NB], rhs[RPT];
  int pos[RPT];  // the row's position in the exchanged order
#pragma unroll
  for (int q = 0; q < RPT; ++q) {
    const int r = tid + q * nt;
    pos[q] = r;
    rhs[q] = r < m ? b[k0 + r] : 0.0;
    // n, k0 and w are even: 16-byte loads
    const double2* __restrict__ row = reinterpret_cast<const double2*>(A + (int64_t)(k0 + (r < m ? r : 0)) * n + k0);
#pragma unroll
    for (int j = 0; j < NB; j += 2) {
      const double2 v = (r < m && j < w) ? row[j / 2] : make_double2(0.0, 0.0);
      a[q][j] = v.x;
      a[q][j + 1] = v.y;
    }
  }
  if (tid == 0) s_moved = 0;
#pragma unroll 1
  for (int c = 0; c < NB; ++c) {
    const bool live = c < w;  // the ragged last panel only rotates its missing columns
    const int t = c & 1;
    int slot = 0;
    if (live) {
      unsigned long long key = 0;
      int p = 0x7fffffff, mine = 0;
#pragma unroll
      for (int q = 0; q < RPT; ++q) {
        const double v = fabs(a[q][0]);
        const unsigned long long kq =
            (pos[q] >= c && pos[q] < m && v == v) ? (unsigned long long)__double_as_longlong(v) : 0;
        if (kq > key || (kq == key && kq != 0 && pos[q] < p)) {
          key = kq;
          p = pos[q];
          mine = q;
        }
      }
      int winner;
      lu_warp_argmax(key, p, winner);
      if (lane == winner) {
        s_key[t][warp] = key;
        s_pos[t][warp] = p;
#pragma unroll
        for (int q = 0; q < RPT; ++q)
          if (q == mine) {
#pragma unroll
            for (int j = 0; j < NB; j += 2)
              *reinterpret_cast<double2*>(&s_u[t][warp][j]) =
                  make_double2(j < NB - c ? a[q][j] : 0.0, j + 1 < NB - c ? a[q][j + 1] : 0.0);
            s_rhs[t][warp] = rhs[q];
          }
      }
      __syncthreads();
      key = lane < nw ? s_key[t][lane] : 0;
      p = lane < nw ? s_pos[t][lane] : 0x7fffffff;
      lu_warp_argmax(key, p, slot);
      if (key == 0) {  // no pivot: uniform over the CTA
        if (tid == 0) status[0] = 1;
        return;
      }
#pragma unroll
      for (int q = 0; q < RPT; ++q) {
        if (pos[q] == p)
          pos[q] = c;
        else if (pos[q] == c)
          pos[q] = p;
      }
    }
    const double* __restrict__ su = s_u[t][slot];
    const double pv = su[0], pr = s_rhs[t][slot];
#pragma unroll
    for (int q = 0; q < RPT; ++q) {
      double l = 0.0, last = a[q][0];
      const bool below = live && pos[q] > c && pos[q] < m;
      if (below && last != 0.0) {  // zeros (outside the band) would take the slow path of the division
        l = last / pv;
        rhs[q] = fma(-l, pr, rhs[q]);
      }
      if (below) last = l;
      // one-column shift with the update; finished columns meet a zero
      if (l != 0.0) {
        a[q][0] = fma(-l, su[1], a[q][1]);
#pragma unroll
        for (int j = 2; j < NB; j += 2) {
          const double2 v = *reinterpret_cast<const double2*>(su + j);
          a[q][j - 1] = fma(-l, v.x, a[q][j]);
          a[q][j] = fma(-l, v.y, a[q][j + 1]);
        }
      } else {
#pragma unroll
        for (int j = 1; j < NB; ++j) a[q][j - 1] = a[q][j];
      }
      a[q][NB - 1] = last;
    }
  }
#pragma unroll
  for (int q = 0; q < RPT; ++q) {
    const int r = tid + q * nt;
    if (r < m) {
      double2* __restrict__ row = reinterpret_cast<double2*>(A + (int64_t)(k0 + pos[q]) * n + k0);
#pragma unroll
      for (int j = 0; j < NB; j += 2)
        if (j < w) row[j / 2] = make_double2(a[q][j], a[q][j + 1]);
      b[k0 + pos[q]] = rhs[q];
      if (pos[q] < w) {
        swaps->src[pos[q]] = k0 + r;
      } else if (pos[q] != r) {  // at most one row per exchange: w of them
        const int e = atomicAdd(&s_moved, 1);
        swaps->dest[e] = k0 + pos[q];
        swaps->from[e] = k0 + r;
      }
    }
  }
  __syncthreads();
  if (tid == 0) swaps->n_moved = s_moved;
}

// Columns k1 .. cend - 1 (k1 = k0 + NB), 32 per CTA: the panel's row exchanges, U12 = L11^-1 A12
// (unit lower L11; a thread per column, its NB values in registers), and with `fused` also
// A22 -= L21 U12 for the rows k1 .. rend - 1.  512 threads.
template <int NB>
__global__ void __launch_bounds__(kLuThreads) beam_lu_trailing_kernel(int n, int k0, int rend, int cend, int fused,
                                                                      double* __restrict__ A,
                                                                      const LuSwaps* __restrict__ swaps,
                                                                      const int* __restrict__ status) {
  constexpr int kRows = 64;  // rows of A22 per pass
  constexpr int kQ = kRows / 16;
  __shared__ double sl[NB][NB + 1];
  __shared__ double sm[kRows][NB + 1];
  __shared__ double su[NB][32 + 1];
  if (status[0] != 0) return;
  const int k1 = k0 + NB, c0 = k1 + blockIdx.x * 32, tid = threadIdx.x;
  const int tx = tid & 31, ty = tid >> 5;  // ty: 0 .. 15
  const int j = c0 + tx;
  const bool on = j < cend;
  constexpr int kMovedPerThread = kLuMaxPanel / 16;
  const int nm = swaps->n_moved;
  double mv[kMovedPerThread];
#pragma unroll
  for (int q = 0; q < kMovedPerThread; ++q) {
    const int e = ty + 16 * q;
    mv[q] = (on && e < nm) ? A[(int64_t)swaps->from[e] * n + j] : 0.0;
  }
  for (int k = ty; k < NB; k += 16) su[k][tx] = on ? A[(int64_t)swaps->src[k] * n + j] : 0.0;
  for (int e = tid; e < NB * NB; e += kLuThreads) sl[e / NB][e % NB] = A[(int64_t)(k0 + e / NB) * n + k0 + e % NB];
  __syncthreads();  // every source row of these columns has been read
#pragma unroll
  for (int q = 0; q < kMovedPerThread; ++q) {
    const int e = ty + 16 * q;
    if (on && e < nm) A[(int64_t)swaps->dest[e] * n + j] = mv[q];
  }
  __syncthreads();  // the moved rows of these columns are visible
  double acc[kQ];
  auto load_pass = [&](int r0) {
    for (int e = tid; e < kRows * NB; e += kLuThreads) {
      const int r = r0 + e / NB;
      sm[e / NB][e % NB] = r < rend ? A[(int64_t)r * n + k0 + e % NB] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < kQ; ++q) {
      const int r = r0 + ty + 16 * q;
      acc[q] = (on && r < rend) ? A[(int64_t)r * n + j] : 0.0;
    }
  };
  if (fused) load_pass(k1);
  if (ty == 0) {
    double u[NB];
#pragma unroll
    for (int k = 0; k < NB; ++k) u[k] = su[k][tx];
#pragma unroll
    for (int k = 0; k < NB; ++k)
#pragma unroll
      for (int i = 0; i < NB; ++i)
        if (i > k) u[i] = fma(-sl[i][k], u[k], u[i]);
#pragma unroll
    for (int k = 0; k < NB; ++k) {
      su[k][tx] = u[k];
      if (on) A[(int64_t)(k0 + k) * n + j] = u[k];
    }
  }
  if (!fused) return;
  for (int r0 = k1; r0 < rend; r0 += kRows) {
    __syncthreads();  // su and sm complete
#pragma unroll 8
    for (int k = 0; k < NB; ++k) {
      const double uk = su[k][tx];
#pragma unroll
      for (int q = 0; q < kQ; ++q) acc[q] = fma(-sm[ty + 16 * q][k], uk, acc[q]);
    }
#pragma unroll
    for (int q = 0; q < kQ; ++q) {
      const int r = r0 + ty + 16 * q;
      if (on && r < rend) A[(int64_t)r * n + j] = acc[q];
    }
    if (r0 + kRows < rend) {
      __syncthreads();  // sm free
      load_pass(r0 + kRows);
    }
  }
}

// A22 -= L21 U12 for the rows k1 .. rend - 1 and columns k1 .. cend - 1: a 32 x 32 tile per CTA
// (32 x 8 threads, four rows each), L21 and U12 tiles staged in shared memory
template <int NB>
__global__ void __launch_bounds__(256) beam_lu_update_kernel(int n, int k0, int rend, int cend,
                                                             double* __restrict__ A, const int* __restrict__ status) {
  __shared__ double sl[32][NB + 1];
  __shared__ double su[NB][32 + 1];
  if (status[0] != 0) return;
  const int k1 = k0 + NB;
  const int r0 = k1 + blockIdx.y * 32, c0 = k1 + blockIdx.x * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int e = threadIdx.x; e < 32 * NB; e += 256) {
    const int r = e / NB, c = e % NB;
    sl[r][c] = r0 + r < rend ? A[(int64_t)(r0 + r) * n + k0 + c] : 0.0;
    const int kr = e / 32, cc = e % 32;
    su[kr][cc] = c0 + cc < cend ? A[(int64_t)(k0 + kr) * n + c0 + cc] : 0.0;
  }
  __syncthreads();
  const int j = c0 + tx;
  if (j >= cend) return;
  double acc[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int i = r0 + ty + 8 * q;
    acc[q] = i < rend ? A[(int64_t)i * n + j] : 0.0;
  }
#pragma unroll
  for (int k = 0; k < NB; ++k)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[q] = fma(-sl[ty + 8 * q][k], su[k][tx], acc[q]);
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int i = r0 + ty + 8 * q;
    if (i < rend) A[(int64_t)i * n + j] = acc[q];
  }
}

// Back substitution with the upper factor (row k ends at column k + 2 kb), in blocks of 32
// unknowns from the bottom, b in shared memory: one warp solves a block (lane i holds row i of its
// triangle), then a thread per row above subtracts the block's columns, the last first; the
// factor's values and reciprocals, which do not depend on x, are ready before the barrier.  One CTA
// of 512 threads; bound by the chain of n quotients.
__global__ void __launch_bounds__(kLuThreads) beam_lu_backsub_kernel(int n, int kb, const double* __restrict__ A,
                                                                     double* __restrict__ b,
                                                                     const int* __restrict__ status) {
  __shared__ double sb[WN_BEAM_DENSE_MAX];
  if (status[0] != 0) return;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < n; i += kLuThreads) sb[i] = b[i];
  double u[32];  // warp 0: the block's triangle; the others: a row above it
  auto load_row = [&](int i, int k0, int w, bool on) {  // n, k0 and w are even: 16-byte loads
    const double2* __restrict__ row = reinterpret_cast<const double2*>(A + (int64_t)i * n + k0);
#pragma unroll
    for (int j = 0; j < 32; j += 2) {
      const double2 v = (on && j < w) ? row[j / 2] : make_double2(0.0, 0.0);
      u[j] = v.x;
      u[j + 1] = v.y;
    }
  };
  for (int k1 = n; k1 > 0; k1 -= 32) {
    const int k0 = max(0, k1 - 32), w = k1 - k0;
    const int lo = max(0, k0 - 2 * kb);  // rows whose factors reach the block
    // warps 1 .. 15 take the rows above, 480 per pass
    int i = lo + tid - 32;
    if (warp == 0)
      load_row(k0 + min(lane, w - 1), k0, w, true);
    else
      load_row(min(i, k0), k0, w, i < k0);
    double diag = 1.0, rec = 1.0;  // the lane's diagonal entry
    if (warp == 0) {
#pragma unroll
      for (int k = 0; k < 32; ++k)
        if (lane == k && k < w) diag = u[k];
      rec = 1.0 / diag;
    }
    __syncthreads();  // sb complete
    if (warp == 0) {
      const double x0 = lane < w ? sb[k0 + lane] : 0.0;
      double x = x0;
      // x_k / u_kk as a product with the reciprocal corrected once by its residual (the correctly
      // rounded quotient wherever the reciprocal is, Markstein 1990): three operations of the chain
      // instead of a division
#pragma unroll
      for (int k = 31; k >= 0; --k) {
        const double q = x * rec;
        const double xk = __shfl_sync(0xffffffffu, fma(fma(-q, diag, x), rec, q), k);
        x = lane == k ? xk : lane < k ? fma(-u[k], xk, x) : x;
      }
      if (__any_sync(0xffffffffu, !isfinite(x))) {  // a reciprocal or product out of range: with divisions
        x = x0;
#pragma unroll 1
        for (int k = w - 1; k >= 0; --k) {
          if (lane == k) x /= diag;
          const double xk = __shfl_sync(0xffffffffu, x, k);
          if (lane < k) x = fma(-A[(int64_t)(k0 + lane) * n + k0 + k], xk, x);
        }
      }
      if (lane < w) sb[k0 + lane] = x;
    }
    __syncthreads();  // the block's unknowns are final
    if (warp != 0)
      for (; i < k0; i += kLuThreads - 32) {
        if (i >= lo + kLuThreads - 32) load_row(i, k0, w, true);
        double x = sb[i];
#pragma unroll
        for (int k = 31; k >= 0; --k)
          if (k < w) x = fma(-u[k], sb[k0 + k], x);
        sb[i] = x;
      }
  }
  __syncthreads();
  for (int i = tid; i < n; i += kLuThreads) b[i] = sb[i];
}

}  // namespace wn

// ---------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------
namespace wn {

struct Beam {
  int device = 0;
  int64_t n_nodes = 0, n_el = 0, nnzb = 0;
  std::vector<int32_t> h_rp, h_ci;
  DArray<double> nodes, props, eref, L0;
  DArray<int32_t> el, rp, ci, block_row, diag_block, gptr, gsrc, inc_ea;
  DArray<int64_t> inc_ptr;
  DArray<uint8_t> fixed;
  DArray<double> fe, ke, K, dinv;
  // BiCGStab workspace
  DArray<double> r, rh, p, v, s, t, y, z, x, part;
  // dense LU workspace (small frames) and the matrix's half bandwidth in DOFs
  DArray<double> dense;
  DArray<int> dstat;
  DArray<LuSwaps> dswaps;
  int half_band = 0;
  bool assembled = false;
};

static int build_beam_pattern(int64_t n_nodes, int64_t n_el, const int32_t* el, Beam& b, std::vector<int32_t>& rp,
                              std::vector<int32_t>& ci, std::vector<int32_t>& brow, std::vector<int32_t>& diag,
                              std::vector<int32_t>& gptr, std::vector<int32_t>& gsrc, std::vector<int64_t>& iptr,
                              std::vector<int32_t>& iea) {
  for (int64_t k = 0; k < n_el * 2; ++k)
    WN_REQUIRE(el[k] >= 0 && el[k] < n_nodes, WN_EMESH, "beam: element node index out of range");
  iptr.assign(n_nodes + 1, 0);
  for (int64_t k = 0; k < n_el * 2; ++k) iptr[el[k] + 1]++;
  for (int64_t i = 0; i < n_nodes; ++i) iptr[i + 1] += iptr[i];
  iea.resize(n_el * 2);
  {
    std::vector<int64_t> pos(iptr.begin(), iptr.end() - 1);
    for (int64_t e = 0; e < n_el; ++e)
      for (int a = 0; a < 2; ++a) iea[pos[el[e * 2 + a]]++] = (int32_t)(e * 2 + a);
  }
  rp.assign(n_nodes + 1, 0);
  std::vector<std::vector<int32_t>> rows(n_nodes);
  for (int64_t i = 0; i < n_nodes; ++i) {
    auto& r = rows[i];
    r.push_back((int32_t)i);  // every node keeps a diagonal block
    for (int64_t q = iptr[i]; q < iptr[i + 1]; ++q) {
      const int32_t e = iea[q] / 2;
      r.push_back(el[e * 2]);
      r.push_back(el[e * 2 + 1]);
    }
    std::sort(r.begin(), r.end());
    r.erase(std::unique(r.begin(), r.end()), r.end());
    rp[i + 1] = rp[i] + (int32_t)r.size();
  }
  const int64_t nnzb = rp[n_nodes];
  ci.resize(nnzb);
  brow.resize(nnzb);
  diag.resize(n_nodes);
  for (int64_t i = 0; i < n_nodes; ++i)
    for (size_t k = 0; k < rows[i].size(); ++k) {
      ci[rp[i] + k] = rows[i][k];
      brow[rp[i] + k] = (int32_t)i;
      if (rows[i][k] == i) diag[i] = rp[i] + (int32_t)k;
    }
  // gather lists in (element, a, b) order
  auto find = [&](int32_t r, int32_t c) {
    return (int32_t)(std::lower_bound(ci.begin() + rp[r], ci.begin() + rp[r + 1], c) - ci.begin());
  };
  std::vector<int32_t> emap(n_el * 4);
  gptr.assign(nnzb + 1, 0);
  for (int64_t e = 0; e < n_el; ++e)
    for (int a = 0; a < 2; ++a)
      for (int c = 0; c < 2; ++c) {
        const int32_t blk = find(el[e * 2 + a], el[e * 2 + c]);
        emap[e * 4 + a * 2 + c] = blk;
        gptr[blk + 1]++;
      }
  for (int64_t k = 0; k < nnzb; ++k) gptr[k + 1] += gptr[k];
  gsrc.resize(n_el * 4);
  std::vector<int32_t> pos(gptr.begin(), gptr.end() - 1);
  for (int64_t e = 0; e < n_el; ++e)
    for (int q = 0; q < 4; ++q) gsrc[pos[emap[e * 4 + q]]++] = (int32_t)(e * 4 + q);
  b.nnzb = nnzb;
  return 0;
}

static Beam* as_beam(void* h) { return reinterpret_cast<Beam*>(h); }

static int beam_dots(Beam* b, const double* a0, const double* b0, const double* a1, const double* b1, double* out2,
                     cudaStream_t st) {
  const int64_t n = b->n_nodes * 6;
  const int g = (int)std::min<int64_t>(256, (n + 255) / 256);
  beam_dot2_kernel<<<g, 256, 0, st>>>(n, a0, b0, a1, b1, b->part.p);
  WN_CUDA(cudaGetLastError());
  std::vector<double> h(2 * g);
  WN_CUDA(cudaMemcpyAsync(h.data(), b->part.p, sizeof(double) * 2 * g, cudaMemcpyDeviceToHost, st));
  WN_CUDA(cudaStreamSynchronize(st));
  out2[0] = out2[1] = 0.0;
  for (int k = 0; k < g; ++k) {  // fixed order
    out2[0] += h[2 * k];
    out2[1] += h[2 * k + 1];
  }
  return 0;
}

}  // namespace wn

using namespace wn;

extern "C" {

int wn_beam_internal_forces(const double* nodes, const int32_t* elements, const double* props, const double* e_ref,
                            const double* L0_arr, const double* U, double* F_int, int n_elements, int n_nodes) {
  WN_REQUIRE(nodes && U && F_int && n_nodes > 0 && n_elements >= 0, WN_EINVAL, "wn_beam_internal_forces: bad argument");
  if (n_elements == 0) return 0;
  WN_REQUIRE(elements && props && e_ref && L0_arr, WN_EINVAL, "wn_beam_internal_forces: null argument");
  void* h = nullptr;
  WN_CHECK(wn_beam_create(n_nodes, n_elements, nodes, elements, props, e_ref, L0_arr, &h));
  Beam* b = as_beam(h);
  int rc = 0;
  DArray<double> dU, dF;
  rc = rc ? rc : dU.upload(U, (int64_t)n_nodes * 6);
  rc = rc ? rc : dF.upload(F_int, (int64_t)n_nodes * 6);
  if (rc == 0) {
    const int64_t ne = b->n_el;
    beam_force_kernel<<<grid_for(ne, 1, 128, 8), 128>>>(ne, b->nodes.p, b->el.p, b->props.p, b->eref.p, b->L0.p, dU.p,
                                                       b->fe.p);
    beam_node_gather_kernel<<<grid_for(n_nodes * 6, 1, 256, 8), 256>>>(n_nodes, b->inc_ptr.p, b->inc_ea.p, b->fe.p, 1,
                                                                       dF.p);
    cudaError_t e = cudaMemcpy(F_int, dF.p, dF.bytes(), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) {
      set_error("wn_beam_internal_forces: %s", cudaGetErrorString(e));
      rc = (int)e;
    }
  }
  wn_beam_destroy(h);
  return rc;
}

int wn_beam_create(int64_t n_nodes, int64_t n_el, const double* nodes, const int32_t* elements, const double* props,
                   const double* e_ref, const double* L0, void** out) {
  WN_REQUIRE(out && nodes && n_nodes > 0 && n_el >= 0 && (n_el == 0 || (elements && props && e_ref && L0)),
             WN_EINVAL, "wn_beam_create: bad argument");
  *out = nullptr;
  auto* b = new Beam();
  WN_CUDA(cudaGetDevice(&b->device));
  b->n_nodes = n_nodes;
  b->n_el = n_el;
  std::vector<int32_t> brow, diag, gptr, gsrc, iea;
  std::vector<int64_t> iptr;
  int rc = build_beam_pattern(n_nodes, n_el, elements, *b, b->h_rp, b->h_ci, brow, diag, gptr, gsrc, iptr, iea);
  const int64_t n = n_nodes * 6;
  int64_t apart = 0;  // nodes, between the ends of a beam
  if (rc == 0)
    for (int64_t e = 0; e < n_el; ++e) apart = std::max<int64_t>(apart, std::abs(elements[2 * e] - elements[2 * e + 1]));
  b->half_band = (int)std::min<int64_t>(6 * apart + 5, WN_BEAM_DENSE_MAX);
  rc = rc ? rc : b->nodes.upload(nodes, n_nodes * 3);
  rc = rc ? rc : b->el.upload(elements, n_el * 2);
  rc = rc ? rc : b->props.upload(props, n_el * 6);
  rc = rc ? rc : b->eref.upload(e_ref, n_el * 9);
  rc = rc ? rc : b->L0.upload(L0, n_el);
  rc = rc ? rc : b->rp.upload(b->h_rp);
  rc = rc ? rc : b->ci.upload(b->h_ci);
  rc = rc ? rc : b->block_row.upload(brow);
  rc = rc ? rc : b->diag_block.upload(diag);
  rc = rc ? rc : b->gptr.upload(gptr);
  rc = rc ? rc : b->gsrc.upload(gsrc);
  rc = rc ? rc : b->inc_ptr.upload(iptr);
  rc = rc ? rc : b->inc_ea.upload(iea);
  rc = rc ? rc : b->fixed.alloc(n);
  rc = rc ? rc : b->fixed.zero();
  rc = rc ? rc : b->fe.alloc(std::max<int64_t>(n_el, 1) * 12);
  rc = rc ? rc : b->ke.alloc(std::max<int64_t>(n_el, 1) * 144);
  rc = rc ? rc : b->K.alloc(b->nnzb * 36);
  rc = rc ? rc : b->dinv.alloc(n_nodes * 36);
  for (DArray<double>* v : {&b->r, &b->rh, &b->p, &b->v, &b->s, &b->t, &b->y, &b->z, &b->x})
    rc = rc ? rc : v->alloc(n);
  rc = rc ? rc : b->part.alloc(512);
  if (rc == 0) {
    cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) {
      set_error("wn_beam_create: %s", cudaGetErrorString(e));
      rc = (int)e;
    }
  }
  if (rc != 0) {
    delete b;
    return rc;
  }
  *out = b;
  return 0;
}

int wn_beam_destroy(void* h) {
  if (h) {
    cudaSetDevice(as_beam(h)->device);
    delete as_beam(h);
  }
  return 0;
}

int wn_beam_info(void* h, int64_t* n_nodes, int64_t* n_el, int64_t* nnzb) {
  WN_REQUIRE(h, WN_EINVAL, "wn_beam_info: null handle");
  Beam* b = as_beam(h);
  if (n_nodes) *n_nodes = b->n_nodes;
  if (n_el) *n_el = b->n_el;
  if (nnzb) *nnzb = b->nnzb;
  return 0;
}

int wn_beam_get_pattern(void* h, int32_t* row_ptr, int32_t* col_idx) {
  WN_REQUIRE(h, WN_EINVAL, "wn_beam_get_pattern: null handle");
  Beam* b = as_beam(h);
  if (row_ptr) memcpy(row_ptr, b->h_rp.data(), sizeof(int32_t) * b->h_rp.size());
  if (col_idx) memcpy(col_idx, b->h_ci.data(), sizeof(int32_t) * b->h_ci.size());
  return 0;
}

int wn_beam_set_fixed(void* h, const uint8_t* fixed_mask) {
  WN_REQUIRE(h, WN_EINVAL, "wn_beam_set_fixed: null handle");
  Beam* b = as_beam(h);
  WN_CUDA(cudaSetDevice(b->device));
  if (fixed_mask)
    WN_CUDA(cudaMemcpy(b->fixed.p, fixed_mask, b->n_nodes * 6, cudaMemcpyHostToDevice));
  else
    WN_CHECK(b->fixed.zero());
  return 0;
}

int wn_beam_evaluate_device(void* h, const double* d_U, double* d_fint, int assemble_tangent, int apply_bcs,
                            uintptr_t stream) {
  WN_REQUIRE(h && d_U, WN_EINVAL, "wn_beam_evaluate_device: null argument");
  Beam* b = as_beam(h);
  WN_CUDA(cudaSetDevice(b->device));
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t ne = b->n_el;
  if (d_fint) {
    if (ne) {
      beam_force_kernel<<<grid_for(ne, 1, 128, 8), 128, 0, st>>>(ne, b->nodes.p, b->el.p, b->props.p, b->eref.p,
                                                                b->L0.p, d_U, b->fe.p);
      WN_CUDA(cudaGetLastError());
    } else {
      WN_CHECK(b->fe.zero(st));
    }
    beam_node_gather_kernel<<<grid_for(b->n_nodes * 6, 1, 256, 8), 256, 0, st>>>(b->n_nodes, b->inc_ptr.p,
                                                                                 b->inc_ea.p, b->fe.p, 0, d_fint);
    WN_CUDA(cudaGetLastError());
  }
  if (assemble_tangent) {
    if (ne) {
      beam_tangent_kernel<<<grid_for(ne * 12, 1, 128, 8), 128, 0, st>>>(ne, b->nodes.p, b->el.p, b->props.p,
                                                                        b->eref.p, b->L0.p, d_U, b->ke.p);
      WN_CUDA(cudaGetLastError());
    }
    beam_gather_kernel<<<grid_for(b->nnzb * 36, 1, 256, 8), 256, 0, st>>>(
        b->nnzb, b->gptr.p, b->gsrc.p, b->ke.p, b->block_row.p, b->ci.p, apply_bcs ? b->fixed.p : nullptr, b->K.p);
    beam_block_inverse_kernel<<<grid_for(b->n_nodes, 1, 128, 8), 128, 0, st>>>(b->n_nodes, b->diag_block.p, b->K.p,
                                                                               b->dinv.p);
    WN_CUDA(cudaGetLastError());
    b->assembled = true;
  }
  return 0;
}

int wn_beam_evaluate(void* h, const double* U, double* fint, int assemble_tangent, int apply_bcs) {
  WN_REQUIRE(h && U, WN_EINVAL, "wn_beam_evaluate: null argument");
  Beam* b = as_beam(h);
  WN_CUDA(cudaSetDevice(b->device));
  const int64_t n = b->n_nodes * 6;
  DArray<double> dU, dF;
  WN_CHECK(dU.upload(U, n));
  if (fint) WN_CHECK(dF.alloc(n));
  WN_CHECK(wn_beam_evaluate_device(h, dU.p, fint ? dF.p : nullptr, assemble_tangent, apply_bcs, 0));
  if (fint) WN_CUDA(cudaMemcpy(fint, dF.p, n * sizeof(double), cudaMemcpyDeviceToHost));
  WN_CUDA(cudaDeviceSynchronize());
  return 0;
}

int wn_beam_get_tangent(void* h, double* values) {
  WN_REQUIRE(h && values, WN_EINVAL, "wn_beam_get_tangent: null argument");
  Beam* b = as_beam(h);
  WN_REQUIRE(b->assembled, WN_ESTATE, "wn_beam_get_tangent: no tangent assembled");
  WN_CUDA(cudaMemcpy(values, b->K.p, b->K.bytes(), cudaMemcpyDeviceToHost));
  return 0;
}

int wn_beam_linear_system(void* h, void** out) {
  WN_REQUIRE(h && out, WN_EINVAL, "wn_beam_linear_system: null argument");
  Beam* b = as_beam(h);
  WN_REQUIRE(b->assembled, WN_ESTATE, "wn_beam_linear_system: assemble the tangent first");
  WN_CUDA(cudaSetDevice(b->device));
  std::vector<double> coords(b->n_nodes * 3);
  std::vector<uint8_t> fixed(b->n_nodes * 6);
  WN_CUDA(cudaMemcpy(coords.data(), b->nodes.p, coords.size() * sizeof(double), cudaMemcpyDeviceToHost));
  WN_CUDA(cudaMemcpy(fixed.data(), b->fixed.p, fixed.size(), cudaMemcpyDeviceToHost));
  bool any = false;
  for (uint8_t f : fixed) any = any || f;
  return make_bsr6_system(b->n_nodes, b->h_rp.data(), b->h_ci.data(), b->K.p, true, coords.data(),
                          any ? fixed.data() : nullptr, out);
}

}  // extern "C"

// one panel of dense_lu of NB columns, rows in registers (RPT per thread)
template <int NB, int RPT>
static void lu_panel(Beam* b, double* d_x, int n, int k0, int rend, int cend, cudaStream_t st) {
  const int m = rend - k0, k1 = std::min(n, k0 + NB);
  const int threads = std::min(kLuThreads, std::max(64, ((m + RPT - 1) / RPT + 31) / 32 * 32));
  beam_lu_panel_kernel<NB, RPT><<<1, threads, 0, st>>>(n, k0, rend, b->dense.p, d_x, b->dswaps.p, b->dstat.p);
  if (cend <= k1) return;
  const int strips = (cend - k1 + 31) / 32, rows = rend - k1;
  const int fused = rows <= kLuFuseRows;
  beam_lu_trailing_kernel<NB><<<strips, kLuThreads, 0, st>>>(n, k0, rend, cend, fused, b->dense.p, b->dswaps.p,
                                                             b->dstat.p);
  if (!fused)
    beam_lu_update_kernel<NB><<<dim3((unsigned)strips, (unsigned)((rows + 31) / 32)), 256, 0, st>>>(
        n, k0, rend, cend, b->dense.p, b->dstat.p);
}

// LU of the dense copy and the solve (d_x: right-hand side in, solution out).  The widest panel
// whose rows fit the registers of one CTA: 32 columns up to 512 rows (64 registers a thread hold
// one row), then 16 columns x 2 rows, 8 x 4 and 8 x 6 (3,072 rows, WN_BEAM_DENSE_MAX); the band
// decides, not n.
static int dense_lu(Beam* b, double* d_x, int n, cudaStream_t st) {
  const int kb = std::min(n - 1, b->half_band);
  const int64_t tall = std::min<int64_t>(n, (int64_t)kb + kLuMaxPanel);
  const int nb = tall <= kLuThreads ? 32 : tall <= 2 * kLuThreads ? 16 : 8;
  for (int k0 = 0; k0 < n; k0 += nb) {
    const int k1 = std::min(n, k0 + nb), rend = std::min(n, k1 + kb), cend = std::min(n, k1 + 2 * kb);
    if (nb == 32)
      lu_panel<32, 1>(b, d_x, n, k0, rend, cend, st);
    else if (nb == 16)
      lu_panel<16, 2>(b, d_x, n, k0, rend, cend, st);
    else if (tall <= 4 * kLuThreads)
      lu_panel<8, 4>(b, d_x, n, k0, rend, cend, st);
    else
      lu_panel<8, 6>(b, d_x, n, k0, rend, cend, st);
  }
  beam_lu_backsub_kernel<<<1, kLuThreads, 0, st>>>(n, kb, b->dense.p, d_x, b->dstat.p);
  WN_CUDA(cudaGetLastError());
  return 0;
}

extern "C" {

int wn_beam_solve_device(void* h, const double* d_b, double* d_x, int method, double rtol, int max_iter, int* iters,
                         double* rel_res, uintptr_t stream) {
  WN_REQUIRE(h && d_b && d_x && rtol > 0 && max_iter > 0 && method >= 0 && method <= 2, WN_EINVAL,
             "wn_beam_solve_device: bad argument");
  Beam* b = as_beam(h);
  WN_REQUIRE(b->assembled, WN_ESTATE, "wn_beam_solve_device: assemble the tangent first");
  WN_CUDA(cudaSetDevice(b->device));
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t n = b->n_nodes * 6;
  if (method == 1 || (method == 0 && n <= WN_BEAM_DENSE_MAX)) {
    WN_REQUIRE(n <= WN_BEAM_DENSE_MAX, WN_ETOOBIG, "wn_beam_solve_device: dense LU limited to %d DOFs",
               WN_BEAM_DENSE_MAX);
    WN_CHECK(b->dense.alloc(n * n));
    WN_CHECK(b->dstat.alloc(1));
    WN_CHECK(b->dswaps.alloc(1));
    WN_CUDA(cudaMemsetAsync(b->dense.p, 0, n * n * sizeof(double), st));
    WN_CUDA(cudaMemsetAsync(b->dstat.p, 0, sizeof(int), st));
    beam_dense_kernel<<<grid_for(n, 1, 256, 8), 256, 0, st>>>(b->n_nodes, b->rp.p, b->ci.p, b->K.p, b->dense.p);
    WN_CUDA(cudaMemcpyAsync(d_x, d_b, n * sizeof(double), cudaMemcpyDeviceToDevice, st));
    WN_CHECK(dense_lu(b, d_x, (int)n, st));
    WN_CUDA(cudaGetLastError());
    int stat = 0;
    WN_CUDA(cudaMemcpyAsync(&stat, b->dstat.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    WN_CUDA(cudaStreamSynchronize(st));
    if (iters) *iters = 1;
    // residual of the direct solve, on the (unfactored) BSR matrix
    WN_CHECK(launch_bsr_spmv_f64(6, 6, b->n_nodes, b->rp.p, b->ci.p, b->K.p, d_x, b->t.p, 1.0, 0.0, st));
    beam_lincomb_kernel<<<grid_for(n, 1, 256, 8), 256, 0, st>>>(n, 1.0, d_b, -1.0, b->t.p, 0.0, nullptr);
    WN_CUDA(cudaGetLastError());
    double d2[2];
    WN_CHECK(beam_dots(b, b->t.p, b->t.p, d_b, d_b, d2, st));
    if (rel_res) *rel_res = d2[1] > 0.0 ? std::sqrt(d2[0] / d2[1]) : 0.0;
    if (stat != 0) set_error("wn_beam_solve_device: singular tangent (zero pivot)");
    return stat == 0 ? 0 : WN_EBREAKDOWN;
  }
  const int gv = grid_for(n, 1, 256, 8);
  auto spmv = [&](const double* x, double* y) {
    return launch_bsr_spmv_f64(6, 6, b->n_nodes, b->rp.p, b->ci.p, b->K.p, x, y, 1.0, 0.0, st);
  };
  auto prec = [&](const double* x, double* y) {
    beam_block_apply_kernel<<<gv, 256, 0, st>>>(b->n_nodes, b->dinv.p, x, y);
    WN_CUDA(cudaGetLastError());
    return 0;
  };
  auto lin = [&](double a, const double* x, double bb, double* y, double c, const double* z) {
    beam_lincomb_kernel<<<gv, 256, 0, st>>>(n, a, x, bb, y, c, z);
    WN_CUDA(cudaGetLastError());
    return 0;
  };
  // preconditioned BiCGStab (van der Vorst 1992), x0 = 0
  double d2[2];
  WN_CUDA(cudaMemsetAsync(b->x.p, 0, n * sizeof(double), st));
  WN_CUDA(cudaMemcpyAsync(b->r.p, d_b, n * sizeof(double), cudaMemcpyDeviceToDevice, st));
  WN_CUDA(cudaMemcpyAsync(b->rh.p, d_b, n * sizeof(double), cudaMemcpyDeviceToDevice, st));
  WN_CUDA(cudaMemsetAsync(b->p.p, 0, n * sizeof(double), st));
  WN_CUDA(cudaMemsetAsync(b->v.p, 0, n * sizeof(double), st));
  WN_CHECK(beam_dots(b, d_b, d_b, nullptr, nullptr, d2, st));
  const double bnorm = std::sqrt(d2[0]);
  double rho = 1.0, alpha = 1.0, omega = 1.0, rn = bnorm;
  int it = 0, status = 0;
  if (bnorm == 0.0 || !std::isfinite(bnorm)) {
    status = std::isfinite(bnorm) ? 0 : WN_EBREAKDOWN;
  } else {
    for (it = 0; it < max_iter; ++it) {
      WN_CHECK(beam_dots(b, b->rh.p, b->r.p, nullptr, nullptr, d2, st));
      const double rho_new = d2[0];
      if (rho_new == 0.0 || !std::isfinite(rho_new)) {
        status = WN_EBREAKDOWN;
        break;
      }
      const double beta = (rho_new / rho) * (alpha / omega);
      rho = rho_new;
      WN_CHECK(lin(-omega * beta, b->v.p, beta, b->p.p, 1.0, b->r.p));  // p = r + beta (p - omega v)
      WN_CHECK(prec(b->p.p, b->y.p));
      WN_CHECK(spmv(b->y.p, b->v.p));
      WN_CHECK(beam_dots(b, b->rh.p, b->v.p, nullptr, nullptr, d2, st));
      alpha = rho / d2[0];
      WN_CHECK(lin(1.0, b->r.p, 0.0, b->s.p, -alpha, b->v.p));  // s = r - alpha v
      WN_CHECK(lin(alpha, b->y.p, 1.0, b->x.p, 0.0, nullptr));  // x += alpha y
      WN_CHECK(beam_dots(b, b->s.p, b->s.p, nullptr, nullptr, d2, st));
      if (std::sqrt(d2[0]) <= rtol * bnorm) {
        rn = std::sqrt(d2[0]);
        ++it;
        break;
      }
      WN_CHECK(prec(b->s.p, b->z.p));
      WN_CHECK(spmv(b->z.p, b->t.p));
      WN_CHECK(beam_dots(b, b->t.p, b->s.p, b->t.p, b->t.p, d2, st));
      omega = d2[1] > 0.0 ? d2[0] / d2[1] : 0.0;
      WN_CHECK(lin(omega, b->z.p, 1.0, b->x.p, 0.0, nullptr));         // x += omega z
      WN_CHECK(lin(1.0, b->s.p, 0.0, b->r.p, -omega, b->t.p));         // r = s - omega t
      WN_CHECK(beam_dots(b, b->r.p, b->r.p, nullptr, nullptr, d2, st));
      rn = std::sqrt(d2[0]);
      if (!std::isfinite(rn)) {
        status = WN_EBREAKDOWN;
        break;
      }
      if (rn <= rtol * bnorm) {
        ++it;
        break;
      }
      if (omega == 0.0) {
        status = WN_EBREAKDOWN;
        break;
      }
    }
    if (status == 0 && rn > rtol * bnorm) status = WN_ENOCONV;
  }
  WN_CUDA(cudaMemcpyAsync(d_x, b->x.p, n * sizeof(double), cudaMemcpyDeviceToDevice, st));
  WN_CUDA(cudaStreamSynchronize(st));
  if (iters) *iters = it;
  if (rel_res) *rel_res = bnorm > 0.0 ? rn / bnorm : 0.0;
  return status;
}

int wn_beam_solve(void* h, const double* rhs, double* x, int method, double rtol, int max_iter, int* iters,
                  double* rel_res) {
  WN_REQUIRE(h && rhs && x, WN_EINVAL, "wn_beam_solve: null argument");
  Beam* b = as_beam(h);
  WN_CUDA(cudaSetDevice(b->device));
  const int64_t n = b->n_nodes * 6;
  DArray<double> db, dx;
  WN_CHECK(db.upload(rhs, n));
  WN_CHECK(dx.alloc(n));
  const int rc = wn_beam_solve_device(h, db.p, dx.p, method, rtol, max_iter, iters, rel_res, 0);
  WN_CUDA(cudaMemcpy(x, dx.p, n * sizeof(double), cudaMemcpyDeviceToHost));
  return rc;
}

}  // extern "C"
