// Multi-right-hand-side PCG: kBatch load cases against one matrix and one AMG hierarchy.  Included
// once per batch width (block_w8.cu, block_w16.cu, block_w32.cu, each defining WN_BATCH).
//
// The reference solves load cases one at a time (each a solve_c3d10_pcg call,
// wnfea/solver/solid_solver.py:197-308); here the batch shares every matrix read.  Each
// load case keeps its own Krylov recurrence -- its own alpha, beta, convergence test and
// iteration count -- so every column reproduces the single-RHS PCG; only the products are
// batched:
//   * block rows are handled by groups of 8 lanes, a lane owning kBatch / 8 load cases (vector
//     loads of the DOF-major n x kBatch vectors), 4 rows per warp;
//   * per-case FP64 dot products are two-stage and deterministic (per-CTA partials of all
//     cases, reduced in a fixed order by a one-CTA scalar kernel);
//   * finished cases take alpha = beta = 0 and stop changing while the rest iterate;
//   * the batched V-cycle mirrors the single-RHS one (Chebyshev smoothing, restriction,
//     prolongation, dense coarsest inverse) in FP32 (mixed) or FP64;
//   * an FP64 refinement loop checks every case on its true residual F - K U and restarts
//     only the cases that are not yet at rtol.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <type_traits>

#include "amg.h"
#include "block.h"
#include "common.cuh"
#include "eft.cuh"
#include "solid.h"
#include "spmv.cuh"
#include "solver.h"

namespace wn {
namespace {

constexpr int kBatch = WN_BATCH;
constexpr int kC = kBatch / 8;  // load cases per lane
using BlockScalars = BlockScalarsT<kBatch>;
using BlockWork = BlockWorkT<kBatch>;
static_assert(kC == 1 || kC == 2 || kC == 4, "batches of 8, 16 or 32 load cases");

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kRowsPerWarp = 4;  // 8 lanes per block row

// Grids of the row and vector kernels: fixed, so that the partial sums of a load case run over the
// same rows in the same order in a batch of any width (its solution does not depend on the batch
// it is solved in), and one resident wave, so that the CTAs sweep the mesh together (row kernels:
// CTAs per SM by block size and type, which are also their launch bounds).
template <typename T, int NB>
constexpr int kRowCtas = sizeof(T) == 4 && NB == 9 ? 3 : 2;
constexpr int kDofGrid = kNumSMs * 8;
inline int part_grid(int64_t work_ctas, int most) {
  return (int)std::max<int64_t>(1, std::min<int64_t>(work_ctas, most));
}
template <typename T, int NB>
inline int row_grid(int64_t work_ctas) {
  return part_grid(work_ctas, kNumSMs * kRowCtas<T, NB>);
}

// ---------------------------------------------------------------------------------------
// case ownership and 4-case vectors
// ---------------------------------------------------------------------------------------
// Lane l (0..7) of an 8-lane group owns kC = kBatch / 8 of the load cases of a DOF row.  The map is
// chosen per kernel by the type M of its widest vectors so that every vector load is one
// coalesced access of up to 16 bytes per lane:
//   kC = 4, M = float : cases 4l .. 4l+3             (one float4 of a float row)
//   kC = 4, M = double: cases 2l, 2l+1, 16+2l, 17+2l (two double2 of a double row, each contiguous
//                                                     over the 8 lanes)
//   kC = 2            : cases 2l, 2l+1
//   kC = 1            : case l
template <typename T>
struct C4 {
  T v[kC];
};
template <typename M>
__device__ __forceinline__ int case_of(int l, int k) {
  if constexpr (kC < 4 || sizeof(M) == 4)
    return kC * l + k;
  else
    return (k < 2) ? 2 * l + k : 16 + 2 * l + (k - 2);
}
// two consecutive cases
__device__ __forceinline__ void ld2(const float* p, float* o) {
  const float2 a = *reinterpret_cast<const float2*>(p);
  o[0] = a.x;
  o[1] = a.y;
}
__device__ __forceinline__ void ld2(const double* p, double* o) {
  const double2 a = *reinterpret_cast<const double2*>(p);
  o[0] = a.x;
  o[1] = a.y;
}
__device__ __forceinline__ void st2(float* p, float a, float b) { *reinterpret_cast<float2*>(p) = make_float2(a, b); }
__device__ __forceinline__ void st2(double* p, double a, double b) {
  *reinterpret_cast<double2*>(p) = make_double2(a, b);
}
template <typename M, typename T>
__device__ __forceinline__ C4<T> ldc(const T* __restrict__ row, int l) {
  C4<T> o;
  if constexpr (kC == 1) {
    o.v[0] = row[l];
  } else if constexpr (kC == 2) {
    ld2(row + 2 * l, o.v);
  } else if constexpr (sizeof(M) == 4 && sizeof(T) == 4) {
    const float4 a = *reinterpret_cast<const float4*>(row + 4 * l);
    o.v[0] = a.x;
    o.v[1] = a.y;
    o.v[2] = a.z;
    o.v[3] = a.w;
  } else if constexpr (sizeof(M) == 4) {
    ld2(row + 4 * l, o.v);
    ld2(row + 4 * l + 2, o.v + 2);
  } else {
    ld2(row + 2 * l, o.v);
    ld2(row + 16 + 2 * l, o.v + 2);
  }
  return o;
}
template <typename M, typename T>
__device__ __forceinline__ void stc(T* row, int l, const C4<T>& v) {
  if constexpr (kC == 1) {
    row[l] = v.v[0];
  } else if constexpr (kC == 2) {
    st2(row + 2 * l, v.v[0], v.v[1]);
  } else if constexpr (sizeof(M) == 4 && sizeof(T) == 4) {
    *reinterpret_cast<float4*>(row + 4 * l) = make_float4(v.v[0], v.v[1], v.v[2], v.v[3]);
  } else if constexpr (sizeof(M) == 4) {
    st2(row + 4 * l, v.v[0], v.v[1]);
    st2(row + 4 * l + 2, v.v[2], v.v[3]);
  } else {
    st2(row + 2 * l, v.v[0], v.v[1]);
    st2(row + 16 + 2 * l, v.v[2], v.v[3]);
  }
}
template <typename TO, typename TI>
__device__ __forceinline__ C4<TO> cvt4(const C4<TI>& a) {
  C4<TO> o;
#pragma unroll
  for (int k = 0; k < kC; ++k) o.v[k] = (TO)a.v[k];
  return o;
}

// ---------------------------------------------------------------------------------------
// loops and per-case reductions
// ---------------------------------------------------------------------------------------
// Defines l (lane in the 8-lane group), `row` (the block row of this group's team) and loops over
// the rows, 4 / S per warp with a team of S groups (S = 1 or 4) per row; `lead` is true in the
// team's first group, which alone runs the epilogue.  `order` (or null): the row at each position,
// n_rows where there is none (BlockSet::order, made for S = 1 and the kernel's grid).  The loop
// bound is warp-uniform so that all 32 lanes reach the row product's shuffles; a body may
// `continue` once the product is done.
#define BATCH_TEAM_LOOP(n_rows, S, order)                                                     \
  const int l = threadIdx.x & 7;                                                              \
  const bool lead = (((threadIdx.x & 31) >> 3) % (S)) == 0;                                   \
  constexpr int kPass = kWarps * (kRowsPerWarp / (S)); /* rows per pass of a CTA */           \
  for (int64_t pass = blockIdx.x, row = 0;                                                    \
       pass * kPass < (n_rows) && (row = batch_row<S>(pass, n_rows, order), true); pass += gridDim.x)
#define BATCH_ROW_LOOP(n_rows, order) BATCH_TEAM_LOOP(n_rows, 1, order)

template <int S>
__device__ __forceinline__ int64_t batch_row(int64_t pass, int64_t n_rows, const int32_t* __restrict__ order) {
  constexpr int kPerWarp = kRowsPerWarp / S;
  const int64_t pos = (pass * kWarps + (threadIdx.x >> 5)) * kPerWarp + ((threadIdx.x & 31) >> 3) / S;
  return order ? (int64_t)__ldg(order + pos) : min(pos, n_rows);
}

// Loop over the DOF rows i of n x kBatch vectors, 8 lanes per row; defines l.  The grid
// stride is a multiple of 8 lanes, so a thread always owns the same cases.
#define BATCH_DOF_LOOP(n)                                                                      \
  const int l = threadIdx.x & 7;                                                               \
  for (int64_t t_ = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, i = t_ >> 3; t_ < (n) * 8; \
       t_ += (int64_t)gridDim.x * blockDim.x, i = t_ >> 3)

// CTA partials of the four per-lane case sums d[0..3] (cases case_of<M>(l, k)) into
// part[blockIdx.x * kBatch + case], in a fixed order.  All threads of the CTA call it.
template <typename M>
__device__ __forceinline__ void write_case_parts(double (&d)[kC], double* __restrict__ part) {
  __shared__ double sh[kThreads / 32][kBatch];
#pragma unroll
  for (int k = 0; k < kC; ++k) {
    d[k] += __shfl_xor_sync(0xffffffffu, d[k], 8);
    d[k] += __shfl_xor_sync(0xffffffffu, d[k], 16);
  }
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane < 8)
#pragma unroll
    for (int k = 0; k < kC; ++k) sh[w][case_of<M>(lane, k)] = d[k];
  __syncthreads();
  if (threadIdx.x < kBatch) {
    double s = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); ++k) s += sh[k][threadIdx.x];
    part[(int64_t)blockIdx.x * kBatch + threadIdx.x] = s;
  }
}

// one-CTA fixed-order sums of nparts x kBatch partials; thread j < kBatch receives case j.  The
// 300 to 1,200 partials of a case are a chain of L2 loads per warp: 32 warps, 8 loads in flight.
constexpr int kScalarThreads = 1024;
__device__ __forceinline__ double reduce_case_parts(const double* __restrict__ part, int nparts) {
  __shared__ double sh[kScalarThreads];
  const int c = threadIdx.x & 31, sub = threadIdx.x >> 5, nsub = blockDim.x >> 5;
  double s = 0.0;
  if (c < kBatch) {
#pragma unroll 8
    for (int k = sub; k < nparts; k += nsub) s += part[(int64_t)k * kBatch + c];
  }
  sh[threadIdx.x] = s;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x < kBatch)
    for (int k = 0; k < nsub; ++k) t += sh[k * 32 + threadIdx.x];
  __syncthreads();
  return t;
}

template <typename M>
__device__ __forceinline__ C4<double> case_scalars(const double* __restrict__ v, int l) {
  C4<double> o;
#pragma unroll
  for (int k = 0; k < kC; ++k) o.v[k] = v[case_of<M>(l, k)];
  return o;
}

// ---------------------------------------------------------------------------------------
// x functors of the batched row product: value of DOF i for this lane's cases
// ---------------------------------------------------------------------------------------
template <typename T, typename M>
struct BLoad {
  const T* __restrict__ x;
  __device__ __forceinline__ C4<T> operator()(int64_t i, int l) const { return ldc<M>(x + i * kBatch, l); }
};
template <typename T, typename M>
struct BD0 {  // first Chebyshev step from zero: dinv_i b_i / theta
  const T* __restrict__ b;
  const T* __restrict__ dinv;
  T inv_theta;
  __device__ __forceinline__ C4<T> operator()(int64_t i, int l) const {
    C4<T> v = ldc<M>(b + i * kBatch, l);
    const T di = dinv[i];
#pragma unroll
    for (int k = 0; k < kC; ++k) v.v[k] = di * v.v[k] * inv_theta;
    return v;
  }
};
template <typename TM>
struct BPNew {  // p_new = z + beta p_old per case (FP64 Krylov, double case map)
  const TM* __restrict__ z;
  const double* __restrict__ p;
  C4<double> beta;
  __device__ __forceinline__ C4<double> operator()(int64_t i, int l) const {
    const C4<double> zz = cvt4<double>(ldc<double>(z + i * kBatch, l));
    const C4<double> pp = ldc<double>(p + i * kBatch, l);
    C4<double> o;
#pragma unroll
    for (int k = 0; k < kC; ++k) o.v[k] = fma(beta.v[k], pp.v[k], zz.v[k]);
    return o;
  }
};

// ---------------------------------------------------------------------------------------
// batched block-row product
// ---------------------------------------------------------------------------------------
// Vector load of W consecutive elements (W * sizeof(T) bytes, naturally aligned).
template <typename T, int W>
struct VLoad;
template <>
struct VLoad<float, 4> {
  static __device__ __forceinline__ void store(float* p, const float (&v)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  }
  static __device__ __forceinline__ void load(const float* p, float (&o)[4]) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(p));
    o[0] = v.x;
    o[1] = v.y;
    o[2] = v.z;
    o[3] = v.w;
  }
  static __device__ __forceinline__ void shared(const float* p, float (&o)[4]) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    o[0] = v.x;
    o[1] = v.y;
    o[2] = v.z;
    o[3] = v.w;
  }
};
template <>
struct VLoad<float, 2> {
  static __device__ __forceinline__ void store(float* p, const float (&v)[2]) {
    *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
  }
  static __device__ __forceinline__ void load(const float* p, float (&o)[2]) {
    const float2 v = __ldg(reinterpret_cast<const float2*>(p));
    o[0] = v.x;
    o[1] = v.y;
  }
};
template <>
struct VLoad<float, 1> {
  static __device__ __forceinline__ void store(float* p, const float (&v)[1]) { p[0] = v[0]; }
  static __device__ __forceinline__ void load(const float* p, float (&o)[1]) { o[0] = __ldg(p); }
};
template <>
struct VLoad<double, 2> {
  static __device__ __forceinline__ void store(double* p, const double (&v)[2]) {
    *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
  }
  static __device__ __forceinline__ void load(const double* p, double (&o)[2]) {
    const double2 v = __ldg(reinterpret_cast<const double2*>(p));
    o[0] = v.x;
    o[1] = v.y;
  }
  static __device__ __forceinline__ void shared(const double* p, double (&o)[2]) {
    const double2 v = *reinterpret_cast<const double2*>(p);
    o[0] = v.x;
    o[1] = v.y;
  }
};
template <>
struct VLoad<double, 1> {
  static __device__ __forceinline__ void store(double* p, const double (&v)[1]) { p[0] = v[0]; }
  static __device__ __forceinline__ void load(const double* p, double (&o)[1]) { o[0] = __ldg(p); }
};

// widest (<= 16 B) load that tiles a block of NB elements of T
template <typename T, int NB>
struct ChunkOf {
  static constexpr int kBlockBytes = NB * (int)sizeof(T);
  static constexpr int kBytes = (kBlockBytes % 16 == 0) ? 16 : (kBlockBytes % 8 == 0) ? 8 : (int)sizeof(T);
  static constexpr int W = kBytes / (int)sizeof(T);  // elements per chunk
  static constexpr int N = kBlockBytes / kBytes;     // chunks per block = chunks per lane per stage
};

// A stage of a row's blocks in shared memory: kBlocks blocks per 8-lane group, a block's values
// row-major with its column behind them.  The strides are odd multiples of 16 bytes, so that 16-byte
// accesses of the 8 lanes to consecutive blocks, and of the 4 groups to one block each, hit
// different banks.
template <int NB, typename T>
struct BStage {
  static constexpr int kBlocks = NB * sizeof(T) <= 80 ? 8 : 4;
  static constexpr int kUnits = (int)((NB * sizeof(T) + 4 + 15) / 16) | 1;  // 16-byte units per block
  static constexpr int kVec = 16 / (int)sizeof(T);
  static constexpr int kStride = kUnits * kVec;                              // elements per block
  static constexpr int kGroup = kBlocks * kStride + kVec;                    // elements per group
  T v[kWarps][4 * kGroup];
  static __device__ __forceinline__ int col(const T* block) { return reinterpret_cast<const int*>(block + NB)[0]; }
};

// Batched block-row product: for every block q of the row and every (r, c) of the block,
// fmacc(r, A(row, q)[r][c], xload(BC col_q + c, l)) -- fmacc accumulates the lane's cases
// (FmaAcc: acc[r][k] += a x[k]).
//
// The 8 lanes of a group walk their row in stages of kBlocks consecutive blocks.  A stage is loaded
// coalesced -- component-major (kSoA): lane i holds block i; block-contiguous (kAoS): the blocks
// are one contiguous span and lane i holds its 16/8/4-byte chunks i, i + 8, ... -- one stage
// ahead, and handed to the group through shared memory, where a lane reads a block's values as
// 16-byte broadcasts.  The x values of TPG blocks are gathered before their multiply-adds
// (blocks past the row end carry zero values and gather node 0), so TPG x BC vector loads per lane
// are in flight at once; trips in which no row of the warp has a block left are skipped.
// All 32 lanes of the warp must call (the 4 groups of a warp work on 4 rows at once);
// `active` = false gives an empty row.
//
// What bounds it is the L1 / shared-memory data path and, with it, L2: the FP32 fine passes of 32
// cases keep it 70 % busy and take 7.6 TB/s from L2 (DRAM 1.7).  Per 32 blocks of 3x3 in FP32 it moves
// 96 wavefronts of x, and moved 72 (FP64: 144) of shuffles when every lane took each value from the
// lane that had loaded it; the broadcasts take 36 (60).  The padding of a warp's rows to the longest
// one, in whole stages, made 37 % of the trips empty; with rows of like length side by side
// (batch_order) and trips of TPG blocks 10 %.  32 cases on the 1M-DOF I-beam, shuffles -> broadcasts
// with the next stage ahead -> rows by length: FP32 pre-smoothing 394 -> 343 -> 259 us, FP64 product
// with FP32 directions 660 -> 670 -> 404 us (375 with the FP32 case map), the 6x6 levels 88 -> 62 us.
template <int BR, int BC, Layout LY, int TPG, int S, typename T, typename XL, typename FA>
__device__ __forceinline__ void batch_row_staged(const int32_t* __restrict__ rp, const int32_t* __restrict__ ci,
                                                 const T* __restrict__ av, int64_t stride, int64_t row, bool active,
                                                 int l, const XL& xload, const FA& fmacc) {
  constexpr int NB = BR * BC;
  constexpr unsigned kFull = 0xffffffffu;
  using ST = BStage<NB, T>;
  constexpr int SB = ST::kBlocks, kTrip = TPG < SB ? TPG : SB;
  static_assert(SB % kTrip == 0, "trips tile a stage");
  using XV = decltype(xload(int64_t(0), 0));
  using CH = ChunkOf<T, NB>;
  constexpr int kChunks = SB * CH::N, kPerLane = (kChunks + 7) / 8;  // kAoS: chunks of a stage, of a lane
  __shared__ __align__(16) ST stage;
  T* const sm = stage.v[threadIdx.x >> 5] + ((threadIdx.x & 31) >> 3) * ST::kGroup;
  int32_t q0 = 0, q1 = 0;
  if (active) {
    q0 = __ldg(rp + row);
    q1 = __ldg(rp + row + 1);
  }
  // a team of S groups shares the row: group h of the team takes stages h, h + S, ...
  const int h = ((threadIdx.x & 31) >> 3) % S;
  const int nst = (q1 - q0 + SB - 1) / SB;
  const int wst = __reduce_max_sync(kFull, nst > h ? (nst - h + S - 1) / S : 0);
  T mv[LY == kSoA ? NB : 1];
  T mc[LY == kSoA ? 1 : kPerLane][CH::W];
  int32_t mcol = 0;
  auto load = [&](int it) {  // this lane's share of the stage's values and columns
    const int32_t qb = q0 + (h + it * S) * SB;
    const int cnt = q1 - qb;  // blocks left (<= 0 once the row is done)
    const int32_t q = qb + l;
    const bool has = l < SB && l < cnt;
    mcol = has ? __ldg(ci + q) : 0;
    if constexpr (LY == kSoA) {
#pragma unroll
      for (int e = 0; e < NB; ++e) mv[e] = has ? __ldg(av + (int64_t)e * stride + q) : T(0);
    } else {
#pragma unroll
      for (int j = 0; j < kPerLane; ++j) {
        const int cidx = l + 8 * j;  // chunk of the stage; chunks never straddle blocks
        if (cidx / CH::N < cnt && cidx < kChunks) {
          VLoad<T, CH::W>::load(av + (int64_t)qb * NB + (int64_t)cidx * CH::W, mc[j]);
        } else {
#pragma unroll
          for (int w = 0; w < CH::W; ++w) mc[j][w] = T(0);
        }
      }
    }
  };
  if (wst > 0) load(0);
  for (int it = 0; it < wst; ++it) {
    __syncwarp();  // the previous stage has been read
    if constexpr (LY == kSoA) {
      static_assert(LY != kSoA || SB == 8, "one block per lane");
      T* o = sm + l * ST::kStride;
#pragma unroll
      for (int e = 0; e < NB; e += ST::kVec) {
        T v[ST::kVec];
#pragma unroll
        for (int w = 0; w < ST::kVec; ++w) v[w] = e + w < NB ? mv[e + w < NB ? e + w : 0] : T(0);
        VLoad<T, ST::kVec>::store(o + e, v);
      }
    } else {
#pragma unroll
      for (int j = 0; j < kPerLane; ++j) {
        const int cidx = l + 8 * j;
        if (cidx < kChunks) {
          T* o = sm + cidx / CH::N * ST::kStride + cidx % CH::N * CH::W;
          VLoad<T, CH::W>::store(o, mc[j]);
        }
      }
    }
    __syncwarp();  // (the column may share a 16-byte store of the last values)
    if (l < SB) reinterpret_cast<int*>(sm + l * ST::kStride + NB)[0] = mcol;
    __syncwarp();
    const int left = max(0, min(SB, q1 - (q0 + (h + it * S) * SB)));
    const int wcnt = __reduce_max_sync(kFull, left);
    if (it + 1 < wst) load(it + 1);
#pragma unroll
    for (int g = 0; g < SB; g += kTrip) {
      if (g < wcnt) {
        XV xv[kTrip][BC];
#pragma unroll
        for (int u = 0; u < kTrip; ++u) {
          const int64_t col = ST::col(sm + (g + u) * ST::kStride);
#pragma unroll
          for (int c = 0; c < BC; ++c) xv[u][c] = xload(col * BC + c, l);
        }
#pragma unroll
        for (int u = 0; u < kTrip; ++u) {
          const T* a = sm + (g + u) * ST::kStride;
#pragma unroll
          for (int e = 0; e < NB; e += ST::kVec) {
            T v[ST::kVec];
            VLoad<T, ST::kVec>::shared(a + e, v);
#pragma unroll
            for (int w = 0; w < ST::kVec; ++w)
              if (e + w < NB) fmacc((e + w) / BC, v[w], xv[u][(e + w) % BC]);
          }
        }
      }
    }
  }
  if constexpr (S > 1) fmacc.template team_reduce<S>();
}

// plain multiply-add accumulation of the lane's four cases
template <int BR, typename T>
struct FmaAcc {
  T (&acc)[BR][kC];
  __device__ __forceinline__ FmaAcc(T (&a)[BR][kC]) : acc(a) {
#pragma unroll
    for (int r = 0; r < BR; ++r)
#pragma unroll
      for (int k = 0; k < kC; ++k) acc[r][k] = T(0);
  }
  template <typename TX>
  __device__ __forceinline__ void operator()(int r, T a, const C4<TX>& x) const {
#pragma unroll
    for (int k = 0; k < kC; ++k) acc[r][k] = fma(a, (T)x.v[k], acc[r][k]);
  }
  // sum over the S groups of a row team (lanes 8 and 16 apart), the same fixed order in
  // every lane
  template <int S>
  __device__ __forceinline__ void team_reduce() const {
#pragma unroll
    for (int r = 0; r < BR; ++r)
#pragma unroll
      for (int k = 0; k < kC; ++k) {
        if constexpr (S >= 2) acc[r][k] += __shfl_xor_sync(0xffffffffu, acc[r][k], 8);
        if constexpr (S >= 4) acc[r][k] += __shfl_xor_sync(0xffffffffu, acc[r][k], 16);
      }
  }
};

template <int BS>
struct BLayout {
  static constexpr Layout value = (BS == 3) ? kSoA : kAoS;
};
// blocks of BC columns whose x is gathered ahead of the multiply-adds (register budget)
template <typename T, int BC>
struct Tpg {
  static constexpr int wide = kC == 1 ? 8 : kC == 2 ? (sizeof(T) == 4 ? 8 : 4) : (sizeof(T) == 4 ? 4 : 2);
  static constexpr int value = BC == 6 && wide > 1 ? wide / 2 : wide;
};

// ---------------------------------------------------------------------------------------
// batched V-cycle kernels (same arithmetic per case as the single-RHS smoother kernels);
// vectors of type T use the case map of T.  Products that are added are written as explicit fma here
// and in all kernels of this file: left to the compiler, the 8-wide build contracted some otherwise
// than the others, and a case's bits must not depend on the batch width.
// ---------------------------------------------------------------------------------------
// xf: the first smoothing step's x, dinv b / theta -- BD0 on the fly, or BLoad of the vector the
// PCG update wrote (the same values)
template <int BS, typename T, int S, typename XF>
__global__ void __launch_bounds__(kThreads, (kRowCtas<T, BS * BS>))
    kb_pre_first(int64_t n_rows, const int32_t* __restrict__ order, const int32_t* __restrict__ rp,
                                                         const int32_t* __restrict__ ci, const T* __restrict__ av,
                                                         int64_t stride, XF xf, const T* __restrict__ b,
                                                         const T* __restrict__ dinv, T inv_theta, int deg, T c1, T c2,
                                                         T* __restrict__ x, T* __restrict__ r, T* __restrict__ d,
                                                         T* __restrict__ res, const int* __restrict__ done) {
  if (*done) return;
  BATCH_TEAM_LOOP(n_rows, S, order) {
    T acc[BS][kC];
    batch_row_staged<BS, BS, BLayout<BS>::value, Tpg<T, BS>::value, S, T>(rp, ci, av, stride, row, row < n_rows, l,
                                                                xf, FmaAcc<BS, T>(acc));
    if (row >= n_rows || !lead) continue;
#pragma unroll
    for (int rr = 0; rr < BS; ++rr) {
      const int64_t i = row * BS + rr;
      const int64_t o = i * kBatch;
      const T di = dinv[i];
      const C4<T> bi = ldc<T>(b + o, l);
      C4<T> xo, ro, dd;
#pragma unroll
      for (int k = 0; k < kC; ++k) {
        const T t = acc[rr][k];
        const T d0 = di * bi.v[k] * inv_theta;
        if (deg == 1) {
          xo.v[k] = d0;
          ro.v[k] = bi.v[k] - t;
        } else {
          const T r1 = fma(-di, t, di * bi.v[k]);
          const T d1 = fma(c1, d0, c2 * r1);
          xo.v[k] = d0 + d1;
          ro.v[k] = r1;
          dd.v[k] = d1;
        }
      }
      stc<T>(x + o, l, xo);
      if (deg == 1) {
        stc<T>(res + o, l, ro);
      } else {
        stc<T>(r + o, l, ro);
        stc<T>(d + o, l, dd);
      }
    }
  }
}

// r -= D^-1 A d_in; d_out = c1 d_in + c2 r; x += d_out; part (if set): b . x per case
template <int BS, typename T, int S>
__global__ void __launch_bounds__(kThreads, (kRowCtas<T, BS * BS>))
    kb_cheb_step(int64_t n_rows, const int32_t* __restrict__ order, const int32_t* __restrict__ rp,
                                                         const int32_t* __restrict__ ci, const T* __restrict__ av,
                                                         int64_t stride, const T* __restrict__ dinv,
                                                         const T* __restrict__ d_in, T* __restrict__ d_out,
                                                         T* __restrict__ r, T* __restrict__ x, T c1, T c2,
                                                         const T* __restrict__ b, double* __restrict__ part,
                                                         const int* __restrict__ done) {
  if (*done) return;
  double dot[kC] = {};
  {
    BATCH_TEAM_LOOP(n_rows, S, order) {
      T acc[BS][kC];
      batch_row_staged<BS, BS, BLayout<BS>::value, Tpg<T, BS>::value, S, T>(rp, ci, av, stride, row, row < n_rows, l,
                                                                  BLoad<T, T>{d_in}, FmaAcc<BS, T>(acc));
      if (row >= n_rows || !lead) continue;
#pragma unroll
      for (int rr = 0; rr < BS; ++rr) {
        const int64_t i = row * BS + rr;
        const int64_t o = i * kBatch;
        const T di = dinv[i];
        const C4<T> rv = ldc<T>(r + o, l), dv = ldc<T>(d_in + o, l), xv = ldc<T>(x + o, l);
        C4<T> ro, dn, xn;
#pragma unroll
        for (int k = 0; k < kC; ++k) {
          ro.v[k] = fma(-di, acc[rr][k], rv.v[k]);
          dn.v[k] = fma(c1, dv.v[k], c2 * ro.v[k]);
          xn.v[k] = xv.v[k] + dn.v[k];
        }
        stc<T>(r + o, l, ro);
        stc<T>(d_out + o, l, dn);
        stc<T>(x + o, l, xn);
        if (part) {
          const C4<T> bv = ldc<T>(b + o, l);
#pragma unroll
          for (int k = 0; k < kC; ++k) dot[k] = fma((double)bv.v[k], (double)xn.v[k], dot[k]);
        }
      }
    }
  }
  if (part) write_case_parts<T>(dot, part);
}

// res = b - A x
template <int BS, typename T, int S>
__global__ void __launch_bounds__(kThreads, (kRowCtas<T, BS * BS>))
    kb_residual(int64_t n_rows, const int32_t* __restrict__ order, const int32_t* __restrict__ rp,
                                                        const int32_t* __restrict__ ci, const T* __restrict__ av,
                                                        int64_t stride, const T* __restrict__ b,
                                                        const T* __restrict__ x, T* __restrict__ res,
                                                        const int* __restrict__ done) {
  if (*done) return;
  BATCH_TEAM_LOOP(n_rows, S, order) {
    T acc[BS][kC];
    batch_row_staged<BS, BS, BLayout<BS>::value, Tpg<T, BS>::value, S, T>(rp, ci, av, stride, row, row < n_rows, l,
                                                                BLoad<T, T>{x}, FmaAcc<BS, T>(acc));
    if (row >= n_rows || !lead) continue;
#pragma unroll
    for (int rr = 0; rr < BS; ++rr) {
      const int64_t o = (row * BS + rr) * kBatch;
      const C4<T> bv = ldc<T>(b + o, l);
      C4<T> ro;
#pragma unroll
      for (int k = 0; k < kC; ++k) ro.v[k] = bv.v[k] - acc[rr][k];
      stc<T>(res + o, l, ro);
    }
  }
}

// first post-smoothing step from x: r0 = D^-1 (b - A x), d0 = r0 / theta, x2 = x + d0
template <int BS, typename T, int S>
__global__ void __launch_bounds__(kThreads, (kRowCtas<T, BS * BS>))
    kb_post_first(int64_t n_rows, const int32_t* __restrict__ order, const int32_t* __restrict__ rp,
                                                          const int32_t* __restrict__ ci, const T* __restrict__ av,
                                                          int64_t stride, const T* __restrict__ b,
                                                          const T* __restrict__ dinv, T inv_theta,
                                                          const T* __restrict__ x, T* __restrict__ x2,
                                                          T* __restrict__ r, T* __restrict__ d,
                                                          double* __restrict__ part, const int* __restrict__ done) {
  if (*done) return;
  double dot[kC] = {};
  {
    BATCH_TEAM_LOOP(n_rows, S, order) {
      T acc[BS][kC];
      batch_row_staged<BS, BS, BLayout<BS>::value, Tpg<T, BS>::value, S, T>(rp, ci, av, stride, row, row < n_rows, l,
                                                                  BLoad<T, T>{x}, FmaAcc<BS, T>(acc));
      if (row >= n_rows || !lead) continue;
#pragma unroll
      for (int rr = 0; rr < BS; ++rr) {
        const int64_t i = row * BS + rr;
        const int64_t o = i * kBatch;
        const T di = dinv[i];
        const C4<T> bv = ldc<T>(b + o, l), xv = ldc<T>(x + o, l);
        C4<T> ro, dd, xn;
#pragma unroll
        for (int k = 0; k < kC; ++k) {
          ro.v[k] = di * (bv.v[k] - acc[rr][k]);
          dd.v[k] = ro.v[k] * inv_theta;
          xn.v[k] = fma(ro.v[k], inv_theta, xv.v[k]);
          if (part) dot[k] = fma((double)bv.v[k], (double)xn.v[k], dot[k]);
        }
        if (r) {  // a Chebyshev step follows
          stc<T>(r + o, l, ro);
          stc<T>(d + o, l, dd);
        }
        stc<T>(x2 + o, l, xn);
      }
    }
  }
  if (part) write_case_parts<T>(dot, part);
}

// ---------------------------------------------------------------------------------------
// streamed fine level (3x3 blocks): the fine matrix comes from its tile-major pack through the
// shared-memory stage ring of stream.cuh (stream_pipeline).  Per tile, a group of 8 lanes per
// block row (4 rows per warp), lane l owning 4 of the 32 cases; the group walks its row's
// blocks in order, two blocks' x gathers in flight, and reads each block's 9 values from the
// stage (the 8 lanes of a group read the same word: a shared-memory broadcast, as the register
// kernels above read the stages that they fill themselves).  The per-case arithmetic and the order
// of every multiply-add are those of the register kernels, so both paths give the same bits.  For
// 32 cases only, and only when switched on (wn_solid_set_stream).
// ---------------------------------------------------------------------------------------
// the fine matrix in one precision as the streamed kernels see it
struct BView {
  const PackTile* tiles;
  int n_tiles;
  const unsigned char* pack;
  StreamCtl ctl;
};
template <typename T>
BView bview(const StreamMat& m) {
  if constexpr (sizeof(T) == 4)
    return {m.d32.p, m.n_tiles, m.p32.p, m.ctl};
  else
    return {m.d64.p, m.n_tiles, m.p64.p, m.ctl};
}

// the per-case partial sums of a CTA of NW warps (cf. write_case_parts)
template <typename M, int NW>
__device__ __forceinline__ void write_case_parts_nw(double (&d)[kC], double* __restrict__ part) {
  __shared__ double sh[NW][kBatch];
#pragma unroll
  for (int k = 0; k < kC; ++k) {
    d[k] += __shfl_xor_sync(0xffffffffu, d[k], 8);
    d[k] += __shfl_xor_sync(0xffffffffu, d[k], 16);
  }
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane < 8)
#pragma unroll
    for (int k = 0; k < kC; ++k) sh[w][case_of<M>(lane, k)] = d[k];
  __syncthreads();
  if (threadIdx.x < kBatch) {
    double s = 0.0;
    for (int k = 0; k < NW; ++k) s += sh[k][threadIdx.x];
    part[(int64_t)blockIdx.x * kBatch + threadIdx.x] = s;
  }
}

// The tile body: rows of the 3x3 fine matrix against DOF-major n x 32 vectors; per row DOF i,
// pre = epi.load(i, l) before the product and epi.store(i, l, pre, acc, dot) after it
template <typename T, typename XF, typename EPI, typename HOOK>
__device__ __forceinline__ void batch_stream_rows(const BView& m, const XF& xf, const EPI& epi, unsigned char* smem,
                                                  BlockScalars* S, bool* skipped, const HOOK& hook,
                                                  double (&dot)[kC]) {
  using Cfg = typename StreamDefault<T, 3, 3>::type;
  constexpr int NCW = Cfg::kWarps;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int l = lane & 7, grp = lane >> 3;
  auto body = [&](int jc, const unsigned char* st, const int4 d, double&) {
    const int r0 = d.x, nr = d.y - d.x, cntp = d.w;
    const T* sv = reinterpret_cast<const T*>(st);
    const int32_t* scol = reinterpret_cast<const int32_t*>(st + pack_col_off<T, 9>(cntp));
    const uint16_t* srp = reinterpret_cast<const uint16_t*>(st + pack_row_off<T, 9>(cntp));
    // warps take the tile's rows in passes of 4, starting from a warp that rotates per tile
    const int wslot = (warp + jc) % NCW;
    for (int base = wslot * 4; base < nr; base += NCW * 4) {
      const int lr = base + grp;
      if (lr >= nr) continue;  // no warp-wide operation below: the groups run independently
      const int rs = srp[lr], re = srp[lr + 1];
      const int64_t i0 = (int64_t)(r0 + lr) * 3;
      typename EPI::Pre pre[3];
#pragma unroll
      for (int r = 0; r < 3; ++r) pre[r] = epi.load(i0 + r, l);
      T acc[3][kC];
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int k = 0; k < kC; ++k) acc[r][k] = T(0);
      auto fma_block = [&](int b, const C4<T> (&x)[3]) {
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const T a = sv[(r * 3 + c) * cntp + b];
#pragma unroll
            for (int k = 0; k < kC; ++k) acc[r][k] = fma(a, x[c].v[k], acc[r][k]);
          }
      };
      int b = rs;
      // two blocks' gathers in flight in FP32; one in FP64 (registers: two CTAs per SM)
      for (; sizeof(T) == 4 && b + 1 < re; b += 2) {
        const int64_t ca = scol[b], cb = scol[b + 1];
        C4<T> xa[3], xb[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          xa[c] = xf(ca * 3 + c, l);
          xb[c] = xf(cb * 3 + c, l);
        }
        fma_block(b, xa);
        fma_block(b + 1, xb);
      }
      for (; b < re; ++b) {
        const int64_t ca = scol[b];
        C4<T> xa[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) xa[c] = xf(ca * 3 + c, l);
        fma_block(b, xa);
      }
#pragma unroll
      for (int r = 0; r < 3; ++r) epi.store(i0 + r, l, pre[r], acc[r], dot);
    }
    return true;
  };
  stream_pipeline<T, 9, Cfg>(m.tiles, m.n_tiles, m.pack, smem, &S->status, &S->done, m.ctl, skipped, hook, body);
}

// epilogues of the streamed fine-level kernels (the arithmetic of kb_pre_first, kb_cheb_step,
// kb_residual, kb_post_first and kb_spmv_dot); like those kernels they read the row's own
// operands after the row product (no registers held across it)
struct BNoPre {};
template <typename T>
struct BEpiPreFirst {
  const T* __restrict__ b;
  const T* __restrict__ dinv;
  T inv_theta;
  int deg;
  T c1, c2;
  T *__restrict__ x, *__restrict__ r, *__restrict__ d, *__restrict__ res;
  using Pre = BNoPre;
  __device__ __forceinline__ Pre load(int64_t, int) const { return {}; }
  __device__ __forceinline__ void store(int64_t i, int l, const Pre&, const T (&acc)[kC], double (&)[kC]) const {
    const int64_t o = i * kBatch;
    const T di = dinv[i];
    const C4<T> bi = ldc<T>(b + o, l);
    C4<T> xo, ro, dd;
#pragma unroll
    for (int k = 0; k < kC; ++k) {
      const T t = acc[k];
      const T d0 = di * bi.v[k] * inv_theta;
      if (deg == 1) {
        xo.v[k] = d0;
        ro.v[k] = bi.v[k] - t;
      } else {
        const T r1 = fma(-di, t, di * bi.v[k]);
        const T d1 = fma(c1, d0, c2 * r1);
        xo.v[k] = d0 + d1;
        ro.v[k] = r1;
        dd.v[k] = d1;
      }
    }
    stc<T>(x + o, l, xo);
    if (deg == 1) {
      stc<T>(res + o, l, ro);
    } else {
      stc<T>(r + o, l, ro);
      stc<T>(d + o, l, dd);
    }
  }
};
template <typename T>
struct BEpiCheb {  // r -= D^-1 A d_in; d_out = c1 d_in + c2 r; x += d_out; dot: b . x
  const T* __restrict__ dinv;
  const T* __restrict__ d_in;
  T *__restrict__ d_out, *__restrict__ r, *__restrict__ x;
  T c1, c2;
  const T* __restrict__ b;
  int want_dot;
  using Pre = BNoPre;
  __device__ __forceinline__ Pre load(int64_t, int) const { return {}; }
  __device__ __forceinline__ void store(int64_t i, int l, const Pre&, const T (&acc)[kC], double (&dot)[kC]) const {
    const int64_t o = i * kBatch;
    const T di = dinv[i];
    const C4<T> rv = ldc<T>(r + o, l), dv = ldc<T>(d_in + o, l), xv = ldc<T>(x + o, l);
    C4<T> ro, dn, xn;
#pragma unroll
    for (int k = 0; k < kC; ++k) {
      ro.v[k] = fma(-di, acc[k], rv.v[k]);
      dn.v[k] = fma(c1, dv.v[k], c2 * ro.v[k]);
      xn.v[k] = xv.v[k] + dn.v[k];
    }
    stc<T>(r + o, l, ro);
    stc<T>(d_out + o, l, dn);
    stc<T>(x + o, l, xn);
    if (want_dot) {
      const C4<T> bv = ldc<T>(b + o, l);
#pragma unroll
      for (int k = 0; k < kC; ++k) dot[k] = fma((double)bv.v[k], (double)xn.v[k], dot[k]);
    }
  }
};
template <typename T>
struct BEpiResidual {  // res = b - A x
  const T* __restrict__ b;
  T* __restrict__ res;
  using Pre = BNoPre;
  __device__ __forceinline__ Pre load(int64_t, int) const { return {}; }
  __device__ __forceinline__ void store(int64_t i, int l, const Pre&, const T (&acc)[kC], double (&)[kC]) const {
    const C4<T> bv = ldc<T>(b + i * kBatch, l);
    C4<T> ro;
#pragma unroll
    for (int k = 0; k < kC; ++k) ro.v[k] = bv.v[k] - acc[k];
    stc<T>(res + i * kBatch, l, ro);
  }
};
template <typename T>
struct BEpiPostFirst {  // r0 = D^-1 (b - A x), d0 = r0 / theta, x2 = x + d0; dot: b . x2
  const T* __restrict__ b;
  const T* __restrict__ dinv;
  T inv_theta;
  const T* __restrict__ x;
  T *__restrict__ x2, *__restrict__ r, *__restrict__ d;
  int want_dot;
  using Pre = BNoPre;
  __device__ __forceinline__ Pre load(int64_t, int) const { return {}; }
  __device__ __forceinline__ void store(int64_t i, int l, const Pre&, const T (&acc)[kC], double (&dot)[kC]) const {
    const int64_t o = i * kBatch;
    const T di = dinv[i];
    const C4<T> bv = ldc<T>(b + o, l), xv = ldc<T>(x + o, l);
    C4<T> ro, dd, xn;
#pragma unroll
    for (int k = 0; k < kC; ++k) {
      ro.v[k] = di * (bv.v[k] - acc[k]);
      dd.v[k] = ro.v[k] * inv_theta;
      xn.v[k] = fma(ro.v[k], inv_theta, xv.v[k]);
      if (want_dot) dot[k] = fma((double)bv.v[k], (double)xn.v[k], dot[k]);
    }
    if (r) {  // a Chebyshev step follows
      stc<T>(r + o, l, ro);
      stc<T>(d + o, l, dd);
    }
    stc<T>(x2 + o, l, xn);
  }
};
template <typename TM>
struct BEpiSpmvDot {  // p_new = z + beta p_old; q = A p_new; dot: p_new . q
  BPNew<TM> pf;
  double *__restrict__ p_new, *__restrict__ q;
  using Pre = BNoPre;
  __device__ __forceinline__ Pre load(int64_t, int) const { return {}; }
  __device__ __forceinline__ void store(int64_t i, int l, const Pre&, const double (&acc)[kC],
                                        double (&dot)[kC]) const {
    const int64_t o = i * kBatch;
    const C4<double> pv = pf(i, l);
    C4<double> qv;
#pragma unroll
    for (int k = 0; k < kC; ++k) {
      qv.v[k] = acc[k];
      dot[k] = fma(pv.v[k], qv.v[k], dot[k]);
    }
    stc<double>(p_new + o, l, pv);
    stc<double>(q + o, l, qv);
  }
};

// the streamed fine-level kernel: a persistent CTA per tile run; part (if set) receives the
// per-case partials of the epilogue's dot
template <typename T>
struct BStreamCtas {
  static constexpr int value = 2;
};
template <typename T, typename XF, typename EPI>
__global__ void __launch_bounds__(kStreamThreads, BStreamCtas<T>::value)
    kbs_rows(BView m, XF xf, EPI epi, double* __restrict__ part, BlockScalars* __restrict__ S) {
  extern __shared__ __align__(128) unsigned char smem[];
  bool skipped = false;
  double dot[kC] = {};
  batch_stream_rows<T>(m, xf, epi, smem, S, &skipped, NoHook{}, dot);
  if (part && !skipped) write_case_parts_nw<T, kStreamThreads / 32>(dot, part);
}
// the PCG product with the FP64 pack: p_new = z + beta p_old on the fly, its case map is the
// FP64 one (cases 2l, 2l+1, 16+2l, 17+2l)
template <typename TM>
__global__ void __launch_bounds__(kStreamThreads, 2)
    kbs_spmv_dot(BView m, const TM* __restrict__ z, const double* __restrict__ p_old, double* __restrict__ p_new,
                 double* __restrict__ q, double* __restrict__ partB, BlockScalars* __restrict__ S) {
  extern __shared__ __align__(128) unsigned char smem[];
  bool skipped = false;
  double dot[kC] = {};
  const int l = threadIdx.x & 7;
  const BPNew<TM> pf{z, p_old, case_scalars<double>(S->beta, l)};
  batch_stream_rows<double>(m, pf, BEpiSpmvDot<TM>{pf, p_new, q}, smem, S, &skipped, NoHook{}, dot);
  if (!skipped) write_case_parts_nw<double, kStreamThreads / 32>(dot, partB);
}

// launch a streamed fine-level kernel; the grid (one persistent wave), 0 if it cannot run here
template <typename T, typename K, typename... Args>
int launch_bs(K kern, const StreamMat& m, cudaStream_t st, Args... args) {
  if (!m.packed || m.br != 3 || m.bc != 3) return 0;
  const size_t smem = stream_smem_bytes<T, 3, 3>();
  const int per_sm = stream_ctas_per_sm(reinterpret_cast<const void*>(kern), kStreamThreads, smem);
  if (per_sm < 1) return 0;
  const int g = std::max(1, std::min(m.n_tiles, kNumSMs * per_sm));
  if (g > BlockWork::kMaxParts) return 0;
  kern<<<g, kStreamThreads, smem, st>>>(args...);
  if (cudaGetLastError() != cudaSuccess) return 0;
  return g;
}

// ---------------------------------------------------------------------------------------
// fine level with each tile's x slice staged in shared memory (32 cases, switched on by
// wn_solid_set_batch_staging).  An x-tile is a run of whole block rows whose blocks name at most kXTileCols
// distinct column nodes (the plan in BlockWork: per tile the sorted column list, per block its
// column as an 8-bit index into that list).  The CTA first writes the x values of the tile's
// columns -- xf(i, l) for the 32 cases of each of their DOFs, the same functor and arithmetic
// as the register kernels' gathers -- into shared memory with coalesced 16-byte loads, many in
// flight at once; then 8-lane groups run the rows in stages of 8 blocks, values component-major and
// coalesced, passed round by shuffles (batch_row_staged hands them over in shared memory; the
// order of every multiply-add is the same, so the bits are too), and read each block's x from shared
// memory by its local column.  A gathered x row served 2-3 blocks of the tile from L1/L2 before (the tiles' column
// lists hold 2.8 M rows against 8.5 M blocks on the I-beam), and the gathers' latency was what
// bound the batched sweeps.
// ---------------------------------------------------------------------------------------
constexpr int kXTileCols = 256;  // columns per x-tile: the 8-bit local column index
struct XTiles {
  const int32_t* rows;     // n_tiles + 1 block-row starts
  const int32_t* col_ptr;  // n_tiles + 1
  const int32_t* cols;     // per tile its distinct column nodes, ascending
  const uint8_t* lcol;     // nnzb: the block's column as an index into its tile's list
  int n_tiles;
};

// How an x functor's slice is staged: the functor's source rows are copied as they are
// (cp.async, 16 bytes per lane, no register round trip) and the functor's arithmetic, if any,
// is applied when a value is read -- the same expression on the same operands, so the same bits.
template <typename XF>
struct XStage;
template <>
struct XStage<BLoad<float, float>> {
  static constexpr bool kDinv = false;
  static __device__ __forceinline__ const float* src(const BLoad<float, float>& f) { return f.x; }
  static __device__ __forceinline__ const float* dinv(const BLoad<float, float>&) { return nullptr; }
  static __device__ __forceinline__ float scale(const BLoad<float, float>&) { return 1.0f; }
};
template <>
struct XStage<BD0<float, float>> {  // dinv_i b_i / theta
  static constexpr bool kDinv = true;
  static __device__ __forceinline__ const float* src(const BD0<float, float>& f) { return f.b; }
  static __device__ __forceinline__ const float* dinv(const BD0<float, float>& f) { return f.dinv; }
  static __device__ __forceinline__ float scale(const BD0<float, float>& f) { return f.inv_theta; }
};

template <bool kDinv>
struct XsLoad {  // x of local DOF u (local column * 3 + component) from the staged slice
  const float* xs;
  const float* sd;  // staged dinv (BD0)
  float it;
  __device__ __forceinline__ C4<float> operator()(int64_t u, int l) const {
    C4<float> v = ldc<float>(xs + u * kBatch, l);
    if constexpr (kDinv) {
      const float di = sd[u];
#pragma unroll
      for (int k = 0; k < kC; ++k) v.v[k] = di * v.v[k] * it;  // BD0's expression
    }
    return v;
  }
};

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

// batch_row_staged for the 3x3 component-major fine matrix with 8-bit local columns
template <typename T, typename XL, typename FA>
__device__ __forceinline__ void batch_row_xs(const int32_t* __restrict__ rp, const uint8_t* __restrict__ lcol,
                                             const T* __restrict__ av, int64_t stride, int64_t row, bool active,
                                             int l, const XL& xload, const FA& fmacc) {
  constexpr unsigned kFull = 0xffffffffu;
  constexpr int TPG = Tpg<T, 3>::value;
  using XV = decltype(xload(int64_t(0), 0));
  const int gbase = threadIdx.x & 24;
  int32_t q0 = 0, q1 = 0;
  if (active) {
    q0 = __ldg(rp + row);
    q1 = __ldg(rp + row + 1);
  }
  const int nst = (q1 - q0 + 7) >> 3;
  const int wst = __reduce_max_sync(kFull, nst);
  for (int it = 0; it < wst; ++it) {
    const int32_t qb = q0 + it * 8;
    const int cnt = q1 - qb;
    const int32_t q = qb + l;
    const int mcol = (l < cnt) ? (int)__ldg(lcol + q) : 0;
    T mv[9];
#pragma unroll
    for (int e = 0; e < 9; ++e) mv[e] = (l < cnt) ? __ldg(av + (int64_t)e * stride + q) : T(0);
#pragma unroll
    for (int g = 0; g < 8; g += TPG) {
      XV xv[TPG][3];
#pragma unroll
      for (int u = 0; u < TPG; ++u) {
        const int col = __shfl_sync(kFull, mcol, gbase | (g + u));
#pragma unroll
        for (int c = 0; c < 3; ++c) xv[u][c] = xload((int64_t)col * 3 + c, l);
      }
#pragma unroll
      for (int u = 0; u < TPG; ++u) {
        const int t = g + u;
#pragma unroll
        for (int r = 0; r < 3; ++r)
#pragma unroll
          for (int c = 0; c < 3; ++c) fmacc(r, __shfl_sync(kFull, mv[r * 3 + c], gbase | t), xv[u][c]);
      }
    }
  }
}

template <typename XF, typename EPI>
__global__ void __launch_bounds__(kThreads, 2) kbx_rows(XTiles xt, const int32_t* __restrict__ rp,
                                                        const float* __restrict__ av, int64_t stride, XF xf, EPI epi,
                                                        double* __restrict__ part, const int* __restrict__ done) {
  if (*done) return;
  using XS = XStage<XF>;
  extern __shared__ __align__(16) unsigned char xsm[];
  float* xs = reinterpret_cast<float*>(xsm);  // kXTileCols x 3 DOFs x 32 cases
  __shared__ int32_t s_cols[kXTileCols];
  __shared__ float s_dinv[XS::kDinv ? kXTileCols * 3 : 1];
  const int warp = threadIdx.x >> 5, grp = (threadIdx.x & 31) >> 3, l = threadIdx.x & 7;
  const float* src = XS::src(xf);
  double dot[kC] = {};
  for (int t = blockIdx.x; t < xt.n_tiles; t += gridDim.x) {
    const int c0 = xt.col_ptr[t], nc = xt.col_ptr[t + 1] - c0;
    for (int k = threadIdx.x; k < nc; k += kThreads) s_cols[k] = xt.cols[c0 + k];
    __syncthreads();
    // the slice: 8 chunks of 16 bytes per DOF row (32 cases), all copies in flight at once
    for (int idx = threadIdx.x; idx < nc * 24; idx += kThreads) {
      const int u = idx >> 3, ch = idx & 7;
      const int64_t dof = (int64_t)s_cols[u / 3] * 3 + u % 3;
      cp_async16(xs + u * kBatch + ch * 4, src + dof * kBatch + ch * 4);
    }
    if constexpr (XS::kDinv)
      for (int u = threadIdx.x; u < nc * 3; u += kThreads) s_dinv[u] = XS::dinv(xf)[(int64_t)s_cols[u / 3] * 3 + u % 3];
    cp_async_wait_all();
    __syncthreads();
    const int r0 = xt.rows[t], r1 = xt.rows[t + 1];
    for (int base = r0 + warp * 4; base < r1; base += (kThreads >> 5) * 4) {  // warp-uniform bound
      const int row = base + grp;
      float acc[3][kC];
      batch_row_xs<float>(rp, xt.lcol, av, stride, row, row < r1, l, XsLoad<XS::kDinv>{xs, s_dinv, XS::scale(xf)},
                          FmaAcc<3, float>(acc));
      if (row >= r1) continue;
#pragma unroll
      for (int r = 0; r < 3; ++r) epi.store((int64_t)row * 3 + r, l, epi.load((int64_t)row * 3 + r, l), acc[r], dot);
    }
    __syncthreads();  // the slice is rewritten for the next tile
  }
  if (part) write_case_parts<float>(dot, part);
}

// host plan of the x-tiles: greedy runs of whole rows with at most kXTileCols distinct columns
int build_x_tiles(Solid* s, BlockWork& W) {
  W.xt_tried = true;
  const int64_t n = s->n_nodes;
  const std::vector<int32_t>& rp = s->h_row_ptr;
  const std::vector<int32_t>& ci = s->h_col_idx;
  if (s->bs != 3 || (int64_t)rp.size() != n + 1 || (int64_t)ci.size() != s->nnzb) return 0;
  std::vector<int32_t> rows{0}, col_ptr{0}, cols;
  std::vector<uint8_t> lcol(s->nnzb);
  std::vector<int32_t> stamp(n, -1), local(n, 0);
  std::vector<int32_t> cur;
  int tile = 0;
  for (int64_t r = 0; r < n;) {
    cur.clear();
    const int64_t r0 = r;
    while (r < n) {
      int add = 0;  // columns of row r new to the tile (a row names each column once)
      for (int32_t q = rp[r]; q < rp[r + 1]; ++q) add += stamp[ci[q]] != tile;
      if ((int)cur.size() + add > kXTileCols) break;
      for (int32_t q = rp[r]; q < rp[r + 1]; ++q)
        if (stamp[ci[q]] != tile) {
          stamp[ci[q]] = tile;
          cur.push_back(ci[q]);
        }
      ++r;
    }
    if (r == r0) return 0;  // one row names more than kXTileCols columns: no plan
    std::sort(cur.begin(), cur.end());
    for (size_t k = 0; k < cur.size(); ++k) local[cur[k]] = (int32_t)k;
    for (int32_t q = rp[r0]; q < rp[r]; ++q) lcol[q] = (uint8_t)local[ci[q]];
    cols.insert(cols.end(), cur.begin(), cur.end());
    rows.push_back((int32_t)r);
    col_ptr.push_back((int32_t)cols.size());
    ++tile;
  }
  WN_CHECK(W.xt_rows.upload(rows));
  WN_CHECK(W.xt_col_ptr.upload(col_ptr));
  WN_CHECK(W.xt_cols.upload(cols));
  WN_CHECK(W.xt_lcol.upload(lcol));
  W.xt_n = tile;
  return 0;
}

// launch a staged-x fine-level kernel (persistent grid); the grid, 0 if no plan, no fit or not
// an FP32 pass with a stageable x functor (an FP64 slice, 192 KB, would leave one CTA per SM)
template <typename XF>
struct Stageable : std::false_type {};
template <>
struct Stageable<BLoad<float, float>> : std::true_type {};
template <>
struct Stageable<BD0<float, float>> : std::true_type {};

template <typename T, typename XF, typename EPI>
int launch_bx(Solid* s, BlockWork& W, const T* av, XF xf, EPI epi, double* part, const int* done, cudaStream_t st) {
  if constexpr (!std::is_same<T, float>::value || !Stageable<XF>::value) {
    return 0;
  } else {
    if (!s->batch_stage_x || W.xt_n == 0) return 0;
    const size_t smem = (size_t)kXTileCols * 3 * kBatch * sizeof(float);
    auto kern = kbx_rows<XF, EPI>;
    const int per_sm = stream_ctas_per_sm(reinterpret_cast<const void*>(kern), kThreads, smem);
    if (per_sm < 1) return 0;
    const int g = std::max(1, std::min(W.xt_n, std::min(kNumSMs * per_sm, BlockWork::kMaxParts)));
    kern<<<g, kThreads, smem, st>>>(XTiles{W.xt_rows.p, W.xt_col_ptr.p, W.xt_cols.p, W.xt_lcol.p, W.xt_n},
                                    s->row_ptr.p, av, s->nnzb, xf, epi, part, done);
    if (cudaGetLastError() != cudaSuccess) return 0;
    return g;
  }
}

// y = A x or y += A x for the block-contiguous transfer operators (BR x BC blocks)
template <int BR, int BC, typename T, int S>
__global__ void __launch_bounds__(kThreads, (kRowCtas<T, BR * BC>))
    kb_level_spmv(int64_t n_rows, const int32_t* __restrict__ order, const int32_t* __restrict__ rp,
                                                          const int32_t* __restrict__ ci, const T* __restrict__ av,
                                                          const T* __restrict__ x, T* __restrict__ y, int accumulate,
                                                          const int* __restrict__ done) {
  if (*done) return;
  BATCH_TEAM_LOOP(n_rows, S, order) {
    T acc[BR][kC];
    batch_row_staged<BR, BC, kAoS, Tpg<T, BC>::value, S, T>(rp, ci, av, 0, row, row < n_rows, l, BLoad<T, T>{x}, FmaAcc<BR, T>(acc));
    if (row >= n_rows || !lead) continue;
#pragma unroll
    for (int rr = 0; rr < BR; ++rr) {
      const int64_t o = (row * BR + rr) * kBatch;
      C4<T> v;
#pragma unroll
      for (int k = 0; k < kC; ++k) v.v[k] = acc[rr][k];
      if (accumulate) {
        const C4<T> yv = ldc<T>(y + o, l);
#pragma unroll
        for (int k = 0; k < kC; ++k) v.v[k] += yv.v[k];
      }
      stc<T>(y + o, l, v);
    }
  }
}

// Coarsest level: X = A_c^-1 B with the dense FP64 inverse.  A CTA takes kCoarseRows rows and cuts
// the columns into 32 runs of equal length, whose sums are added in order at the end (the same in a
// batch of any width).  A warp's lane is a case: kBatch = 32 walks 4 runs per warp side by side,
// 16 two and 8 one, so every b loaded serves kCoarseRows rows and the loads of several columns are
// in flight (32 cases at n = 1,482: 105 us with one chain of n dependent loads per row, 43 us).
constexpr int kCoarseRows = 4;
template <typename T>
__global__ void __launch_bounds__(kThreads) kb_coarse(int64_t n, const double* __restrict__ inv,
                                                      const T* __restrict__ b, T* __restrict__ x,
                                                      const int* __restrict__ done) {
  if (*done) return;
  constexpr int kRuns = 32, kPerLane = kRuns / 8 * kBatch / 32;  // runs of a warp: 4; of a lane
  __shared__ double sh[kRuns][kCoarseRows][kBatch];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int j = lane % kBatch, sub = lane / kBatch;
  const int64_t r0 = (int64_t)blockIdx.x * kCoarseRows;
  const int64_t len = (n + kRuns - 1) / kRuns;
  double s[kPerLane][kCoarseRows] = {};
  const double* rowp[kCoarseRows];
#pragma unroll
  for (int r = 0; r < kCoarseRows; ++r) rowp[r] = inv + min(r0 + r, n - 1) * n;
#pragma unroll(16 / kPerLane)
  for (int64_t c = 0; c < len; ++c) {
#pragma unroll
    for (int u = 0; u < kPerLane; ++u) {
      const int64_t col = (warp * 4 + sub * kPerLane + u) * len + c;
      if (col < n) {
        const double bv = (double)b[col * kBatch + j];
#pragma unroll
        for (int r = 0; r < kCoarseRows; ++r) s[u][r] = fma(__ldg(rowp[r] + col), bv, s[u][r]);
      }
    }
  }
#pragma unroll
  for (int u = 0; u < kPerLane; ++u)
#pragma unroll
    for (int r = 0; r < kCoarseRows; ++r) sh[warp * 4 + sub * kPerLane + u][r][j] = s[u][r];
  __syncthreads();
  for (int t = threadIdx.x; t < kCoarseRows * kBatch; t += kThreads) {
    const int r = t / kBatch, c = t % kBatch;
    if (r0 + r >= n) continue;
    double v = 0.0;
    for (int u = 0; u < kRuns; ++u) v += sh[u][r][c];
    x[(r0 + r) * kBatch + c] = (T)v;
  }
}

// ---------------------------------------------------------------------------------------
// batched PCG kernels (FP64 Krylov vectors: double case map)
// ---------------------------------------------------------------------------------------

// r = b, x = 0, rm = (TM) b (if rm), partC = b . b per case
template <typename TM>
__global__ void __launch_bounds__(kThreads) kb_init_vecs(int64_t n, const double* __restrict__ b,
                                                         double* __restrict__ x, double* __restrict__ r,
                                                         TM* __restrict__ rm, double* __restrict__ partC) {
  double dot[kC] = {};
  {
    BATCH_DOF_LOOP(n) {
      const int64_t o = i * kBatch;
      const C4<double> v = ldc<double>(b + o, l);
      stc<double>(r + o, l, v);
      stc<double>(x + o, l, C4<double>{});
      if (rm) stc<double>(rm + o, l, cvt4<TM>(v));
#pragma unroll
      for (int k = 0; k < kC; ++k) dot[k] = fma(v.v[k], v.v[k], dot[k]);
    }
  }
  write_case_parts<double>(dot, partC);
}

// per-case targets; cases with rtol_j >= 1 (already converged outside) or a zero right-hand
// side start finished
__global__ void kb_init_scalars(BlockScalars* S, const double* __restrict__ partC, int nparts,
                                const double* __restrict__ rtol, int max_iter) {
  const double bb = reduce_case_parts(partC, nparts);
  __shared__ int sdone[kBatch];
  if (threadIdx.x < kBatch) {
    const int j = threadIdx.x;
    const bool finite = isfinite(bb);
    S->bnorm2[j] = bb;
    S->tol2[j] = rtol[j] * rtol[j] * bb;
    S->rr[j] = bb;
    S->rz[j] = 0.0;
    S->alpha[j] = 0.0;
    S->beta[j] = 0.0;
    S->col_iters[j] = 0;
    S->col_status[j] = finite ? 0 : WN_EBREAKDOWN;
    const int d = (bb == 0.0 || !finite || rtol[j] >= 1.0) ? 1 : 0;
    S->col_done[j] = d;
    sdone[j] = d;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int all = 1;
    for (int j = 0; j < kBatch; ++j) all &= sdone[j];
    S->done = all;
    S->iters = 0;
    S->status = 0;
    S->max_iter = max_iter;
  }
}

// z = D^-1 r (jacobi) or z = r; partA = r . z per case
template <typename T>
__global__ void __launch_bounds__(kThreads) kb_prec_vec(int64_t n, const T* __restrict__ r,
                                                        const T* __restrict__ dinv, int jacobi, T* __restrict__ z,
                                                        double* __restrict__ partA, const int* __restrict__ done) {
  if (*done) return;
  double dot[kC] = {};
  {
    BATCH_DOF_LOOP(n) {
      const int64_t o = i * kBatch;
      const C4<T> rv = ldc<T>(r + o, l);
      const T di = jacobi ? dinv[i] : T(1);
      C4<T> zv;
#pragma unroll
      for (int k = 0; k < kC; ++k) {
        zv.v[k] = jacobi ? di * rv.v[k] : rv.v[k];
        dot[k] = fma((double)rv.v[k], (double)zv.v[k], dot[k]);
      }
      stc<T>(z + o, l, zv);
    }
  }
  write_case_parts<T>(dot, partA);
}

// rz_new = r . z (partA); beta = rz_new / rz (0 at the first iteration and for finished cases)
__global__ void kb_beta(BlockScalars* S, const double* __restrict__ partA, int nparts, int first) {
  if (S->done) return;
  const double rz_new = reduce_case_parts(partA, nparts);
  __shared__ int sdone[kBatch];
  if (threadIdx.x < kBatch) {
    const int j = threadIdx.x;
    int d = S->col_done[j];
    double beta = 0.0;
    if (!d) {
      if (!isfinite(rz_new)) {
        S->col_status[j] = WN_EBREAKDOWN;
        d = 1;
      } else if (!first) {
        const double rz = S->rz[j];
        beta = rz != 0.0 ? rz_new / rz : 0.0;
      }
    }
    S->rz[j] = rz_new;
    S->beta[j] = d ? 0.0 : beta;
    S->col_done[j] = d;
    sdone[j] = d;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int all = 1;
    for (int j = 0; j < kBatch; ++j) all &= sdone[j];
    S->done = all;
  }
}

// p_new = z + beta p_old; q = A p_new (fine matrix, component-major FP64); partB = p_new . q
template <typename TM>
__global__ void __launch_bounds__(kThreads, (kRowCtas<double, 9>))
    kb_spmv_dot(int64_t n_rows, const int32_t* __restrict__ order, const int32_t* __restrict__ rp,
                                                        const int32_t* __restrict__ ci, const double* __restrict__ av,
                                                        int64_t stride, const TM* __restrict__ z,
                                                        const double* __restrict__ p_old, double* __restrict__ p_new,
                                                        double* __restrict__ q, double* __restrict__ partB,
                                                        const BlockScalars* __restrict__ S) {
  if (S->done) return;
  double dot[kC] = {};
  {
    BATCH_ROW_LOOP(n_rows, order) {
      const BPNew<TM> pf{z, p_old, case_scalars<double>(S->beta, l)};
      double acc[3][kC];
      batch_row_staged<3, 3, kSoA, Tpg<double, 3>::value, 1, double>(rp, ci, av, stride, row, row < n_rows, l, pf,
                                                               FmaAcc<3, double>(acc));
      if (row >= n_rows) continue;
#pragma unroll
      for (int rr = 0; rr < 3; ++rr) {
        const int64_t i = row * 3 + rr;
        const int64_t o = i * kBatch;
        const C4<double> pv = pf(i, l);
        C4<double> qv;
#pragma unroll
        for (int k = 0; k < kC; ++k) {
          qv.v[k] = acc[rr][k];
          dot[k] = fma(pv.v[k], qv.v[k], dot[k]);
        }
        stc<double>(p_new + o, l, pv);
        stc<double>(q + o, l, qv);
      }
    }
  }
  write_case_parts<double>(dot, partB);
}

// The mixed batch (FP32 V-cycle) keeps its search directions in FP32: p = z + beta p is formed
// once per iteration in FP64 and rounded (kb_pnew32), and the product gathers those FP32
// values (12 bytes per column DOF and case pair instead of the 8-byte p and 4-byte z of the
// fused kb_spmv_dot) into FP64 sums with the FP64 matrix.  x is updated with the same rounded p
// whose product gave q, so r = b - A x still holds to FP64 rounding; only the A-conjugacy of the
// directions carries the FP32 rounding (on the I-beam the iteration counts did not change).
template <typename TM>
__global__ void __launch_bounds__(kThreads) kb_pnew32(int64_t n, const TM* __restrict__ z, float* __restrict__ p,
                                                      const BlockScalars* __restrict__ S) {
  if (S->done) return;
  const int l0 = threadIdx.x & 7;
  const C4<double> b = case_scalars<float>(S->beta, l0);
  BATCH_DOF_LOOP(n) {
    const int64_t o = i * kBatch;
    const C4<double> zz = cvt4<double>(ldc<float>(z + o, l));
    const C4<float> pp = ldc<float>(p + o, l);
    C4<float> pn;
#pragma unroll
    for (int k = 0; k < kC; ++k) pn.v[k] = (float)fma(b.v[k], (double)pp.v[k], zz.v[k]);
    stc<float>(p + o, l, pn);
  }
}

// q = A p (fine matrix, component-major FP64; p FP32, widened by FmaAcc); partB = p . q.  The case map
// is the FP32 one: a gathered case row is then one 128-byte line per load of an 8-lane group (with
// the FP64 map two loads of half a line each, 36 L1 wavefronts per 4 blocks instead of 12).
__global__ void __launch_bounds__(kThreads, (kRowCtas<double, 9>))
    kb_spmv_dot32(int64_t n_rows, const int32_t* __restrict__ order, const int32_t* __restrict__ rp,
                                                          const int32_t* __restrict__ ci,
                                                          const double* __restrict__ av, int64_t stride,
                                                          const float* __restrict__ p, double* __restrict__ q,
                                                          double* __restrict__ partB,
                                                          const BlockScalars* __restrict__ S) {
  if (S->done) return;
  double dot[kC] = {};
  {
    BATCH_ROW_LOOP(n_rows, order) {
      const BLoad<float, float> pf{p};
      double acc[3][kC];
      batch_row_staged<3, 3, kSoA, Tpg<float, 3>::value, 1, double>(rp, ci, av, stride, row, row < n_rows, l, pf,
                                                              FmaAcc<3, double>(acc));
      if (row >= n_rows) continue;
#pragma unroll
      for (int rr = 0; rr < 3; ++rr) {
        const int64_t i = row * 3 + rr;
        const C4<double> pv = cvt4<double>(pf(i, l));
        C4<double> qv;
#pragma unroll
        for (int k = 0; k < kC; ++k) {
          qv.v[k] = acc[rr][k];
          dot[k] = fma(pv.v[k], qv.v[k], dot[k]);
        }
        stc<float>(q + i * kBatch, l, qv);
      }
    }
  }
  write_case_parts<float>(dot, partB);
}

// alpha = rz / (p . q) for the running cases; a non-positive curvature ends that case
__global__ void kb_alpha(BlockScalars* S, const double* __restrict__ partB, int nparts) {
  if (S->done) return;
  const double gamma = reduce_case_parts(partB, nparts);
  if (threadIdx.x < kBatch) {
    const int j = threadIdx.x;
    double alpha = 0.0;
    if (!S->col_done[j]) {
      alpha = S->rz[j] / gamma;
      if (!(gamma > 0.0) || !isfinite(alpha)) {
        S->col_status[j] = WN_EBREAKDOWN;
        S->col_done[j] = 1;
        alpha = 0.0;
      }
    }
    S->alpha[j] = alpha;
  }
}

// x += alpha p; r -= alpha q; rm = (TM) r (if rm); partC = r . r per case (p: FP64, or the mixed
// batch's FP32 search directions, widened)
template <typename TM, typename TP = double>
__global__ void __launch_bounds__(kThreads) kb_update(int64_t n, double* __restrict__ x, double* __restrict__ r,
                                                      TM* __restrict__ rm, const TP* __restrict__ p,
                                                      const double* __restrict__ q, double* __restrict__ partC,
                                                      const BlockScalars* __restrict__ S, TM* __restrict__ d0,
                                                      const TM* __restrict__ dinv, TM inv_theta) {
  if (S->done) return;
  double dot[kC] = {};
  {
    const int l0 = threadIdx.x & 7;
    const C4<double> a = case_scalars<double>(S->alpha, l0);
    BATCH_DOF_LOOP(n) {
      const int64_t o = i * kBatch;
      C4<double> xv = ldc<double>(x + o, l), rv = ldc<double>(r + o, l);
      const C4<double> pv = cvt4<double>(ldc<double>(p + o, l)), qv = ldc<double>(q + o, l);
#pragma unroll
      for (int k = 0; k < kC; ++k) {
        if (a.v[k] != 0.0) {  // finished cases keep x and r exactly (their p may be anything)
          xv.v[k] = fma(a.v[k], pv.v[k], xv.v[k]);
          rv.v[k] = fma(-a.v[k], qv.v[k], rv.v[k]);
        }
        dot[k] = fma(rv.v[k], rv.v[k], dot[k]);
      }
      stc<double>(x + o, l, xv);
      stc<double>(r + o, l, rv);
      const C4<TM> rt = cvt4<TM>(rv);
      if (rm) stc<double>(rm + o, l, rt);
      if (d0) {  // the V-cycle's first smoothing input, BD0's expression on the same values
        const TM di = dinv[i];
        C4<TM> dv;
#pragma unroll
        for (int k = 0; k < kC; ++k) dv.v[k] = di * rt.v[k] * inv_theta;
        stc<double>(d0 + o, l, dv);
      }
    }
  }
  write_case_parts<double>(dot, partC);
}

// convergence test of every running case; the batch ends when all cases are finished or
// the iteration limit is reached (the unfinished cases then report WN_ENOCONV)
__global__ void kb_check(BlockScalars* S, const double* __restrict__ partC, int nparts) {
  if (S->done) return;
  const double rr = reduce_case_parts(partC, nparts);
  __shared__ int sdone[kBatch];
  const int it = S->iters + 1;
  if (threadIdx.x < kBatch) {
    const int j = threadIdx.x;
    int d = S->col_done[j];
    if (!d) {
      S->rr[j] = rr;
      S->col_iters[j] += 1;
      if (!isfinite(rr)) {
        S->col_status[j] = WN_EBREAKDOWN;
        d = 1;
      } else if (rr <= S->tol2[j]) {
        d = 1;
      } else if (it >= S->max_iter) {
        S->col_status[j] = WN_ENOCONV;
      }
    }
    S->col_done[j] = d;
    sdone[j] = d;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int all = 1;
    for (int j = 0; j < kBatch; ++j) all &= sdone[j];
    S->iters = it;
    if (!all && it >= S->max_iter) {
      S->status = WN_ENOCONV;
      all = 1;
    }
    S->done = all;
  }
}

// ---------------------------------------------------------------------------------------
// extra-precise refinement: U = U_hi + U_lo (double-double), R = F - K U with compensated
// products and sums
// ---------------------------------------------------------------------------------------
// (two_sum / two_prod: error-free transformations, eft.cuh)
struct DD4 {
  C4<double> hi, lo;
};
template <typename M>
struct DDLoad {
  const double* __restrict__ hi;
  const double* __restrict__ lo;
  __device__ __forceinline__ DD4 operator()(int64_t i, int l) const {
    return {ldc<M>(hi + i * kBatch, l), ldc<M>(lo + i * kBatch, l)};
  }
};
// compensated accumulation (Dot2 of Ogita-Rump-Oishi): s + c carries about twice the FP64
// precision of a plain sum of a (x_hi + x_lo)
template <int BR>
struct DdAcc {
  double (&s)[BR][kC];
  double (&c)[BR][kC];
  __device__ __forceinline__ DdAcc(double (&s_)[BR][kC], double (&c_)[BR][kC]) : s(s_), c(c_) {
#pragma unroll
    for (int r = 0; r < BR; ++r)
#pragma unroll
      for (int k = 0; k < kC; ++k) s[r][k] = c[r][k] = 0.0;
  }
  __device__ __forceinline__ void operator()(int r, double a, const DD4& x) const {
#pragma unroll
    for (int k = 0; k < kC; ++k) {
      double p, ep, t, es;
      two_prod(a, x.hi.v[k], p, ep);
      two_sum(s[r][k], p, t, es);
      s[r][k] = t;
      c[r][k] += fma(a, x.lo.v[k], ep + es);
    }
  }
};

// R = F - K (U_hi + U_lo), rounded to FP64 from the compensated sum; partC = R . R per case
__global__ void __launch_bounds__(kThreads, (kRowCtas<double, 9>))
    kb_outer_residual(int64_t n_rows, const int32_t* __restrict__ order, const int32_t* __restrict__ rp,
                                                              const int32_t* __restrict__ ci,
                                                              const double* __restrict__ av, int64_t stride,
                                                              const double* __restrict__ F,
                                                              const double* __restrict__ Uhi,
                                                              const double* __restrict__ Ulo, double* __restrict__ R,
                                                              double* __restrict__ partC) {
  double dot[kC] = {};
  {
    BATCH_ROW_LOOP(n_rows, order) {
      double s[3][kC], c[3][kC];
      batch_row_staged<3, 3, kSoA, 1, 1, double>(rp, ci, av, stride, row, row < n_rows, l,
                                              DDLoad<double>{Uhi, Ulo}, DdAcc<3>(s, c));
      if (row >= n_rows) continue;
#pragma unroll
      for (int rr = 0; rr < 3; ++rr) {
        const int64_t o = (row * 3 + rr) * kBatch;
        const C4<double> fv = ldc<double>(F + o, l);
        C4<double> rv;
#pragma unroll
        for (int k = 0; k < kC; ++k) {
          double t, e;
          two_sum(fv.v[k], -s[rr][k], t, e);
          rv.v[k] = t + (e - c[rr][k]);
          dot[k] = fma(rv.v[k], rv.v[k], dot[k]);
        }
        stc<double>(R + o, l, rv);
      }
    }
  }
  write_case_parts<double>(dot, partC);
}

// (U_hi, U_lo) += X, renormalised so that U_hi = fl(U_hi + U_lo)
__global__ void kb_accumulate(int64_t n, double* __restrict__ Uhi, double* __restrict__ Ulo,
                              const double* __restrict__ X) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n * kBatch;
       i += (int64_t)gridDim.x * blockDim.x) {
    double s, e, h, g;
    two_sum(Uhi[i], X[i], s, e);
    two_sum(s, __dadd_rn(Ulo[i], e), h, g);
    Uhi[i] = h;
    Ulo[i] = g;
  }
}

// part = a . b per case (the r . z of a hierarchy that is only its coarsest level)
template <typename T>
__global__ void __launch_bounds__(kThreads) kb_dot_pair(int64_t n, const T* __restrict__ a, const T* __restrict__ b,
                                                        double* __restrict__ part, const int* __restrict__ done) {
  if (*done) return;
  double dot[kC] = {};
  {
    BATCH_DOF_LOOP(n) {
      const C4<T> av = ldc<T>(a + i * kBatch, l), bv = ldc<T>(b + i * kBatch, l);
#pragma unroll
      for (int k = 0; k < kC; ++k) dot[k] = fma((double)av.v[k], (double)bv.v[k], dot[k]);
    }
  }
  write_case_parts<T>(dot, part);
}

// partC = x . x per case
__global__ void __launch_bounds__(kThreads) kb_dot_self(int64_t n, const double* __restrict__ x,
                                                        double* __restrict__ partC) {
  double dot[kC] = {};
  {
    BATCH_DOF_LOOP(n) {
      const C4<double> v = ldc<double>(x + i * kBatch, l);
#pragma unroll
      for (int k = 0; k < kC; ++k) dot[k] = fma(v.v[k], v.v[k], dot[k]);
    }
  }
  write_case_parts<double>(dot, partC);
}

// S->rr[j] = sum of partC (one CTA)
__global__ void kb_reduce_rr(BlockScalars* S, const double* __restrict__ partC, int nparts) {
  const double rr = reduce_case_parts(partC, nparts);
  if (threadIdx.x < kBatch) S->rr[threadIdx.x] = rr;
}

// pack columns [j0, j0 + m) of a row-major n x ld matrix into the n x kBatch batch (zero
// padding), and back
__global__ void kb_pack(int64_t n, const double* __restrict__ src, int64_t ld, int64_t j0, int m,
                        double* __restrict__ dst) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n * kBatch;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = i / kBatch;
    const int j = (int)(i - row * kBatch);
    dst[i] = j < m ? src[row * ld + j0 + j] : 0.0;
  }
}
__global__ void kb_unpack(int64_t n, const double* __restrict__ src, int64_t ld, int64_t j0, int m,
                          double* __restrict__ dst) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n * kBatch;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = i / kBatch;
    const int j = (int)(i - row * kBatch);
    if (j < m) dst[row * ld + j0 + j] = src[i];
  }
}

// 1 / diag of the fine matrix (component-major values), the rule of solid_solver.py:230
__global__ void kb_fill_dinv(int64_t n_rows, int64_t nnzb, const int32_t* __restrict__ diag_block,
                             const double* __restrict__ k64, double* __restrict__ d64, float* __restrict__ d32) {
  for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n_rows * 3;
       t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t row = t / 3;
    const int c = (int)(t - row * 3);
    const double dv = k64[(int64_t)(c * 4) * nnzb + diag_block[row]];
    const double inv = (fabs(dv) > 1e-12) ? 1.0 / dv : 1.0;
    d64[t] = inv;
    d32[t] = (float)inv;
  }
}

// ---------------------------------------------------------------------------------------
// host orchestration
// ---------------------------------------------------------------------------------------
inline int rows_work(int64_t n_rows) { return (int)((n_rows * (32 / kRowsPerWarp) + kThreads - 1) / kThreads); }
inline int quads_work(int64_t n) { return (int)((n * 8 + kThreads - 1) / kThreads); }

template <typename T>
struct BPrec;
template <>
struct BPrec<float> {
  static const float* A0(Solid* s) { return s->k32.p; }
  static const float* Av(DevLevel& L) { return L.A.v32.p; }
  static const float* Pv(DevLevel& L) { return L.P.v32.p; }
  static const float* Rv(DevLevel& L) { return L.R.v32.p; }
  static const float* dinv(DevLevel& L) { return L.dinv32.p; }
  static BatchLevelVecs<float>& lv(BlockWork& W, int l) { return W.lv32[l]; }
  static float* cb(BlockWork& W) { return W.cb32.p; }
  static float* cx(BlockWork& W) { return W.cx32.p; }
  static const float* fine_dinv(BlockWork& W) { return W.dinv32.p; }
  static float* z(BlockWork& W) { return W.z32.p; }
  static float* rm(BlockWork& W) { return W.r32.p; }  // r in FP32 for the V-cycle
  static float* d0(BlockWork& W) { return W.d0_32.p; }
};
template <>
struct BPrec<double> {
  static const double* A0(Solid* s) { return s->k64.p; }
  static const double* Av(DevLevel& L) { return L.A.v64.p; }
  static const double* Pv(DevLevel& L) { return L.P.v64.p; }
  static const double* Rv(DevLevel& L) { return L.R.v64.p; }
  static const double* dinv(DevLevel& L) { return L.dinv64.p; }
  static BatchLevelVecs<double>& lv(BlockWork& W, int l) { return W.lv64[l]; }
  static double* cb(BlockWork& W) { return W.cb64.p; }
  static double* cx(BlockWork& W) { return W.cx64.p; }
  static const double* fine_dinv(BlockWork& W) { return W.dinv64.p; }
  static double* z(BlockWork& W) { return W.z64.p; }
  static double* rm(BlockWork&) { return nullptr; }  // the V-cycle reads the FP64 r directly
  static double* d0(BlockWork& W) { return W.d0_64.p; }
};

// long rows (>= 4 stages of 8 blocks on average) are shared by the 4 groups of a warp
template <int BR, int BC, typename T>
void batch_level_spmv(const DevBsr& M, const int32_t* order, const T* vals, const T* x, T* y, int accumulate,
                      const int* done, cudaStream_t st) {
  const bool team = M.n_rows > 0 && M.nnzb >= 32 * M.n_rows;
  if (team) {
    auto k = kb_level_spmv<BR, BC, T, 4>;
    k<<<row_grid<T, BR * BC>(rows_work(M.n_rows * 4)), kThreads, 0, st>>>(M.n_rows, order, M.rp.p, M.ci.p, vals, x,
                                                                                y, accumulate, done);
  } else {
    auto k = kb_level_spmv<BR, BC, T, 1>;
    k<<<row_grid<T, BR * BC>(rows_work(M.n_rows)), kThreads, 0, st>>>(M.n_rows, order, M.rp.p, M.ci.p, vals, x, y,
                                                                            accumulate, done);
  }
}

// one batched V-cycle at level lvl: out = V(b); part (if set) receives b . out per case
template <typename T>
int batch_vcycle(Solid* s, AmgHierarchy& H, BlockWork& W, int lvl, const T* b, T* out, double* part,
                 BlockScalars* S, cudaStream_t st, const T* d0 = nullptr) {
  const int* done = &S->done;
  const int nlev = (int)H.levels.size();
  if (lvl == nlev) {
    kb_coarse<T><<<(unsigned)((H.n_coarse + kCoarseRows - 1) / kCoarseRows), kThreads, 0, st>>>(
        H.n_coarse, H.coarse_inv.p, b, out, done);
    W.launches++;
    if (part) {  // a hierarchy without levels: the PCG's r . z comes from here
      const int g = part_grid(quads_work(H.n_coarse), kDofGrid);
      W.npA = g;
      kb_dot_pair<T><<<g, kThreads, 0, st>>>(H.n_coarse, b, out, part, done);
      W.launches++;
    }
    WN_CUDA(cudaGetLastError());
    return 0;
  }
  DevLevel& L = H.levels[lvl];
  BatchLevelVecs<T>& V = BPrec<T>::lv(W, lvl);
  const int64_t nr = L.n_nodes;
  const T* dinv = (lvl == 0) ? BPrec<T>::fine_dinv(W) : BPrec<T>::dinv(L);
  const int deg = H.degree;
  const T it = (T)L.inv_theta;
  const int64_t sd = (lvl == 0) ? s->nnzb : 0;
  auto run = [&](auto bs_tag) -> int {
    constexpr int BS = decltype(bs_tag)::value;
    constexpr int SG = (BS == 3) ? 1 : 4;  // coarse 6x6 levels: rows of ~50-250 blocks, one warp each
    const int work = rows_work(nr * SG);
    auto rg = [&](auto) { return row_grid<T, BS * BS>(work); };
    const int32_t* order = lvl == 0 ? s->batch->order[kRowCtas<T, 9> - 2].p : nullptr;
    const int32_t* rp = lvl == 0 ? s->row_ptr.p : L.A.rp.p;
    const int32_t* ci = lvl == 0 ? s->col_idx.p : L.A.ci.p;
    const T* av = lvl == 0 ? BPrec<T>::A0(s) : BPrec<T>::Av(L);
    const T c1 = deg >= 2 ? (T)L.c1[0] : T(0), c2 = deg >= 2 ? (T)L.c2[0] : T(0);
    // the fine level streams its matrix from the tile-major pack when it has one
    const bool fine_stream = lvl == 0 && BS == 3 && s->fine.packed && s->stream_batched;
    const BView fv = bview<T>(s->fine);
    // the fine level: streamed from the pack when batched streaming is on, else with each
    // tile's x slice staged in shared memory (when the plan exists), else the register kernels
    auto streamed = [&](auto xf, auto epi, double* part_out) -> int {
      if constexpr (kBatch == 32) {  // the dispatcher takes the widest batch for these paths
        int g = fine_stream ? launch_bs<T>(kbs_rows<T, decltype(xf), decltype(epi)>, s->fine, st, fv, xf, epi,
                                           part_out, S)
                            : 0;
        if (g == 0 && lvl == 0 && BS == 3) g = launch_bx<T>(s, W, av, xf, epi, part_out, done, st);
        return g;
      } else {
        return 0;
      }
    };
    // the first step's x: dinv b / theta, read from d0 when the PCG update wrote it
    const BEpiPreFirst<T> epf{b, dinv, it, deg, c1, c2, V.x.p, V.r.p, V.d.p, V.res.p};
    if (d0 && lvl == 0) {
      if (!streamed(BLoad<T, T>{d0}, epf, nullptr)) {
        auto k = kb_pre_first<BS, T, SG, BLoad<T, T>>;
        k<<<rg(k), kThreads, 0, st>>>(nr, order, rp, ci, av, sd, BLoad<T, T>{d0}, b, dinv, it, deg, c1, c2, V.x.p, V.r.p,
                                      V.d.p, V.res.p, done);
      }
    } else if (!streamed(BD0<T, T>{b, dinv, it}, epf, nullptr)) {
      auto k = kb_pre_first<BS, T, SG, BD0<T, T>>;
      k<<<rg(k), kThreads, 0, st>>>(nr, order, rp, ci, av, sd, BD0<T, T>{b, dinv, it}, b, dinv, it, deg, c1, c2, V.x.p,
                                    V.r.p, V.d.p, V.res.p, done);
    }
    W.launches++;
    T* din = V.d.p;
    T* dout = V.d2.p;
    for (int k = 2; k < deg; ++k) {
      const T ck1 = (T)L.c1[k - 1], ck2 = (T)L.c2[k - 1];
      if (!streamed(BLoad<T, T>{din}, BEpiCheb<T>{dinv, din, dout, V.r.p, V.x.p, ck1, ck2, b, 0}, nullptr))
        kb_cheb_step<BS, T, SG><<<rg(kb_cheb_step<BS, T, SG>), kThreads, 0, st>>>(nr, order, rp, ci, av, sd, dinv, din, dout,
                                                                          V.r.p, V.x.p, ck1, ck2, b, nullptr, done);
      W.launches++;
      std::swap(din, dout);
    }
    if (deg >= 2) {
      if (!streamed(BLoad<T, T>{V.x.p}, BEpiResidual<T>{b, V.res.p}, nullptr))
        kb_residual<BS, T, SG><<<rg(kb_residual<BS, T, SG>), kThreads, 0, st>>>(nr, order, rp, ci, av, sd, b, V.x.p, V.res.p,
                                                                         done);
      W.launches++;
    }
    const bool last = lvl + 1 >= nlev;
    T* bc = last ? BPrec<T>::cb(W) : BPrec<T>::lv(W, lvl + 1).b.p;
    T* xc = last ? BPrec<T>::cx(W) : BPrec<T>::lv(W, lvl + 1).x2.p;
    batch_level_spmv<6, BS, T>(L.R, nullptr, BPrec<T>::Rv(L), V.res.p, bc, 0, done, st);
    W.launches++;
    WN_CHECK(batch_vcycle<T>(s, H, W, lvl + 1, bc, xc, nullptr, S, st));
    batch_level_spmv<BS, 6, T>(L.P, nullptr, BPrec<T>::Pv(L), xc, V.x.p, 1, done, st);
    W.launches++;
    double* part_last = (deg == 1) ? part : nullptr;
    T* r_post = deg == 1 ? nullptr : V.r.p;
    int gpf = streamed(BLoad<T, T>{V.x.p},
                       BEpiPostFirst<T>{b, dinv, it, V.x.p, out, r_post, V.d.p, part_last != nullptr}, part_last);
    if (gpf == 0) {
      gpf = rg(kb_post_first<BS, T, SG>);
      kb_post_first<BS, T, SG><<<gpf, kThreads, 0, st>>>(nr, order, rp, ci, av, sd, b, dinv, it, V.x.p, out, r_post, V.d.p,
                                                          part_last, done);
    }
    if (part_last) W.npA = gpf;
    W.launches++;
    din = V.d.p;
    dout = V.d2.p;
    for (int k = 1; k < deg; ++k) {
      double* pk = (k == deg - 1) ? part : nullptr;
      const T ck1 = (T)L.c1[k - 1], ck2 = (T)L.c2[k - 1];
      int gcs = streamed(BLoad<T, T>{din}, BEpiCheb<T>{dinv, din, dout, V.r.p, out, ck1, ck2, b, pk != nullptr},
                         pk);
      if (gcs == 0) {
        gcs = rg(kb_cheb_step<BS, T, SG>);
        kb_cheb_step<BS, T, SG><<<gcs, kThreads, 0, st>>>(nr, order, rp, ci, av, sd, dinv, din, dout, V.r.p, out, ck1, ck2, b,
                                                      pk, done);
      }
      if (pk) W.npA = gcs;
      W.launches++;
      std::swap(din, dout);
    }
    return 0;
  };
  WN_CHECK(L.bs == 3 ? run(std::integral_constant<int, 3>{}) : run(std::integral_constant<int, 6>{}));
  WN_CUDA(cudaGetLastError());
  return 0;
}

// z = M r for all cases, partA = r . z per case
template <typename TM>
int batch_prec(Solid* s, BlockWork& W, int precond, const TM* r, TM* z, BlockScalars* S, cudaStream_t st,
               const TM* d0 = nullptr) {
  const int* done = &S->done;
  if (precond == 2) return batch_vcycle<TM>(s, *s->amg, W, 0, r, z, W.partA.p, S, st, d0);
  const int g = part_grid(quads_work(W.n), kDofGrid);
  W.npA = g;
  kb_prec_vec<TM><<<g, kThreads, 0, st>>>(W.n, r, BPrec<TM>::fine_dinv(W), precond == 1 ? 1 : 0, z, W.partA.p,
                                          done);
  W.launches++;
  WN_CUDA(cudaGetLastError());
  return 0;
}

template <typename TM>
const TM* prec_input(BlockWork& W) {
  if constexpr (std::is_same<TM, double>::value)
    return W.r.p;
  else
    return W.r32.p;
}

// FP32 search directions (kb_pnew32 / kb_spmv_dot32): the mixed batch on the register fine
// level; the FP64 batch and the streamed fine level keep FP64 directions
template <typename TM>
bool fp32_directions(const Solid* s) {
  return std::is_same<TM, float>::value && !s->stream_batched;
}

// one batched PCG iteration (parity k & 1 selects the p buffers)
template <typename TM>
int batch_iteration(Solid* s, BlockWork& W, int precond, int k, BlockScalars* S, cudaStream_t st) {
  const int par = k & 1;
  double* p_new = par ? W.p1.p : W.p0.p;
  double* p_old = par ? W.p0.p : W.p1.p;
  const bool p32 = fp32_directions<TM>(s);
  float* p_f = reinterpret_cast<float*>(W.p0.p);  // the FP32 directions, in place
  // the fine FP64 matrix streamed from its pack when batched streaming is on, else the
  // register kernel
  int gsd = 0;
  if constexpr (kBatch == 32) {
    if (s->stream_batched && !p32)
      gsd = launch_bs<double>(kbs_spmv_dot<TM>, s->fine, st, bview<double>(s->fine), (const TM*)BPrec<TM>::z(W),
                              (const double*)p_old, p_new, W.q.p, W.partB.p, S);
  }
  if (p32) {
    kb_pnew32<TM><<<part_grid(quads_work(W.n), kDofGrid), kThreads, 0, st>>>(
        W.n, BPrec<TM>::z(W), p_f, S);
    gsd = row_grid<double, 9>(rows_work(s->n_nodes));
    kb_spmv_dot32<<<gsd, kThreads, 0, st>>>(s->n_nodes, s->batch->order[kRowCtas<double, 9> - 2].p, s->row_ptr.p, s->col_idx.p, s->k64.p, s->nnzb, p_f, W.q.p,
                                            W.partB.p, S);
    W.launches++;
  } else if (gsd == 0) {
    gsd = row_grid<double, 9>(rows_work(s->n_nodes));
    kb_spmv_dot<TM><<<gsd, kThreads, 0, st>>>(s->n_nodes, s->batch->order[kRowCtas<double, 9> - 2].p, s->row_ptr.p, s->col_idx.p, s->k64.p, s->nnzb,
                                              BPrec<TM>::z(W), p_old, p_new, W.q.p, W.partB.p, S);
  }
  W.npB = gsd;
  kb_alpha<<<1, kScalarThreads, 0, st>>>(S, W.partB.p, W.npB);
  // with the AMG preconditioner the update also writes the V-cycle's first smoothing input
  TM* d0 = (precond == 2 && s->amg && !s->amg->levels.empty()) ? BPrec<TM>::d0(W) : nullptr;
  const TM it0 = d0 ? (TM)s->amg->levels[0].inv_theta : TM(0);
  const int gup = part_grid(quads_work(W.n), kDofGrid);
  if (p32)
    kb_update<TM, float><<<gup, kThreads, 0, st>>>(W.n, W.x.p, W.r.p, BPrec<TM>::rm(W), p_f, W.q.p, W.partC.p, S,
                                                   d0, BPrec<TM>::fine_dinv(W), it0);
  else
    kb_update<TM><<<gup, kThreads, 0, st>>>(W.n, W.x.p, W.r.p, BPrec<TM>::rm(W), p_new, W.q.p, W.partC.p, S, d0,
                                            BPrec<TM>::fine_dinv(W), it0);
  W.npC = gup;
  kb_check<<<1, kScalarThreads, 0, st>>>(S, W.partC.p, W.npC);
  W.launches += 4;
  WN_CUDA(cudaGetLastError());
  WN_CHECK(batch_prec<TM>(s, W, precond, prec_input<TM>(W), BPrec<TM>::z(W), S, st, d0));
  kb_beta<<<1, kScalarThreads, 0, st>>>(S, W.partA.p, W.npA, 0);
  W.launches++;
  WN_CUDA(cudaGetLastError());
  return 0;
}

// batched PCG on b (n x kBatch) from x = 0 with the per-case targets in W.rtol_cols
template <typename TM>
int batch_pcg(Solid* s, BlockWork& W, int vmode, const double* b, int max_iter, int precond, int chunk,
              int use_graph, BlockScalars* S, cudaStream_t st, BlockScalars* hS) {
  // first iteration: p = z + 0 * p_old
  const size_t vb = (size_t)W.n * kBatch * (fp32_directions<TM>(s) ? sizeof(float) : sizeof(double));
  WN_CUDA(cudaMemsetAsync(W.p0.p, 0, vb, st));
  if (!fp32_directions<TM>(s)) WN_CUDA(cudaMemsetAsync(W.p1.p, 0, vb, st));
  W.npC = part_grid(quads_work(W.n), kDofGrid);
  kb_init_vecs<TM><<<W.npC, kThreads, 0, st>>>(W.n, b, W.x.p, W.r.p, BPrec<TM>::rm(W), W.partC.p);
  kb_init_scalars<<<1, kScalarThreads, 0, st>>>(S, W.partC.p, W.npC, W.rtol_cols.p, max_iter);
  W.launches += 2;
  WN_CUDA(cudaGetLastError());
  WN_CHECK(batch_prec<TM>(s, W, precond, prec_input<TM>(W), BPrec<TM>::z(W), S, st));
  kb_beta<<<1, kScalarThreads, 0, st>>>(S, W.partA.p, W.npA, 1);
  W.launches++;
  chunk = std::max(2, chunk + (chunk & 1));  // even: the parity pattern repeats per chunk
  GraphCache& G = W.graphs[vmode][precond];
  const int64_t key = chunk;
  int k0 = 0;
  while (true) {
    WN_CUDA(cudaMemcpyAsync(hS, S, sizeof(BlockScalars), cudaMemcpyDeviceToHost, st));
    WN_CUDA(cudaStreamSynchronize(st));
    if (hS->done || k0 >= max_iter) break;
    if (use_graph) {
      if (G.key != key || G.stream != st || !G.exec || G.fine_epoch != s->fine.epoch) {
        G.reset();
        cudaGraph_t graph;
        const int64_t before = W.launches;
        WN_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        int rc = 0;
        for (int k = 0; k < chunk && rc == 0; ++k) rc = batch_iteration<TM>(s, W, precond, k, S, st);
        cudaError_t e = cudaStreamEndCapture(st, &graph);
        WN_CHECK(rc);
        WN_CUDA(e);
        e = cudaGraphInstantiate(&G.exec, graph, 0);
        cudaGraphDestroy(graph);
        WN_CUDA(e);
        G.key = key;
        G.stream = st;
        G.fine_epoch = s->fine.epoch;
        G.kernels = W.launches - before;
        W.launches = before;
      }
      WN_CUDA(cudaGraphLaunch(G.exec, st));
      W.launches += G.kernels;
    } else {
      for (int k = 0; k < chunk; ++k) WN_CHECK(batch_iteration<TM>(s, W, precond, k0 + k, S, st));
    }
    k0 += chunk;
  }
  return 0;
}

// the set's workspace of this width
BlockWork* block_work(BlockSet& B) {
  std::unique_ptr<BlockWork>& w = B.width<kBatch>();
  if (!w) w.reset(new BlockWork());
  return w.get();
}

int ensure_block_work(Solid* s, int vmode, int precond) {
  BlockWork& W = *block_work(*s->batch);
  BatchStore& M = s->batch->store;
  const int64_t n = s->n_nodes * 3, nb = n * kBatch;
  const int64_t np = (int64_t)BlockWork::kMaxParts * kBatch;
  if (precond == 2 && M.hierarchy_id != s->amg->id) {
    M.release_from(kVecHierarchy);
    M.hierarchy_id = s->amg->id;
  }
  W.n = n;
  WN_CHECK(W.partA.take(M, kVecPartA, np));
  WN_CHECK(W.partB.take(M, kVecPartB, np));
  WN_CHECK(W.partC.take(M, kVecPartC, np));
  WN_CHECK(W.F.take(M, kVecF, nb));
  WN_CHECK(W.U.take(M, kVecU, nb));
  WN_CHECK(W.Ulo.take(M, kVecUlo, nb));
  WN_CHECK(W.R.take(M, kVecR, nb));
  WN_CHECK(W.x.take(M, kVecX, nb));
  WN_CHECK(W.r.take(M, kVecRes, nb));
  WN_CHECK(W.q.take(M, kVecQ, nb));
  WN_CHECK(W.dinv64.take(M, kVecDinv64, n));
  WN_CHECK(W.dinv32.take(M, kVecDinv32, n));
  // search directions: one FP32 vector in place, or two FP64 ones
  const bool p32 = vmode == 1 && fp32_directions<float>(s);
  WN_CHECK(W.p0.take(M, kVecP0, p32 ? (nb + 1) / 2 : nb));
  if (!p32) WN_CHECK(W.p1.take(M, kVecP1, nb));
  if (vmode == 1) {
    WN_CHECK(W.z32.take(M, kVecZ32, nb));
    WN_CHECK(W.r32.take(M, kVecR32, nb));
    if (precond == 2) WN_CHECK(W.d0_32.take(M, kVecD32, nb));
  } else {
    WN_CHECK(W.z64.take(M, kVecZ64, nb));
    if (precond == 2) WN_CHECK(W.d0_64.take(M, kVecD64, nb));
  }
  WN_CHECK(W.scal.alloc(2));
  WN_CHECK(W.rtol_cols.alloc(kBatch));
  W.h_rtol.assign(kBatch, 1.0);
  if (precond == 2) {
    AmgHierarchy& H = *s->amg;
    const size_t nl = H.levels.size();
    auto levels = [&](auto& lv, auto& cb, auto& cx, int id) -> int {
      lv.resize(nl);
      for (size_t l = 0; l < nl; ++l)
        WN_CHECK(lv[l].take(M, (int)l, H.levels[l].n_nodes * H.levels[l].bs * kBatch, H.degree));
      WN_CHECK(cb.take(M, id, H.n_coarse * kBatch));
      return cx.take(M, id + 1, H.n_coarse * kBatch);
    };
    WN_CHECK(vmode == 1 ? levels(W.lv32, W.cb32, W.cx32, kVecCb32) : levels(W.lv64, W.cb64, W.cx64, kVecCb64));
  }
  if (W.epoch != M.epoch) {  // some vector has moved since the graphs were captured
    W.epoch = M.epoch;
    for (auto& a : W.graphs)
      for (auto& g : a) g.reset();
  }
  if (kBatch == 32 && s->batch_stage_x && !W.xt_tried) WN_CHECK(build_x_tiles(s, W));
  return 0;
}

// per-case norms of an n x kBatch FP64 vector into host rr[]
int case_norms2(BlockWork& W, const double* v, BlockScalars* S1, cudaStream_t st, BlockScalars* hS) {
  W.npC = part_grid(quads_work(W.n), kDofGrid);
  kb_dot_self<<<W.npC, kThreads, 0, st>>>(W.n, v, W.partC.p);
  kb_reduce_rr<<<1, kScalarThreads, 0, st>>>(S1, W.partC.p, W.npC);
  W.launches += 2;
  WN_CUDA(cudaGetLastError());
  WN_CUDA(cudaMemcpyAsync(hS, S1, sizeof(BlockScalars), cudaMemcpyDeviceToHost, st));
  WN_CUDA(cudaStreamSynchronize(st));
  return 0;
}

// Refinement over the batch in W.F (m live cases): U = 0, R = F; while some case has
// ||R_j|| > rtol ||F_j||: batched PCG on R with per-case inner targets, U += X, R = F - K U.
// U is kept as a double-double pair and R is evaluated with compensated products and sums,
// so the test resolves residuals below the FP64 rounding level of K U (which for load cases
// with large displacements lies near 1e-8 of ||F||); U_hi is returned.
template <typename TM>
int batch_outer(Solid* s, BlockWork& W, int vmode, int m, const wn_solve_params& prm, int chunk, cudaStream_t st,
                BatchResult& res) {
  const int64_t n = W.n;
  const size_t vb = (size_t)n * kBatch * sizeof(double);
  BlockScalars* S = W.scal.p;
  BlockScalars* S1 = W.scal.p + 1;
  BlockScalars hS{};
  WN_CHECK(case_norms2(W, W.F.p, S1, st, &hS));
  double fnorm[kBatch], rr[kBatch];
  for (int j = 0; j < kBatch; ++j) {
    fnorm[j] = std::sqrt(hS.rr[j]);
    rr[j] = hS.rr[j];
  }
  WN_CUDA(cudaMemsetAsync(W.U.p, 0, vb, st));
  WN_CUDA(cudaMemsetAsync(W.Ulo.p, 0, vb, st));
  WN_CUDA(cudaMemcpyAsync(W.R.p, W.F.p, vb, cudaMemcpyDeviceToDevice, st));
  const int max_outer = prm.max_outer > 0 ? prm.max_outer : 10;
  bool first = true;
  while (true) {
    if (!first) {
      W.npC = row_grid<double, 9>(rows_work(s->n_nodes));
      kb_outer_residual<<<W.npC, kThreads, 0, st>>>(s->n_nodes, s->batch->order[kRowCtas<double, 9> - 2].p, s->row_ptr.p, s->col_idx.p, s->k64.p, s->nnzb,
                                                    W.F.p, W.U.p, W.Ulo.p, W.R.p, W.partC.p);
      kb_reduce_rr<<<1, kScalarThreads, 0, st>>>(S1, W.partC.p, W.npC);
      W.launches += 2;
      WN_CUDA(cudaGetLastError());
      WN_CUDA(cudaMemcpyAsync(&hS, S1, sizeof(BlockScalars), cudaMemcpyDeviceToHost, st));
      WN_CUDA(cudaStreamSynchronize(st));
      for (int j = 0; j < kBatch; ++j) rr[j] = hS.rr[j];
    }
    first = false;
    bool all = true;
    for (int j = 0; j < kBatch; ++j) {
      double t = 1.0;  // 1 = case finished (or padding)
      if (j < m) {
        const double rn = std::sqrt(rr[j]);
        if (!std::isfinite(fnorm[j]) || !std::isfinite(rr[j])) {
          res.case_status[j] = WN_EBREAKDOWN;  // corrupt load case or diverged: not iterated on
        } else if (fnorm[j] > 0.0 && res.case_status[j] != WN_EBREAKDOWN && rn > prm.rtol * fnorm[j]) {
          t = std::min(0.5, 0.5 * prm.rtol * fnorm[j] / rn);
          all = false;
        }
      }
      W.h_rtol[j] = t;
    }
    if (all) break;
    if (res.outer >= max_outer || res.iterations >= prm.max_iter) {
      res.status = WN_ENOCONV;
      break;
    }
    WN_CUDA(cudaMemcpyAsync(W.rtol_cols.p, W.h_rtol.data(), kBatch * sizeof(double), cudaMemcpyHostToDevice, st));
    WN_CHECK((batch_pcg<TM>(s, W, vmode, W.R.p, prm.max_iter - res.iterations, prm.precond, chunk, prm.use_graph, S,
                            st, &hS)));
    res.iterations += hS.iters;
    ++res.outer;
    for (int j = 0; j < m; ++j) {
      res.case_iters[j] += hS.col_iters[j];
      if (hS.col_status[j] == WN_EBREAKDOWN) res.case_status[j] = WN_EBREAKDOWN;
    }
    kb_accumulate<<<grid_for(n * kBatch, 1, kThreads, 8), kThreads, 0, st>>>(n, W.U.p, W.Ulo.p, W.x.p);
    W.launches++;
    WN_CUDA(cudaGetLastError());
  }
  for (int j = 0; j < m; ++j) {
    res.case_rel[j] = fnorm[j] > 0.0 ? std::sqrt(rr[j]) / fnorm[j] : 0.0;
    const bool ok = res.case_rel[j] <= prm.rtol;
    if (res.case_status[j] == 0 && !ok) res.case_status[j] = WN_ENOCONV;
    if (res.case_status[j] == WN_EBREAKDOWN) res.status = WN_EBREAKDOWN;
    else if (res.case_status[j] == WN_ENOCONV && res.status == 0) res.status = WN_ENOCONV;
  }
  return 0;
}

}  // namespace

template <>
int solve_batch<kBatch>(Solid* s, const double* F, double* U, int n_rhs, int j0, int m, const wn_solve_params& prm,
                        BatchResult& res, cudaStream_t st) {
  const int vmode = prm.precision == 1 ? 1 : 0;
  WN_CHECK(ensure_block_work(s, vmode, prm.precond));
  BlockWork& W = *block_work(*s->batch);
  W.launches = 0;
  const int64_t n = W.n;
  const int chunk = prm.chunk > 0 ? prm.chunk : 8;
  kb_fill_dinv<<<grid_for(n, 1, kThreads, 8), kThreads, 0, st>>>(s->n_nodes, s->nnzb, s->diag_block.p, s->k64.p,
                                                                 W.dinv64.p, W.dinv32.p);
  kb_pack<<<grid_for(n * kBatch, 1, kThreads, 8), kThreads, 0, st>>>(n, F, n_rhs, j0, m, W.F.p);
  W.launches += 2;
  WN_CUDA(cudaGetLastError());
  if (vmode == 1)
    WN_CHECK(batch_outer<float>(s, W, vmode, m, prm, chunk, st, res));
  else
    WN_CHECK(batch_outer<double>(s, W, vmode, m, prm, chunk, st, res));
  kb_unpack<<<grid_for(n * kBatch, 1, kThreads, 8), kThreads, 0, st>>>(n, W.U.p, n_rhs, j0, m, U);
  W.launches++;
  WN_CUDA(cudaGetLastError());
  res.launches = W.launches;
  return 0;
}

}  // namespace wn
