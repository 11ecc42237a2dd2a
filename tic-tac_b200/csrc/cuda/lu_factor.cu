// Blocked right-looking LU with partial pivoting of the complex Faddeev kernel
// matrix 1 - A G (row-major, in place).  Replaces the LAPACK zgetrf of the
// reference's dense solver (CPP/General_functions/matrix_routines.cpp:73-80).
//
// Outer panels of NB columns (512 for the complex64 / tensor-core path, 128
// for complex128).  Each panel is factored in IB = 32 column sub-panels:
//   k_subpanel_ll  each block's rows on chip and no grid barrier: tries pivots
//                from the 32 x 32 diagonal block, checked against all rows, else
//                every block posts its best pivot row of a column in tagged
//                records that the others poll; also the sub-panel's interchanges
//                on the rest of the panel (k_subpanel: from global memory with a
//                grid barrier per column, for sub-panels too tall for shared
//                memory)
//   k_trsm_rows  U = L^{-1} U for the unit-lower diagonal block
//   the update of the remaining panel columns
// then the panel's interchanges outside the panel (k_laswp2), the triangular
// solve for U12 and the trailing update A22 -= L21 U12 (tcgen05 for complex64,
// FP64 tensor cores for complex128).
#include <cooperative_groups.h>

#include <algorithm>
#include <functional>
#include <map>
#include <mutex>
#include <type_traits>
#include <vector>

#include "ll_record.cuh"
#include "tc2_pack.cuh"
#include "tt_kernels.h"
#include "tt_lu_internal.h"

namespace cg = cooperative_groups;

namespace tt {
namespace {

template <typename T>
struct Real;
template <>
struct Real<double2> {
  using R = double;
};
template <>
struct Real<float2> {
  using R = float;
};

template <typename T>
__device__ __forceinline__ T cdiv_smith(T a, T b) {
  using R = typename Real<T>::R;
  T r;
  if (fabs((double)b.x) >= fabs((double)b.y)) {
    const R t = b.y / b.x, d = b.x + b.y * t;
    r.x = (a.x + a.y * t) / d;
    r.y = (a.y - a.x * t) / d;
  } else {
    const R t = b.x / b.y, d = b.y + b.x * t;
    r.x = (a.x * t + a.y) / d;
    r.y = (a.y * t - a.x) / d;
  }
  return r;
}

// acc -= a b and acc += a b, complex: two fused multiply-adds a component
template <typename T>
__device__ __forceinline__ void cfma_sub(T& acc, T a, T b) {
  acc.x -= a.x * b.x;
  acc.x += a.y * b.y;
  acc.y -= a.x * b.y;
  acc.y -= a.y * b.x;
}
template <typename T>
__device__ __forceinline__ void cfma_add(T& acc, T a, T b) {
  acc.x += a.x * b.x;
  acc.x -= a.y * b.y;
  acc.y += a.x * b.y;
  acc.y += a.y * b.x;
}
template <typename T>
__device__ __forceinline__ T cmul(T a, T b) {
  T r;
  r.x = a.x * b.x - a.y * b.y;
  r.y = a.x * b.y + a.y * b.x;
  return r;
}

constexpr int IB = 32;
constexpr int SP = IB + 1;                     // shared-memory row stride of a staged sub-panel
constexpr size_t kSubpanelSmem = 226 * 1024;  // shared memory of a CTA of the on-chip sub-panel kernel
constexpr int SP_WARPS = 16;                  // most warps of a CTA of the on-chip sub-panel kernel

template <typename T>
struct PivotScratch {
  double* val;              // [2][G]
  int* idx;                 // [2][G]
  T* row;                   // [2][G][IB]
  T* top;                   // [2][IB]
};

// Matrices of equal n factored together: the sub-panel grid is split into B
// equal groups of blocks, group b working on matrix b (the exchange of the
// pivot, not the work, bounds a sub-panel column).
constexpr int kMaxBatch = 4;
template <typename T>
struct SubpanelBatch {
  T* A[kMaxBatch];
  int32_t* ipiv[kMaxBatch];
  int* info;                           // [B]
  int* err;                            // set when a wait ran out
  int* tries;                          // [B][2] sub-panels to come without a try, and how many after the next failure
  unsigned char* verdict;              // [B][CTAs of a matrix] records: this CTA's rows agree with the try
  int B;
};
// a[i] by predicated selects: a runtime index into a kernel parameter array
// would copy the whole parameter struct to local memory
template <typename P>
__device__ __forceinline__ P batch_pick(const P (&a)[kMaxBatch], int i) {
  P r = a[0];
#pragma unroll
  for (int q = 1; q < kMaxBatch; q++)
    if (i == q) r = a[q];
  return r;
}

// Sub-panel rows [c0, n), columns [c0, c0+w), w <= IB.
template <typename T>
__global__ void __launch_bounds__(256) k_subpanel(T* __restrict__ A, int n, int c0, int w, int32_t* __restrict__ ipiv,
                                                  PivotScratch<T> scr, int* __restrict__ info) {
  cg::grid_group grid = cg::this_grid();
  const int G = gridDim.x;
  const int m = n - c0;
  const int chunk = (m + G - 1) / G;
  const int lo = c0 + blockIdx.x * chunk;
  const int hi = min(n, lo + chunk);
  __shared__ double s_val[256];
  __shared__ int s_idx[256];
  __shared__ T s_prow[IB];
  __shared__ int s_grp[256];
  __shared__ int s_piv;
  __shared__ int s_zero;
  __shared__ int s_win;
  for (int jj = 0; jj < w; jj++) {
    const int j = c0 + jj;  // diagonal row/column
    const int buf = jj & 1;
    // 1. local candidate among own rows >= j
    double best = -1.0;
    int bidx = -1;
    for (int i = max(lo, j) + threadIdx.x; i < hi; i += blockDim.x) {
      const T v = A[(size_t)i * n + j];
      const double a = fabs((double)v.x) + fabs((double)v.y);
      if (a > best || (a == best && i < bidx)) {
        best = a;
        bidx = i;
      }
    }
    s_val[threadIdx.x] = best;
    s_idx[threadIdx.x] = bidx;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
      if (threadIdx.x < s) {
        const double o = s_val[threadIdx.x + s];
        const int oi = s_idx[threadIdx.x + s];
        const double mv = s_val[threadIdx.x];
        const int mi = s_idx[threadIdx.x];
        if (oi >= 0 && (mi < 0 || o > mv || (o == mv && oi < mi))) {
          s_val[threadIdx.x] = o;
          s_idx[threadIdx.x] = oi;
        }
      }
      __syncthreads();
    }
    const int cand = s_idx[0];
    if (threadIdx.x == 0) {
      scr.val[buf * G + blockIdx.x] = s_val[0];
      scr.idx[buf * G + blockIdx.x] = cand;
    }
    if (cand >= 0 && threadIdx.x < w) scr.row[((size_t)buf * G + blockIdx.x) * IB + threadIdx.x] = A[(size_t)cand * n + c0 + threadIdx.x];
    if (j >= lo && j < hi && threadIdx.x < w) scr.top[buf * IB + threadIdx.x] = A[(size_t)j * n + c0 + threadIdx.x];
    grid.sync();
    // 2. global pivot: every block reduces the G candidates in parallel (same rule everywhere)
    {
      double v = -1.0;
      int vi = -1, vg = -1;
      for (int g = threadIdx.x; g < G; g += blockDim.x) {
        const int ci = scr.idx[buf * G + g];
        if (ci < 0) continue;
        const double cv = scr.val[buf * G + g];
        if (vi < 0 || cv > v || (cv == v && ci < vi)) {
          v = cv;
          vi = ci;
          vg = g;
        }
      }
      s_val[threadIdx.x] = v;
      s_idx[threadIdx.x] = vi;
      s_grp[threadIdx.x] = vg;
      __syncthreads();
      for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) {
          const double o = s_val[threadIdx.x + s];
          const int oi = s_idx[threadIdx.x + s];
          const double mv = s_val[threadIdx.x];
          const int mi = s_idx[threadIdx.x];
          if (oi >= 0 && (mi < 0 || o > mv || (o == mv && oi < mi))) {
            s_val[threadIdx.x] = o;
            s_idx[threadIdx.x] = oi;
            s_grp[threadIdx.x] = s_grp[threadIdx.x + s];
          }
        }
        __syncthreads();
      }
      if (threadIdx.x == 0) {
        s_piv = s_idx[0];
        s_zero = !(s_val[0] > 0.0);
        if (blockIdx.x == 0) {
          ipiv[j] = s_zero ? j : s_idx[0];
          if (s_zero && *info == 0) *info = j + 1;
        }
        s_win = s_grp[0];
      }
      __syncthreads();
    }
    const int piv = s_piv;
    if (s_zero) {
      __syncthreads();
      continue;
    }
    const int winner = s_win;
    if (threadIdx.x < w) s_prow[threadIdx.x] = scr.row[((size_t)buf * G + winner) * IB + threadIdx.x];
    __syncthreads();
    // 3. the two owners exchange rows j and piv (sub-panel columns only)
    if (piv != j) {
      if (piv >= lo && piv < hi && threadIdx.x < w)
        A[(size_t)piv * n + c0 + threadIdx.x] = scr.top[buf * IB + threadIdx.x];
      if (j >= lo && j < hi && threadIdx.x < w) A[(size_t)j * n + c0 + threadIdx.x] = s_prow[threadIdx.x];
    } else if (j >= lo && j < hi && threadIdx.x < w) {
      A[(size_t)j * n + c0 + threadIdx.x] = s_prow[threadIdx.x];
    }
    __syncthreads();
    // 4. eliminate below the diagonal in own rows
    const T d = s_prow[jj];
    const int r0 = max(lo, j + 1);
    const int ncol = w - jj - 1;
    for (int i = r0 + threadIdx.x; i < hi; i += blockDim.x) {
      T* row = A + (size_t)i * n + c0;
      const T l = cdiv_smith(row[jj], d);
      row[jj] = l;
      for (int c = 1; c <= ncol; c++) {
        const T u = s_prow[jj + c];
        T a = row[jj + c];
        a.x -= l.x * u.x - l.y * u.y;
        a.y -= l.x * u.y + l.y * u.x;
        row[jj + c] = a;
      }
    }
    __syncthreads();
  }
}

// ---- sub-panel resident on chip
//
// The CTAs of a matrix hold its sub-panel rows, one thread per row (two where
// the rows outnumber the threads), columns in register blocks of CB: within a
// block a column's elimination touches registers only; the columns right of the
// block wait in shared memory and take all CB pivots in one rank-CB update.
// Every element still sees the pivots one after another in ascending order.
//
// What bounds a column is the exchange of its pivot.  Each CTA posts its best
// row as 16-byte records {element, tag, row index}, one atomic store each: the
// tag (column + 1) tells a reader that the record is this column's, so there is
// no barrier, no fence and no flag beside the data.  Up to LL_ONE_HOP CTAs a
// matrix, every CTA reads all posted rows and picks the winner itself: one
// store-to-load trip through L2.  With more, the rows would cost more L2
// traffic than a second trip, so it reads the candidates' own elements, then the
// winner's row.  The diagonal row always lives in the matrix's first CTA, which
// posts it for the interchange; a matrix of one CTA exchanges in shared memory.
// Records are double-buffered by column parity: a CTA posts column j + 2 only
// after it has seen every CTA's column j + 1, posted after their reads of j.
//
// Of a column's 2.5 to 6 thousand cycles the trips through L2 take about 1,200
// each; the rest is the latency of its own instructions.
//
// The matrices are 1 - A G: all 32 pivots of a sub-panel mostly lie in its 32 x 32 diagonal
// block, nearly always on the diagonal (in 96 to 100% of the sub-panels of channels of
// n = 8,496 to 42,300; two in three at n = 512 of Malfliet-Tjon s-waves).  So the kernel
// first tries that, without any exchange: every CTA factors the diagonal block for
// itself (sp_factor_diag, and with interchanges in the block, sp_factor_block, where the
// diagonal will not do), takes its own rows through the block's U (sp_try_row) and looks
// at each element before its division: none may exceed the pivot of its column by the
// same keys that the search compares.  One verdict a CTA, one trip, and if all agree these
// are pivots that the search may choose (its elements differ in their rounding, so near
// ties may fall the other way).  Else the rows, still unchanged in A, are read
// again for the search; a matrix whose tries fail in a row goes 1, 3, 7, then 15
// sub-panels without one, so that a try (a fifth of a search) is lost on few.
// Bound: the latency of the block's 32 steps (~5 us) and the rows' FP32 multiply-adds.
//
// Per sub-panel of 32 columns, search alone -> with tries, two complex64 matrices:
// n = 10,944 82 -> 22 us, n = 16,128 80 -> 20 us, n = 42,300 113 -> 31 us; four at
// n = 20,160 93 -> 28 us; one complex128 at n = 8,496 90 -> 29 us.
// Rows of a CTA: 224 (eight warps, the count the block needs) against 480: channel of
// n = 16,128 11.7 -> 10.3 ms in all, n = 42,300 43.5 -> 40.5 ms, complex128 17.6 -> 15.5.
// Waits end after LL_SPINS polls: the error word is set and the rest of the
// launch runs without waiting.
constexpr int LL_ONE_HOP = 32;
constexpr int LL_SPINS = 1 << 20;
constexpr size_t SP_CLUSTER_ROWS = 256;  // most rows of a CTA in a cluster
constexpr int SP_ROWS = 224;  // rows of a CTA, where the CTAs suffice: one per thread of 7 warps
constexpr int TRY_LD = IB + 2, TRY_THREADS = 256;  // row stride of the tried diagonal block; threads it takes
constexpr int LL_PER_WARP = 4;  // posted rows that a warp gathers, the diagonal row among them

// Pivot candidates as keys: 0 for none (NaN magnitudes included), else the bits
// of |re| + |im| plus one, which order as the magnitudes do; ties go to the
// lower row, as in LAPACK's izamax.
__device__ __forceinline__ unsigned pivot_key(float2 v) {
  const float m = fabsf(v.x) + fabsf(v.y);
  return m >= 0 ? __float_as_uint(m) + 1u : 0u;
}
__device__ __forceinline__ unsigned long long pivot_key(double2 v) {
  const double m = fabs(v.x) + fabs(v.y);
  return m >= 0 ? (unsigned long long)__double_as_longlong(m) + 1ull : 0ull;
}
__device__ __forceinline__ unsigned warp_max(unsigned k) { return __reduce_max_sync(0xffffffffu, k); }
__device__ __forceinline__ unsigned long long warp_max(unsigned long long k) {
  const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(k >> 32));
  const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(k >> 32) == hi ? (unsigned)k : 0u);
  return ((unsigned long long)hi << 32) | lo;
}
// the warp's best (key, row) to every lane, the lower row on ties; returns the lane that held it
template <typename K>
__device__ __forceinline__ int warp_best(K& key, int& row) {
  const K best = warp_max(key);
  unsigned who = __ballot_sync(0xffffffffu, key == best);
  if (who & (who - 1)) {
    const int r = (int)__reduce_min_sync(0xffffffffu, key == best ? (unsigned)row : 0x7fffffffu);
    who = __ballot_sync(0xffffffffu, key == best && row == r);
  }
  const int lane = __ffs(who) - 1;
  key = best;
  row = __shfl_sync(0xffffffffu, row, lane);
  return lane;
}

// 1 / b by one reciprocal, b scaled by a power of two where |b|^2 would leave the
// range it is formed in without loss
__device__ __forceinline__ float2 pivot_recip(float2 b) {
  const float big = fmaxf(fabsf(b.x), fabsf(b.y));
  float x = b.x, y = b.y, r = __frcp_rn(fmaf(x, x, y * y));
  if (!(big > 0x1p-50f && big < 0x1p50f)) {
    const int e = min(max((int)(__float_as_uint(big) >> 23) - 127, -126), 126);
    const float sc = __uint_as_float((unsigned)(127 - e) << 23);
    x *= sc;
    y *= sc;
    r = sc * __frcp_rn(fmaf(x, x, y * y));
  }
  return make_float2(x * r, -y * r);
}
__device__ __forceinline__ double2 pivot_recip(double2 b) {
  const double big = fmax(fabs(b.x), fabs(b.y));
  double x = b.x, y = b.y, r = __drcp_rn(fma(x, x, y * y));
  if (!(big > 0x1p-400 && big < 0x1p400)) {
    const int e = min(max((int)(((unsigned long long)__double_as_longlong(big)) >> 52) - 1023, -1022), 1022);
    const double sc = __longlong_as_double((long long)((unsigned long long)(1023 - e) << 52));
    x *= sc;
    y *= sc;
    r = sc * __drcp_rn(fma(x, x, y * y));
  }
  return make_double2(x * r, -y * r);
}

// a column's U elements of a block, by 16-byte loads
__device__ __forceinline__ void load_u(const float2* p, float2 (&u)[8]) {
#pragma unroll
  for (int c = 0; c < 4; c++) {
    const float4 f = reinterpret_cast<const float4*>(p)[c];
    u[2 * c] = make_float2(f.x, f.y);
    u[2 * c + 1] = make_float2(f.z, f.w);
  }
}
__device__ __forceinline__ void load_u(const double2* p, double2 (&u)[4]) {
#pragma unroll
  for (int c = 0; c < 4; c++) u[c] = p[c];
}

template <typename T>
struct SubpanelCfg {
  using Key = decltype(pivot_key(T{}));
  static constexpr int CB = sizeof(T) == 8 ? 8 : 4;  // columns of a register block
  static constexpr int RW = IB + CB;                 // padded row: a block read past column 31 stays inside
  // shared memory beside the rows: the gathered rows and diagonal rows (two
  // columns' worth), the block's U rows, candidates and pivots
  static constexpr size_t EXTRA = sizeof(T) * (2 * SP_WARPS * RW + 2 * RW + CB * IB) +
                                  2 * SP_WARPS * 2 * (sizeof(Key) + sizeof(int)) + IB * sizeof(int) + 16;
  static constexpr int MAX_ROWS = (int)((kSubpanelSmem - EXTRA) / (SP * sizeof(T)));
};
// rows per thread of a CTA of `rows` rows, and its threads: the row warps and one more
inline int sp_rpt(int rows) { return rows > 32 * (SP_WARPS - 1) ? 2 : 1; }
inline int sp_threads(int rows) {
  return std::max(TRY_THREADS, 32 * ((rows + 32 * sp_rpt(rows) - 1) / (32 * sp_rpt(rows)) + 1));
}

// Barrier of the warps that factor the diagonal block.  Its aligned form is for converged
// warps, and inline code is not converged by the compiler: lanes that took different
// branches meet first.
__device__ __forceinline__ void sp_block_sync() {
  __syncwarp();
  asm volatile("bar.sync 1, %0;" ::"n"(TRY_THREADS) : "memory");
}

// LU of the sub-panel's w x w diagonal block in sD (row stride TRY_LD), every pivot on the
// diagonal; false (to some thread) if an element of the block would have been the pivot.
// Thread t of 256 keeps row t / 8, columns 4 (t % 8) to + 3.  A step takes four columns:
// every thread factors their 4 x 4 diagonal block for itself, solves its own L row and U
// columns against it and updates its four elements; what the next step reads goes to
// shared memory, one barrier a step.  sRd, sBest: the pivots' reciprocals and keys.
// Bound: the chain of 32 reciprocals.
template <typename T, typename Key>
__device__ __forceinline__ bool sp_factor_diag(T* sD, T* sRd, Key* sBest, int w, int tid) {
  constexpr int W = 4;
  const int i = tid >> 3, g = tid & 7, warp = tid >> 5;
  bool ok = true;
  T a[W];
#pragma unroll
  for (int c = 0; c < W; c++) a[c] = sD[i * TRY_LD + W * g + c];
#pragma unroll 1
  for (int s = 0; W * s < w; s++) {
    const int j0 = W * s;
    if (warp >= s && g >= s) {
      T d[W][W], rd[W], l[W];
#pragma unroll
      for (int r = 0; r < W; r++)
#pragma unroll
        for (int c = 0; c < W; c++) d[r][c] = sD[(j0 + r) * TRY_LD + j0 + c];
#pragma unroll
      for (int c = 0; c < W; c++) l[c] = sD[i * TRY_LD + j0 + c];
      Key best[W];
#pragma unroll
      for (int k = 0; k < W; k++) {
        rd[k] = pivot_recip(d[k][k]);
        best[k] = pivot_key(d[k][k]);
#pragma unroll
        for (int r = k + 1; r < W; r++) {
          ok &= pivot_key(d[r][k]) <= best[k];
          d[r][k] = cmul(d[r][k], rd[k]);
#pragma unroll
          for (int c = k + 1; c < W; c++) cfma_sub(d[r][c], d[r][k], d[k][c]);
        }
      }
      // row i takes the pivots above it: all four below the diagonal block
#pragma unroll
      for (int k = 0; k < W; k++)
        if (k < i - j0) {
          ok &= pivot_key(l[k]) <= best[k];
          l[k] = cmul(l[k], rd[k]);
#pragma unroll
          for (int c = k + 1; c < W; c++) cfma_sub(l[c], l[k], d[k][c]);
        }
      if (g > s) {
#pragma unroll
        for (int c = 0; c < W; c++) {
          T u[W];
#pragma unroll
          for (int r = 0; r < W; r++) {
            u[r] = sD[(j0 + r) * TRY_LD + W * g + c];
#pragma unroll
            for (int k = 0; k < r; k++) cfma_sub(u[r], d[r][k], u[k]);
          }
#pragma unroll
          for (int k = 0; k < W; k++)
            if (k < i - j0) cfma_sub(a[c], l[k], u[k]);
        }
        if (warp > s)
#pragma unroll
          for (int c = 0; c < W; c++) sD[i * TRY_LD + W * g + c] = a[c];
      } else {
#pragma unroll
        for (int c = 0; c < W; c++) a[c] = l[c];
        if (i == j0)
#pragma unroll
          for (int k = 0; k < W; k++) {
            sRd[j0 + k] = rd[k];
            sBest[j0 + k] = best[k];
          }
      }
    }
    sp_block_sync();
  }
#pragma unroll
  for (int c = 0; c < W; c++) sD[i * TRY_LD + W * g + c] = a[c];
  return ok;
}

// Pivoted LU of the sub-panel's w x w diagonal block in sD (row stride TRY_LD) by warps
// 0 to 7, warp q the columns 4q to 4q + 3, lane = row.  The owner of four columns takes
// them in registers and leaves their multipliers in shared memory; the other warps then
// interchange and update theirs: a barrier every four columns.  sPiv[j]: pivot row within
// the block, sRd[j]: its reciprocal, sBest[j]: its key.  Bound by latency.
template <typename T, typename Key>
__device__ __forceinline__ void sp_factor_block(T* sD, T* sRd, Key* sBest, int* sPiv, int w, int lane, int warp) {
  constexpr int CW = 4;  // columns of a warp
  auto shfl = [&](T v, int src) {
    T r;
    r.x = __shfl_sync(0xffffffffu, v.x, src);
    r.y = __shfl_sync(0xffffffffu, v.y, src);
    return r;
  };
  T a[CW];
#pragma unroll
  for (int k = 0; k < CW; k++) a[k] = sD[lane * TRY_LD + CW * warp + k];
  sp_block_sync();  // the block is in registers, sD holds multipliers from here on
#pragma unroll 1
  for (int q = 0; CW * q < w; q++) {
    T* mult = sD + (q & 1) * CW * IB;  // [CW][IB]
    if (warp == q) {
#pragma unroll
      for (int k = 0; k < CW; k++) {
        const int j = CW * q + k;
        if (j >= w) break;
        const Key key = lane >= j && lane < w ? pivot_key(a[k]) : Key(0);
        const Key best = warp_max(key);
        const int p = __ffs(__ballot_sync(0xffffffffu, key == best && lane >= j)) - 1;
        if (p != j) {
          const int src = lane == j ? p : lane == p ? j : lane;
#pragma unroll
          for (int c = 0; c < CW; c++) a[c] = shfl(a[c], src);
        }
        const T rd = pivot_recip(shfl(a[k], j));
        T l = T{0, 0};
        if (lane > j) {
          l.x = a[k].x * rd.x - a[k].y * rd.y;
          l.y = a[k].x * rd.y + a[k].y * rd.x;
          a[k] = l;
        }
        mult[k * IB + lane] = l;
        if (lane == 0) {
          sPiv[j] = p;
          sRd[j] = rd;
          sBest[j] = best;
        }
#pragma unroll
        for (int c = k + 1; c < CW; c++) {
          const T u = shfl(a[c], j);
          if (lane > j) {
            a[c].x -= l.x * u.x - l.y * u.y;
            a[c].y -= l.x * u.y + l.y * u.x;
          }
        }
      }
    }
    sp_block_sync();
    if (warp != q) {
#pragma unroll
      for (int k = 0; k < CW; k++) {
        const int j = CW * q + k;
        if (j >= w) break;
        const int p = sPiv[j];
        if (p != j) {
          const int src = lane == j ? p : lane == p ? j : lane;
#pragma unroll
          for (int c = 0; c < CW; c++) a[c] = shfl(a[c], src);
        }
        if (warp > q) {
          const T l = mult[k * IB + lane];
#pragma unroll
          for (int c = 0; c < CW; c++) {
            const T u = shfl(a[c], j);
            if (lane > j) {
              a[c].x -= l.x * u.x - l.y * u.y;
              a[c].y -= l.x * u.y + l.y * u.x;
            }
          }
        }
      }
    }
  }
  sp_block_sync();
#pragma unroll
  for (int k = 0; k < CW; k++) sD[lane * TRY_LD + CW * warp + k] = a[k];
}

// A row below the diagonal block, x <- x U^{-1} in shared memory, CB columns at a time in
// registers, each element taking the pivots in ascending order; false if one of its
// elements would have been the column's pivot.
//
// a[c] -= l[d] u[d][c] over CB x CB; complex64 in packed pairs, P = a - sum l.x u and
// Q = sum l.y u, so that a = (P.x + Q.y, P.y - Q.x)
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  return (unsigned long long)__float_as_uint(x) | ((unsigned long long)__float_as_uint(y) << 32);
}
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
template <int CB>
struct TryAcc {
  unsigned long long P[CB], Q[CB];
  __device__ __forceinline__ void start(const float2* row) {
#pragma unroll
    for (int c = 0; c < CB; c++) {
      P[c] = pack2(row[c].x, row[c].y);
      Q[c] = 0;
    }
  }
  __device__ __forceinline__ void add(float2 l, const float2* u) {
    const unsigned long long x = pack2(-l.x, -l.x), y = pack2(l.y, l.y);
#pragma unroll
    for (int c = 0; c < CB; c += 2) {
      const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(u + c);
      fma2(P[c], x, v.x);
      fma2(Q[c], y, v.x);
      fma2(P[c + 1], x, v.y);
      fma2(Q[c + 1], y, v.y);
    }
  }
  __device__ __forceinline__ float2 value(int c) const {
    return make_float2(__uint_as_float((unsigned)P[c]) + __uint_as_float((unsigned)(Q[c] >> 32)),
                       __uint_as_float((unsigned)(P[c] >> 32)) - __uint_as_float((unsigned)Q[c]));
  }
};
template <int CB>
struct TryAccD {
  double2 a[CB];
  __device__ __forceinline__ void start(const double2* row) {
#pragma unroll
    for (int c = 0; c < CB; c++) a[c] = row[c];
  }
  __device__ __forceinline__ void add(double2 l, const double2* u) {
#pragma unroll
    for (int c = 0; c < CB; c++) cfma_sub(a[c], l, u[c]);
  }
  __device__ __forceinline__ double2 value(int c) const { return a[c]; }
};
template <typename T, typename Key>
__device__ __forceinline__ bool sp_try_row(T* row, const T* sD, const T* sRd, const Key* sBest) {
  constexpr int CB = sizeof(T) == 8 ? 8 : 4;
  bool ok = true;
#pragma unroll 1
  for (int k0 = 0; k0 < IB; k0 += CB) {
    std::conditional_t<sizeof(T) == 8, TryAcc<CB>, TryAccD<CB>> acc;
    acc.start(row + k0);
#pragma unroll 1
    for (int j0 = 0; j0 < k0; j0 += CB) {
      T l[CB];
#pragma unroll
      for (int d = 0; d < CB; d++) l[d] = row[j0 + d];
#pragma unroll
      for (int d = 0; d < CB; d++) acc.add(l[d], sD + (j0 + d) * TRY_LD + k0);
    }
    T a[CB];
#pragma unroll
    for (int c = 0; c < CB; c++) a[c] = acc.value(c);
#pragma unroll
    for (int d = 0; d < CB; d++) {
      ok &= pivot_key(a[d]) <= sBest[k0 + d];
      a[d] = cmul(a[d], sRd[k0 + d]);
      T u[CB];
      load_u(sD + (k0 + d) * TRY_LD + k0, u);
#pragma unroll
      for (int c = d + 1; c < CB; c++) cfma_sub(a[c], a[d], u[c]);
    }
#pragma unroll
    for (int c = 0; c < CB; c++) row[k0 + c] = a[c];
  }
  return ok;
}

// Sub-panel rows [c0, n), columns [c0, c0 + w) of bt.B matrices, Gb = gridDim.x / B
// consecutive CTAs each (group b works on matrix b); at least IB rows in the first.
// Warps but the last own rows, the last solves the block's U rows meanwhile.
// With pk0 < pk1, the sub-panel's interchanges are also applied to the other
// columns [pk0, c0) and [c0 + w, pk1) of its panel.  rec: [2][B][Gb + 1][IB]
// records, zero before the factorisation.
// CLUSTER: a matrix's CTAs are one cluster of up to 16, which exchanges the rows
// through distributed shared memory: the owner warp stores its row into every CTA,
// and one cluster barrier takes the place of the records' trip through L2.  Taken for
// 225 to 4,096 rows, a row per thread: 84 -> 67 us a search there, complex128 101 ->
// 84 us, and a verdict costs 900 cycles against 2,500 to 5,000.  Taller sub-panels would
// need more rows a CTA than SP_ROWS, and meet in L2.
__device__ __forceinline__ void sp_cluster_sync() {
  __syncwarp();  // an aligned barrier, as sp_block_sync's
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t sp_remote(const void* p, int rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  return r;
}
__device__ __forceinline__ void sp_store_remote(uint32_t a, float2 v) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y) : "memory");
}
__device__ __forceinline__ void sp_store_remote(uint32_t a, double2 v) {
  asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v.x), "d"(v.y) : "memory");
}
__device__ __forceinline__ void sp_store_remote(uint32_t a, int v) {
  asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

template <typename T>
__device__ __forceinline__ void sp_cp_async(T* dst, const T* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "n"(sizeof(T))
               : "memory");
}

template <typename T, int RPT, bool CLUSTER>
__global__ void __launch_bounds__(32 * SP_WARPS, 1) k_subpanel_ll(SubpanelBatch<T> bt, int n, int c0, int w, int pk0,
                                                                  int pk1, unsigned char* __restrict__ rec) {
  using CF = SubpanelCfg<T>;
  using Key = typename CF::Key;
  constexpr int CB = CF::CB, RW = CF::RW, NONE = 0x7fffffff;
  extern __shared__ __align__(16) unsigned char sp_raw[];
  const int Gb = gridDim.x / bt.B, grp = blockIdx.x / Gb, cta = blockIdx.x - grp * Gb;
  T* __restrict__ A = batch_pick(bt.A, grp);
  pdl_wait();
  pdl_launch_next();
  const int m = n - c0;
  const int chunk = (m + Gb - 1) / Gb;
  const int lo = cta * chunk;  // first row of this CTA, from c0
  const int nr = max(0, min(m, lo + chunk) - lo);
  T* sRow = reinterpret_cast<T*>(sp_raw);                  // [2][SP_WARPS][RW] gathered rows
  T* sTop = sRow + 2 * SP_WARPS * RW;                      // [2][RW] diagonal row
  T* sU = sTop + 2 * RW;                                   // [IB][CB] solved pivot rows of the block, by column
  Key* sKey = reinterpret_cast<Key*>(sU + CB * IB);        // [2][2][SP_WARPS] candidates: own, gathered
  int* sIdx = reinterpret_cast<int*>(sKey + 4 * SP_WARPS);  // [2][2][SP_WARPS]
  int* sPiv = sIdx + 4 * SP_WARPS;                         // [IB]
  int* sFlag = sPiv + IB;                                  // a wait ran out
  T* sA = reinterpret_cast<T*>(sp_raw + CF::EXTRA);        // [chunk][SP]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int NW = blockDim.x >> 5, NWR = NW - 1;
  const bool helper = warp == NWR;
  const int col = min(lane, w - 1);
  auto slot = [&](int buf, int g) { return rec + (((size_t)buf * bt.B + grp) * (Gb + 1) + g) * IB * LL<T>::BYTES; };
  auto load_rows = [&]() {
    if (lane < w)
      for (int r = warp; r < nr; r += NW) sp_cp_async(sA + r * SP + lane, A + (size_t)(c0 + lo + r) * n + c0 + lane);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto load_diag = [&](T* sD) {
    if (warp < TRY_THREADS / 32)
#pragma unroll
      for (int q = 0; q < IB * 32 / TRY_THREADS; q++) {
        const int r = warp + q * (TRY_THREADS / 32);
        if (r < w && lane < w)
          sp_cp_async(sD + r * TRY_LD + lane, A + (size_t)(c0 + r) * n + c0 + lane);
        else
          sD[r * TRY_LD + lane] = T{0, 0};
      }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  int* tries = bt.tries + 2 * grp;
  const bool trying = tries[0] == 0 && (w == IB || w == m);
  bool tried = false;  // ... and every pivot lies in the diagonal block
  T* sD = sRow;        // the diagonal block
  if (trying) load_diag(sD);
  load_rows();
  if (trying)
    asm volatile("cp.async.wait_group 1;" ::: "memory");  // the block; the rows come meanwhile
  else
    asm volatile("cp.async.wait_group 0;" ::: "memory");
  if (tid == 0) *sFlag = *(volatile int*)bt.err;
  if (CLUSTER) sp_cluster_sync();  // every CTA's shared memory exists before the first store into it
  else __syncthreads();
  // a[i][k]: column jj + k of this thread's row i, jj the column at work.  The
  // registers move down by one each column, so that one copy of the code serves
  // all of them; finished columns are in shared memory.
  T a[RPT][CB];
  auto row_of = [&](int i) { return (warp * RPT + i) * 32 + lane; };  // local row i of this thread
  auto owner_warp = [&](int r) { return r / (32 * RPT); };
  // local row r whole, lane = column, in its owner's warp: the block's columns
  // [jj, end) from the owner's registers, the others from shared memory
  auto row_values = [&](int r, int jj, int end) -> T {
    T v = sA[r * SP + col];
    const int src = r & 31;
    const bool second = RPT == 2 && (r >> 5 & 1);
#pragma unroll
    for (int k = 0; k < CB; k++) {
      const T x = second ? a[RPT - 1][k] : a[0][k];
      const T y = T{__shfl_sync(0xffffffffu, x.x, src), __shfl_sync(0xffffffffu, x.y, src)};
      if (lane == jj + k && lane < end) v = y;
    }
    return v;
  };
  // local row r replaced, in its owner's warp
  auto set_row = [&](int r, const T* row, int jj) {
    if (lane < w) sA[r * SP + lane] = row[lane];
#pragma unroll
    for (int i = 0; i < RPT; i++)
      if (row_of(i) == r)
#pragma unroll
        for (int k = 0; k < CB; k++) a[i][k] = row[jj + k];
  };
  auto load_block = [&](int b0) {
#pragma unroll
    for (int i = 0; i < RPT; i++)
#pragma unroll
      for (int k = 0; k < CB; k++) {
        a[i][k] = T{0, 0};
        if (!helper && row_of(i) < nr && b0 + k < w) a[i][k] = sA[row_of(i) * SP + b0 + k];
      }
  };
  // poll until every lane's record is this column's, at most LL_SPINS times
  auto wait_row = [&](const unsigned char* p, unsigned tag, T& v, unsigned long long& hi) {
    for (int spin = 0;; spin++) {
      const bool ok = LL<T>::poll(p, v, hi, tag);
      if (__all_sync(0xffffffffu, ok)) return;
      if (spin >= LL_SPINS || *(volatile int*)sFlag) {
        if (lane == 0) {
          *(volatile int*)sFlag = 1;
          atomicExch(bt.err, 1);
        }
        return;
      }
    }
  };
  // the diagonal row to every CTA, one warp
  auto post_top = [&](T v, T* top, int buf, unsigned tag) {
    if (CLUSTER) {
      for (int g = 0; g < Gb; g++) sp_store_remote(sp_remote(top + lane, g), v);
    } else if (Gb > 1) {
      LL<T>::post(slot(buf, Gb) + lane * LL<T>::BYTES, v, tag);
    } else {
      top[lane] = v;
    }
  };
  const bool one_hop = Gb <= LL_ONE_HOP && Gb < LL_PER_WARP * NW;
  if (trying) {
    T* sRd = sTop;
    Key* sBest = sKey;
    bool ok = true;
    if (warp < TRY_THREADS / 32) ok = sp_factor_diag(sD, sRd, sBest, w, tid);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (tid < IB) sPiv[tid] = tid;
    if (!__syncthreads_and(ok)) {
      load_diag(sD);
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
      if (warp < TRY_THREADS / 32) sp_factor_block(sD, sRd, sBest, sPiv, w, lane, warp);
      __syncthreads();
    }
    ok = sBest[col] > 1;  // a column without a pivot is left to the full search
    if (!helper)
#pragma unroll 1
      for (int i = 0; i < RPT; i++)
        if (row_of(i) < nr && lo + row_of(i) >= w) ok = sp_try_row(sA + row_of(i) * SP, sD, sRd, sBest) && ok;
    ok = __syncthreads_and(ok);
    if (CLUSTER) {
      // sIdx[g] of every CTA: CTA g agrees
      if (tid < Gb) sp_store_remote(sp_remote(sIdx + cta, tid), (int)ok);
      sp_cluster_sync();
      tried = __syncthreads_and(tid >= Gb || sIdx[tid]);
    } else if (Gb > 1) {
      unsigned char* v = bt.verdict + (size_t)grp * Gb * LL<float2>::BYTES;
      const unsigned tag = (unsigned)c0 + 1u;
      if (tid == 0) LL<float2>::post(v + cta * LL<float2>::BYTES, make_float2(ok ? 1.0f : 0.0f, 0.0f), tag);
      if (tid < Gb) {
        float2 r = make_float2(0, 0);
        unsigned long long hi;
        for (int spin = 0; !LL<float2>::poll(v + tid * LL<float2>::BYTES, r, hi, tag); spin++)
          if (spin >= LL_SPINS || *(volatile int*)sFlag) {
            *(volatile int*)sFlag = 1;
            atomicExch(bt.err, 1);
            break;
          }
        ok = r.x != 0.0f;
      }
      tried = __syncthreads_and(ok);
    } else {
      tried = ok;
    }
    if (tried) {
      if (cta == 0 && warp < TRY_THREADS / 32 && lane < w)
        for (int r = warp; r < w; r += TRY_THREADS / 32) sA[r * SP + lane] = sD[r * TRY_LD + lane];
      if (tid < w) sPiv[tid] += c0;
    } else {
      load_rows();
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
    }
  }
  if (!tried) load_block(0);
  for (int b0 = tried ? w : 0; b0 < w; b0 += CB) {
    const int end = min(b0 + CB, w);
#pragma unroll 1
    for (int jj = b0; jj < end; jj++) {
      const int buf = jj & 1;
      const unsigned tag = (unsigned)(c0 + jj) + 1u;
      Key* kOwn = sKey + buf * 2 * SP_WARPS;
      Key* kAll = kOwn + SP_WARPS;
      int* iOwn = sIdx + buf * 2 * SP_WARPS;
      int* iAll = iOwn + SP_WARPS;
      T* rows = sRow + buf * SP_WARPS * RW;
      T* top = sTop + buf * RW;
      // ---- this CTA's candidate among its rows from the diagonal on
      Key key = 0;
      int idx = NONE;
      if (!helper) {
#pragma unroll
        for (int i = 0; i < RPT; i++) {
          const int r = row_of(i);
          if (r < nr && lo + r >= jj) {
            const Key k = pivot_key(a[i][0]);
            if (k > key) {
              key = k;
              idx = lo + r;
            }
          }
        }
        warp_best(key, idx);
        if (lane == 0) {
          kOwn[warp] = key;
          iOwn[warp] = idx;
        }
      }
      __syncthreads();
      key = lane < NWR ? kOwn[lane] : Key(0);
      idx = lane < NWR ? iOwn[lane] : NONE;
      warp_best(key, idx);
      const bool have = key != 0;
      const bool diag_best = cta == 0 && have && idx == jj;  // one row to post, as candidate and diagonal row
      if (warp == (have ? owner_warp(idx - lo) : 0)) {
        T v = T{0, 0};
        if (have) v = row_values(idx - lo, jj, end);
        if (CLUSTER) {
#pragma unroll 4
          for (int g = 0; g < Gb; g++) {
            sp_store_remote(sp_remote(rows + cta * RW + lane, g), v);
            if (lane == 0) sp_store_remote(sp_remote(iAll + cta, g), have ? idx : NONE);
          }
        } else if (Gb > 1) {
          LL<T>::post(slot(buf, cta) + lane * LL<T>::BYTES, v,
                      (unsigned long long)tag | ((unsigned long long)(unsigned)(have ? idx : NONE) << 32));
        } else {
          rows[lane] = v;
        }
        if (diag_best) post_top(v, top, buf, tag);
      }
      if (cta == 0 && !diag_best && warp == owner_warp(jj)) post_top(row_values(jj, jj, end), top, buf, tag);
      // ---- the column's pivot row and the diagonal row, from all CTAs
      if (!CLUSTER && Gb > 1) {
        Key bk = 0;
        int bi = NONE;
        if (one_hop) {
          // all of this warp's slots are asked for before the first is waited for
          T v[LL_PER_WARP], bv = T{0, 0};
          unsigned long long hi[LL_PER_WARP];
          bool ok[LL_PER_WARP];
#pragma unroll
          for (int k = 0; k < LL_PER_WARP; k++) {
            const int g = warp + k * NW;
            ok[k] = true;
            if (g <= Gb) ok[k] = LL<T>::poll(slot(buf, g) + lane * LL<T>::BYTES, v[k], hi[k], tag);
          }
#pragma unroll
          for (int k = 0; k < LL_PER_WARP; k++) {
            const int g = warp + k * NW;
            if (g <= Gb) {
              if (!__all_sync(0xffffffffu, ok[k])) {
                T tv;
                unsigned long long th;
                wait_row(slot(buf, g) + lane * LL<T>::BYTES, tag, tv, th);
                v[k] = tv;
                hi[k] = th;
              }
              if (g == Gb) {
                top[lane] = v[k];
              } else {
                const int gi = (int)(hi[k] >> 32);
                T d;
                d.x = __shfl_sync(0xffffffffu, v[k].x, jj);
                d.y = __shfl_sync(0xffffffffu, v[k].y, jj);
                const Key gk = gi != NONE ? pivot_key(d) : Key(0);
                if (gk > bk || (gk == bk && gi < bi)) {
                  bk = gk;
                  bi = gi;
                  bv = v[k];
                }
              }
            }
          }
          rows[warp * RW + lane] = bv;
        } else if (helper) {
          T v;
          unsigned long long hi;
          wait_row(slot(buf, Gb) + lane * LL<T>::BYTES, tag, v, hi);
          top[lane] = v;
        } else {
          for (int g0 = warp * 32; g0 < Gb; g0 += NWR * 32) {
            const int g = min(g0 + lane, Gb - 1);
            T v;
            unsigned long long hi;
            wait_row(slot(buf, g) + jj * LL<T>::BYTES, tag, v, hi);
            const int gi = (int)(hi >> 32);
            const Key gk = gi != NONE ? pivot_key(v) : Key(0);
            if (gk > bk || (gk == bk && gi < bi)) {
              bk = gk;
              bi = gi;
            }
          }
          warp_best(bk, bi);
        }
        if (lane == 0) {
          kAll[warp] = bk;
          iAll[warp] = bi;
        }
      }
      if (CLUSTER) sp_cluster_sync();
      else __syncthreads();
      int ww = 0;
      if (CLUSTER) {
        idx = lane < Gb ? iAll[lane] : NONE;
        key = idx != NONE ? pivot_key(rows[lane * RW + jj]) : Key(0);
        ww = warp_best(key, idx);
      } else if (Gb > 1) {
        key = lane < NW ? kAll[lane] : Key(0);
        idx = lane < NW ? iAll[lane] : NONE;
        ww = warp_best(key, idx);
        if (!one_hop) {
          // the second trip: one warp fetches the winner's row (more readers of
          // these few lines of L2 make it slower)
          if (helper && key != 0) {
            T v;
            unsigned long long hi;
            wait_row(slot(buf, min(idx / chunk, Gb - 1)) + lane * LL<T>::BYTES, tag, v, hi);
            rows[ww * RW + lane] = v;
          }
          __syncthreads();
        }
      }
      const bool zero = key <= 1;  // no candidate, or a column of zeros
      const int piv = zero ? jj : min(idx, m - 1);  // within the matrix whatever a run-out wait left
      const T* prow = zero ? top : rows + ww * RW;
      if (helper) {
        // the pivot row solved with the block's earlier pivots, for the columns right of the block
        T v = prow[lane], us[CB];
        load_u(sU + lane * CB, us);
#pragma unroll
        for (int d = 0; d < CB; d++) {
          const T l = prow[b0 + d];
          if (d < jj - b0) {
            v.x -= l.x * us[d].x - l.y * us[d].y;
            v.y -= l.x * us[d].y + l.y * us[d].x;
          }
        }
        sU[lane * CB + jj - b0] = v;
        if (lane == 0) {
          sPiv[jj] = c0 + piv;
          if (cta == 0 && zero && bt.info[grp] == 0) bt.info[grp] = c0 + jj + 1;
        }
        continue;
      }
      // ---- interchange
      if (piv != jj) {
        const int rp = piv - lo;
        if (rp >= 0 && rp < nr && warp == owner_warp(rp)) set_row(rp, top, jj);
        if (cta == 0 && warp == owner_warp(jj)) set_row(jj, prow, jj);
      }
      // ---- eliminate within the block; column jj goes to shared memory
      const T rd = pivot_recip(prow[jj]);
      T u[CB];
#pragma unroll
      for (int k = 1; k < CB; k++) u[k] = prow[jj + k];
#pragma unroll
      for (int i = 0; i < RPT; i++) {
        const int r = row_of(i);
        const bool on = r < nr && lo + r > jj && !zero;
        T l = T{0, 0};
        if (on) {
          l.x = a[i][0].x * rd.x - a[i][0].y * rd.y;
          l.y = a[i][0].x * rd.y + a[i][0].y * rd.x;
        }
        if (r < nr) sA[r * SP + jj] = on ? l : a[i][0];
#pragma unroll
        for (int k = 1; k < CB; k++) {
          a[i][k - 1] = a[i][k];
          if (on) {
            a[i][k - 1].x -= l.x * u[k].x - l.y * u[k].y;
            a[i][k - 1].y -= l.x * u[k].y + l.y * u[k].x;
          }
        }
      }
    }
    // ---- the columns right of the block take its CB pivots
    __syncthreads();
    if (!helper && b0 + CB < w) {
      // (a block followed by another has all its CB columns)
      T l[RPT][CB];
#pragma unroll
      for (int i = 0; i < RPT; i++)
#pragma unroll
        for (int c = 0; c < CB; c++) l[i][c] = row_of(i) < nr ? sA[row_of(i) * SP + b0 + c] : T{0, 0};
      // QU columns at a time: independent chains, since few warps share a scheduler
      constexpr int QU = 4;
      for (int q0 = b0 + CB; q0 < w; q0 += QU) {
        T v[RPT][QU];
#pragma unroll
        for (int i = 0; i < RPT; i++)
#pragma unroll
          for (int j = 0; j < QU; j++) v[i][j] = row_of(i) < nr ? sA[row_of(i) * SP + min(q0 + j, IB)] : T{0, 0};
#pragma unroll
        for (int j = 0; j < QU; j++) {
          T us[CB];
          load_u(sU + min(q0 + j, IB - 1) * CB, us);
#pragma unroll
          for (int i = 0; i < RPT; i++)
#pragma unroll
            for (int c = 0; c < CB; c++) {
              v[i][j].x -= l[i][c].x * us[c].x - l[i][c].y * us[c].y;
              v[i][j].y -= l[i][c].x * us[c].y + l[i][c].y * us[c].x;
            }
        }
#pragma unroll
        for (int i = 0; i < RPT; i++) {
          const int r = row_of(i), gr = lo + r;
          if (r >= nr || gr < b0) continue;
#pragma unroll
          for (int j = 0; j < QU; j++)
            if (q0 + j < w)  // a pivot row of this block takes its solved values
              sA[r * SP + q0 + j] = gr < b0 + CB ? sU[(q0 + j) * CB + gr - b0] : v[i][j];
        }
      }
      load_block(b0 + CB);
    }
  }
  __syncthreads();
  for (int r0 = warp; r0 < nr; r0 += 8 * NW) {
    T v[8];  // read before the first is written
#pragma unroll
    for (int q = 0; q < 8; q++) v[q] = sA[min(r0 + q * NW, nr - 1) * SP + col];
#pragma unroll
    for (int q = 0; q < 8; q++)
      if (r0 + q * NW < nr && lane < w) A[(size_t)(c0 + lo + r0 + q * NW) * n + c0 + lane] = v[q];
  }
  if (cta == 0 && tid < w) batch_pick(bt.ipiv, grp)[c0 + tid] = sPiv[tid];
  if (cta == 0 && tid == 0) {
    // (every CTA has read them by now: its records were waited for)  After a failure in a
    // row the next 1, 3, 7, then 15 sub-panels go without a try
    if (!trying) {
      tries[0] = max(tries[0] - 1, 0);
    } else if (tried) {
      tries[1] = 0;
    } else {
      tries[0] = tries[1];
      tries[1] = min(2 * tries[1] + 1, 15);
    }
  }
  if (pk1 - pk0 > w) {
    const unsigned moves = __ballot_sync(0xffffffffu, lane < w && sPiv[col] != c0 + lane);
    const int nl = c0 - pk0, nc = nl + (pk1 - (c0 + w));
    for (int t = cta * blockDim.x + tid; t < nc; t += Gb * blockDim.x) {
      const int q = t < nl ? pk0 + t : c0 + w + (t - nl);
      for (unsigned left = moves; left; left &= left - 1) {
        const int jj = __ffs(left) - 1;
        T* x = A + (size_t)(c0 + jj) * n + q;
        T* y = A + (size_t)sPiv[jj] * n + q;
        const T v = *x;
        *x = *y;
        *y = v;
      }
    }
  }
}

// X = L^{-1} for the w x w unit-lower block L at (r0, r0) of A (ld n),
// w <= INV_MAX, into X[w][w] (row-major, ld w), by recursive doubling:
// k_inv_diag32 inverts the 32 x 32 diagonal blocks (one CTA each), then per
// level s = 64, 128, .. every pair of inverted s/2 blocks is joined,
//   [X11 0; X21 X22] with X21 = -X22 (L21 X11),
// first T = L21 X11, then X21 = -X22 T, one CTA per tile (k_inv_join), all pairs
// of a level in the same two launches.  Entries above the diagonal are written as zero.
constexpr int INV_MAX = 512;

constexpr int INV32_LD = 34, INV32_SCRATCH = 256;  // of inv_unit32

// One level of inv_unit32: per 32 x 32 block, the pairs of inverted H x H blocks are
// joined by S = L21 X11, X21 = -X22 S, an output a thread.
template <int NB, int H, int LD, typename T>
__device__ __forceinline__ void inv_unit32_join(const T* L, T* X, T* S) {
  constexpr int PAIRS = 16 / H, XLD = INV32_LD;
#pragma unroll
  for (int step = 0; step < 2; step++) {
    for (int o = threadIdx.x; o < NB * PAIRS * H * H; o += 256) {
      const int p = o / (H * H), r = o / H % H, c = o % H, q = p / PAIRS, i0 = p % PAIRS * 2 * H;
      const T* a = step == 0 ? L + (32 * q + i0 + H + r) * LD + 32 * q + i0 : X + (32 * q + i0 + H + r) * XLD + i0 + H;
      const T* b = step == 0 ? X + (32 * q + i0) * XLD + i0 + c : S + p * H * H + c;
      T v[2];
      v[0].x = v[0].y = v[1].x = v[1].y = 0;
#pragma unroll
      for (int k = 0; k < H; k++) {
        if (step == 0)
          cfma_add(v[k & 1], a[k], b[k * XLD]);
        else
          cfma_sub(v[k & 1], a[k], b[k * H]);
      }
      v[0].x += v[1].x;
      v[0].y += v[1].y;
      if (step == 0)
        S[o] = v[0];
      else
        X[(32 * q + i0 + H + r) * XLD + i0 + c] = v[0];
    }
    __syncthreads();
  }
}

// Inverses of the NB unit-lower 32 x 32 diagonal blocks of L (shared, row stride LD,
// only entries below the diagonal are read) into X[NB 32][INV32_LD], zeros above the
// diagonal; S: scratch of INV32_SCRATCH NB elements; 256 threads, synchronised at the
// end.  Bound: latency.  A column a lane through all 32 rows took 21,000 clocks, each
// row waiting for its sums over shared memory; 8 x 8 blocks in registers and two joins
// take a tenth of that.
template <int NB, int LD, typename T>
__device__ __forceinline__ void inv_unit32(const T* L, T* X, T* S) {
  if (threadIdx.x < NB * 32) {
    const int c = threadIdx.x & 31, e = c & ~7, row0 = threadIdx.x & ~31;
    const T* l = L + (row0 + e) * LD + row0 + e;
    T v[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      v[i].x = e + i == c ? 1 : 0;
      v[i].y = 0;
#pragma unroll
      for (int j = 0; j < i; j++) cfma_sub(v[i], l[i * LD + j], v[j]);
    }
    T zero;
    zero.x = zero.y = 0;
    for (int i = 0; i < e; i++) X[(row0 + i) * INV32_LD + c] = zero;
#pragma unroll
    for (int i = 0; i < 8; i++) X[(row0 + e + i) * INV32_LD + c] = v[i];
  }
  __syncthreads();
  inv_unit32_join<NB, 8, LD>(L, X, S);
  inv_unit32_join<NB, 16, LD>(L, X, S);
}

// Matrices whose unit-lower blocks are inverted in the same launches: block
// (blockIdx.y for the diagonal blocks, blockIdx.z / pairs for the joins)
// picks matrix b, whose inverse is X + b w w and join scratch T + b w w / 2.
template <typename T>
struct InvBatch {
  const T* A[4];
};

template <typename T>
__global__ void __launch_bounds__(256) k_inv_diag32(InvBatch<T> ib, int n, int r0, int w, T* __restrict__ X) {
  __shared__ T sL[32][33];
  __shared__ T sX[32][INV32_LD];
  __shared__ T sS[INV32_SCRATCH];
  const T* __restrict__ A = ib.A[blockIdx.y];
  X += (size_t)blockIdx.y * w * w;
  const int i0 = blockIdx.x * 32, hi = min(32, w - i0);
#pragma unroll
  for (int t = threadIdx.x; t < 32 * 32; t += 256) {
    const int i = t >> 5, j = t & 31;
    T l;
    l.x = 0;
    l.y = 0;
    if (i < hi && j < hi) l = A[(size_t)(r0 + i0 + i) * n + r0 + i0 + j];
    sL[i][j] = l;
  }
  __syncthreads();
  inv_unit32<1, 33>(&sL[0][0], &sX[0][0], sS);
  // the whole 32-row band of X: the diagonal block, zeros elsewhere in the band
  for (int i = threadIdx.x >> 5; i < hi; i += 8) {
    T* row = X + (size_t)(i0 + i) * w;
    const int lane = threadIdx.x & 31;
    T zero;
    zero.x = zero.y = 0;
    const T v = lane <= i ? sX[i][lane] : zero;
#pragma unroll 4
    for (int c = lane; c < w; c += 32) row[c] = c - lane == i0 ? v : zero;
  }
}

// Level s: pair p joins the blocks [p s, p s + h) and [p s + h, p s + s), h = s / 2
// (the second may be shorter at the end of w) in two launches of one CTA per tile of
// 32 rows of block 2 (ty) and 16 columns of block 1 (tx):
//   k_inv_join<.., false>:  Tp = L21 X11     (X11 lower: k from the tile's column)
//   k_inv_join<.., true>:   X21 = -X22 Tp    (X22 lower: k up to the tile's row)
// Tp is the pair's h x h scratch at T + p h h.  The whole depth of both operands is
// asked for at once (cp.async), a thread then sums two elements.  Bound: latency and,
// from h = 128 on, FP32 issue.  The eight joins of a 512 x 512 block, two matrices,
// against 32 x 32 tiles staged 32 deep one after another: 127 -> 54 us (n = 16,128).
constexpr int JT_M = 32, JT_N = 16;
template <typename T>
size_t inv_join_smem(int h) {
  return sizeof(T) * ((size_t)JT_M * (h + 2) + (size_t)h * (JT_N + 1));
}
template <typename T, bool SECOND>
__global__ void __launch_bounds__(256) k_inv_join(InvBatch<T> ib, int n, int r0, int w, int s, T* __restrict__ X,
                                                  T* __restrict__ Tsc) {
  extern __shared__ __align__(16) unsigned char join_raw[];
  const int h = s / 2, lda = h + 2, ldb = JT_N + 1;
  T* sa = reinterpret_cast<T*>(join_raw);  // [JT_M][lda]
  T* sb = sa + JT_M * lda;                 // [h][ldb]
  const int pairs = (w + s - 1) / s, mb = blockIdx.z / pairs;
  const int p = blockIdx.z - mb * pairs, base = p * s;
  const T* __restrict__ A = ib.A[mb];
  X += (size_t)mb * w * w;
  T* Tp = Tsc + (size_t)mb * w * w / 2 + (size_t)p * h * h;
  const int h2 = min(h, w - base - h);  // rows of the second block, a multiple of 32
  const int i0 = blockIdx.y * JT_M, c0 = blockIdx.x * JT_N;
  if (i0 >= h2) return;
  const int k0 = SECOND ? 0 : c0 & ~31, k1 = SECOND ? i0 + JT_M : h;  // multiples of 32
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const T* a = SECOND ? X + (size_t)(base + h + i0) * w + base + h : A + (size_t)(r0 + base + h + i0) * n + r0 + base;
  const T* b = SECOND ? Tp + c0 : X + (size_t)base * w + base + c0;
  const int la = SECOND ? w : n, lb = SECOND ? h : w;
  for (int i = warp; i < JT_M; i += 8)
    for (int k = k0 + lane; k < k1; k += 32) sp_cp_async(sa + i * lda + k, a + (size_t)i * la + k);
  const int col = tid % JT_N, row = tid / JT_N;
  for (int k = k0 + row; k < k1; k += 256 / JT_N) sp_cp_async(sb + k * ldb + col, b + (size_t)k * lb + col);
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  T v[2][2];  // two rows, two partial sums each
#pragma unroll
  for (int u = 0; u < 2; u++) v[u][0] = v[u][1] = T{0, 0};
  const T *x = sa + row * lda, *y = x + JT_M / 2 * lda;
#pragma unroll 4
  for (int k = k0; k < k1; k += 2) {
    const T b0 = sb[k * ldb + col], b1 = sb[(k + 1) * ldb + col];
    cfma_add(v[0][0], x[k], b0);
    cfma_add(v[1][0], y[k], b0);
    cfma_add(v[0][1], x[k + 1], b1);
    cfma_add(v[1][1], y[k + 1], b1);
  }
#pragma unroll
  for (int u = 0; u < 2; u++) {
    const int i = i0 + row + u * (JT_M / 2);
    const T r = T{v[u][0].x + v[u][1].x, v[u][0].y + v[u][1].y};
    if (SECOND)
      X[(size_t)(base + h + i) * w + base + c0 + col] = T{-r.x, -r.y};
    else
      Tp[(size_t)i * h + c0 + col] = r;
  }
}

// Interchanges of pivots [p0, p1), at most LS_MAX, applied to columns [a0, a1) and
// [b0, b1) of the batch's matrices (blockIdx.y).  Most pivots of 1 - A G lie on the
// diagonal: a CTA first lists the actual moves, in order, then its threads, a column
// each, make them four at a time, all eight loads before the stores, where the four
// touch no row twice.  Bound: latency of the moves.  512 pivots of four
// matrices, n = 20,160: 159 -> 3.6 us (a dependent step per pivot, a launch a matrix,
// before).
constexpr int LS_MAX = 512, LS_THREADS = 256;
template <typename T>
__global__ void __launch_bounds__(LS_THREADS) k_laswp2(SubpanelBatch<T> bt, int n, int p0, int p1, int a0, int a1,
                                                       int b0, int b1) {
  __shared__ int s_piv[LS_MAX];
  __shared__ int2 s_move[LS_MAX + 4];
  __shared__ int s_count;
  const int32_t* ipiv = batch_pick(bt.ipiv, blockIdx.y);
  const int np = p1 - p0;
  for (int i = threadIdx.x; i < np; i += LS_THREADS) s_piv[i] = ipiv[p0 + i];
  __syncthreads();
  if (threadIdx.x < 32) {
    int cnt = 0;
    for (int i0 = 0; i0 < np; i0 += 32) {
      const int i = i0 + threadIdx.x, p = i < np ? s_piv[i] : p0 + i;
      const unsigned moves = __ballot_sync(0xffffffffu, p != p0 + i);
      if (p != p0 + i) s_move[cnt + __popc(moves & ((1u << threadIdx.x) - 1u))] = make_int2(p0 + i, p);
      cnt += __popc(moves);
    }
    if (threadIdx.x == 0) s_count = cnt;
  }
  __syncthreads();
  const int t = blockIdx.x * LS_THREADS + threadIdx.x;
  const int na = a1 - a0;
  int c;
  if (t < na) c = a0 + t;
  else if (t - na < b1 - b0) c = b0 + (t - na);
  else return;
  T* A = batch_pick(bt.A, blockIdx.y) + c;
  const int cnt = s_count;
  for (int i = 0; i < cnt; i += 4) {
    int2 m[4];
    bool apart = i + 4 <= cnt;
#pragma unroll
    for (int u = 0; u < 4; u++) m[u] = s_move[i + u];
    // the diagonal rows differ; a pivot row may be another move's pivot or diagonal row
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
      for (int v = 0; v < 4; v++)
        if (v != u) apart = apart && m[u].y != m[v].x && (v < u || m[u].y != m[v].y);
    if (apart) {
      T x[4], y[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        x[u] = A[(size_t)m[u].x * n];
        y[u] = A[(size_t)m[u].y * n];
      }
#pragma unroll
      for (int u = 0; u < 4; u++) {
        A[(size_t)m[u].x * n] = y[u];
        A[(size_t)m[u].y * n] = x[u];
      }
    } else {
      for (int u = 0; u < 4 && i + u < cnt; u++) {
        const int2 mv = s_move[i + u];
        const T x = A[(size_t)mv.x * n];
        A[(size_t)mv.x * n] = A[(size_t)mv.y * n];
        A[(size_t)mv.y * n] = x;
      }
    }
  }
}

// The matrices of a batch whose same 32-row block is solved in one launch
// (blockIdx.y = matrix); matrix b's operand planes start at WB + b plane.
template <typename T>
struct TrsmBatch {
  T* A[4];
  unsigned char* WB;
  size_t plane;
};

// X <- L^{-1} X for the h x h unit-lower block (h = 32 NB <= 128) at (r0, r0) of each
// matrix of the batch (blockIdx.y), X = rows [r0, r0 + h) of columns [cb, ce),
// complex64, also packed as the B operand of the update that follows.  A CTA inverts
// the 32 x 32 diagonal blocks (inv_unit32), then takes chunks of 8 columns: block by
// block x_j = D_j^{-1} b_j, an element a thread, and L x_j off the rows below, L as
// 16-byte broadcasts.  Bound: latency of these steps (8 columns a CTA, as narrow as a
// 64-byte row segment allows).  It stands for the explicit inverse of a mid-panel's
// block, a pack, a tensor-core product and another pack (66 -> 13 us on average at 128 x up to
// 384, n = 16,128) and for a substitution row by row (10 -> 4 us at 32 x up to 96).
// complex128 (h = 32, not packed): 11.5 -> 7.2 us on average over the factorisation of
// n = 8,496.
constexpr int TR_MAX = 128, TR_COLS = 8, TR_XLD = TR_COLS + 1;
template <typename T, int NB>
constexpr size_t trsm_rows_smem() {
  return sizeof(T) * (32 * NB * (32 * NB + 2) + 32 * NB * TR_XLD + 32 * NB * INV32_LD + INV32_SCRATCH * NB);
}
// two neighbouring elements of shared memory, the first on a 2-element boundary
__device__ __forceinline__ void load_pair(const float2* p, float2& a, float2& b) {
  const float4 f = *reinterpret_cast<const float4*>(p);
  a = make_float2(f.x, f.y);
  b = make_float2(f.z, f.w);
}
__device__ __forceinline__ void load_pair(const double2* p, double2& a, double2& b) {
  a = p[0];
  b = p[1];
}
template <typename T, int NB>
__global__ void __launch_bounds__(256) k_trsm_rows(TrsmBatch<T> tb, int n, int r0, int cb, int ce, int pack_mode) {
  constexpr int H = 32 * NB, LD = H + 2;
  extern __shared__ __align__(16) unsigned char tr_raw[];
  T* sL = reinterpret_cast<T*>(tr_raw);  // [H][LD]
  T* sX = sL + H * LD;                   // [H][TR_XLD]
  T* sD = sX + H * TR_XLD;               // [H][INV32_LD]
  T* sS = sD + H * INV32_LD;
  T* A = tb.A[blockIdx.y];
  void* WB = tb.WB ? tb.WB + tb.plane * blockIdx.y : nullptr;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row = threadIdx.x / TR_COLS, col = threadIdx.x % TR_COLS;
  pdl_wait();
  pdl_launch_next();
  for (int i = warp; i < H; i += 8)
    for (int q = 0; q <= i / 32; q++)
      sp_cp_async(sL + i * LD + 32 * q + lane, A + (size_t)(r0 + i) * n + r0 + 32 * q + lane);
  for (int c0 = cb + blockIdx.x * TR_COLS; c0 < ce; c0 += gridDim.x * TR_COLS) {
    const int c = c0 + col;
#pragma unroll
    for (int q = 0; q < NB; q++) {
      const int i = 32 * q + row;
      if (c < ce)
        sp_cp_async(sX + i * TR_XLD + col, A + (size_t)(r0 + i) * n + c);
      else
        sX[i * TR_XLD + col] = T{0, 0};
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    if (c0 == cb + (int)blockIdx.x * TR_COLS) inv_unit32<NB, LD>(sL, sD, sS);
#pragma unroll
    for (int j = 0; j < NB; j++) {
      const T* Y = sD + (32 * j + row) * INV32_LD;
      const T* xj = sX + 32 * j * TR_XLD + col;
      T v[2] = {T{0, 0}, T{0, 0}};
#pragma unroll 4
      for (int k = 0; k < warp * 4; k += 2) {
        T y0, y1;
        load_pair(Y + k, y0, y1);
        cfma_add(v[0], y0, xj[k * TR_XLD]);
        cfma_add(v[1], y1, xj[(k + 1) * TR_XLD]);
      }
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (warp * 4 + u <= row) cfma_add(v[u & 1], Y[warp * 4 + u], xj[(warp * 4 + u) * TR_XLD]);
      __syncthreads();
      sX[(32 * j + row) * TR_XLD + col] = T{v[0].x + v[1].x, v[0].y + v[1].y};
      __syncthreads();
      if (j + 1 < NB) {
        constexpr int REST = NB > 1 ? NB - 1 : 1;
        T a[REST];
#pragma unroll
        for (int u = 0; u < REST; u++)
          if (j + 1 + u < NB) a[u] = sX[(32 * (j + 1 + u) + row) * TR_XLD + col];
#pragma unroll 4
        for (int k = 0; k < 32; k += 2) {
          const T b0 = xj[k * TR_XLD], b1 = xj[(k + 1) * TR_XLD];
#pragma unroll
          for (int u = 0; u < REST; u++)
            if (j + 1 + u < NB) {
              T l0, l1;
              load_pair(sL + (32 * (j + 1 + u) + row) * LD + 32 * j + k, l0, l1);
              cfma_sub(a[u], l0, b0);
              cfma_sub(a[u], l1, b1);
            }
        }
#pragma unroll
        for (int u = 0; u < REST; u++)
          if (j + 1 + u < NB) sX[(32 * (j + 1 + u) + row) * TR_XLD + col] = a[u];
        __syncthreads();
      }
    }
#pragma unroll
    for (int q = 0; q < NB; q++)
      if (c < ce) A[(size_t)(r0 + 32 * q + row) * n + c] = sX[(32 * q + row) * TR_XLD + col];
    if constexpr (sizeof(T) == sizeof(float2)) {
      if (pack_mode && c0 + warp < ce) {
#pragma unroll
        for (int q = 0; q < NB; q++)
          tc2_pack_b(pack_mode, WB, ce - cb, H, c0 + warp - cb, 32 * q + lane, sX[(32 * q + lane) * TR_XLD + warp]);
      }
    }
    __syncthreads();
  }
}

// C[M x N] -= L[M x K] U[K x N], complex, leading dimensions ld*; 64 x 64 tiles.
template <typename T>
__global__ void __launch_bounds__(256) k_gemm_sub(T* __restrict__ C, int ldc, const T* __restrict__ L, int ldl,
                                                  const T* __restrict__ U, int ldu, int M, int N, int K) {
  using R = typename Real<T>::R;
  constexpr int BM = 64, BN = 64, BK = 16;
  __shared__ T sA[BK][BM + 1];
  __shared__ T sB[BK][BN + 1];
  const int r0 = blockIdx.y * BM, c0 = blockIdx.x * BN;
  const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
  R ar[4][4], ai[4][4];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) ar[i][j] = ai[i][j] = 0;
  for (int k0 = 0; k0 < K; k0 += BK) {
    for (int t = threadIdx.x; t < BM * BK; t += 256) {
      const int i = t / BK, q = t % BK;
      T v;
      v.x = 0;
      v.y = 0;
      if (r0 + i < M && k0 + q < K) v = L[(size_t)(r0 + i) * ldl + k0 + q];
      sA[q][i] = v;
    }
    for (int t = threadIdx.x; t < BK * BN; t += 256) {
      const int q = t / BN, j = t % BN;
      T v;
      v.x = 0;
      v.y = 0;
      if (c0 + j < N && k0 + q < K) v = U[(size_t)(k0 + q) * ldu + c0 + j];
      sB[q][j] = v;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < BK; q++) {
      T a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; i++) a[i] = sA[q][ty + 16 * i];
#pragma unroll
      for (int j = 0; j < 4; j++) b[j] = sB[q][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
          ar[i][j] += a[i].x * b[j].x - a[i].y * b[j].y;
          ai[i][j] += a[i].x * b[j].y + a[i].y * b[j].x;
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int r = r0 + ty + 16 * i;
    if (r >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int c = c0 + tx + 16 * j;
      if (c >= N) continue;
      T v = C[(size_t)r * ldc + c];
      v.x -= ar[i][j];
      v.y -= ai[i][j];
      C[(size_t)r * ldc + c] = v;
    }
  }
}

template <typename T>
int gemm_sub(T* C, int ldc, const T* L, int ldl, const T* U, int ldu, int M, int N, int K, cudaStream_t st) {
  if (M <= 0 || N <= 0 || K <= 0) return TT_OK;
  if constexpr (sizeof(T) == sizeof(double2))
    return zgemm_sub_dmma(reinterpret_cast<double2*>(C), ldc, reinterpret_cast<const double2*>(L), ldl,
                          reinterpret_cast<const double2*>(U), ldu, M, N, K, st);
  dim3 grid(ceil_div(N, 64), ceil_div(M, 64));
  ProfScope prof(TT_PROF_SIMT_UPDATE, st, 8.0 * M * N * K, 2.0 * M * N * sizeof(T) + ((double)M + N) * K * sizeof(T));
  k_gemm_sub<T><<<grid, 256, 0, st>>>(C, ldc, L, ldl, U, ldu, M, N, K);
  count_launch();
  TT_CUDA_TRY(cudaGetLastError());
  return TT_OK;
}

template <typename T>
int laswp2(T* const* As, int B, int n, int32_t* const* ipivs, int p0, int p1, int a0, int a1, int b0, int b1,
           cudaStream_t st) {
  const int cols = std::max(0, a1 - a0) + std::max(0, b1 - b0);
  if (cols <= 0 || p1 <= p0) return TT_OK;
  SubpanelBatch<T> bt{};
  for (int b = 0; b < B; b++) {
    bt.A[b] = As[b];
    bt.ipiv[b] = ipivs[b];
  }
  ProfScope prof(TT_PROF_LASWP, st, 0.0, 4.0 * (p1 - p0) * cols * sizeof(T) * B);
  for (int p = p0; p < p1; p += LS_MAX) {
    k_laswp2<T><<<dim3(ceil_div(cols, LS_THREADS), B), LS_THREADS, 0, st>>>(bt, n, p, std::min(p1, p + LS_MAX), a0,
                                                                           std::max(a0, a1), b0, std::max(b0, b1));
    count_launch();
    TT_CUDA_TRY(cudaGetLastError());
  }
  return TT_OK;
}

// X: B w w elements (inverse of matrix b at X + b w w, ld w); Tsc: scratch of
// at least B w w / 2 elements.  B <= 4.
template <typename T>
int inv_unit_lower(const T* const* As, int B, int n, int r0, int w, T* X, T* Tsc, cudaStream_t st) {
  if (w <= 0) return TT_OK;
  InvBatch<T> ib{};
  for (int b = 0; b < B; b++) ib.A[b] = As[b];
  if (w > INV_MAX || w % 32 != 0) {
    set_error("unit-lower inverse of a block of " + std::to_string(w) + " rows (multiples of 32 up to " +
              std::to_string(INV_MAX) + ")");
    return TT_ERR_BADARG;
  }
  ProfScope prof(TT_PROF_PANEL_TRSM, st, 8.0 / 6.0 * w * (double)w * w * B, 2.0 * w * (double)w * sizeof(T) * B);
  k_inv_diag32<T><<<dim3(w / 32, B), 256, 0, st>>>(ib, n, r0, w, X);
  count_launch();
  TT_CUDA_TRY(cudaGetLastError());
  const int join_smem = (int)inv_join_smem<T>(INV_MAX / 2);
  TT_TRY(smem_limit_once((const void*)k_inv_join<T, false>, join_smem));
  TT_TRY(smem_limit_once((const void*)k_inv_join<T, true>, join_smem));
  for (int s = 64; s / 2 < w; s *= 2) {
    const int h = s / 2;
    const dim3 grid(h / JT_N, h / JT_M, ((w + s - 1) / s) * B);
    const size_t smem = inv_join_smem<T>(h);
    k_inv_join<T, false><<<grid, 256, smem, st>>>(ib, n, r0, w, s, X, Tsc);
    count_launch();
    TT_CUDA_TRY(cudaGetLastError());
    k_inv_join<T, true><<<grid, 256, smem, st>>>(ib, n, r0, w, s, X, Tsc);
    count_launch();
    TT_CUDA_TRY(cudaGetLastError());
  }
  return TT_OK;
}

// k_trsm_rows of B <= 4 matrices, h a multiple of 32 up to TR_MAX; no more CTAs than fit
// at once, as a CTA's block inverses serve all its chunks
template <typename T, int NB>
int launch_trsm_rows(const TrsmBatch<T>& tb, int B, int n, int r0, int cb, int ce, int pack_mode, cudaStream_t st) {
  constexpr size_t smem = trsm_rows_smem<T, NB>();
  constexpr int resident = std::max(1, std::min(4, (int)(200 * 1024 / smem)));
  const int chunks = ceil_div(ce - cb, TR_COLS), per = std::max(1, resident * device_sm_count() / B);
  TT_TRY(smem_limit_once((const void*)k_trsm_rows<T, NB>, (int)smem));
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1] = {pdl_attribute()};
  cfg.gridDim = dim3(ceil_div(chunks, ceil_div(chunks, per)), B);
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  TT_CUDA_TRY(cudaLaunchKernelEx(&cfg, k_trsm_rows<T, NB>, tb, n, r0, cb, ce, pack_mode));
  count_launch();
  return TT_OK;
}
// Pack_mode: matrix b's solved rows also go to its operand planes at WB + b plane.
// Panels, mid-panels and their halves are multiples of 32 wide; only the matrix's last
// sub-panel is narrower, with nothing behind it.
template <typename T>
int trsm_rows_batched(T* const* As, int B, int n, int r0, int h, int cb, int ce, cudaStream_t st, int pack_mode = 0,
                      unsigned char* WB = nullptr, size_t plane = 0) {
  if (ce <= cb) return TT_OK;
  if (h % IB != 0 || h > (sizeof(T) == sizeof(float2) ? TR_MAX : IB)) {
    set_error("block row solve of " + std::to_string(h) + " rows");
    return TT_ERR_BADARG;
  }
  ProfScope prof(TT_PROF_PANEL_TRSM, st, 4.0 * h * h * (double)(ce - cb) * B,
                 2.0 * h * (double)(ce - cb) * sizeof(T) * B);
  TrsmBatch<T> tb{};
  for (int b = 0; b < B; b++) tb.A[b] = As[b];
  tb.WB = WB;
  tb.plane = plane;
  if constexpr (sizeof(T) == sizeof(float2)) {
    switch (h / 32) {
      case 2: return launch_trsm_rows<T, 2>(tb, B, n, r0, cb, ce, pack_mode, st);
      case 3: return launch_trsm_rows<T, 3>(tb, B, n, r0, cb, ce, pack_mode, st);
      case 4: return launch_trsm_rows<T, 4>(tb, B, n, r0, cb, ce, pack_mode, st);
    }
  }
  return launch_trsm_rows<T, 1>(tb, B, n, r0, cb, ce, pack_mode, st);
}

// C -= L U on the tensor cores in the factorisation's product mode when K is
// a multiple of the mode's k-chunk, else on the CUDA cores
template <typename T>
int panel_gemm_sub(int mode, T* C, int ldc, const T* L, int ldl, const T* U, int ldu, int M, int N, int K,
                   cudaStream_t st) {
  if (M <= 0 || N <= 0 || K <= 0) return TT_OK;
  if (mode == TC_LEGACY_BF16X3 && K % 32 == 0)
    return tc_gemm_sub(reinterpret_cast<float2*>(C), ldc, reinterpret_cast<const float2*>(L), ldl,
                       reinterpret_cast<const float2*>(U), ldu, M, N, K, st);
  if ((mode == TC_TF32 || mode == TC_BF16X3) && K % 16 == 0)
    return tc2_gemm_sub(mode, reinterpret_cast<float2*>(C), ldc, reinterpret_cast<const float2*>(L), ldl,
                        reinterpret_cast<const float2*>(U), ldu, M, N, K, st);
  return gemm_sub(C, ldc, L, ldl, U, ldu, M, N, K, st);
}

// Largest cluster of full-size sub-panel CTAs the current device runs: 16, 8 or 1
template <typename T>
int query_subpanel_cluster() {
  const void* k = (const void*)k_subpanel_ll<T, 1, true>;
  if (smem_limit_once(k, (int)kSubpanelSmem) != TT_OK ||
      cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
    cudaGetLastError();
    return 1;
  }
  for (int g : {16, 8}) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = g;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.gridDim = dim3(g);
    cfg.blockDim = dim3(32 * SP_WARPS);
    cfg.dynamicSmemBytes = kSubpanelSmem;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k, &cfg) == cudaSuccess && n > 0) return g;
    cudaGetLastError();
  }
  return 1;
}
// ... asked once per device
template <typename T>
int subpanel_cluster() {
  static std::mutex mu;
  static std::map<int, int> largest;
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(mu);
  const auto it = largest.find(dev);
  return it != largest.end() ? it->second : largest[dev] = query_subpanel_cluster<T>();
}

}  // namespace

template <typename T>
int lu_factor_batched_device(T* const* As, int B, int n, int32_t* const* ipivs, cudaStream_t st, int use_tc,
                             int* info, bool blocked_order, int panel, int inv_block, bool cta_pairs, int mid) {
  const int mode = use_tc;
  const bool tc = mode != 0;
  if (mode < 0 || mode > TC_BF16X3) {
    set_error("unknown tensor-core product mode " + std::to_string(mode));
    return TT_ERR_BADARG;
  }
  if (tc && sizeof(T) != sizeof(float2)) {
    set_error("tensor-core trailing update is only defined for the complex64 factorisation");
    return TT_ERR_UNSUPPORTED;
  }
  if (B < 1 || B > kMaxBatch) {
    set_error("LU batch of " + std::to_string(B) + " matrices (1.." + std::to_string(kMaxBatch) + ")");
    return TT_ERR_BADARG;
  }
  if (panel < 0 || panel > INV_MAX || panel % IB != 0) {
    set_error("panel width " + std::to_string(panel) + " (a multiple of 32 up to 512)");
    return TT_ERR_BADARG;
  }
  if (mid < 0 || mid % IB != 0) {
    set_error("mid-panel width " + std::to_string(mid) + " (0 or a multiple of 32)");
    return TT_ERR_BADARG;
  }
  if (inv_block < 0 || inv_block > INV_MAX || inv_block % IB != 0) {
    set_error("inverse block " + std::to_string(inv_block) + " (a multiple of 32 up to 512)");
    return TT_ERR_BADARG;
  }
  const int IVB = inv_block ? inv_block : INV_MAX;
  // the update kernel's tile shape for this factorisation (restored on return)
  struct PairScope {
    explicit PairScope(bool on) { tc2_set_pairs(on); }
    ~PairScope() { tc2_set_pairs(false); }
  } pair_scope(cta_pairs);
  const int NB = panel ? panel : (sizeof(T) == sizeof(float2)) ? 512 : 128;
  const int G = device_sm_count();
  DevBuf<double> sval;
  DevBuf<int> sidx, d_info;
  DevBuf<T> srow, stop;
  DevBuf<unsigned char> srec;
  TT_TRY(sval.alloc(2 * (size_t)G));
  TT_TRY(sidx.alloc(2 * (size_t)G));
  TT_TRY(srow.alloc(2 * (size_t)G * IB));
  TT_TRY(stop.alloc(2 * (size_t)kMaxBatch * IB));
  // records of B matrices in one launch, or of each matrix in its own: one
  // region per matrix, since the matrices of separate launches share the tags
  const size_t rec_region = 2 * ((size_t)G + kMaxBatch) * IB * LL<T>::BYTES, rec_bytes = rec_region * B;
  const size_t verdicts = (size_t)G * LL<float2>::BYTES;  // of a matrix, behind the records
  TT_TRY(srec.alloc(rec_bytes + verdicts * B));
  TT_TRY(d_info.alloc(3 * B + 1));  // [B] first zero pivots, the sub-panels' error word, [B][2] tries
  TT_CUDA_TRY(cudaMemsetAsync(d_info.ptr, 0, sizeof(int) * (3 * B + 1), st));
  TT_CUDA_TRY(cudaMemsetAsync(srec.ptr, 0, rec_bytes + verdicts * B, st));
  PivotScratch<T> scr{sval.ptr, sidx.ptr, srow.ptr, stop.ptr};
  using SC = SubpanelCfg<T>;
  // rows per thread: complex128 rows fill shared memory before they outnumber the threads,
  // and a cluster's CTA holds at most SP_CLUSTER_ROWS
  constexpr int RPT2 = sizeof(T) == 8 ? 2 : 1;
  static_assert(SP_CLUSTER_ROWS <= 32 * (SP_WARPS - 1), "a row per thread in a cluster");
  const void* sp_kernel[2][2] = {{(const void*)k_subpanel_ll<T, 1, false>, (const void*)k_subpanel_ll<T, RPT2, false>},
                                 {(const void*)k_subpanel_ll<T, 1, true>, nullptr}};
  for (const void* k : {sp_kernel[0][0], sp_kernel[0][1], sp_kernel[1][0]})
    TT_TRY(smem_limit_once(k, (int)kSubpanelSmem));
  const int max_cluster = subpanel_cluster<T>();
  const size_t one_row = std::min(SP_ROWS, SC::MAX_ROWS);  // rows of a CTA with a row per thread
  auto cluster_ctas = [&](size_t m) { return subpanel_cluster_ctas(m, one_row, SP_CLUSTER_ROWS, max_cluster); };
  // CTAs of a matrix of m rows, of at most `most`: one while its shared memory
  // holds them (no exchange through L2), else about SP_ROWS rows each; 0: too tall
  auto ctas = [&](size_t m, int most) -> int {
    const size_t need = (m + SC::MAX_ROWS - 1) / SC::MAX_ROWS;
    if (need <= 1) return 1;
    if (need > (size_t)most) return 0;
    return (int)std::min<size_t>(most, std::max<size_t>(need, (m + SP_ROWS - 1) / SP_ROWS));
  };
  // the sub-panel of matrices [b0, b0 + nb) in one launch of gb CTAs each (gb < 0: a
  // cluster of -gb), cooperative where they meet in L2
  auto subpanel = [&](int b0, int nb, int j0, int w, int pk0, int pk1, int gb) -> int {
    SubpanelBatch<T> bt{};
    for (int b = 0; b < nb; b++) {
      bt.A[b] = As[b0 + b];
      bt.ipiv[b] = ipivs[b0 + b];
    }
    bt.info = d_info.ptr + b0;
    bt.err = d_info.ptr + B;
    bt.tries = d_info.ptr + B + 1 + 2 * b0;
    bt.verdict = srec.ptr + rec_bytes + verdicts * b0;
    bt.B = nb;
    int nn = n, cc0 = j0, ww = w, p0 = pk0, p1 = pk1;
    unsigned char* rec = srec.ptr + rec_region * b0;
    void* args[] = {&bt, &nn, &cc0, &ww, &p0, &p1, &rec};
    const bool cluster = gb < 0;  // -gb CTAs of one cluster
    if (cluster) gb = -gb;
    const int chunk = (n - j0 + gb - 1) / gb;
    const void* kernel = sp_kernel[cluster][sp_rpt(chunk) - 1];
    const size_t smem = (size_t)chunk * SP * sizeof(T) + SC::EXTRA;
    if (cluster) {
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute attr[2] = {};
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = gb;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      attr[1] = pdl_attribute();
      cfg.gridDim = dim3(gb * nb);
      cfg.blockDim = dim3(sp_threads(chunk));
      cfg.dynamicSmemBytes = smem;
      cfg.stream = st;
      cfg.attrs = attr;
      cfg.numAttrs = 2;
      TT_CUDA_TRY(cudaLaunchKernelExC(&cfg, kernel, args));
    } else {
      TT_CUDA_TRY(cudaLaunchCooperativeKernel(kernel, dim3(gb * nb), dim3(sp_threads(chunk)), args, smem, st));
    }
    count_launch();
    return TT_OK;
  };
  // pivoted factorisation of columns [j0, j0 + w), w <= IB, rows [j0, n), of all B matrices,
  // with its interchanges applied to the panel's other columns [pk0, j0) and [j0 + w, pk1)
  auto leaf = [&](int j0, int w, int pk0, int pk1) -> int {
    const size_t m = (size_t)(n - j0);
    const int together = ctas(m, G / B), alone = ctas(m, G);
    ProfScope prof(TT_PROF_SUBPANEL, st, 4.0 * m * w * w * B, 2.0 * m * w * sizeof(T) * B);
    if (const int c = cluster_ctas(m)) return subpanel(0, B, j0, w, pk0, pk1, -c);
    if (together) return subpanel(0, B, j0, w, pk0, pk1, together);
    for (int b = 0; b < B; b++) {
      if (alone) {
        TT_TRY(subpanel(b, 1, j0, w, pk0, pk1, alone));
      } else {
        T* Ap = As[b];
        int nn = n, cc0 = j0, ww = w;
        int32_t* ip = ipivs[b];
        int* inf = d_info.ptr + b;
        void* args[] = {&Ap, &nn, &cc0, &ww, &ip, &scr, &inf};
        TT_CUDA_TRY(cudaLaunchCooperativeKernel((void*)k_subpanel<T>, dim3(G), dim3(256), args, 0, st));
        count_launch();
        TT_TRY(laswp2(As + b, 1, n, ipivs + b, j0, j0 + w, pk0, j0, j0 + w, pk1, st));
      }
    }
    return TT_OK;
  };
  // split of a block of h rows or columns: the largest multiple of IB not above h / 2, at least IB
  auto half = [](int h) { return std::max(IB, (h / 2) / IB * IB); };
  // the tensor-core modes solve a block row with the explicit inverse of its
  // unit-lower block: X = L^{-1} once, then U = X A in one product
  const bool inv_solve = (mode == TC_TF32 || mode == TC_BF16X3);
  DevBuf<T> Xinv, Tinv;
  if (inv_solve) {
    const size_t wmax = (size_t)std::min(NB, IVB);
    TT_TRY(Xinv.alloc(wmax * wmax * B));
    TT_TRY(Tinv.alloc(wmax * wmax * B / 2));
  }
  // rows [r0, r0 + h) of columns [cb, ce) <- L^{-1} of them, L the unit-lower h x h block at (r0, r0):
  // halves recursively, so that most of the work is one update of depth h / 2
  std::function<int(T*, int, int, int, int)> trsm_rec = [&](T* A, int r0, int h, int cb, int ce) -> int {
    if (h <= IB) return trsm_rows_batched(&A, 1, n, r0, h, cb, ce, st);
    if (inv_solve && h % 32 == 0 && h <= IVB) {
      const T* A1 = A;
      TT_TRY(inv_unit_lower(&A1, 1, n, r0, h, Xinv.ptr, Tinv.ptr, st));
      return tc2_gemm_sub(mode, reinterpret_cast<float2*>(A) + (size_t)r0 * n + cb, n,
                          reinterpret_cast<const float2*>(Xinv.ptr), h,
                          reinterpret_cast<const float2*>(A) + (size_t)r0 * n + cb, n, h, ce - cb, h, st, 1);
    }
    const int h1 = half(h);
    TT_TRY(trsm_rec(A, r0, h1, cb, ce));
    TT_TRY(panel_gemm_sub(mode, A + (size_t)(r0 + h1) * n + cb, n, A + (size_t)(r0 + h1) * n + r0, n,
                          A + (size_t)r0 * n + cb, n, h - h1, ce - cb, h1, st));
    return trsm_rec(A, r0 + h1, h - h1, cb, ce);
  };
  // trsm_rec of the same block in all B matrices: one set of inverse launches
  // for all of them when the block is solved through its explicit inverse
  auto trsm_all = [&](int r0, int h, int cb, int ce) -> int {
    if (!(inv_solve && h > IB && h % 32 == 0 && h <= IVB)) {
      for (int b = 0; b < B; b++) TT_TRY(trsm_rec(As[b], r0, h, cb, ce));
      return TT_OK;
    }
    const T* Ac[kMaxBatch];
    for (int b = 0; b < B; b++) Ac[b] = As[b];
    TT_TRY(inv_unit_lower(Ac, B, n, r0, h, Xinv.ptr, Tinv.ptr, st));
    float2* Cs[kMaxBatch];
    const float2* Ls[kMaxBatch];
    const float2* Us[kMaxBatch];
    for (int b = 0; b < B; b++) {
      Cs[b] = reinterpret_cast<float2*>(As[b]) + (size_t)r0 * n + cb;
      Ls[b] = reinterpret_cast<const float2*>(Xinv.ptr + (size_t)b * h * h);
      Us[b] = Cs[b];
    }
    return tc2_gemm_sub_batched(mode, B, Cs, n, Ls, h, Us, n, h, ce - cb, h, st, 1);
  };
  // C -= L U at the same offsets of all B matrices (row/column offsets of C,
  // L and U given as (row, col) pairs): one batched tensor-core launch in the
  // real-row modes, else one update per matrix
  auto gemm_all = [&](int cr, int cc, int lr, int lc, int ur, int uc, int M, int N, int K) -> int {
    if (M <= 0 || N <= 0 || K <= 0) return TT_OK;
    if ((mode == TC_TF32 || mode == TC_BF16X3) && K % 16 == 0) {
      float2* Cs[kMaxBatch];
      const float2* Ls[kMaxBatch];
      const float2* Us[kMaxBatch];
      for (int b = 0; b < B; b++) {
        float2* A = reinterpret_cast<float2*>(As[b]);
        Cs[b] = A + (size_t)cr * n + cc;
        Ls[b] = A + (size_t)lr * n + lc;
        Us[b] = A + (size_t)ur * n + uc;
      }
      return tc2_gemm_sub_batched(mode, B, Cs, n, Ls, n, Us, n, M, N, K, st);
    }
    for (int b = 0; b < B; b++) {
      T* A = As[b];
      TT_TRY(panel_gemm_sub(mode, A + (size_t)cr * n + cc, n, A + (size_t)lr * n + lc, n, A + (size_t)ur * n + uc, n,
                            M, N, K, st));
    }
    return TT_OK;
  };
  // columns [c0, c0 + w) of the panel [k, k + kb) factored by recursive halving:
  // left half, its U block and the update of the right half (depth w / 2), right half
  std::function<int(int, int, int, int)> factor_cols = [&](int k, int kb, int c0, int w) -> int {
    if (w <= IB) {
      return leaf(c0, w, k, k + kb);
    }
    const int h = half(w);
    TT_TRY(factor_cols(k, kb, c0, h));
    for (int b = 0; b < B; b++) {
      T* A = As[b];
      TT_TRY(trsm_rec(A, c0, h, c0 + h, c0 + w));
      TT_TRY(panel_gemm_sub(mode, A + (size_t)(c0 + h) * n + (c0 + h), n, A + (size_t)(c0 + h) * n + c0, n,
                            A + (size_t)c0 * n + (c0 + h), n, n - c0 - h, w - h, h, st));
    }
    return factor_cols(k, kb, c0 + h, w - h);
  };
  const bool blocked = blocked_order || mode == TC_LEGACY_BF16X3;
  for (int k = 0; k < n; k += NB) {
    const int kb = std::min(NB, n - k);
    const int rest = n - k - kb;
    if (!blocked) {
      TT_TRY(factor_cols(k, kb, k, kb));
      for (int b = 0; b < B; b++) {
        T* A = As[b];
        // ---- interchanges outside the panel, U12 = L11^{-1} A12, trailing update
        TT_TRY(laswp2(As + b, 1, n, ipivs + b, k, k + kb, 0, k, k + kb, n, st));
        if (rest <= 0) continue;
        TT_TRY(trsm_rec(A, k, kb, k + kb, n));
        if (tc)
          TT_TRY(tc2_gemm_sub(mode, reinterpret_cast<float2*>(A) + (size_t)(k + kb) * n + (k + kb), n,
                              reinterpret_cast<const float2*>(A) + (size_t)(k + kb) * n + k, n,
                              reinterpret_cast<const float2*>(A) + (size_t)k * n + (k + kb), n, rest, rest, kb, st));
        else
          TT_TRY(gemm_sub(A + (size_t)(k + kb) * n + (k + kb), n, A + (size_t)(k + kb) * n + k, n,
                          A + (size_t)k * n + (k + kb), n, rest, rest, kb, st));
      }
      continue;
    }
    // ---- panel [k, k+kb) in mid-panels of MB columns (MB = kb: one level),
    // each in sub-panels of IB columns updated within the mid-panel, then the
    // mid-panel's U block row and the update of the panel's columns right of it
    const int MB = (mid > 0 && mid < kb) ? mid : kb;
    for (int m0 = k; m0 < k + kb; m0 += MB) {
      const int mw = std::min(MB, k + kb - m0);
      for (int j0 = m0; j0 < m0 + mw; j0 += IB) {
        const int w = std::min(IB, m0 + mw - j0);
        TT_TRY(leaf(j0, w, k, k + kb));
        const int right = m0 + mw - (j0 + w);
        if (right > 0 && inv_solve && w % 16 == 0) {
          // the solved block rows are written straight into the update's
          // operand planes, then one update for all matrices
          int ws = TT_OK;
          unsigned char* WB = static_cast<unsigned char*>(tc2_b_workspace(mode, right, w, &ws, B));
          TT_TRY(ws);
          const size_t plane = tc2_b_plane_bytes(mode, right, w);
          float2* Cs[kMaxBatch];
          const float2* Ls[kMaxBatch];
          const float2* Us[kMaxBatch];
          float2* Af[kMaxBatch];
          for (int b = 0; b < B; b++) Af[b] = reinterpret_cast<float2*>(As[b]);
          TT_TRY(trsm_rows_batched(As, B, n, j0, w, j0 + w, m0 + mw, st, mode, WB, plane));
          for (int b = 0; b < B; b++) {
            float2* A = Af[b];
            Cs[b] = A + (size_t)(j0 + w) * n + (j0 + w);
            Ls[b] = A + (size_t)(j0 + w) * n + j0;
            Us[b] = A + (size_t)j0 * n + (j0 + w);
          }
          TT_TRY(tc2_gemm_sub_batched(mode, B, Cs, n, Ls, n, Us, n, n - j0 - w, right, w, st, 0, true));
        } else if (right > 0) {
          for (int b = 0; b < B; b++) {
            T* A = As[b];
            TT_TRY(trsm_rows_batched(&A, 1, n, j0, w, j0 + w, m0 + mw, st));
            TT_TRY(panel_gemm_sub(mode, A + (size_t)(j0 + w) * n + (j0 + w), n, A + (size_t)(j0 + w) * n + j0, n,
                                  A + (size_t)j0 * n + (j0 + w), n, n - j0 - w, right, w, st));
          }
        }
      }
      const int right_out = k + kb - (m0 + mw);
      if (right_out > 0) {
        if (inv_solve && mw <= std::min(TR_MAX, IVB) && mw % 32 == 0) {
          int ws = TT_OK;
          unsigned char* WB = static_cast<unsigned char*>(tc2_b_workspace(mode, right_out, mw, &ws, B));
          TT_TRY(ws);
          float2* Cs[kMaxBatch];
          const float2* Ls[kMaxBatch];
          const float2* Us[kMaxBatch];
          float2* Af[kMaxBatch];
          for (int b = 0; b < B; b++) {
            float2* A = Af[b] = reinterpret_cast<float2*>(As[b]);
            Cs[b] = A + (size_t)(m0 + mw) * n + (m0 + mw);
            Ls[b] = A + (size_t)(m0 + mw) * n + m0;
            Us[b] = A + (size_t)m0 * n + (m0 + mw);
          }
          TT_TRY(trsm_rows_batched(Af, B, n, m0, mw, m0 + mw, k + kb, st, mode, WB,
                                  tc2_b_plane_bytes(mode, right_out, mw)));
          TT_TRY(tc2_gemm_sub_batched(mode, B, Cs, n, Ls, n, Us, n, n - m0 - mw, right_out, mw, st, 0, true));
        } else {
          TT_TRY(trsm_all(m0, mw, m0 + mw, k + kb));
          TT_TRY(gemm_all(m0 + mw, m0 + mw, m0 + mw, m0, m0, m0 + mw, n - m0 - mw, right_out, mw));
        }
      }
    }
    // ---- interchanges outside the panel; U12 = L11^{-1} A12 with the
    // explicit inverse in the tensor-core modes (all matrices together)
    TT_TRY(laswp2(As, B, n, ipivs, k, k + kb, 0, k, k + kb, n, st));
    if (rest > 0 && inv_solve) TT_TRY(trsm_all(k, kb, k + kb, n));
    for (int b = 0; b < B; b++) {
      T* A = As[b];
      if (rest <= 0) continue;
      // ---- U12 blocked by IB without tensor cores
      if (!inv_solve) for (int i0 = k; i0 < k + kb; i0 += IB) {
        const int wi = std::min(IB, k + kb - i0);
        TT_TRY(trsm_rows_batched(&A, 1, n, i0, wi, k + kb, n, st));
        const int below = k + kb - (i0 + wi);
        if (below > 0)
          TT_TRY(panel_gemm_sub(mode, A + (size_t)(i0 + wi) * n + (k + kb), n, A + (size_t)(i0 + wi) * n + i0, n,
                                A + (size_t)i0 * n + (k + kb), n, below, rest, wi, st));
      }
      // ---- trailing update (the real-row modes: below, all matrices in one launch)
      if (mode == TC_LEGACY_BF16X3)
        TT_TRY(lu_update_tc(reinterpret_cast<float2*>(A), n, k, kb, st));
      else if (!tc)
        TT_TRY(gemm_sub(A + (size_t)(k + kb) * n + (k + kb), n, A + (size_t)(k + kb) * n + k, n,
                        A + (size_t)k * n + (k + kb), n, rest, rest, kb, st));
    }
    if (rest > 0 && (mode == TC_TF32 || mode == TC_BF16X3))
      TT_TRY(gemm_all(k + kb, k + kb, k + kb, k, k, k + kb, rest, rest, kb));
  }
  if (mode == TC_LEGACY_BF16X3) TT_TRY(tc_check_error(st));
  if (mode == TC_TF32 || mode == TC_BF16X3) TT_TRY(tc2_check_error(st));
  std::vector<int> h_info(B + 1);
  TT_CUDA_TRY(cudaMemcpyAsync(h_info.data(), d_info.ptr, sizeof(int) * (B + 1), cudaMemcpyDeviceToHost, st));
  TT_CUDA_TRY(cudaStreamSynchronize(st));
  if (h_info[B]) {
    set_error("sub-panel factorisation timed out waiting for a pivot row");
    return TT_ERR_CUDA;
  }
  if (info) std::copy(h_info.begin(), h_info.begin() + B, info);
  return TT_OK;
}
template int lu_factor_batched_device<double2>(double2* const*, int, int, int32_t* const*, cudaStream_t, int, int*,
                                               bool, int, int, bool, int);
template int lu_factor_batched_device<float2>(float2* const*, int, int, int32_t* const*, cudaStream_t, int, int*,
                                              bool, int, int, bool, int);

template <typename T>
int lu_factor_device(T* A, int n, int32_t* ipiv, cudaStream_t st, int use_tc, int* info) {
  return lu_factor_batched_device<T>(&A, 1, n, &ipiv, st, use_tc, info);
}
template int lu_factor_device<double2>(double2*, int, int32_t*, cudaStream_t, int, int*);
template int lu_factor_device<float2>(float2*, int, int32_t*, cudaStream_t, int, int*);

}  // namespace tt
