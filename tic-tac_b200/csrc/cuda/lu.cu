// Triangular solves with the LU factor of lu_factor.cu (the zgetrs half of the
// reference's LAPACK solve, General_functions/matrix_routines.cpp:73-80), for a
// few right-hand sides at a time: forward substitution with the unit lower
// factor and back substitution with the upper factor.
//
// The factor is read once per substitution, as a stream: after each
// factorisation the 128 x 128 diagonal blocks of L and U are inverted (one CTA
// per block, in shared memory); each substitution is then one cooperative kernel
// whose CTAs pass the solved blocks on in tagged records (k_trsv).
#include <algorithm>
#include <cstring>
#include <vector>

#include "ll_record.cuh"
#include "tt_kernels.h"
#include "tt_lu_internal.h"

namespace tt {

template <typename T>
struct CT;
template <>
struct CT<double2> {
  using R = double;
};
template <>
struct CT<float2> {
  using R = float;
};

constexpr int TW = 128;       // diagonal block of the substitution (both element types)
constexpr int TSB = TW / 2;   // its halves are inverted, then joined
constexpr int TLD = TSB + 1;  // padded shared-memory row of a 64 x 64 tile

template <typename T>
__device__ __forceinline__ T cmul(T a, T b) {
  T r;
  r.x = a.x * b.x - a.y * b.y;
  r.y = a.x * b.y + a.y * b.x;
  return r;
}
template <typename T>
__device__ __forceinline__ T crecip(T b) {
  using R = typename CT<T>::R;
  // Smith's algorithm for 1 / b
  T r;
  if (fabs((double)b.x) >= fabs((double)b.y)) {
    const R t = b.y / b.x, d = b.x + b.y * t;
    r.x = R(1) / d;
    r.y = -t / d;
  } else {
    const R t = b.x / b.y, d = b.y + b.x * t;
    r.x = t / d;
    r.y = R(-1) / d;
  }
  return r;
}

// Blocks in sweep order: block q of the forward sweep starts at row TW q, of the
// backward one it ends TW q rows before n; only the last can be shorter.
__host__ __device__ __forceinline__ int blk_rows(int n, int q) { return n - q * TW < TW ? n - q * TW : TW; }
template <bool UPPER>
__host__ __device__ __forceinline__ int blk_start(int n, int q) {
  return UPPER ? n - q * TW - blk_rows(n, q) : q * TW;
}

// ---------------------------------------------------------------------------
// Inverses of the diagonal blocks, inv[q] (128 x 128, row-major), of a factor's
// lower and upper triangle (blockIdx.y = 0, 1), with a unit diagonal or the
// stored one.  The factor of L U keeps the unit lower and the upper triangle; its
// transpose (TRANSPOSED, for transposed solves) keeps the non-unit lower and the
// unit upper triangle.  Rows and columns past the block are the identity's.
// An upper triangle is taken with its rows and columns in reverse order, as a lower
// one.  A CTA inverts the block's two 64 x 64 diagonal halves at once, 256 threads
// each, in place in shared memory: 8 x 8 blocks in registers, a column a thread, then
// pairs of inverted blocks joined three times, and the halves once,
//   [X11 0; X21 X22] with X21 = -X22 (L21 X11).
// Bound: latency; the 64 steps of a right-looking inversion, three barriers each, took
// 84 us for a factor of order 512 against 34 now, 100 against 38 at 1,859, 142 against
// 66 for a complex128 one of order 8,496.
template <typename T>
__device__ __forceinline__ void cfma(T& acc, T a, T b) {
  acc.x += a.x * b.x;
  acc.x -= a.y * b.y;
  acc.y += a.x * b.y;
  acc.y += a.y * b.x;
}

// One join of H x H blocks of a half (256 threads, t the thread), H / 8 elements each;
// L21 X11 waits in the zeros above the diagonal
template <int H, typename T>
__device__ __forceinline__ void inv_join(T* M, int t) {
  constexpr int U = H / 8;
  const int i0 = t / (8 * H) * 2 * H, r = t / 8 % H, c = t % 8;
  T* X11 = M + i0 * TLD + i0;
  T *S = X11 + H, *X21 = X11 + H * TLD, *X22 = X21 + H;
  auto product = [&](const T* a, const T* b, T* out, bool minus) {
    T acc[U];
#pragma unroll
    for (int u = 0; u < U; u++) acc[u] = T{0, 0};
#pragma unroll 8
    for (int k = 0; k < H; k++) {
      const T x = a[r * TLD + k];
#pragma unroll
      for (int u = 0; u < U; u++) cfma(acc[u], x, b[k * TLD + c + 8 * u]);
    }
#pragma unroll
    for (int u = 0; u < U; u++) out[r * TLD + c + 8 * u] = minus ? T{-acc[u].x, -acc[u].y} : acc[u];
  };
  product(X21, X11, S, false);
  __syncthreads();
  product(X22, S, X21, true);
  __syncthreads();
#pragma unroll
  for (int u = 0; u < U; u++) S[r * TLD + c + 8 * u] = T{0, 0};
  __syncthreads();
}

template <typename T, bool UPPER, bool UNIT>
__device__ void inv_block(const T* __restrict__ LU, int n, int q, T* __restrict__ out, T* sm) {
  const int tid = threadIdx.x, half = tid >> 8, t = tid & 255;
  const int r0 = blk_start<UPPER>(n, q), rows = blk_rows(n, q);
  const T zero = {0, 0}, one = {1, 0};
  T* M = sm + half * TSB * TLD;   // this half's diagonal tile
  T* O = sm + 2 * TSB * TLD;      // the tile below the first half's
  const int h0 = half * TSB;
  // row (column) i of the lower triangle worked on is row at(i) of the block
  auto at = [&](int i) { return UPPER && i < rows ? rows - 1 - i : i; };
#pragma unroll 4
  for (int e = t; e < TSB * TSB; e += 256) {
    const int r = e / TSB, c = e % TSB;
    T v = (r == c) ? one : zero;
    if (h0 + r < rows && h0 + c < rows && (UNIT ? c < r : c <= r))
      v = LU[(size_t)(r0 + at(h0 + r)) * n + r0 + at(h0 + c)];
    M[r * TLD + c] = v;
  }
#pragma unroll 4
  for (int e = tid; e < TSB * TSB; e += 512) {
    const int r = e / TSB + TSB, c = e % TSB;
    O[(e / TSB) * TLD + c] = (r < rows && c < rows) ? LU[(size_t)(r0 + at(r)) * n + r0 + at(c)] : zero;
  }
  __syncthreads();
  if (t < TSB) {
    const int c = t & 7;
    T* B = M + (t & ~7) * (TLD + 1);
    T v[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      v[i] = i == c ? one : zero;
#pragma unroll
      for (int j = 0; j < i; j++) {
        const T m = B[i * TLD + j];
        cfma(v[i], T{-m.x, -m.y}, v[j]);
      }
      if (!UNIT) v[i] = cmul(v[i], crecip(B[i * TLD + i]));
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; i++) B[i * TLD + c] = v[i];
  }
  __syncthreads();
  inv_join<8>(M, t);
  inv_join<16>(M, t);
  inv_join<32>(M, t);
  // join of the halves: 8 elements a thread, row tr, columns tc + 8 u
  const T* X1 = sm;               // inverse of the first half
  const T* X2 = sm + TSB * TLD;   // of the second
  const int tr = tid >> 3, tc = tid & 7;
  auto product = [&](const T* a, const T* b, T(&acc)[8]) {
#pragma unroll
    for (int u = 0; u < 8; u++) acc[u] = zero;
#pragma unroll 4
    for (int k = 0; k < TSB; k++) {
      const T x = a[tr * TLD + k];
#pragma unroll
      for (int u = 0; u < 8; u++) cfma(acc[u], x, b[k * TLD + tc + 8 * u]);
    }
  };
  T acc[8];
  product(O, X1, acc);
  __syncthreads();
#pragma unroll
  for (int u = 0; u < 8; u++) O[tr * TLD + tc + 8 * u] = acc[u];
  __syncthreads();
  product(X2, O, acc);
  T* o = out + (size_t)q * TW * TW;
  const int i1 = at(tr) * TW, i2 = at(tr + TSB) * TW;
#pragma unroll
  for (int u = 0; u < 8; u++) {
    const int c = tc + 8 * u, j1 = at(c), j2 = at(c + TSB);
    o[(size_t)i2 + j1] = T{-acc[u].x, -acc[u].y};
    o[(size_t)i1 + j2] = zero;
    o[(size_t)i1 + j1] = X1[tr * TLD + c];
    o[(size_t)i2 + j2] = X2[tr * TLD + c];
  }
}
template <typename T, bool TRANSPOSED>
__global__ void __launch_bounds__(512) k_inv_blocks(const T* __restrict__ LU, int n, T* __restrict__ invL,
                                                    T* __restrict__ invU) {
  extern __shared__ __align__(16) unsigned char ism[];
  T* sm = reinterpret_cast<T*>(ism);  // [3][TSB][TLD]
  if (blockIdx.y == 0) inv_block<T, false, !TRANSPOSED>(LU, n, blockIdx.x, invL, sm);
  else inv_block<T, true, TRANSPOSED>(LU, n, blockIdx.x, invU, sm);
}

// ---------------------------------------------------------------------------
// One substitution (forward with L when !UPPER, backward with U when UPPER) for
// kn <= RHS right-hand sides, of B factors (Gb CTAs each), cooperative.  Blocks of
// 128 rows are visited in sweep order q = 0, 1, ..  Arithmetic is in the factor's
// precision (FP32 for the complex64 factor, whose solves only feed the
// FP64-residual refinement; FP64 for the complex128 factor); the vectors are
// complex128.
//  - LEADS lead CTAs solve the blocks: when block q's right-hand side y is
//    complete, they form x_q = inv[q] y, 32 rows each, the rows of inv asked for
//    while y is awaited.
//  - The other CTAs own the rows, two neighbouring ones at a time in turn, and keep
//    their values in shared memory.  When x_q is there, a warp applies block column q
//    to four of its CTA's unsolved rows at a time; those of block q + 1 come first
//    and are posted at once, so the leads solve block q + 1 while the rest of the
//    column is applied.
// y and x pass through tagged records (ll_record.cuh), so a step costs two trips
// through L2 and no grid barrier.  Slots are reused: y_q's for y_{q+2}, posted by
// owners that have all of x_{q+1}, so every lead has read y_q; x_q's for
// x_{q+X_SLOTS}.  Every owner that still waits for x_q has its next pair of rows in
// a block no later than q + 1 + (GO - 1) / 64, and x_{q+X_SLOTS} needs that block's y,
// so X_SLOTS = 4 serves up to 192 owners.  Bound: the factor read once from HBM where its rows
// are long, else the two trips (about 2 us a block of 128).  Per sweep, against
// blocks of 64 with a grid barrier each: n = 512 (2 factors) 28 -> 11 us, 1,859 (4)
// 115 -> 46 us, 10,944 (1) 670 -> 303 us, 16,128 (2) 1.42 -> 0.68 ms, 20,160 (4)
// 2.57 -> 1.44 ms, 42,300 (2) 6.5 -> 3.65 ms; complex128 n = 8,496 755 -> 530 us.
constexpr int RHS = 4;
constexpr int TRSV_THREADS = 512;
constexpr int LEADS = 4;
constexpr int X_SLOTS = 4;
constexpr int TRSV_SPINS = 1 << 20;

// reduce 2 M values over the 32 lanes of a warp by halving the values each round;
// value i ends complete in lane i (M = 16) or in lanes 2i and 2i + 1 (M = 8)
template <int M, typename C>
__device__ __forceinline__ C butterfly(C (&acc)[2 * M], int lane) {
#pragma unroll
  for (int o = 16, m = M; m >= 1; o >>= 1, m >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int j = 0; j < m; j++) {
      const C send = up ? acc[j] : acc[j + m];
      const C keep = up ? acc[j + m] : acc[j];
      acc[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  if (M == 8) return acc[0] + __shfl_xor_sync(0xffffffffu, acc[0], 1);
  return acc[0];
}

// Up to kMaxSweeps factors swept in one cooperative launch.
constexpr int kMaxSweeps = 4;
template <typename T>
struct TrsvBatch {
  const T* LU[kMaxSweeps];
  const T* inv[kMaxSweeps];
  const double2* in[kMaxSweeps];      // right-hand sides [k][n], row r read at in_perm[r]
  double2* out[kMaxSweeps];           // solutions [k][n], row r written at out_perm[r]
  const int32_t* in_perm[kMaxSweeps];
  const int32_t* out_perm[kMaxSweeps];
  unsigned char* rec[kMaxSweeps];     // [2 of y, X_SLOTS of x][RHS][TW] records
  unsigned epoch[kMaxSweeps];         // tags of this sweep are above it
  int* err[kMaxSweeps];
  int B;
};

// the 4 elements of a 128-column row segment that a lane holds: pairs of
// neighbours where 16-byte loads of complex64 are possible (WIDE), else every 32nd
template <typename T, bool WIDE>
__device__ __forceinline__ void load_seg(const T* __restrict__ row, int lane, T (&v)[4]) {
  if constexpr (WIDE && sizeof(T) == 8) {
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const float4 f = __ldcs(reinterpret_cast<const float4*>(row) + lane + 32 * u);
      v[2 * u] = T{f.x, f.y};
      v[2 * u + 1] = T{f.z, f.w};
    }
  } else {
#pragma unroll
    for (int u = 0; u < 4; u++) v[u] = __ldcs(row + lane + 32 * u);
  }
}
template <typename T, bool WIDE>
__device__ __forceinline__ void smem_seg(const T* row, int lane, T (&v)[4]) {
  if constexpr (WIDE && sizeof(T) == 8) {
#pragma unroll
    for (int u = 0; u < 2; u++) {
      const float4 f = reinterpret_cast<const float4*>(row)[lane + 32 * u];
      v[2 * u] = T{f.x, f.y};
      v[2 * u + 1] = T{f.z, f.w};
    }
  } else {
#pragma unroll
    for (int u = 0; u < 4; u++) v[u] = row[lane + 32 * u];
  }
}

template <typename T, bool UPPER, bool WIDE>
__global__ void __launch_bounds__(TRSV_THREADS, 1) k_trsv(TrsvBatch<T> bt, int n, int kn) {
  using C = typename CT<T>::R;
  const int Gb = gridDim.x / bt.B, grp = blockIdx.x / Gb, local = blockIdx.x - grp * Gb;
  const T* __restrict__ LU = bt.LU[grp];
  unsigned char* rec = bt.rec[grp];
  const unsigned epoch = bt.epoch[grp];
  extern __shared__ __align__(16) unsigned char tsm[];
  T* vs = reinterpret_cast<T*>(tsm);  // [2][RHS][TW]: y (leads) or x (owners) of this step, double-buffered
  T* xo = vs + 2 * RHS * TW;          // owners: [pairs][2][RHS]
  __shared__ int s_dead;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int nb = (n + TW - 1) / TW;
  auto slot = [&](int which, int q) {
    return rec + (size_t)(which ? 2 + q % X_SLOTS : q & 1) * RHS * TW * LL<T>::BYTES;
  };
  int* err = bt.err[grp];
  if (t == 0) s_dead = *(volatile int*)err;
  // this thread's element of a posted block into vs; RHS * TW threads
  const int ek = t / TW, ej = t % TW;
  auto collect = [&](int which, int q) {
    T v = {0, 0};
    if (ek < kn && ej < blk_rows(n, q)) {
      unsigned long long hi;
      const unsigned char* p = slot(which, q) + t * LL<T>::BYTES;
      const unsigned tag = epoch + (unsigned)q + 1u;
      for (int spin = 0; !LL<T>::poll(p, v, hi, tag); spin++) {
        if (spin >= TRSV_SPINS || *(volatile int*)&s_dead) {
          *(volatile int*)&s_dead = 1;
          atomicExch(err, 1);
          break;
        }
      }
    }
    vs[(q & 1) * RHS * TW + t] = v;
  };
  __syncthreads();

  if (local < LEADS) {
    const int row = local * (TW / LEADS) + warp * 2;  // two rows a warp
    T a[2][4];
    auto load_inv = [&](int q) {
#pragma unroll
      for (int h = 0; h < 2; h++) load_seg<T, WIDE>(bt.inv[grp] + (size_t)q * TW * TW + (size_t)(row + h) * TW, lane, a[h]);
    };
    load_inv(0);
    for (int q = 0; q < nb; q++) {
      collect(0, q);
      __syncthreads();
      C acc[16];
#pragma unroll
      for (int k = 0; k < RHS; k++) {
        C sr[2] = {0, 0}, si[2] = {0, 0};
        if (k < kn) {
          T y[4];
          smem_seg<T, WIDE>(vs + ((q & 1) * RHS + k) * TW, lane, y);
#pragma unroll
          for (int h = 0; h < 2; h++)
#pragma unroll
            for (int u = 0; u < 4; u++) {
              sr[h] += a[h][u].x * y[u].x - a[h][u].y * y[u].y;
              si[h] += a[h][u].x * y[u].y + a[h][u].y * y[u].x;
            }
        }
#pragma unroll
        for (int h = 0; h < 2; h++) {
          acc[(h * RHS + k) * 2] = sr[h];
          acc[(h * RHS + k) * 2 + 1] = si[h];
        }
      }
      if (q + 1 < nb) load_inv(q + 1);
      const C v = butterfly<8>(acc, lane);
      const C im = __shfl_down_sync(0xffffffffu, v, 2);
      const int i = lane >> 1, h = i >> 3, k = (i >> 1) & 3, j = row + h;
      if ((lane & 3) == 0 && k < kn && j < blk_rows(n, q)) {
        LL<T>::post(slot(1, q) + (k * TW + j) * LL<T>::BYTES, T{v, im}, epoch + (unsigned)q + 1u);
        const int r = blk_start<UPPER>(n, q) + j;
        bt.out[grp][(size_t)k * n + (bt.out_perm[grp] ? bt.out_perm[grp][r] : r)] = make_double2((double)v, (double)im);
      }
    }
    return;
  }

  // owners: pair p of sweep rows 2 p, 2 p + 1 belongs to CTA LEADS + p % GO
  const int GO = Gb - LEADS, me = local - LEADS;
  const int npairs = (n + 1) / 2;
  const int mine = me < npairs ? (npairs - me + GO - 1) / GO : 0;
  auto row_of = [&](int pl, int h) {  // row of local pair pl, or -1
    const int i = 2 * (me + pl * GO) + h;
    return i < n ? (UPPER ? n - 1 - i : i) : -1;
  };
  for (int e = t; e < mine * 2 * RHS; e += TRSV_THREADS) {
    const int k = e % RHS, h = (e / RHS) & 1, pl = e / (2 * RHS), r = row_of(pl, h);
    T v = {0, 0};
    if (k < kn && r >= 0) {
      const double2 d = bt.in[grp][(size_t)k * n + (bt.in_perm[grp] ? bt.in_perm[grp][r] : r)];
      v = T{(C)d.x, (C)d.y};
      if (2 * (me + pl * GO) < TW)  // block 0 is complete as it is
        LL<T>::post(slot(0, 0) + (k * TW + r - blk_start<UPPER>(n, 0)) * LL<T>::BYTES, v, epoch + 1u);
    }
    xo[e] = v;
  }
  // first local pair of block q or later
  auto first_pair = [&](int q) {
    const int p0 = q * (TW / 2);
    return p0 > me ? (p0 - me + GO - 1) / GO : 0;
  };
  constexpr int NW = TRSV_THREADS / 32;
  for (int q = 0; q + 1 < nb && first_pair(q + 1) < mine; q++) {
    const int c0 = blk_start<UPPER>(n, q);
    const int y0 = blk_start<UPPER>(n, q + 1), yn = blk_rows(n, q + 1);
    // two pairs (four rows) a warp at a time, the next ones asked for ahead
    const int p0 = first_pair(q + 1) + 2 * warp;
    T a[4][4], an[4][4];
    auto load = [&](int p, T(&d)[4][4]) {
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int pl = p + (i >> 1), r = pl < mine ? row_of(pl, i & 1) : -1;
        if (r >= 0) {
          load_seg<T, WIDE>(LU + (size_t)r * n + c0, lane, d[i]);
        } else {
#pragma unroll
          for (int u = 0; u < 4; u++) d[i][u] = T{0, 0};
        }
      }
    };
    constexpr bool AHEAD = sizeof(T) == 8;  // two sets of complex128 rows do not fit in registers
    if (p0 < mine) load(p0, a);
    collect(1, q);
    __syncthreads();
    const T* xs = vs + (q & 1) * RHS * TW;
    for (int p = p0; p < mine; p += 2 * NW) {
      const bool more = p + 2 * NW < mine;
      if (AHEAD && more) load(p + 2 * NW, an);
      C acc[32];
#pragma unroll
      for (int k = 0; k < RHS; k++) {
        T x[4];
        if (k < kn) smem_seg<T, WIDE>(xs + k * TW, lane, x);
#pragma unroll
        for (int i = 0; i < 4; i++) {
          C sr = 0, si = 0;
          if (k < kn) {
#pragma unroll
            for (int u = 0; u < 4; u++) {
              sr += a[i][u].x * x[u].x - a[i][u].y * x[u].y;
              si += a[i][u].x * x[u].y + a[i][u].y * x[u].x;
            }
          }
          acc[(i * RHS + k) * 2] = sr;
          acc[(i * RHS + k) * 2 + 1] = si;
        }
      }
      const C v = butterfly<16>(acc, lane);  // lane = (row i, k, part)
      C* d = reinterpret_cast<C*>(xo + (size_t)p * 2 * RHS) + lane;
      const int i = lane >> 3, k = (lane >> 1) & 3, pl = p + (i >> 1);
      C val = 0;
      if (pl < mine) {
        val = *d - v;
        *d = val;
      }
      const C im = __shfl_down_sync(0xffffffffu, val, 1);
      const int r = pl < mine ? row_of(pl, i & 1) : -1;
      if ((lane & 1) == 0 && k < kn && r >= y0 && r < y0 + yn)
        LL<T>::post(slot(0, q + 1) + (k * TW + r - y0) * LL<T>::BYTES, T{val, im}, epoch + (unsigned)q + 2u);
      if (more) {
        if (AHEAD) {
#pragma unroll
          for (int x = 0; x < 4; x++)
#pragma unroll
            for (int u = 0; u < 4; u++) a[x][u] = an[x][u];
        } else {
          load(p + 2 * NW, a);
        }
      }
    }
  }
}

int lu_permutation(const int32_t* d_ipiv, int n, std::vector<int32_t>& perm, cudaStream_t st) {
  std::vector<int32_t> ipiv(n);
  TT_CUDA_TRY(cudaMemcpyAsync(ipiv.data(), d_ipiv, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, st));
  TT_CUDA_TRY(cudaStreamSynchronize(st));
  perm.resize(n);
  for (int i = 0; i < n; i++) perm[i] = i;
  for (int j = 0; j < n; j++) {
    const int p = ipiv[j];
    if (p < 0 || p >= n) {
      set_error("corrupt pivot sequence");
      return TT_ERR_CUDA;
    }
    std::swap(perm[j], perm[p]);
  }
  return TT_OK;
}

template <typename T>
int lu_trsv_prepare(const T* d_LU, int n, TrsvBlocks<T>& blk, cudaStream_t st, bool transposed) {
  const int nb = (n + TW - 1) / TW;
  const size_t need = (size_t)nb * TW * TW;
  if (blk.invL.count < need) {
    TT_TRY(blk.invL.alloc(need));
    TT_TRY(blk.invU.alloc(need));
  }
  if (!blk.rec.ptr) {
    const size_t bytes = (size_t)(2 + X_SLOTS) * RHS * TW * LL<T>::BYTES;
    TT_TRY(blk.rec.alloc(bytes));
    TT_TRY(blk.err.alloc(1));
    TT_CUDA_TRY(cudaMemsetAsync(blk.err.ptr, 0, sizeof(int), st));
    TT_CUDA_TRY(cudaMemsetAsync(blk.rec.ptr, 0, bytes, st));
    blk.epoch = 0;
  }
  blk.n = n;
  ProfScope prof(TT_PROF_SUBST_PREP, st, 0.0, 2.0 * (double)n * TW * sizeof(T));
  const size_t smem = (size_t)3 * TSB * TLD * sizeof(T);
  const dim3 grid(nb, 2);
  if (!transposed) {
    TT_TRY(smem_limit_once((const void*)k_inv_blocks<T, false>, (int)smem));
    k_inv_blocks<T, false><<<grid, 512, smem, st>>>(d_LU, n, blk.invL.ptr, blk.invU.ptr);
  } else {
    TT_TRY(smem_limit_once((const void*)k_inv_blocks<T, true>, (int)smem));
    k_inv_blocks<T, true><<<grid, 512, smem, st>>>(d_LU, n, blk.invL.ptr, blk.invU.ptr);
  }
  count_launch();
  TT_CUDA_TRY(cudaGetLastError());
  return TT_OK;
}
template int lu_trsv_prepare<double2>(const double2*, int, TrsvBlocks<double2>&, cudaStream_t, bool);
template int lu_trsv_prepare<float2>(const float2*, int, TrsvBlocks<float2>&, cudaStream_t, bool);

// Forward then backward substitution of the right-hand sides x_b [k][n] in place,
// for the B factors of a batch (one cooperative launch per sweep for all of them):
// row r of the forward sweep's right-hand side is row in_perm[r] of x_b, row r of
// the solution goes to out_perm[r] (null: r).
template <typename T>
int trsv_sweeps(int B, const T* const* d_LU, int n, TrsvBlocks<T>* const* blk, double2* const* x,
                const int32_t* const* in_perm, const int32_t* const* out_perm, int nrhs, cudaStream_t st) {
  if (B < 1 || B > kMaxSweeps) {
    set_error("substitution batch of " + std::to_string(B) + " factors (1.." + std::to_string(kMaxSweeps) + ")");
    return TT_ERR_BADARG;
  }
  for (int b = 0; b < B; b++)
    if (blk[b]->n != n || !blk[b]->invL.ptr) {
      set_error("triangular solve called without the inverted diagonal blocks of this factor");
      return TT_ERR_BADARG;
    }
  // CTAs of a factor: the leads, and owners of at least 64 rows (one turn of their warps)
  const int most = device_sm_count() / B;
  const int Gb = LEADS + std::max(1, std::min({most - LEADS, (n + 63) / 64, (X_SLOTS - 1) * TW / 2}));
  const int pairs = ceil_div((n + 1) / 2, Gb - LEADS);
  const size_t smem = ((size_t)2 * RHS * TW + (size_t)pairs * 2 * RHS) * sizeof(T);
  constexpr size_t kMaxSmem = 224 * 1024;
  if (smem > kMaxSmem) {
    if (B > 1) {
      // fewer owners per factor would not hold their rows: one factor at a time
      for (int b = 0; b < B; b++)
        TT_TRY(trsv_sweeps<T>(1, d_LU + b, n, blk + b, x + b, in_perm + b, out_perm + b, nrhs, st));
      return TT_OK;
    }
    set_error("triangular solve: n = " + std::to_string(n) + " needs " + std::to_string(smem) +
              " bytes of shared memory per CTA (limit " + std::to_string(kMaxSmem) + ")");
    return TT_ERR_UNSUPPORTED;
  }
  // a lane's pairs of complex64 need rows on 16-byte boundaries
  bool wide = n % 2 == 0;
  for (int b = 0; b < B; b++) wide = wide && (uintptr_t)d_LU[b] % 16 == 0;
  const void* lower = wide ? (const void*)k_trsv<T, false, true> : (const void*)k_trsv<T, false, false>;
  const void* upper = wide ? (const void*)k_trsv<T, true, true> : (const void*)k_trsv<T, true, false>;
  TT_TRY(smem_limit_once(lower, (int)kMaxSmem));
  TT_TRY(smem_limit_once(upper, (int)kMaxSmem));
  DevBuf<double2> mid;  // between the sweeps
  TT_TRY(mid.alloc((size_t)B * n * std::min(nrhs, RHS)));
  const unsigned nb = (unsigned)((n + TW - 1) / TW);
  for (int k0 = 0; k0 < nrhs; k0 += RHS) {
    int kn = std::min(RHS, nrhs - k0);
    TrsvBatch<T> bl{}, bu{};
    bl.B = bu.B = B;
    for (int b = 0; b < B; b++) {
      if (blk[b]->epoch > 0xF0000000u) {  // tags about to run out: start over
        TT_CUDA_TRY(cudaMemsetAsync(blk[b]->rec.ptr, 0, blk[b]->rec.count, st));
        blk[b]->epoch = 0;
      }
      bl.LU[b] = bu.LU[b] = d_LU[b];
      bl.inv[b] = blk[b]->invL.ptr;
      bu.inv[b] = blk[b]->invU.ptr;
      bl.in[b] = x[b] + (size_t)k0 * n;
      bl.in_perm[b] = in_perm[b];
      bl.out[b] = mid.ptr + (size_t)b * n * std::min(nrhs, RHS);
      bu.in[b] = bl.out[b];
      bu.out[b] = x[b] + (size_t)k0 * n;
      bu.out_perm[b] = out_perm[b];
      bl.err[b] = bu.err[b] = blk[b]->err.ptr;
      bl.rec[b] = bu.rec[b] = blk[b]->rec.ptr;
      bl.epoch[b] = blk[b]->epoch;
      bu.epoch[b] = blk[b]->epoch + nb;
      blk[b]->epoch += 2 * nb;
    }
    int nn = n;
    void* argsL[] = {&bl, &nn, &kn};
    TT_CUDA_TRY(cudaLaunchCooperativeKernel(lower, dim3(Gb * B), dim3(TRSV_THREADS), argsL, smem, st));
    count_launch();
    void* argsU[] = {&bu, &nn, &kn};
    TT_CUDA_TRY(cudaLaunchCooperativeKernel(upper, dim3(Gb * B), dim3(TRSV_THREADS), argsU, smem, st));
    count_launch();
  }
  return TT_OK;
}

template <typename T>
int lu_trsv_check(const TrsvBlocks<T>& blk, cudaStream_t st) {
  if (!blk.err.ptr) return TT_OK;
  int bad = 0;
  TT_CUDA_TRY(cudaMemcpyAsync(&bad, blk.err.ptr, sizeof(int), cudaMemcpyDeviceToHost, st));
  TT_CUDA_TRY(cudaStreamSynchronize(st));
  if (bad) {
    set_error("triangular solve timed out waiting for a block of the solution");
    return TT_ERR_CUDA;
  }
  return TT_OK;
}
template int lu_trsv_check<float2>(const TrsvBlocks<float2>&, cudaStream_t);
template int lu_trsv_check<double2>(const TrsvBlocks<double2>&, cudaStream_t);

template <typename T>
int lu_solve_batched_device(int B, const T* const* d_LU, int n, TrsvBlocks<T>* const* blk,
                            const int32_t* const* d_perm, double* const* d_x, int nrhs, cudaStream_t st) {
  if (n <= 0 || nrhs <= 0 || B <= 0) return TT_OK;
  ProfScope prof(TT_PROF_TRSV, st, 8.0 * n * (double)n * nrhs * B, (double)n * n * sizeof(T) * B);
  double2* xs[kMaxSweeps];
  const int32_t* none[kMaxSweeps] = {};
  for (int b = 0; b < std::min(B, kMaxSweeps); b++) xs[b] = reinterpret_cast<double2*>(d_x[b]);
  return trsv_sweeps<T>(B, d_LU, n, blk, xs, d_perm, none, nrhs, st);
}
template int lu_solve_batched_device<float2>(int, const float2* const*, int, TrsvBlocks<float2>* const*,
                                             const int32_t* const*, double* const*, int, cudaStream_t);

template <typename T>
int lu_solve_device(const T* d_LU, int n, TrsvBlocks<T>& blk, const int32_t* d_perm, double* d_x, int nrhs,
                    cudaStream_t st) {
  TrsvBlocks<T>* pb = &blk;
  return lu_solve_batched_device<T>(1, &d_LU, n, &pb, &d_perm, &d_x, nrhs, st);
}

template <typename T>
int lu_solve_transposed_device(const T* d_LUt, int n, TrsvBlocks<T>& blkT, const int32_t* d_perm, double* d_x,
                               int nrhs, cudaStream_t st) {
  if (n <= 0 || nrhs <= 0) return TT_OK;
  ProfScope prof(TT_PROF_TRSV, st, 8.0 * n * (double)n * nrhs, (double)n * n * sizeof(T));
  // x[perm[r]] = row r: the row interchanges applied backwards
  TrsvBlocks<T>* pb = &blkT;
  double2* x = reinterpret_cast<double2*>(d_x);
  const int32_t* none = nullptr;
  return trsv_sweeps<T>(1, &d_LUt, n, &pb, &x, &none, &d_perm, nrhs, st);
}
template int lu_solve_transposed_device<double2>(const double2*, int, TrsvBlocks<double2>&, const int32_t*, double*,
                                                 int, cudaStream_t);
template int lu_solve_transposed_device<float2>(const float2*, int, TrsvBlocks<float2>&, const int32_t*, double*, int,
                                                cudaStream_t);
template int lu_solve_device<double2>(const double2*, int, TrsvBlocks<double2>&, const int32_t*, double*, int,
                                      cudaStream_t);
template int lu_solve_device<float2>(const float2*, int, TrsvBlocks<float2>&, const int32_t*, double*, int,
                                     cudaStream_t);

}  // namespace tt
