// Pade resummation of the Neumann coefficients on the device
// (pade_method_solve, CPP/solve_faddeev.cpp:440-1444): the coefficients of all
// elements stay in device memory, and each order's [N/N] approximants and
// stopping criteria are evaluated there, one warp per element.
#include "tt_kernels.h"

namespace tt {
namespace {

constexpr int PD_MAX = 14;               // highest order
constexpr int PD_TERMS = 2 * PD_MAX + 1;
constexpr int PD_S = PD_MAX + 1;         // largest determinant
constexpr int PD_WARPS = 8;

// complex arithmetic in separately rounded operations, as a host compiler
// without contraction evaluates std::complex<double>: the determinants cancel
// and amplify whatever rounding they get
__device__ __forceinline__ double2 zmul(double2 a, double2 b) {
  return make_double2(__dsub_rn(__dmul_rn(a.x, b.x), __dmul_rn(a.y, b.y)),
                      __dadd_rn(__dmul_rn(a.x, b.y), __dmul_rn(a.y, b.x)));
}
__device__ __forceinline__ double2 zsub(double2 a, double2 b) {
  return make_double2(__dsub_rn(a.x, b.x), __dsub_rn(a.y, b.y));
}
// Smith's division
__device__ __forceinline__ double2 zdiv(double2 a, double2 b) {
  if (fabs(b.x) < fabs(b.y)) {
    const double t = __ddiv_rn(b.x, b.y), d = __dadd_rn(__dmul_rn(b.x, t), b.y);
    return make_double2(__ddiv_rn(__dadd_rn(__dmul_rn(a.x, t), a.y), d),
                        __ddiv_rn(__dsub_rn(__dmul_rn(a.y, t), a.x), d));
  }
  const double t = __ddiv_rn(b.y, b.x), d = __dadd_rn(__dmul_rn(b.y, t), b.x);
  return make_double2(__ddiv_rn(__dadd_rn(__dmul_rn(a.y, t), a.x), d),
                      __ddiv_rn(__dsub_rn(a.y, __dmul_rn(a.x, t)), d));
}

// Determinant of the S x S matrix m (row stride PD_S) by LU with partial
// pivoting, pivots by |re| + |im| as LAPACK's zgetrf chooses them
// (CPP/General_functions/matrix_routines.cpp:82-101); lane i holds row i.
__device__ double2 warp_det(double2* m, int S, int lane) {
  double2 det = make_double2(1.0, 0.0);
  for (int k = 0; k < S; k++) {
    __syncwarp();
    double v = -1.0;
    if (lane >= k && lane < S) {
      const double2 x = m[lane * PD_S + k];
      const double mag = __dadd_rn(fabs(x.x), fabs(x.y));
      v = mag > v ? mag : v;  // a NaN is never chosen
    }
    int p = v >= 0 ? lane : PD_S + k;  // none: the diagonal
    for (int o = 16; o > 0; o >>= 1) {
      const double ov = __shfl_xor_sync(0xffffffffu, v, o);
      const int op = __shfl_xor_sync(0xffffffffu, p, o);
      if (ov > v || (ov == v && op < p)) {
        v = ov;
        p = op;
      }
    }
    if (v < 0) p = k;
    const double2 piv = m[p * PD_S + k];
    __syncwarp();  // every lane has it before the rows change places
    if (piv.x == 0.0 && piv.y == 0.0) return make_double2(0.0, 0.0);
    if (p != k) {
      if (lane >= k && lane < S) {
        const double2 t = m[k * PD_S + lane];
        m[k * PD_S + lane] = m[p * PD_S + lane];
        m[p * PD_S + lane] = t;
      }
      det = make_double2(-det.x, -det.y);
      __syncwarp();
    }
    det = zmul(det, piv);
    if (lane > k && lane < S) {
      const double2 l = zdiv(m[lane * PD_S + k], piv);
      for (int c = k + 1; c < S; c++) m[lane * PD_S + c] = zsub(m[lane * PD_S + c], zmul(l, m[k * PD_S + c]));
    }
  }
  return det;
}

// Coefficient `term` of the elements still open: a[e][term] = R[row[e]][col[e]]
__global__ void k_pade_term(const double2* __restrict__ R, int n, const int32_t* __restrict__ row,
                            const int32_t* __restrict__ col, int nel, int term, const uint8_t* __restrict__ done,
                            double2* __restrict__ a) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e < nel && !done[e]) a[(size_t)e * PD_TERMS + term] = R[(size_t)row[e] * n + col[e]];
}

// The [N/N] approximant at z = 1 of each open element
// (pade_approximant, CPP/solve_faddeev.cpp:271-296) and the reference's stopping
// criteria: order 14; no better difference in the last 4 orders; smallest
// difference of consecutive approximants below 1e-6 |best| or 1e-7.  A finished
// element's value and relative difference go to out and diff; *open counts the
// others.  Evaluated on the host, 3,660 breakup cells took 35 of a 70 ms solve.
__global__ void __launch_bounds__(32 * PD_WARPS) k_pade_order(int N, int nel, const double2* __restrict__ a,
                                                              double2* __restrict__ pa, uint8_t* __restrict__ done,
                                                              double2* __restrict__ out, double* __restrict__ diff,
                                                              int* __restrict__ open) {
  extern __shared__ double2 pd_sm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int e = blockIdx.x * PD_WARPS + warp;
  if (e >= nel || done[e]) return;
  double2* P = pd_sm + (size_t)warp * 2 * PD_S * PD_S;
  double2* Q = P + PD_S * PD_S;
  const double2* ae = a + (size_t)e * PD_TERMS;
  const int S = N + 1;
  for (int i = lane; i < N * S; i += 32) {
    const int r = i / S, c = i - r * S;
    P[r * PD_S + c] = Q[r * PD_S + c] = ae[1 + r + c];
  }
  if (lane < S) {
    // last rows: ones, and the partial sums a_0 + .. + a_c
    double2 s = make_double2(0.0, 0.0);
    for (int j = 0; j <= lane; j++) s = make_double2(__dadd_rn(s.x, ae[j].x), __dadd_rn(s.y, ae[j].y));
    P[N * PD_S + lane] = s;
    Q[N * PD_S + lane] = make_double2(1.0, 0.0);
  }
  __syncwarp();
  const double2 num = warp_det(P, S, lane);
  const double2 den = warp_det(Q, S, lane);
  if (lane != 0) return;
  double2* p = pa + (size_t)e * PD_S;
  p[N] = zdiv(num, den);
  int best = 0;
  double least = 1.0;
  for (int k = 0; k <= N; k++) {
    // the reference compares approximant 0 with the slot before it, zero here
    const double2 q = k > 0 ? p[k - 1] : make_double2(0.0, 0.0);
    const double d = hypot(p[k].x - q.x, p[k].y - q.y);
    if (d < least && d > 1e-15) {
      best = k;
      least = d;
    }
  }
  const double mag = hypot(p[best].x, p[best].y);
  if (N == PD_MAX || N - best > 4 || least < 1e-6 * mag || least < 1e-7) {
    done[e] = 1;
    out[e] = p[best];
    diff[e] = least / fmax(1e-300, mag);
  } else {
    atomicAdd(open, 1);
  }
}

}  // namespace

int PadeSeries::init(const std::vector<int32_t>& row, const std::vector<int32_t>& col, cudaStream_t st) {
  nel = (int)row.size();
  TT_TRY(row_.upload(row, st));
  TT_TRY(col_.upload(col, st));
  TT_TRY(a_.alloc((size_t)2 * nel * PD_TERMS));
  TT_TRY(pa_.alloc((size_t)2 * nel * PD_S));
  TT_TRY(out_.alloc((size_t)2 * nel));
  TT_TRY(diff_.alloc(nel));
  TT_TRY(done_.alloc(nel));
  TT_TRY(open_.alloc(1));
  TT_CUDA_TRY(cudaMemsetAsync(done_.ptr, 0, nel, st));
  return TT_OK;
}

int PadeSeries::term(const double* d_R, int n, int t, cudaStream_t st) {
  k_pade_term<<<ceil_div(nel, 128), 128, 0, st>>>(reinterpret_cast<const double2*>(d_R), n, row_.ptr, col_.ptr, nel, t,
                                                  done_.ptr, reinterpret_cast<double2*>(a_.ptr));
  count_launch();
  TT_CUDA_TRY(cudaGetLastError());
  return TT_OK;
}

int PadeSeries::order(int N, int* open, cudaStream_t st) {
  const size_t smem = sizeof(double2) * PD_WARPS * 2 * PD_S * PD_S;
  TT_TRY(smem_limit_once((const void*)k_pade_order, (int)smem));
  TT_CUDA_TRY(cudaMemsetAsync(open_.ptr, 0, sizeof(int), st));
  k_pade_order<<<ceil_div(nel, PD_WARPS), 32 * PD_WARPS, smem, st>>>(
      N, nel, reinterpret_cast<const double2*>(a_.ptr), reinterpret_cast<double2*>(pa_.ptr), done_.ptr,
      reinterpret_cast<double2*>(out_.ptr), diff_.ptr, open_.ptr);
  count_launch();
  TT_CUDA_TRY(cudaGetLastError());
  TT_CUDA_TRY(cudaMemcpyAsync(open, open_.ptr, sizeof(int), cudaMemcpyDeviceToHost, st));
  TT_CUDA_TRY(cudaStreamSynchronize(st));
  return TT_OK;
}

int PadeSeries::result(std::vector<double>& out, std::vector<double>& diff, cudaStream_t st) {
  out.resize((size_t)2 * nel);
  diff.resize(nel);
  TT_CUDA_TRY(cudaMemcpyAsync(out.data(), out_.ptr, sizeof(double) * out.size(), cudaMemcpyDeviceToHost, st));
  TT_CUDA_TRY(cudaMemcpyAsync(diff.data(), diff_.ptr, sizeof(double) * nel, cudaMemcpyDeviceToHost, st));
  TT_CUDA_TRY(cudaStreamSynchronize(st));
  return TT_OK;
}

}  // namespace tt
