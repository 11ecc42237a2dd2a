// Kernels of the Faddeev-solve stage other than the LU factorisation and the
// A build (a_build.cu): resolvent diagonals, L = 1 - A diag(G), right-hand
// sides and the FP64 refinement residual.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <map>
#include <utility>

#include "tt_kernels.h"

namespace tt {

constexpr double kMp_d = 938.272;
constexpr double kMn_d = 939.565;

int DeviceLayout::upload(const ChannelLayout& L, const std::vector<double>& qwp, cudaStream_t st) {
  Nalpha = L.Nalpha;
  Np = L.Np;
  Nq = L.Nq;
  n = L.Nalpha * L.Np * L.Nq;
  TT_TRY(blk.upload(L.blk, st));
  TT_TRY(part.upload(L.part, st));
  TT_TRY(dim.upload(L.dim, st));
  TT_TRY(cpl_off.upload(L.cpl_off, st));
  TT_TRY(cpl.upload(L.cpl, st));
  TT_TRY(blk_off.upload(L.blk_off, st));
  TT_TRY(blk_dim.upload(L.blk_dim, st));
  TT_TRY(C.upload(L.C, st));
  TT_TRY(VC.upload(L.VC, st));
  TT_TRY(e_off.upload(L.e_off, st));
  TT_TRY(e_swp.upload(L.e_swp, st));
  TT_TRY(q_WP.upload(qwp, st));
  return TT_OK;
}

namespace {

__device__ __forceinline__ double heaviside(double v) { return v < 0 ? 0.0 : 1.0; }

// make_resolvent.cpp:14-80 (bound-continuum and continuum-continuum terms)
__global__ void k_resolvent(int Na, int Nq, int Np, const int32_t* __restrict__ e_off,
                            const double* __restrict__ e_swp, const double* __restrict__ qwp,
                            const double* __restrict__ E, int nE, double2* __restrict__ G) {
  const int n = Na * Nq * Np;
  const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= (size_t)n * nE) return;
  const int j = (int)(tid / n), idx = (int)(tid % n);
  const int a = idx / (Nq * Np), q = (idx / Np) % Nq, p = idx % Np;
  const double e_lo = e_swp[e_off[a] + p], e_hi = e_swp[e_off[a] + p + 1];
  const double q_lo = qwp[q], q_hi = qwp[q + 1];
  const double En = E[j];
  double re, im;
  if (e_lo < 0) {
    const double Eb = e_lo;
    const double mu1 = kMn_d * (kMn_d + kMp_d + Eb) / (kMn_d + kMn_d + kMp_d + Eb);
    const double Eq_lo = q_lo * q_lo / (2 * mu1), Eq_hi = q_hi * q_hi / (2 * mu1);
    const double Dq = Eq_hi - Eq_lo;
    re = log(fabs((Eq_lo + Eb - En) / (Eq_hi + Eb - En))) / (Dq);
    im = (heaviside(Eq_hi + Eb - En) - heaviside(Eq_lo + Eb - En)) * (-M_PI) / (Dq);
  } else {
    const double Eb = 0;
    const double mu1 = kMn_d * (kMn_d + kMp_d + Eb) / (kMn_d + kMn_d + kMp_d + Eb);
    const double Eq_lo = q_lo * q_lo / (2 * mu1), Eq_hi = q_hi * q_hi / (2 * mu1);
    const double Ep = 0.5 * (e_lo + e_hi), Eq = 0.5 * (Eq_lo + Eq_hi);
    const double Dq = Eq_hi - Eq_lo, Dp = e_hi - e_lo;
    const double DM = 0.5 * (Dp - Dq), DP = 0.5 * (Dp + Dq), D = Ep + Eq - En;
    re = ((D + DM) * log(fabs(D + DM)) + (D - DM) * log(fabs(D - DM)) - (D + DP) * log(fabs(D + DP)) -
          (D - DP) * log(fabs(D - DP))) /
         (Dp * Dq);
    im = ((D + DM) * heaviside(D + DM) + (D - DM) * heaviside(D - DM) - (D + DP) * heaviside(D + DP) -
          (D - DP) * heaviside(D - DP)) *
         M_PI / (Dp * Dq);
  }
  G[tid] = make_double2(re, im);
}

// First-order change dG of the resolvents of k_resolvent for a change de of
// the SWP energy boundaries (layout of e_swp; a bound state's lower boundary
// is E_bound, which also sets the n-d reduced mass of its bins) and dEn of the
// energies E_j = E_com,j + E_bound (make_resolvent.cpp:14-80 differentiated;
// d(x ln|x|) = (ln|x| + 1) dx, d(x theta(x)) = theta(x) dx).
__global__ void k_dresolvent(int Na, int Nq, int Np, const int32_t* __restrict__ e_off,
                             const double* __restrict__ e_swp, const double* __restrict__ de_swp,
                             const double* __restrict__ qwp, const double* __restrict__ E, int nE, double dEn,
                             double2* __restrict__ dG) {
  const int n = Na * Nq * Np;
  const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= (size_t)n * nE) return;
  const int j = (int)(tid / n), idx = (int)(tid % n);
  const int a = idx / (Nq * Np), q = (idx / Np) % Nq, p = idx % Np;
  const double e_lo = e_swp[e_off[a] + p], e_hi = e_swp[e_off[a] + p + 1];
  const double de_lo = de_swp[e_off[a] + p], de_hi = de_swp[e_off[a] + p + 1];
  const double q_lo = qwp[q], q_hi = qwp[q + 1];
  const double En = E[j], dE = dEn;
  double dre, dim;
  if (e_lo < 0) {
    const double Eb = e_lo, dEbl = de_lo;
    const double den = kMn_d + kMn_d + kMp_d + Eb;
    const double mu1 = kMn_d * (kMn_d + kMp_d + Eb) / den;
    const double dmu1 = kMn_d * kMn_d / (den * den) * dEbl;
    const double Eq_lo = q_lo * q_lo / (2 * mu1), Eq_hi = q_hi * q_hi / (2 * mu1);
    const double dEq_lo = -Eq_lo * dmu1 / mu1, dEq_hi = -Eq_hi * dmu1 / mu1;
    const double Dq = Eq_hi - Eq_lo, dDq = dEq_hi - dEq_lo;
    const double x = Eq_lo + Eb - En, y = Eq_hi + Eb - En;
    const double dx = dEq_lo + dEbl - dE, dy = dEq_hi + dEbl - dE;
    const double re = log(fabs(x / y)) / Dq;
    const double im = (heaviside(y) - heaviside(x)) * (-M_PI) / Dq;
    dre = (dx / x - dy / y) / Dq - re * dDq / Dq;
    dim = -im * dDq / Dq;
  } else {
    const double mu1 = kMn_d * (kMn_d + kMp_d) / (kMn_d + kMn_d + kMp_d);
    const double Eq_lo = q_lo * q_lo / (2 * mu1), Eq_hi = q_hi * q_hi / (2 * mu1);
    const double Ep = 0.5 * (e_lo + e_hi), Eq = 0.5 * (Eq_lo + Eq_hi);
    const double Dq = Eq_hi - Eq_lo, Dp = e_hi - e_lo;
    const double DM = 0.5 * (Dp - Dq), DP = 0.5 * (Dp + Dq), D = Ep + Eq - En;
    const double dDp = de_hi - de_lo, dD = 0.5 * (de_lo + de_hi) - dE;
    const double xs[4] = {D + DM, D - DM, D + DP, D - DP};
    const double dxs[4] = {dD + 0.5 * dDp, dD - 0.5 * dDp, dD + 0.5 * dDp, dD - 0.5 * dDp};
    const double sg[4] = {1.0, 1.0, -1.0, -1.0};
    double nre = 0, nim = 0, dnre = 0, dnim = 0;
    for (int t = 0; t < 4; t++) {
      nre += sg[t] * xs[t] * log(fabs(xs[t]));
      nim += sg[t] * xs[t] * heaviside(xs[t]);
      dnre += sg[t] * (log(fabs(xs[t])) + 1.0) * dxs[t];
      dnim += sg[t] * heaviside(xs[t]) * dxs[t];
    }
    const double re = nre / (Dp * Dq), im = nim * M_PI / (Dp * Dq);
    dre = dnre / (Dp * Dq) - re * dDp / Dp;
    dim = dnim * M_PI / (Dp * Dq) - im * dDp / Dp;
  }
  dG[tid] = make_double2(dre, dim);
}

template <typename T>
__device__ __forceinline__ T make_c(double re, double im);
template <>
__device__ __forceinline__ double2 make_c<double2>(double re, double im) { return make_double2(re, im); }
template <>
__device__ __forceinline__ float2 make_c<float2>(double re, double im) {
  return make_float2((float)re, (float)im);
}

// L_b = 1 - A diag(G_b) for NB resolvents in one pass over A.  A thread keeps the
// NB resolvents of its VEC columns (2 where rows are 16-byte aligned: even n) for
// FL_ROWS rows, four rows' loads at a time.  Bound: A read once, every L written
// once.  n = 42,300, 2 resolvents: 13.9 -> 7.0 ms (6.1 TB/s); n = 20,160, 4: 6.3 ->
// 2.6 ms (one pass over A each before).
constexpr int FL_ROWS = 32;
template <typename T>
struct FormL {
  T* L[4];
};
template <typename T, int NB, int VEC>
__global__ void __launch_bounds__(256) k_form_L(const double* __restrict__ A, const double2* __restrict__ G, int n,
                                                FormL<T> out) {
  const int c = (blockIdx.x * 256 + threadIdx.x) * VEC;
  if (c >= n) return;
  double2 g[NB][VEC];
#pragma unroll
  for (int b = 0; b < NB; b++)
#pragma unroll
    for (int v = 0; v < VEC; v++) g[b][v] = G[(size_t)b * n + c + v];
  const int r0 = blockIdx.y * FL_ROWS, r1 = min(n, r0 + FL_ROWS);
  for (int r = r0; r < r1; r += 4) {
    double a[4][VEC];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const double* p = A + (size_t)min(r + u, r1 - 1) * n + c;
      if constexpr (VEC == 2) {
        const double2 t = __ldcs(reinterpret_cast<const double2*>(p));
        a[u][0] = t.x;
        a[u][1] = t.y;
      } else {
        a[u][0] = __ldcs(p);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      if (r + u >= r1) break;
#pragma unroll
      for (int b = 0; b < NB; b++) {
        T v[VEC];
#pragma unroll
        for (int x = 0; x < VEC; x++)
          v[x] = make_c<T>((r + u == c + x ? 1.0 : 0.0) - a[u][x] * g[b][x].x, -a[u][x] * g[b][x].y);
        T* o = out.L[b] + (size_t)(r + u) * n + c;
        if constexpr (VEC == 2 && sizeof(T) == 8) {
          *reinterpret_cast<float4*>(o) = make_float4(v[0].x, v[0].y, v[1].x, v[1].y);
        } else {
#pragma unroll
          for (int x = 0; x < VEC; x++) o[x] = v[x];
        }
      }
    }
  }
}
template <typename T, int NB>
void launch_form_L(const double* A, const double2* G, int n, const FormL<T>& out, bool wide, cudaStream_t st) {
  const int rows = ceil_div(n, FL_ROWS);
  if (wide) k_form_L<T, NB, 2><<<dim3(ceil_div(n, 512), rows), 256, 0, st>>>(A, G, n, out);
  else k_form_L<T, NB, 1><<<dim3(ceil_div(n, 256), rows), 256, 0, st>>>(A, G, n, out);
}

__global__ void k_gather_rhs(const double* __restrict__ A, int n, const int32_t* __restrict__ cols, int nrhs,
                             double2* __restrict__ b) {
  const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= (size_t)n * nrhs) return;
  const int k = (int)(tid / n), i = (int)(tid % n);
  b[tid] = make_double2(A[(size_t)i * n + cols[k]], 0.0);
}

// part[slab][v] = A y_v over the slab's columns, for nv <= 4 NT vectors in one pass over
// A: a real n x n by n x 8 NT product on the FP64 tensor cores (m8n8k4), the real and
// imaginary parts of a vector being two columns.  A warp takes 16 rows; a lane's four
// neighbouring columns of a row serve as the k = lane % 4 elements of four products, so
// A goes from HBM to registers in 16-byte loads (VEC = 2, even n; else 8-byte), asked
// for two steps of 16 columns ahead, and y comes through shared memory, transposed, 128
// columns at a time.  Slabs of columns even out the last wave of CTAs: two an SM, their
// number chosen in residual_slabs.  Bound: A read once.  FMA kernels of up to 4 vectors
// a launch before: six vectors, n = 16,128 0.87 -> 0.36 ms,
// n = 42,300 5.6 -> 2.5 ms (5.8 TB/s); twelve at n = 20,160 2.97 -> 0.80 ms.
constexpr int RM_ROWS = 128, RM_COLS = 128, RM_LD = RM_COLS + 2, RM_NT = 3, RM_SLABS = 16;
__device__ __forceinline__ void mma884(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}
template <int NT, int VEC>
__global__ void __launch_bounds__(256, 2) k_residual(const double* __restrict__ A, int n,
                                                     const double2* __restrict__ y, int nv, int slabs,
                                                     double2* __restrict__ part) {
  __shared__ __align__(16) double sy[8 * NT][RM_LD];
  constexpr int AHEAD = 2, STEP = 16, PER = RM_COLS / STEP;
  const int tid = threadIdx.x, warp = tid >> 5, r = (tid & 31) >> 2, q = tid & 3;
  const int chunks = (n + RM_COLS - 1) / RM_COLS;
  const int c_lo = (int)((long long)chunks * blockIdx.y / slabs) * RM_COLS;
  const int c_hi = min(n, (int)((long long)chunks * (blockIdx.y + 1) / slabs) * RM_COLS);
  const int64_t row0 = (int64_t)blockIdx.x * RM_ROWS + warp * 16 + r;
  const double* Ar[2];  // rows past the last read it again
#pragma unroll
  for (int m = 0; m < 2; m++) Ar[m] = A + min(row0 + 8 * m, (int64_t)n - 1) * n + 4 * q;
  auto load = [&](int c, double(&a)[2][4]) {
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
      for (int h = 0; h < 4; h += VEC) {
        const bool in = c + 4 * q + h < c_hi;
        if constexpr (VEC == 2) {
          const double2 t = in ? __ldcs(reinterpret_cast<const double2*>(Ar[m] + c + h)) : make_double2(0.0, 0.0);
          a[m][h] = t.x;
          a[m][h + 1] = t.y;
        } else {
          a[m][h] = in ? __ldcs(Ar[m] + c + h) : 0.0;
        }
      }
  };
  double acc[2][NT][2] = {};
  double a[AHEAD + 1][2][4];
#pragma unroll
  for (int d = 0; d < AHEAD; d++) load(c_lo + d * STEP, a[d + 1]);
  for (int c0 = c_lo; c0 < c_hi; c0 += RM_COLS) {
    __syncthreads();
#pragma unroll
    for (int e = tid; e < 4 * NT * RM_COLS; e += 256) {
      const int v = e / RM_COLS, i = e % RM_COLS;
      const double2 z = v < nv && c0 + i < n ? y[(size_t)v * n + c0 + i] : make_double2(0.0, 0.0);
      sy[2 * v][i] = z.x;
      sy[2 * v + 1][i] = z.y;
    }
    __syncthreads();
    const int s1 = min(PER, (c_hi - c0 + STEP - 1) / STEP);
#pragma unroll 2
    for (int s = 0; s < s1; s++) {
#pragma unroll
      for (int d = 0; d < AHEAD; d++)
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
          for (int h = 0; h < 4; h++) a[d][m][h] = a[d + 1][m][h];
      load(c0 + (s + AHEAD) * STEP, a[AHEAD]);
#pragma unroll
      for (int j = 0; j < NT; j++) {
        const double2* p = reinterpret_cast<const double2*>(&sy[8 * j + r][s * STEP + 4 * q]);
        const double2 b0 = p[0], b1 = p[1];
#pragma unroll
        for (int m = 0; m < 2; m++) {
          mma884(acc[m][j], a[0][m][0], b0.x);
          mma884(acc[m][j], a[0][m][1], b0.y);
          mma884(acc[m][j], a[0][m][2], b1.x);
          mma884(acc[m][j], a[0][m][3], b1.y);
        }
      }
    }
  }
#pragma unroll
  for (int m = 0; m < 2; m++)
#pragma unroll
    for (int j = 0; j < NT; j++)
      if (row0 + 8 * m < n && 4 * j + q < nv)
        part[((size_t)blockIdx.y * nv + 4 * j + q) * n + row0 + 8 * m] = make_double2(acc[m][j][0], acc[m][j][1]);
}

// r = b - x + the sum of the slabs, in order
__global__ void k_residual_sum(const double2* __restrict__ part, int slabs, size_t total,
                               const double2* __restrict__ b, const double2* __restrict__ x, double2* __restrict__ r) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total) return;
  double2 s = part[t];
  for (int i = 1; i < slabs; i++) {
    const double2 p = part[(size_t)i * total + t];
    s.x += p.x;
    s.y += p.y;
  }
  r[t] = make_double2(b[t].x - x[t].x + s.x, b[t].y - x[t].y + s.y);
}

// Slabs of columns: the number whose CTAs fill their last wave best, each costing a
// pass over the vectors, about a hundredth of a CTA's work
int residual_slabs(int n) {
  const int rows = ceil_div(n, RM_ROWS), slots = 2 * device_sm_count();
  int best = 1;
  double least = 1e30;
  for (int s = 1; s <= std::min((int)ceil_div(n, RM_COLS), RM_SLABS); s++) {
    const double t = (double)ceil_div((size_t)rows * s, slots) / s + 0.01 * s * rows / slots;
    if (t < least) {
      least = t;
      best = s;
    }
  }
  return best;
}

template <int VEC>
void launch_residual(const double* A, int n, const double2* y, int nv, int slabs, double2* part, cudaStream_t st) {
  const dim3 grid(ceil_div(n, RM_ROWS), slabs);
  switch ((nv + 3) / 4) {
    case 1: k_residual<1, VEC><<<grid, 256, 0, st>>>(A, n, y, nv, slabs, part); break;
    case 2: k_residual<2, VEC><<<grid, 256, 0, st>>>(A, n, y, nv, slabs, part); break;
    default: k_residual<3, VEC><<<grid, 256, 0, st>>>(A, n, y, nv, slabs, part); break;
  }
}

__global__ void k_hadamard(const double2* __restrict__ G, const int32_t* __restrict__ rhs_e, int n,
                           const double2* __restrict__ x, int nrhs, double2* __restrict__ y) {
  const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= (size_t)n * nrhs) return;
  const int k = (int)(tid / n), c = (int)(tid % n);
  const double2 g = G[(size_t)rhs_e[k] * n + c];
  const double2 v = x[tid];
  y[tid] = make_double2(g.x * v.x - g.y * v.y, g.x * v.y + g.y * v.x);
}

__global__ void k_axpy_norm(double2* __restrict__ x, const double2* __restrict__ d, int n, int nrhs,
                            unsigned long long* __restrict__ dmax, unsigned long long* __restrict__ xmax) {
  const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  double ad = 0.0, ax = 0.0;
  int k = 0;
  if (tid < (size_t)n * nrhs) {
    k = (int)(tid / n);
    const double2 dv = d[tid];
    double2 xv = x[tid];
    xv.x += dv.x;
    xv.y += dv.y;
    x[tid] = xv;
    ad = fmax(fabs(dv.x), fabs(dv.y));
    ax = fmax(fabs(xv.x), fabs(xv.y));
  }
  if (tid < (size_t)n * nrhs) {
    // non-negative doubles order like their bit patterns
    atomicMax(&dmax[k], (unsigned long long)__double_as_longlong(ad));
    atomicMax(&xmax[k], (unsigned long long)__double_as_longlong(ax));
  }
}

// On-shell entries after the update: out[k nrows + r] = (|d_k[rows[r]]|, |x_k[rows[r]]|)
__global__ void k_onshell_pick(const double2* __restrict__ x, const double2* __restrict__ d, int n, int nrhs,
                               const int32_t* __restrict__ rows, int nrows, double2* __restrict__ out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nrhs * nrows) return;
  const int k = t / nrows, r = t % nrows;
  const size_t i = (size_t)k * n + rows[r];
  out[t] = make_double2(hypot(d[i].x, d[i].y), hypot(x[i].x, x[i].y));
}

}  // namespace

int resolvent_device(const DeviceLayout& L, const double* d_E, int nE, double* d_G, cudaStream_t st) {
  const size_t total = (size_t)L.n * nE;
  if (total == 0) return TT_OK;
  ProfScope prof(TT_PROF_VECTOR, st, 0.0, 16.0 * (double)total);
  k_resolvent<<<ceil_div(total, 256), 256, 0, st>>>(L.Nalpha, L.Nq, L.Np, L.e_off.ptr, L.e_swp.ptr, L.q_WP.ptr, d_E,
                                                    nE, reinterpret_cast<double2*>(d_G));
  count_launch();
  TT_CUDA_TRY(cudaGetLastError());
  return TT_OK;
}

int dresolvent_device(const DeviceLayout& L, const double* d_de, double dE, const double* d_E, int nE, double* d_dG,
                      cudaStream_t st) {
  const size_t total = (size_t)L.n * nE;
  if (total == 0) return TT_OK;
  k_dresolvent<<<ceil_div(total, 256), 256, 0, st>>>(L.Nalpha, L.Nq, L.Np, L.e_off.ptr, L.e_swp.ptr, d_de, L.q_WP.ptr,
                                                     d_E, nE, dE, reinterpret_cast<double2*>(d_dG));
  count_launch();
  TT_CUDA_TRY(cudaGetLastError());
  return TT_OK;
}

int resolvent_device_tables(int Na, int Nq, int Np, const int32_t* e_off, const double* e_swp, const double* q_WP,
                            const double* d_E, int nE, double* d_G, cudaStream_t st) {
  const size_t total = (size_t)Na * Nq * Np * nE;
  if (total == 0) return TT_OK;
  k_resolvent<<<ceil_div(total, 256), 256, 0, st>>>(Na, Nq, Np, e_off, e_swp, q_WP, d_E, nE,
                                                    reinterpret_cast<double2*>(d_G));
  count_launch();
  TT_CUDA_TRY(cudaGetLastError());
  return TT_OK;
}

template <typename T>
int form_L_device(const double* d_A, const double* d_G, int n, T* const* d_L, int nb, cudaStream_t st) {
  if (n <= 0) return TT_OK;
  const double total = (double)n * n;
  ProfScope prof(TT_PROF_FORM_L, st, 2.0 * total * nb, (8.0 + nb * sizeof(T)) * total);
  const double2* G = reinterpret_cast<const double2*>(d_G);
  FormL<T> out{};
  bool wide = n % 2 == 0;
  for (int b = 0; b < nb; b++) {
    out.L[b] = d_L[b];
    wide = wide && (uintptr_t)d_L[b] % 16 == 0;
  }
  switch (nb) {
    case 1: launch_form_L<T, 1>(d_A, G, n, out, wide, st); break;
    case 2: launch_form_L<T, 2>(d_A, G, n, out, wide, st); break;
    case 3: launch_form_L<T, 3>(d_A, G, n, out, wide, st); break;
    case 4: launch_form_L<T, 4>(d_A, G, n, out, wide, st); break;
    default: set_error("1 - A G for " + std::to_string(nb) + " energies (1..4)"); return TT_ERR_BADARG;
  }
  count_launch();
  TT_CUDA_TRY(cudaGetLastError());
  return TT_OK;
}
template int form_L_device<double2>(const double*, const double*, int, double2* const*, int, cudaStream_t);
template int form_L_device<float2>(const double*, const double*, int, float2* const*, int, cudaStream_t);

int gather_rhs_device(const double* d_A, int n, const int32_t* d_cols, int nrhs, double* d_b, cudaStream_t st) {
  ProfScope prof(TT_PROF_VECTOR, st, 0.0, 24.0 * (double)n * nrhs);
  k_gather_rhs<<<ceil_div((size_t)n * nrhs, 256), 256, 0, st>>>(d_A, n, d_cols, nrhs, reinterpret_cast<double2*>(d_b));
  count_launch();
  TT_CUDA_TRY(cudaGetLastError());
  return TT_OK;
}

int hadamard_device(const double* d_G, const int32_t* d_rhs_e, int n, const double* d_x, int nrhs, double* d_y,
                    cudaStream_t st) {
  ProfScope prof(TT_PROF_VECTOR, st, 6.0 * (double)n * nrhs, 48.0 * (double)n * nrhs);
  k_hadamard<<<ceil_div((size_t)n * nrhs, 256), 256, 0, st>>>(reinterpret_cast<const double2*>(d_G), d_rhs_e, n,
                                                             reinterpret_cast<const double2*>(d_x), nrhs,
                                                             reinterpret_cast<double2*>(d_y));
  count_launch();
  TT_CUDA_TRY(cudaGetLastError());
  return TT_OK;
}

int residual_multi_device(const double* d_A, int n, const double* d_y, const double* d_b, const double* d_x, int nrhs,
                          double* d_r, cudaStream_t st) {
  // one pass over A per group of up to 4 RM_NT vectors
  constexpr int GROUP = 4 * RM_NT;
  ProfScope prof(TT_PROF_RESIDUAL, st, 4.0 * n * (double)n * nrhs, 8.0 * n * (double)n * ceil_div(nrhs, GROUP));
  const int slabs = residual_slabs(n);
  DevBuf<double2> part;
  TT_TRY(part.alloc((size_t)slabs * std::min(nrhs, GROUP) * n));
  for (int v0 = 0; v0 < nrhs; v0 += GROUP) {
    const int nv = std::min(GROUP, nrhs - v0);
    const size_t o = (size_t)v0 * n, total = (size_t)nv * n;
    const double2* y = reinterpret_cast<const double2*>(d_y) + o;
    if (n % 2 == 0) launch_residual<2>(d_A, n, y, nv, slabs, part.ptr, st);
    else launch_residual<1>(d_A, n, y, nv, slabs, part.ptr, st);
    count_launch();
    TT_CUDA_TRY(cudaGetLastError());
    k_residual_sum<<<ceil_div(total, 256), 256, 0, st>>>(part.ptr, slabs, total,
                                                        reinterpret_cast<const double2*>(d_b) + o,
                                                        reinterpret_cast<const double2*>(d_x) + o,
                                                        reinterpret_cast<double2*>(d_r) + o);
    count_launch();
    TT_CUDA_TRY(cudaGetLastError());
  }
  return TT_OK;
}

int axpy_norms_device(double* d_x, const double* d_d, int n, int nrhs, double* h_ratio, cudaStream_t st,
                      const int32_t* d_rows, int nrows, double* h_elem) {
  if (!d_rows || !h_elem) nrows = 0;
  // [2 nrhs] maxima as ordered bit patterns, then nrhs x nrows (|d|, |x|) pairs
  const size_t words = 2 * (size_t)nrhs + 2 * (size_t)nrhs * nrows;
  DevBuf<unsigned long long> mx;
  TT_TRY(mx.alloc(words));
  TT_CUDA_TRY(cudaMemsetAsync(mx.ptr, 0, sizeof(unsigned long long) * 2 * nrhs, st));
  ProfScope prof(TT_PROF_VECTOR, st, 4.0 * (double)n * nrhs, 48.0 * (double)n * nrhs);
  k_axpy_norm<<<ceil_div((size_t)n * nrhs, 256), 256, 0, st>>>(reinterpret_cast<double2*>(d_x),
                                                              reinterpret_cast<const double2*>(d_d), n, nrhs, mx.ptr,
                                                              mx.ptr + nrhs);
  count_launch();
  TT_CUDA_TRY(cudaGetLastError());
  if (nrows > 0) {
    k_onshell_pick<<<ceil_div((size_t)nrhs * nrows, 64), 64, 0, st>>>(
        reinterpret_cast<const double2*>(d_x), reinterpret_cast<const double2*>(d_d), n, nrhs, d_rows, nrows,
        reinterpret_cast<double2*>(mx.ptr + 2 * nrhs));
    count_launch();
    TT_CUDA_TRY(cudaGetLastError());
  }
  std::vector<unsigned long long> h(words);
  TT_CUDA_TRY(cudaMemcpyAsync(h.data(), mx.ptr, sizeof(unsigned long long) * words, cudaMemcpyDeviceToHost, st));
  TT_CUDA_TRY(cudaStreamSynchronize(st));
  for (int k = 0; k < nrhs; k++) {
    double dm, xm;
    memcpy(&dm, &h[k], 8);
    memcpy(&xm, &h[nrhs + k], 8);
    h_ratio[k] = xm > 0 ? dm / xm : dm;
  }
  if (nrows > 0) {
    // each on-shell entry's own |dx| / |x|; entries below kOnshellZeroFloor of
    // the largest on-shell |x| of their right-hand side are zero by symmetry
    // up to rounding and are measured against that floor instead
    const double* pr = reinterpret_cast<const double*>(h.data() + 2 * nrhs);
    for (int k = 0; k < nrhs; k++) {
      double big = 0;
      for (int r = 0; r < nrows; r++) big = std::max(big, pr[2 * ((size_t)k * nrows + r) + 1]);
      for (int r = 0; r < nrows; r++) {
        const double dv = pr[2 * ((size_t)k * nrows + r)], xv = pr[2 * ((size_t)k * nrows + r) + 1];
        const double den = std::max(xv, kOnshellZeroFloor * big);
        h_elem[(size_t)k * nrows + r] = den > 0 ? dv / den : dv;
      }
    }
  }
  return TT_OK;
}

int smem_limit_once(const void* kernel, int bytes) {
  static std::mutex mu;
  static std::map<std::pair<const void*, int>, int> limit;  // (kernel, device) -> limit set so far
  int dev = 0;
  TT_CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lock(mu);
  int& cur = limit[std::make_pair(kernel, dev)];
  if (bytes <= cur) return TT_OK;  // only ever raised: a launch needing less still fits
  TT_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  cur = bytes;
  return TT_OK;
}

int device_sm_count() {
  static int sms = -1;
  if (sms < 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 148;
  }
  return sms;
}

}  // namespace tt
