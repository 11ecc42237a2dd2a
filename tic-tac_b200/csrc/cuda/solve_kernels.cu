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

// r_v = b_v - x_v + A y_v for NV <= 4 vectors in one pass over A.  A CTA owns 32
// rows, 4 per warp; a lane takes VEC columns of each row at a step (2 where rows
// are 16-byte aligned: even n), and asks for A two steps ahead.  y comes through
// shared memory, 512 columns at a time, read from L2 once per 32 rows.  Bound: A
// read once; the loads in flight (two steps x 4 rows x 16 warps an SM, 64 KB)
// carry on across the refills of y.  n = 42,300: 2 vectors 3.00 -> 2.41 ms
// (5.9 TB/s), 4 vectors 3.48 -> 3.16 ms (their accumulators leave one step ahead).
constexpr int R2_ROWS = 32, R2_COLS = 512;
template <int NV, int VEC>
__global__ void __launch_bounds__(256, 2) k_residual(const double* __restrict__ A, int n,
                                                     const double2* __restrict__ y, const double2* __restrict__ b,
                                                     const double2* __restrict__ x, double2* __restrict__ r) {
  __shared__ double2 sy[NV][R2_COLS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t row0 = (int64_t)blockIdx.x * R2_ROWS + warp * 4;
  const double* Ar = A + (size_t)min(row0, (int64_t)n - 1) * n + lane * VEC;
  int64_t off[4];  // rows past the last read it again
#pragma unroll
  for (int h = 0; h < 4; h++) off[h] = row0 + h < n ? (int64_t)h * n : 0;
  double sr[4][NV], si[4][NV];
#pragma unroll
  for (int h = 0; h < 4; h++)
#pragma unroll
    for (int v = 0; v < NV; v++) sr[h][v] = si[h][v] = 0.0;
  constexpr int STEP = 32 * VEC, PER = R2_COLS / STEP;
  const int steps = (n + STEP - 1) / STEP;
  auto load = [&](int s, double(&a)[4][VEC]) {
    const int c = s * STEP;
    const bool in = c + lane * VEC < n;
#pragma unroll
    for (int h = 0; h < 4; h++) {
      if constexpr (VEC == 2) {
        const double2 t = in ? __ldcs(reinterpret_cast<const double2*>(Ar + off[h] + c)) : make_double2(0.0, 0.0);
        a[h][0] = t.x;
        a[h][1] = t.y;
      } else {
        a[h][0] = in ? __ldcs(Ar + off[h] + c) : 0.0;
      }
    }
  };
  // steps in flight beyond the present one, as the accumulators leave registers
  constexpr int AHEAD = NV > 2 ? 1 : 2;
  double a[AHEAD + 1][4][VEC];
#pragma unroll
  for (int d = 0; d < AHEAD; d++) load(d, a[d + 1]);
  for (int s0 = 0; s0 < steps; s0 += PER) {
    __syncthreads();
#pragma unroll
    for (int v = 0; v < NV; v++)
      for (int i = threadIdx.x; i < R2_COLS; i += 256) {
        const int c = s0 * STEP + i;
        sy[v][i] = c < n ? y[(size_t)v * n + c] : make_double2(0.0, 0.0);
      }
    __syncthreads();
    const int s1 = min(PER, steps - s0);
#pragma unroll 2
    for (int s = 0; s < s1; s++) {
#pragma unroll
      for (int d = 0; d < AHEAD; d++)
#pragma unroll
        for (int h = 0; h < 4; h++)
#pragma unroll
          for (int q = 0; q < VEC; q++) a[d][h][q] = a[d + 1][h][q];
      load(s0 + s + AHEAD, a[AHEAD]);
#pragma unroll
      for (int v = 0; v < NV; v++)
#pragma unroll
        for (int q = 0; q < VEC; q++) {
          const double2 t = sy[v][s * STEP + lane * VEC + q];
#pragma unroll
          for (int h = 0; h < 4; h++) {
            sr[h][v] += a[0][h][q] * t.x;
            si[h][v] += a[0][h][q] * t.y;
          }
        }
    }
  }
#pragma unroll
  for (int h = 0; h < 4; h++)
#pragma unroll
    for (int v = 0; v < NV; v++)
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        sr[h][v] += __shfl_xor_sync(0xffffffffu, sr[h][v], o);
        si[h][v] += __shfl_xor_sync(0xffffffffu, si[h][v], o);
      }
  if (lane == 0) {
#pragma unroll
    for (int h = 0; h < 4; h++) {
      if (row0 + h >= n) break;
#pragma unroll
      for (int v = 0; v < NV; v++) {
        const size_t o = (size_t)v * n + row0 + h;
        r[o] = make_double2(b[o].x - x[o].x + sr[h][v], b[o].y - x[o].y + si[h][v]);
      }
    }
  }
}

template <int VEC>
void launch_residual(int nv, const double* A, int n, const double2* y, const double2* b, const double2* x, double2* r,
                     cudaStream_t st) {
  const unsigned grid = ceil_div((size_t)n, R2_ROWS);
  switch (nv) {
    case 1: k_residual<1, VEC><<<grid, 256, 0, st>>>(A, n, y, b, x, r); break;
    case 2: k_residual<2, VEC><<<grid, 256, 0, st>>>(A, n, y, b, x, r); break;
    case 3: k_residual<3, VEC><<<grid, 256, 0, st>>>(A, n, y, b, x, r); break;
    default: k_residual<4, VEC><<<grid, 256, 0, st>>>(A, n, y, b, x, r); break;
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
  // one pass over A per group of up to 4 vectors
  ProfScope prof(TT_PROF_RESIDUAL, st, 4.0 * n * (double)n * nrhs, 8.0 * n * (double)n * ((nrhs + 3) / 4));
  for (int v0 = 0; v0 < nrhs; v0 += 4) {
    const int nv = std::min(4, nrhs - v0);
    const size_t o = (size_t)v0 * n;
    const double2* y = reinterpret_cast<const double2*>(d_y) + o;
    const double2* b = reinterpret_cast<const double2*>(d_b) + o;
    const double2* x = reinterpret_cast<const double2*>(d_x) + o;
    double2* r = reinterpret_cast<double2*>(d_r) + o;
    if (n % 2 == 0) launch_residual<2>(nv, d_A, n, y, b, x, r, st);
    else launch_residual<1>(nv, d_A, n, y, b, x, r, st);
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
