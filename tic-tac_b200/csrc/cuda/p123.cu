// Device builder of the sparse wave-packet permutation matrix P123 of one 3N
// channel, in CSR.  Restates calculate_WP_overlap and
// calculate_permutation_elements_for_3N_channel
// (CPP/make_permutation_matrix.cpp:160-255, 324-943) and the cell integral and
// geometric function of CPP/auxiliary.cpp:660-746, 950-1067 as a pipeline of
// kernels:
//
//   1. k_overlap      boolean WP-cell overlap mask over (q',p',q,p)
//   2. k_cell_weights quadrature weights of each overlapping cell on the
//                     (phi, x) mesh: wx wphi cos sin (kmax^2-kmin^2)/(2 z1 z2)
//   3. k_legendre     spharm tables at cos(theta1), cos(theta2) per (phi, x)
//   4. k_orbital      F_f(phi, x) per bra cell (q',p'), the orbital parts of
//                     Gtilde (tt_p123.h)
//   5. k_contract     Q[f][cell] = sum_k F[f][k] W[cell][k]
//   6. k_row_count / k_row_fill   CSR rows (alpha', q', p'), columns ascending,
//                     P = sum_t c_t Q[f_t] / cell norm
//
// All geometric decisions (kmin < kmax tests) use explicitly rounded
// intrinsics on host-computed sin/cos tables, so they are bit-identical to the
// reference's host arithmetic.
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <cmath>

#include "../host/tt_p123.h"
#include "tt_device.h"
#include "tt_kernels.h"

namespace tt {
namespace {

// std::max / std::min semantics: max(a,b) = (a<b)?b:a, min(a,b) = (b<a)?b:a
__device__ __forceinline__ double smax(double a, double b) { return (a < b) ? b : a; }
__device__ __forceinline__ double smin(double a, double b) { return (b < a) ? b : a; }

// pi1_tilde / pi2_tilde (auxiliary.cpp:453-462), never contracted into FMA
__device__ __forceinline__ double pi1_tilde(double p, double q, double x) {
  double t1 = __dmul_rn(__dmul_rn(0.25, p), p);
  double t2 = __dmul_rn(__dmul_rn(9.0 / 16.0, q), q);
  double t3 = __dmul_rn(__dmul_rn(__dmul_rn(0.75, p), q), x);
  return __dsqrt_rn(__dadd_rn(__dadd_rn(t1, t2), t3));
}
__device__ __forceinline__ double pi2_tilde(double p, double q, double x) {
  double t1 = __dmul_rn(p, p);
  double t2 = __dmul_rn(__dmul_rn(0.25, q), q);
  double t3 = __dmul_rn(__dmul_rn(p, q), x);
  return __dsqrt_rn(__dsub_rn(__dadd_rn(t1, t2), t3));
}

// One CTA per bra cell (q', p').  Cell (q, p) overlaps it when at some mesh
// point the lower radial bounds of all four bins lie below the upper ones
// (make_permutation_matrix.cpp:188-243).  A thread takes mesh points: the bins'
// bounds qb / z2 and pb / z1 rise with the bin (rounded division is monotone),
// so the bins that reach into (kmin, kmax) are neighbours, found by bisection,
// and only those cells are tested, with the reference's own comparison.  Testing
// every cell at every point divides 4 Nq Np times a point instead of about 20.
// Bound: FP64 divide latency.  N = 24: 7.0 ms -> 0.07 ms.
__global__ void __launch_bounds__(256) k_overlap(const double* __restrict__ pb, const double* __restrict__ qb, int Np,
                                                 int Nq, const double* __restrict__ x, int Nx,
                                                 const uint8_t* __restrict__ phi_ok,
                                                 const double* __restrict__ sinphi,
                                                 const double* __restrict__ cosphi, int Nphi,
                                                 uint8_t* __restrict__ mask) {
  const int nrow = Nq * Np;
  const int row = blockIdx.x;
  uint8_t* m = mask + (size_t)row * nrow;
  for (int i = threadIdx.x; i < nrow; i += blockDim.x) m[i] = 0;
  __syncthreads();
  if (!phi_ok[row]) return;
  const int qp = row / Np, pp = row % Np;
  const double qp_l = qb[qp], qp_u = qb[qp + 1], pp_l = pb[pp], pp_u = pb[pp + 1];
  for (int k = threadIdx.x; k < Nphi * Nx; k += blockDim.x) {
    const int ip = k / Nx, ix = k % Nx;
    const double s = sinphi[(size_t)row * Nphi + ip], c = cosphi[(size_t)row * Nphi + ip];
    const double kmin = smax(__ddiv_rn(pp_l, s), __ddiv_rn(qp_l, c));
    const double kmax = smin(__ddiv_rn(pp_u, s), __ddiv_rn(qp_u, c));
    if (!(kmin < kmax)) continue;
    const double xv = x[ix];
    const double z1 = pi1_tilde(s, c, xv), z2 = pi2_tilde(s, c, xv);
    // the first bin whose upper bound lies above kmin
    auto first_above = [&](const double* __restrict__ edges, int N, double z) {
      int lo = 0, hi = N;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__ddiv_rn(edges[mid + 1], z) > kmin) hi = mid;
        else lo = mid + 1;
      }
      return lo;
    };
    const int q0 = first_above(qb, Nq, z2), p0 = first_above(pb, Np, z1);
    for (int q = q0; q < Nq; q++) {
      const double q_l = __ddiv_rn(qb[q], z2), q_u = __ddiv_rn(qb[q + 1], z2);
      if (!(q_l < kmax)) break;
      for (int p = p0; p < Np; p++) {
        const double p_l = __ddiv_rn(pb[p], z1);
        if (!(p_l < kmax) || !(p_l < q_u)) break;
        const double p_u = __ddiv_rn(pb[p + 1], z1);
        const double hl = smax(p_l, q_l), hu = smin(p_u, q_u);
        if (hl < hu) {
          const double kpmin = smax(kmin, hl), kpmax = smin(kmax, hu);
          if (kpmin < kpmax) m[q * Np + p] = 1;
        }
      }
    }
  }
}

// One block per overlapping cell; threads over the Nphi*Nx mesh (k = iphi*Nx + ix).
__global__ void k_cell_weights(const int32_t* __restrict__ cells, const double* __restrict__ pb,
                               const double* __restrict__ qb, int Np, const double* __restrict__ x,
                               const double* __restrict__ wx, int Nx, const double* __restrict__ sinphi,
                               const double* __restrict__ cosphi, const double* __restrict__ wphi, int Nphi,
                               double* __restrict__ W) {
  const int c = blockIdx.x;
  const int qp = cells[4 * c + 0], pp = cells[4 * c + 1], q = cells[4 * c + 2], p = cells[4 * c + 3];
  const double qp_l = qb[qp], qp_u = qb[qp + 1], pp_l = pb[pp], pp_u = pb[pp + 1];
  const double q_l = qb[q], q_u = qb[q + 1], p_l = pb[p], p_u = pb[p + 1];
  const size_t row = (size_t)qp * Np + pp;
  const int K = Nphi * Nx;
  for (int k = threadIdx.x; k < K; k += blockDim.x) {
    const int ip = k / Nx, ix = k % Nx;
    const double s = sinphi[row * Nphi + ip], co = cosphi[row * Nphi + ip];
    const double xv = x[ix];
    const double z1 = pi1_tilde(s, co, xv), z2 = pi2_tilde(s, co, xv);
    // kmin/kmax over the four bin constraints (auxiliary.cpp:713-717)
    double kmin = __ddiv_rn(pp_l, s);
    kmin = smax(kmin, __ddiv_rn(qp_l, co));
    kmin = smax(kmin, __ddiv_rn(p_l, z1));
    kmin = smax(kmin, __ddiv_rn(q_l, z2));
    double kmax = __ddiv_rn(pp_u, s);
    kmax = smin(kmax, __ddiv_rn(qp_u, co));
    kmax = smin(kmax, __ddiv_rn(p_u, z1));
    kmax = smin(kmax, __ddiv_rn(q_u, z2));
    double w = 0.0;
    if (!(kmin > kmax)) {
      const double a = __dmul_rn(__dmul_rn(__dmul_rn(wx[ix], wphi[row * Nphi + ip]), co), s);
      const double dk = __dsub_rn(__dmul_rn(kmax, kmax), __dmul_rn(kmin, kmin));
      w = __ddiv_rn(__dmul_rn(a, dk), __dmul_rn(__dmul_rn(2.0, z1), z2));
    }
    W[(size_t)c * K + k] = w;
  }
}

// out[i * ld] = i-th entry of the spharm table at x
__device__ void spharm_row(int lmax, double x, double* out, size_t ld) {
  const double s = sqrt((1.0 - x) * (1.0 + x));
  double ymm = 1.0 / sqrt(4.0 * M_PI);
  for (int m = 0; m <= lmax; m++) {
    if (m > 0) ymm = -sqrt((2.0 * m + 1.0) / (2.0 * m)) * s * ymm;
    out[(size_t)(m * (m + 1) / 2 + m) * ld] = ymm;
    if (m + 1 > lmax) continue;
    double ylm1 = ymm;
    double yl = x * sqrt(2.0 * m + 3.0) * ymm;
    out[(size_t)((m + 1) * (m + 2) / 2 + m) * ld] = yl;
    for (int l = m + 2; l <= lmax; l++) {
      const double a = sqrt((4.0 * l * l - 1.0) / ((double)l * l - (double)m * m));
      const double b = sqrt(((double)(l - 1) * (l - 1) - (double)m * m) / (4.0 * (l - 1) * (l - 1) - 1.0));
      const double yn = a * (x * yl - b * ylm1);
      ylm1 = yl;
      yl = yn;
      out[(size_t)(l * (l + 1) / 2 + m) * ld] = yl;
    }
  }
}

// spharm tables of cos(theta1) (lmax = max L12) and cos(theta2) (lmax = max l3)
// for a batch of bra rows, plm[row][i][k]; make_permutation_matrix.cpp:554-592.
__global__ void k_legendre(int row0, int nrows, const double* __restrict__ x, int Nx,
                           const double* __restrict__ sinphi, const double* __restrict__ cosphi, int Nphi,
                           int maxL, int lenL, int maxl, int lenl, double* __restrict__ plm2,
                           double* __restrict__ plm3) {
  const int K = Nphi * Nx;
  const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= (size_t)nrows * K) return;
  const int b = (int)(tid / K), k = (int)(tid % K);
  const size_t row = (size_t)(row0 + b);
  const int ip = k / Nx, ix = k % Nx;
  const double p = sinphi[row * Nphi + ip], q = cosphi[row * Nphi + ip], xv = x[ix];
  const double pi1 = pi1_tilde(p, q, xv), pi2 = pi2_tilde(p, q, xv);
  double ct1 = -(0.5 * p + 0.75 * q * xv) / pi1;
  double ct2 = (p - 0.5 * q * xv) / pi2;
  ct1 = ct1 > 1 ? 1 : (ct1 < -1 ? -1 : ct1);
  ct2 = ct2 > 1 ? 1 : (ct2 < -1 ? -1 : ct2);
  spharm_row(maxL, ct1, plm2 + (size_t)b * lenL * K + k, K);
  spharm_row(maxl, ct2, plm3 + (size_t)b * lenl * K + k, K);
}

// F[b][f][k] of a batch of bra rows (tt_p123.h): CTA = 32 mesh points (the
// lanes) of one row.  Per phase the warps share out its B, kept in shared
// memory, then its F.  Every table read is a broadcast (the term lists) or 32
// neighbouring doubles, and each B is made once for all alpha pairs; evaluating
// every pair's own term list (gathers from the spharm tables) took 624 ms of the
// 63-wave channel at N = 16 and 70 ms of the 31-wave one at N = 24, this takes
// 2.0 and 0.9 ms.  Bound: latency of the term lists and table reads (58% of the issue
// slots busy, F stored at 1.1 TB/s at n = 9,072).
constexpr int ORB_K = 32, ORB_THREADS = 256;
constexpr size_t kOrbSmem = 220 * 1024;
// STAGED: the spharm columns in shared memory (up to l = 25 or so); else read
// where they are.
template <bool STAGED>
__global__ void __launch_bounds__(ORB_THREADS) k_orbital(int K, int Nx, int n_phases,
                                                         const int32_t* __restrict__ phase_b,
                                                         const int32_t* __restrict__ phase_f,
                                                         const int32_t* __restrict__ b_off,
                                                         const BTerm* __restrict__ b_terms,
                                                         const int32_t* __restrict__ f_off,
                                                         const FTerm* __restrict__ f_terms, int n_f,
                                                         const double* __restrict__ plm1, int lenl,
                                                         const double* __restrict__ plm2, int lenL,
                                                         const double* __restrict__ plm3, double* __restrict__ F) {
  extern __shared__ double orb_sm[];
  double* sB = orb_sm + (STAGED ? (lenL + lenl) * ORB_K : 0);  // [max_phase_b][32]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int NW = ORB_THREADS / 32;
  const int k = blockIdx.x * ORB_K + lane, kc = min(k, K - 1);
  const size_t b = blockIdx.y;
  const double* s2 = plm2 + b * lenL * K + kc;
  const double* s3 = plm3 + b * lenl * K + kc;
  const int ld = STAGED ? ORB_K : K;
  if (STAGED) {
    for (int i = warp; i < lenL; i += NW) orb_sm[i * ORB_K + lane] = s2[(size_t)i * K];
    for (int i = warp; i < lenl; i += NW) orb_sm[(lenL + i) * ORB_K + lane] = s3[(size_t)i * K];
    s2 = orb_sm + lane;
    s3 = orb_sm + lenL * ORB_K + lane;
  }
  const double* P1 = plm1 + kc % Nx;
  for (int ph = 0; ph < n_phases; ph++) {
    const int b0 = phase_b[ph], b1 = phase_b[ph + 1];
    __syncthreads();
    for (int y = b0 + warp; y < b1; y += NW) {
      double v = 0.0;
      for (int t = b_off[y]; t < b_off[y + 1]; t++) {
        const BTerm g = b_terms[t];
        v += g.c * s2[(size_t)g.i2 * ld] * s3[(size_t)g.i3 * ld];
      }
      sB[(y - b0) * ORB_K + lane] = v;
    }
    __syncthreads();
    for (int f = phase_f[ph] + warp; f < phase_f[ph + 1]; f += NW) {
      double v = 0.0;
      for (int t = f_off[f]; t < f_off[f + 1]; t++) {
        const FTerm g = f_terms[t];
        v += g.c * P1[(size_t)g.i1 * Nx] * sB[g.y * ORB_K + lane];
      }
      if (k < K) F[(b * n_f + f) * K + k] = v;
    }
  }
}

// Q[f][c] = sum_k F[row][f][k] W[c][k] for the cells of one bra row, on the FP64
// tensor cores (mma m8n8k4): CTA = 64 f of one row and up to 64 cells at a time,
// K staged 32 deep in two cp.async buffers; warp w owns the 8 f of tile w and
// all cell tiles, so a row's work follows its number of cells (10 .. 60) in
// steps of 8.  Row stride 36 doubles: a fragment's 8 x 4 elements fall in
// different banks.  Contracting the F instead of every alpha pair, and DMMA
// instead of FMA tiles: 31 waves at N = 24 16.0 ms -> 0.71 ms, 63 waves at N = 16
// 23.9 ms -> below 0.9 ms.  Q of row r starts at Q + n_f row_cell_off[r], [n_f][cells].
constexpr int CT_F = 64, CT_C = 64, CT_K = 32, CT_LD = CT_K + 4;
template <int BYTES>
__device__ __forceinline__ void cp_async_zfill(void* dst, const void* src, bool in) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  const int n = in ? BYTES : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(d), "l"(src), "n"(BYTES), "r"(n) : "memory");
}
// VEC doubles per copy: 2 where the mesh rows are 16-byte aligned (even K)
template <int VEC>
__global__ void __launch_bounds__(256) k_contract(int row0, const int32_t* __restrict__ row_cell_off, int n_f, int K,
                                                  const double* __restrict__ W, const double* __restrict__ F,
                                                  double* __restrict__ Q) {
  extern __shared__ __align__(16) double ct_sm[];  // [2][CT_F + CT_C][CT_LD]
  const int row = row0 + blockIdx.y;
  const int c_lo = row_cell_off[row], nc = row_cell_off[row + 1] - c_lo;
  const int f0 = blockIdx.x * CT_F;
  const double* Fb = F + (size_t)blockIdx.y * n_f * K;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gid = lane >> 2, tig = lane & 3;
  const int chunks = (K + CT_K - 1) / CT_K;
  for (int cb = 0; cb < nc; cb += CT_C) {
    const int ct = min(CT_C, nc - cb), nt = (ct + 7) >> 3;
    auto stage = [&](int ch) {
      double* sF = ct_sm + (ch & 1) * (CT_F + CT_C) * CT_LD;
      const int k0 = ch * CT_K;
      constexpr int PR = CT_K / VEC;  // copies per row
      for (int i = threadIdx.x; i < (CT_F + nt * 8) * PR; i += 256) {
        const int r = i / PR, kk = (i % PR) * VEC, k = k0 + kk;
        const bool isF = r < CT_F;
        const bool in = k < K && (isF ? f0 + r < n_f : r - CT_F < ct);
        const double* src = isF ? Fb + (size_t)(f0 + r) * K + k : W + (size_t)(c_lo + cb + r - CT_F) * K + k;
        cp_async_zfill<VEC * 8>(sF + r * CT_LD + kk, in ? src : F, in);
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    double acc[CT_C / 8][2];
#pragma unroll
    for (int j = 0; j < CT_C / 8; j++) acc[j][0] = acc[j][1] = 0.0;
    stage(0);
    for (int ch = 0; ch < chunks; ch++) {
      if (ch + 1 < chunks) {
        stage(ch + 1);
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
      } else {
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
      }
      __syncthreads();
      const double* sF = ct_sm + (ch & 1) * (CT_F + CT_C) * CT_LD + (warp * 8 + gid) * CT_LD + tig;
      const double* sW = ct_sm + (ch & 1) * (CT_F + CT_C) * CT_LD + (CT_F + gid) * CT_LD + tig;
#pragma unroll
      for (int kk = 0; kk < CT_K; kk += 4) {
        const double a = sF[kk];
#pragma unroll
        for (int j = 0; j < CT_C / 8; j++) {
          if (j >= nt) break;
          const double w = sW[j * 8 * CT_LD + kk];
          asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                       : "+d"(acc[j][0]), "+d"(acc[j][1])
                       : "d"(a), "d"(w));
        }
      }
      __syncthreads();
    }
    const int f = f0 + warp * 8 + gid;
    if (f < n_f) {
      double* Qf = Q + (size_t)c_lo * n_f + (size_t)f * nc + cb;
#pragma unroll
      for (int j = 0; j < CT_C / 8; j++) {
        const int c = j * 8 + 2 * tig;
        if (c < ct) Qf[c] = acc[j][0];
        if (c + 1 < ct) Qf[c + 1] = acc[j][1];
      }
    }
  }
}

// P (before the cell norm) of pair pr and the i-th of a row's nc cells, Qr the row's Q
__device__ __forceinline__ double pair_value(const int32_t* __restrict__ pair_off, const int32_t* __restrict__ pair_f,
                                             const double* __restrict__ pair_c, int pr,
                                             const double* __restrict__ Qr, int nc, int i) {
  double v = 0.0;
  for (int t = pair_off[pr]; t < pair_off[pr + 1]; t++) v = __fma_rn(pair_c[t], Qr[(size_t)pair_f[t] * nc + i], v);
  return v;
}

// One warp per CSR row (alpha', q', p'): entries (alpha, q, p) over the active
// pairs of alpha' (ascending alpha) x the cells of the bra row (ascending q,p).
__global__ void k_row_count(int Na, int Nq, int Np, const int32_t* __restrict__ ap_pair_lo,
                            const int32_t* __restrict__ row_cell_off, const int32_t* __restrict__ pair_off,
                            const int32_t* __restrict__ pair_f, const double* __restrict__ pair_c, int n_f,
                            const double* __restrict__ Q, int64_t* __restrict__ counts) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) / 32, lane = threadIdx.x % 32;
  const int nrows = Na * Nq * Np;
  if (warp >= nrows) return;
  const int ap = warp / (Nq * Np), brow = warp % (Nq * Np);
  const int pr0 = ap_pair_lo[ap], pr1 = ap_pair_lo[ap + 1];
  const int c0 = row_cell_off[brow], c1 = row_cell_off[brow + 1];
  const int nc = c1 - c0;
  const double* Qr = Q + (size_t)c0 * n_f;
  int64_t cnt = 0;
  for (int i = lane; i < (pr1 - pr0) * nc; i += 32)
    if (pair_value(pair_off, pair_f, pair_c, pr0 + i / nc, Qr, nc, i % nc) != 0.0) cnt++;
  for (int o = 16; o > 0; o >>= 1) cnt += __shfl_down_sync(0xffffffffu, cnt, o);
  if (lane == 0) counts[warp] = cnt;
}

__global__ void k_row_fill(int Na, int Nq, int Np, const int32_t* __restrict__ ap_pair_lo,
                           const int32_t* __restrict__ pair_a, const int32_t* __restrict__ row_cell_off,
                           const int32_t* __restrict__ cells, const double* __restrict__ cell_norm,
                           const int32_t* __restrict__ pair_off, const int32_t* __restrict__ pair_f,
                           const double* __restrict__ pair_c, int n_f, const double* __restrict__ Q,
                           const int64_t* __restrict__ rowptr, int32_t* __restrict__ col, double* __restrict__ val) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) / 32, lane = threadIdx.x % 32;
  const int nrows = Na * Nq * Np;
  if (warp >= nrows) return;
  const int ap = warp / (Nq * Np), brow = warp % (Nq * Np);
  const int pr0 = ap_pair_lo[ap], pr1 = ap_pair_lo[ap + 1];
  const int c0 = row_cell_off[brow], c1 = row_cell_off[brow + 1];
  const int nc = c1 - c0;
  int64_t pos = rowptr[warp];
  const int total = (pr1 - pr0) * nc;
  const double* Qr = Q + (size_t)c0 * n_f;
  for (int base = 0; base < total; base += 32) {
    const int i = base + lane;
    double v = 0.0;
    int pr = 0, c = 0;
    if (i < total) {
      pr = pr0 + i / nc;
      c = c0 + i % nc;
      v = pair_value(pair_off, pair_f, pair_c, pr, Qr, nc, i % nc);
    }
    const bool nz = (i < total) && (v != 0.0);
    const unsigned bal = __ballot_sync(0xffffffffu, nz);
    if (nz) {
      const int off = __popc(bal & ((1u << lane) - 1u));
      const int a = pair_a[pr];
      const int q = cells[4 * c + 2], p = cells[4 * c + 3];
      col[pos + off] = a * Nq * Np + q * Np + p;
      val[pos + off] = v / cell_norm[c];
    }
    pos += __popc(bal);
  }
}

}  // namespace

int p123_build_device(const P123Tables& t, DeviceCSR& out, cudaStream_t st, P123Stats* stats) {
  const int Np = t.Np, Nq = t.Nq, Na = t.Nalpha, Nphi = t.Nphi, Nx = t.Nx;
  const int K = Nphi * Nx;
  const size_t nrow = (size_t)Nq * Np;
  const int n = Na * Nq * Np;
  if (!t.production_run) {
    set_error("production_run=false is not supported by the device P123 builder");
    return TT_ERR_UNSUPPORTED;
  }
  DevBuf<double> d_pb, d_qb, d_x, d_wx, d_sin, d_cos, d_wphi, d_plm1;
  DevBuf<uint8_t> d_phi_ok, d_mask;
  TT_TRY(d_pb.upload(t.p_WP, st));
  TT_TRY(d_qb.upload(t.q_WP, st));
  TT_TRY(d_x.upload(t.x, st));
  TT_TRY(d_wx.upload(t.wx, st));
  TT_TRY(d_sin.upload(t.sinphi, st));
  TT_TRY(d_cos.upload(t.cosphi, st));
  TT_TRY(d_wphi.upload(t.wphi, st));
  TT_TRY(d_plm1.upload(t.plm1, st));
  std::vector<uint8_t> phi_ok(nrow);
  for (int qp = 0; qp < Nq; qp++)
    for (int pp = 0; pp < Np; pp++) {
      const double lo = std::atan(t.p_WP[pp] / t.q_WP[qp + 1]);
      const double hi = std::atan(t.p_WP[pp + 1] / t.q_WP[qp]);
      phi_ok[(size_t)qp * Np + pp] = lo < hi ? 1 : 0;
    }
  TT_TRY(d_phi_ok.upload(phi_ok, st));
  const size_t ncell_all = nrow * nrow;
  TT_TRY(d_mask.alloc(ncell_all));
  k_overlap<<<(unsigned)nrow, 256, 0, st>>>(d_pb.ptr, d_qb.ptr, Np, Nq, d_x.ptr, Nx, d_phi_ok.ptr, d_sin.ptr,
                                            d_cos.ptr, Nphi, d_mask.ptr);
  count_launch();
  TT_CUDA_TRY(cudaGetLastError());
  std::vector<uint8_t> mask(ncell_all);
  TT_CUDA_TRY(cudaMemcpyAsync(mask.data(), d_mask.ptr, ncell_all, cudaMemcpyDeviceToHost, st));
  TT_CUDA_TRY(cudaStreamSynchronize(st));
  // cell list per bra row, (q,p) ascending; WP normalisation per cell
  std::vector<int32_t> cells, row_cell_off(nrow + 1, 0);
  std::vector<double> cell_norm;
  for (size_t r = 0; r < nrow; r++) {
    const int qp = (int)(r / Np), pp = (int)(r % Np);
    for (int q = 0; q < Nq; q++)
      for (int p = 0; p < Np; p++) {
        if (!mask[r * nrow + (size_t)q * Np + p]) continue;
        cells.push_back(qp);
        cells.push_back(pp);
        cells.push_back(q);
        cells.push_back(p);
        const double nw = std::sqrt(t.q_WP[q + 1] - t.q_WP[q]) * std::sqrt(t.p_WP[p + 1] - t.p_WP[p]) *
                          std::sqrt(t.q_WP[qp + 1] - t.q_WP[qp]) * std::sqrt(t.p_WP[pp + 1] - t.p_WP[pp]);
        cell_norm.push_back(nw);
      }
    row_cell_off[r + 1] = (int32_t)(cells.size() / 4);
  }
  const int ncell = (int)(cells.size() / 4);
  const int npairs = (int)t.pair_ap.size();
  if (stats) {
    stats->n_cells = ncell;
    stats->n_pairs = npairs;
  }
  out.n = n;
  TT_TRY(out.rowptr.alloc((size_t)n + 1));
  if (ncell == 0 || npairs == 0) {
    TT_CUDA_TRY(cudaMemsetAsync(out.rowptr.ptr, 0, sizeof(int64_t) * (n + 1), st));
    out.nnz = 0;
    return TT_OK;
  }
  const int n_f = t.n_f, n_phases = (int)t.phase_b.size() - 1;
  DevBuf<int32_t> d_cells, d_rco, d_pair_off, d_pair_f, d_pair_a, d_ap_lo, d_phase_b, d_phase_f, d_b_off, d_f_off;
  DevBuf<double> d_cnorm, d_W, d_Q, d_pair_c;
  DevBuf<BTerm> d_b_terms;
  DevBuf<FTerm> d_f_terms;
  TT_TRY(d_cells.upload(cells, st));
  TT_TRY(d_rco.upload(row_cell_off, st));
  TT_TRY(d_cnorm.upload(cell_norm, st));
  TT_TRY(d_pair_off.upload(t.pair_off, st));
  TT_TRY(d_pair_f.upload(t.pair_f, st));
  TT_TRY(d_pair_c.upload(t.pair_c, st));
  TT_TRY(d_pair_a.upload(t.pair_a, st));
  TT_TRY(d_phase_b.upload(t.phase_b, st));
  TT_TRY(d_phase_f.upload(t.phase_f, st));
  TT_TRY(d_b_off.upload(t.b_off, st));
  TT_TRY(d_f_off.upload(t.f_off, st));
  TT_TRY(d_b_terms.upload(t.b_terms, st));
  TT_TRY(d_f_terms.upload(t.f_terms, st));
  std::vector<int32_t> ap_lo(Na + 1, 0);
  {
    int pr = 0;
    for (int ap = 0; ap < Na; ap++) {
      ap_lo[ap] = pr;
      while (pr < npairs && t.pair_ap[pr] == ap) pr++;
    }
    ap_lo[Na] = npairs;
  }
  TT_TRY(d_ap_lo.upload(ap_lo, st));
  TT_TRY(d_W.alloc((size_t)ncell * K));
  k_cell_weights<<<ncell, 256, 0, st>>>(d_cells.ptr, d_pb.ptr, d_qb.ptr, Np, d_x.ptr, d_wx.ptr, Nx, d_sin.ptr,
                                        d_cos.ptr, d_wphi.ptr, Nphi, d_W.ptr);
  count_launch();
  TT_CUDA_TRY(cudaGetLastError());
  TT_TRY(d_Q.alloc((size_t)ncell * n_f));
  // batches of bra rows so that F stays within ~4 GB
  const size_t f_row_bytes = (size_t)n_f * K * sizeof(double);
  int batch = (int)std::max<size_t>(1, std::min<size_t>(nrow, ((size_t)4 << 30) / std::max<size_t>(1, f_row_bytes)));
  batch = std::min(batch, 65535);
  DevBuf<double> d_F, d_plm2, d_plm3;
  TT_TRY(d_F.alloc((size_t)batch * n_f * K));
  TT_TRY(d_plm2.alloc((size_t)batch * K * t.lenL));
  TT_TRY(d_plm3.alloc((size_t)batch * K * t.lenl));
  const size_t orb_b = sizeof(double) * ORB_K * t.max_phase_b;
  const size_t orb_all = orb_b + sizeof(double) * ORB_K * ((size_t)t.lenL + t.lenl);
  const bool orb_staged = orb_all <= kOrbSmem;
  TT_TRY(smem_limit_once((const void*)k_orbital<true>, (int)std::min(orb_all, kOrbSmem)));
  TT_TRY(smem_limit_once((const void*)k_orbital<false>, (int)orb_b));
  const size_t ct_smem = sizeof(double) * 2 * (CT_F + CT_C) * CT_LD;
  TT_TRY(smem_limit_once((const void*)k_contract<1>, (int)ct_smem));
  TT_TRY(smem_limit_once((const void*)k_contract<2>, (int)ct_smem));
  for (size_t r0 = 0; r0 < nrow; r0 += batch) {
    const int nb = (int)std::min<size_t>(batch, nrow - r0);
    if (row_cell_off[r0 + nb] == row_cell_off[r0]) continue;  // no overlapping cells in this batch
    k_legendre<<<ceil_div((size_t)nb * K, 128), 128, 0, st>>>((int)r0, nb, d_x.ptr, Nx, d_sin.ptr, d_cos.ptr, Nphi,
                                                             t.max_L12, t.lenL, t.max_l3, t.lenl, d_plm2.ptr,
                                                             d_plm3.ptr);
    count_launch();
    TT_CUDA_TRY(cudaGetLastError());
    const dim3 go(ceil_div(K, ORB_K), nb);
    if (orb_staged)
      k_orbital<true><<<go, ORB_THREADS, orb_all, st>>>(K, Nx, n_phases, d_phase_b.ptr, d_phase_f.ptr, d_b_off.ptr,
                                                        d_b_terms.ptr, d_f_off.ptr, d_f_terms.ptr, n_f, d_plm1.ptr,
                                                        t.lenl, d_plm2.ptr, t.lenL, d_plm3.ptr, d_F.ptr);
    else
      k_orbital<false><<<go, ORB_THREADS, orb_b, st>>>(K, Nx, n_phases, d_phase_b.ptr, d_phase_f.ptr, d_b_off.ptr,
                                                       d_b_terms.ptr, d_f_off.ptr, d_f_terms.ptr, n_f, d_plm1.ptr,
                                                       t.lenl, d_plm2.ptr, t.lenL, d_plm3.ptr, d_F.ptr);
    count_launch();
    TT_CUDA_TRY(cudaGetLastError());
    const dim3 gc(ceil_div(n_f, CT_F), nb);
    if (K % 2 == 0)
      k_contract<2><<<gc, 256, ct_smem, st>>>((int)r0, d_rco.ptr, n_f, K, d_W.ptr, d_F.ptr, d_Q.ptr);
    else
      k_contract<1><<<gc, 256, ct_smem, st>>>((int)r0, d_rco.ptr, n_f, K, d_W.ptr, d_F.ptr, d_Q.ptr);
    count_launch();
    TT_CUDA_TRY(cudaGetLastError());
  }
  DevBuf<int64_t> d_counts;
  TT_TRY(d_counts.alloc((size_t)n + 1));
  TT_CUDA_TRY(cudaMemsetAsync(d_counts.ptr + n, 0, sizeof(int64_t), st));
  k_row_count<<<ceil_div((size_t)n * 32, 256), 256, 0, st>>>(Na, Nq, Np, d_ap_lo.ptr, d_rco.ptr, d_pair_off.ptr,
                                                           d_pair_f.ptr, d_pair_c.ptr, n_f, d_Q.ptr, d_counts.ptr);
  count_launch();
  TT_CUDA_TRY(cudaGetLastError());
  size_t tmp_bytes = 0;
  TT_CUDA_TRY(cub::DeviceScan::ExclusiveSum(nullptr, tmp_bytes, d_counts.ptr, out.rowptr.ptr, n + 1, st));
  DevBuf<uint8_t> d_tmp;
  TT_TRY(d_tmp.alloc(tmp_bytes));
  TT_CUDA_TRY(cub::DeviceScan::ExclusiveSum(d_tmp.ptr, tmp_bytes, d_counts.ptr, out.rowptr.ptr, n + 1, st));
  int64_t nnz = 0;
  TT_CUDA_TRY(cudaMemcpyAsync(&nnz, out.rowptr.ptr + n, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  TT_CUDA_TRY(cudaStreamSynchronize(st));
  out.nnz = nnz;
  TT_TRY(out.col.alloc((size_t)std::max<int64_t>(nnz, 1)));
  TT_TRY(out.val.alloc((size_t)std::max<int64_t>(nnz, 1)));
  k_row_fill<<<ceil_div((size_t)n * 32, 256), 256, 0, st>>>(Na, Nq, Np, d_ap_lo.ptr, d_pair_a.ptr, d_rco.ptr,
                                                          d_cells.ptr, d_cnorm.ptr, d_pair_off.ptr, d_pair_f.ptr,
                                                          d_pair_c.ptr, n_f, d_Q.ptr, out.rowptr.ptr, out.col.ptr,
                                                          out.val.ptr);
  count_launch();
  TT_CUDA_TRY(cudaGetLastError());
  TT_CUDA_TRY(cudaStreamSynchronize(st));
  return TT_OK;
}

}  // namespace tt
