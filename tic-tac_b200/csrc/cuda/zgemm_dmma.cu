// Complex128 update C[M x N] -= L[M x K] U[K x N] on the FP64 tensor cores
// (mma.sync m8n8k4 f64, the only FP64 matrix instruction of sm_100a), for the
// trailing and panel updates of the FP64 factorisation.
//
// CTA tile 64 x 64 complex, 8 warps of 32 x 16 (4 x 2 m8n8 tiles), two CTAs an SM,
// k tiles of 16 in a ring of cp.async stages.  Elements stay interleaved, 16 bytes each: one
// shared-memory load brings a fragment's re and im, and row strides of 20 (L) and
// 66 (U) elements put the 8 lanes of a load phase into different banks.  Per k4
// step a warp loads 6 fragments and issues 32 DMMAs:
//   Re += Lr Ur + Li (-Ui),   Im += Lr Ui + Li Ur
// Bound: the FP64 tensor pipe (79% busy); 4 warps a scheduler cover the fragments'
// latency, with the second CTA's products under the first's epilogue.  M = N = 8,368, K = 128:
// 3.2 -> 2.42 ms (29.6 TFLOP/s; 64 x 128 tiles on 2 warps a scheduler before, on 4
// warps 2.69, without the prefetch of C 2.48).
#include <algorithm>

#include "tt_kernels.h"
#include "tt_lu_internal.h"

namespace tt {
namespace dmma {

constexpr int BM = 64, BN = 64, BK = 16;
constexpr int AS = BK + 4;  // row stride of the L tile [BM][AS], in elements
constexpr int BS = BN + 2;  // and of the U tile [BK][BS]
constexpr int STAGES = 3, THREADS = 256;
constexpr int STAGE = BM * AS + BK * BS;  // elements
constexpr int SMEM_BYTES = STAGES * STAGE * 16;

__device__ __forceinline__ void mma884(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

__device__ __forceinline__ void cp16(double2* dst, const double2* src, bool in) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(in ? 16 : 0) : "memory");
}

__global__ void __launch_bounds__(THREADS, 2) k_zgemm_dmma(double2* __restrict__ C, int ldc,
                                                           const double2* __restrict__ L, int ldl,
                                                           const double2* __restrict__ U, int ldu, int M, int N,
                                                           int K) {
  extern __shared__ double2 dsm[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int gid = lane >> 2, tig = lane & 3;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int wm0 = (warp >> 2) * 32, wn0 = (warp & 3) * 16;
  const int kt = (K + BK - 1) / BK;
  auto stage = [&](int t) {
    if (t < kt) {
      double2* sA = dsm + (t % STAGES) * STAGE;
      double2* sB = sA + BM * AS;
      const int k0 = t * BK;
#pragma unroll
      for (int e = 0; e < BM * BK / THREADS; e++) {
        const int i = tid + THREADS * e, r = i / BK, c = i % BK;
        const bool in = m0 + r < M && k0 + c < K;
        cp16(sA + r * AS + c, in ? L + (size_t)(m0 + r) * ldl + k0 + c : L, in);
      }
#pragma unroll
      for (int e = 0; e < BK * BN / THREADS; e++) {
        const int i = tid + THREADS * e, r = i / BN, c = i % BN;
        const bool in = k0 + r < K && n0 + c < N;
        cp16(sB + r * BS + c, in ? U + (size_t)(k0 + r) * ldu + n0 + c : U, in);
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  double accr[4][2][2], acci[4][2][2];
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 2; j++) accr[i][j][0] = accr[i][j][1] = acci[i][j][0] = acci[i][j][1] = 0.0;
#pragma unroll
  for (int t = 0; t < STAGES - 1; t++) stage(t);
  // the tile of C into L2 meanwhile, a 128-byte line per access
  for (int i = tid; i < BM * BN / 8; i += THREADS) {
    const int r = m0 + i / (BN / 8), c = n0 + i % (BN / 8) * 8;
    if (r < M && c < N) asm volatile("prefetch.global.L2 [%0];" ::"l"(C + (size_t)r * ldc + c));
  }
  for (int t = 0; t < kt; t++) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
    __syncthreads();  // tile t is there, and tile t - 1 has been read by all
    stage(t + STAGES - 1);
    const double2* sA = dsm + (t % STAGES) * STAGE + (wm0 + gid) * AS + tig;
    const double2* sB = dsm + (t % STAGES) * STAGE + BM * AS + tig * BS + wn0 + gid;
#pragma unroll
    for (int kk = 0; kk < BK; kk += 4) {
      double2 a[4], b[2];
#pragma unroll
      for (int i = 0; i < 4; i++) a[i] = sA[i * 8 * AS + kk];
#pragma unroll
      for (int j = 0; j < 2; j++) b[j] = sB[kk * BS + j * 8];
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const double nbi = -b[j].y;
#pragma unroll
        for (int i = 0; i < 4; i++) {
          mma884(accr[i][j], a[i].x, b[j].x);
          mma884(acci[i][j], a[i].x, b[j].y);
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
          mma884(accr[i][j], a[i].y, nbi);
          mma884(acci[i][j], a[i].y, b[j].x);
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int row = m0 + wm0 + i * 8 + gid;
    if (row >= M) continue;
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        const int col = n0 + wn0 + j * 8 + 2 * tig + e;
        if (col < N) {
          double2* p = &C[(size_t)row * ldc + col];
          const double2 v = *p;
          *p = make_double2(v.x - accr[i][j][e], v.y - acci[i][j][e]);
        }
      }
  }
}

}  // namespace dmma

int zgemm_sub_dmma(double2* C, int ldc, const double2* L, int ldl, const double2* U, int ldu, int M, int N, int K,
                   cudaStream_t st) {
  if (M <= 0 || N <= 0 || K <= 0) return TT_OK;
  TT_TRY(smem_limit_once((const void*)dmma::k_zgemm_dmma, dmma::SMEM_BYTES));
  dim3 grid(ceil_div(N, dmma::BN), ceil_div(M, dmma::BM));
  ProfScope prof(TT_PROF_FP64_UPDATE, st, 8.0 * M * N * K, 32.0 * M * N + 16.0 * ((double)M + N) * K);
  dmma::k_zgemm_dmma<<<grid, dmma::THREADS, dmma::SMEM_BYTES, st>>>(C, ldc, L, ldl, U, ldu, M, N, K);
  count_launch();
  TT_CUDA_TRY(cudaGetLastError());
  return TT_OK;
}

}  // namespace tt
