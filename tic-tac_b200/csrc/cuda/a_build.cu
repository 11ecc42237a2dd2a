// The dense kernel matrix of one 3N channel,
//   A = C^T (2 P123) (V C)                      (solve_faddeev.cpp:4-181),
// in one pass over P123 that writes each element of A once.
//
// Index of a state: (alpha, q, p) -> (alpha Nq + q) Np + p.  C and V C are
// block diagonal over the 2N blocks: alpha couples only with the partners of
// its coupling list (itself and at most one other partial wave of the same 2N
// block), and
//   A[(ar,q,pr), (ac,q',pc)] = sum_{ai in cpl(ar)} sum_pi Ct(ar,ai)[pr][pi] T_ai[(q,pi), (q',pc)],
//   T_ai[(q,pi), (q',pc)]     = 2 sum_{aj in cpl(ac)} sum_pj P[(ai,q,pi), (aj,q',pj)] VC[(aj,pj), (ac,pc)].
// The reference forms the product column by column (calculate_PVC_col,
// calculate_CPVC_col); here one CTA owns a row block (ar, q) and a column
// partial wave ac, walks the P123 rows (ai, q, pi) of the coupled ai once over
// the q' range of the coupled aj (sorted columns; each row's start of every
// alpha range is tabulated once per channel), accumulates T for a chunk of q'
// in shared memory, contracts it with Ct and streams the chunk of A out.
// No n x n intermediate: HBM traffic is the A written once plus P123 read
// (twice per coupled pair).
#include <algorithm>
#include <climits>

#include "tt_kernels.h"

namespace tt {
namespace {

constexpr int AB_THREADS = 256;
constexpr int AB_CAP = 32;  // staged nonzeros of a range: one per lane

__device__ __forceinline__ int64_t first_col_at_least(const int32_t* __restrict__ col, int64_t lo, int64_t hi,
                                                      int32_t key) {
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (col[mid] < key) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// aoff[r * (Na + 1) + a] = first nonzero of row r with column >= a Nq Np,
// relative to rowptr[r], for a = 0 .. Na
__global__ void k_alpha_offsets(int n, int Na, int NqNp, const int64_t* __restrict__ rowptr,
                                const int32_t* __restrict__ col, int32_t* __restrict__ aoff) {
  const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (tid >= (size_t)n * (Na + 1)) return;
  const int r = (int)(tid / (Na + 1)), a = (int)(tid % (Na + 1));
  const int64_t lo = rowptr[r], hi = rowptr[r + 1];
  aoff[tid] = (int32_t)(first_col_at_least(col, lo, hi, a * NqNp) - lo);
}

// Shared memory of k_abuild: T [RTP][LD], and per (T row, coupled aj) range a
// window of its nonzeros, for T of `ncr` partial waves.  QW values of q' a chunk,
// as many as leave room for two CTAs an SM: a row block of one partial wave takes
// longer chunks.  LD = 4 or 12 mod 16 doubles: an 8 x 4 fragment of T falls in
// different banks.
struct AbLayout {
  int QW, CW, LD, RTP, RT2;
  size_t val, base, end, pos, col, bytes;
  AbLayout(int Np, int Nq, int ncr) {
    constexpr size_t kTwoPerSM = 112 * 1024;
    RTP = (ncr * Np + 3) / 4 * 4;
    RT2 = 2 * ncr * Np;
    for (QW = Nq; QW >= 1; QW--) {
      CW = QW * Np;
      LD = (CW + 15) / 16 * 16 + 4;
      if (CW % 16 > 0 && CW % 16 <= 4) LD -= 16;
      else if (CW % 16 > 4 && CW % 16 <= 12) LD -= 8;
      val = sizeof(double) * ((size_t)RTP * LD + 8);  // a tile may read past the last row's end
      base = val + sizeof(double) * RT2 * AB_CAP;
      end = base + sizeof(int64_t) * RT2;
      pos = end + sizeof(int64_t) * RT2;
      col = pos + sizeof(int32_t) * RT2;
      bytes = col + sizeof(int32_t) * RT2 * AB_CAP;
      if (bytes <= kTwoPerSM) break;
    }
    QW = QW < 1 ? 1 : QW;
  }
};

// One CTA per (row block R = ar Nq + q, column partial wave ac), chunk by chunk
// of q'.  A warp builds whole T rows: the nonzeros of a range sit one per lane
// (from the staged window, refilled where a range outlasts it), and their VC
// rows, read through L1, are added up in registers while q' stays the same.  Then
// the warps contract the chunk with Ct on the FP64 tensor cores (mma m8n8k4); the
// Ct fragments stay in registers for all chunks.  MT row tiles of 8 (4 for
// Np <= 32, 8 for Np <= 64).  Bound: latency of the T rows and the FP64 tensor
// pipe (28% busy at Np = 30); the two resident CTAs overlap them.  n = 24,300 10.9 -> 6.0 ms,
// n = 42,300 35.5 -> 19.4 ms, n = 16,128 9.1 -> 4.0 ms (64-column chunks, a read-add-write of T per nonzero,
// Ct read from it per chunk before).
template <int MT>
__global__ void __launch_bounds__(AB_THREADS, 2) k_abuild(AbLayout ly1, AbLayout ly2, int Na, int Nq, int Np,
                                                          const int64_t* __restrict__ rowptr,
                                                          const int32_t* __restrict__ col,
                                                          const double* __restrict__ val,
                                                          const int32_t* __restrict__ aoff,
                                                          const int32_t* __restrict__ blk,
                                                          const int32_t* __restrict__ part,
                                                          const int32_t* __restrict__ cpl_off,
                                                          const int32_t* __restrict__ cpl,
                                                          const int64_t* __restrict__ blk_off,
                                                          const int32_t* __restrict__ blk_dim,
                                                          const double* __restrict__ Cm,
                                                          const double* __restrict__ VC, double* __restrict__ A) {
  extern __shared__ __align__(16) unsigned char ab_raw[];
  const int n = Na * Nq * Np, NqNp = Nq * Np;
  const int R = blockIdx.x, ac = blockIdx.y;
  const int ar = R / Nq, q = R % Nq;
  const int cr0 = cpl_off[ar], ncr = cpl_off[ar + 1] - cr0;
  const int cc0 = cpl_off[ac], ncc = cpl_off[ac + 1] - cc0;
  const AbLayout ly = ncr > 1 ? ly2 : ly1;
  double* sT = reinterpret_cast<double*>(ab_raw);                  // [RTP][LD]
  double* sVal = reinterpret_cast<double*>(ab_raw + ly.val);       // [rr 2 + t2][CAP]
  int64_t* sBase = reinterpret_cast<int64_t*>(ab_raw + ly.base);   // first nonzero of the window
  int64_t* sEnd = reinterpret_cast<int64_t*>(ab_raw + ly.end);
  int32_t* sPos = reinterpret_cast<int32_t*>(ab_raw + ly.pos);     // next nonzero in the window
  int32_t* sCol = reinterpret_cast<int32_t*>(ab_raw + ly.col);
  constexpr int NWARP = AB_THREADS / 32, KMAX = MT * 4;            // k steps of 4: 2 Np / 4
  const int QW = ly.QW, LD = ly.LD;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int RT = ncr * Np, KS = (RT + 3) / 4;  // rows of T, k steps
  // the range of every (T row, coupled aj) in its P123 row
  for (int i = tid; i < RT * 2; i += AB_THREADS) {
    const int rr = i >> 1, t2 = i & 1;
    int64_t e0 = 0, e1 = 0;
    if (t2 < ncc) {
      const int t = rr >= Np, ai = cpl[cr0 + t], pi = rr - t * Np, aj = cpl[cc0 + t2];
      const int r = (ai * Nq + q) * Np + pi;
      const int64_t rp = rowptr[r];
      e0 = rp + aoff[(size_t)r * (Na + 1) + aj];
      e1 = rp + aoff[(size_t)r * (Na + 1) + aj + 1];
    }
    sBase[i] = e0;
    sEnd[i] = e1;
    sPos[i] = 0;
  }
  for (int i = RT * LD + tid; i < KS * 4 * LD; i += AB_THREADS) sT[i] = 0.0;  // the last k step's rows past RT
  // Ct(ar, ai)[pr][pi] = C[(part_i, pi), (part_r, pr)] of ar's 2N block: fragment
  // row pr = 8 mt + lane / 4, column k = 4 ks + lane % 4 over (ai, pi)
  const int gid = lane >> 2, tig = lane & 3, mt = warp % MT, prow = mt * 8 + gid;
  double ct[KMAX];
  {
    const int b = blk[ar], dimb = blk_dim[b];
    const double* Cb = Cm + blk_off[b] + part[ar] * Np + prow;
    const int pi0 = part[cpl[cr0]] * Np, pi1 = ncr > 1 ? part[cpl[cr0 + 1]] * Np : 0;
#pragma unroll
    for (int ks = 0; ks < KMAX; ks++) {
      const int k = ks * 4 + tig, t = k >= Np;
      ct[ks] = (k < RT && prow < Np) ? Cb[(size_t)((t ? pi1 : pi0) + k - t * Np) * dimb] : 0.0;
    }
  }
  __syncthreads();
  // the first window of every range
#pragma unroll 4
  for (int p = warp; p < RT * 2; p += NWARP) {
    const int64_t e = sBase[p] + lane;
    const bool in = e < sEnd[p];
    sCol[p * AB_CAP + lane] = in ? col[e] : INT_MAX;
    sVal[p * AB_CAP + lane] = in ? val[e] : 0.0;
  }
  const int bc = blk[ac], dimc = blk_dim[bc];
  const float rNp = 1.0f / (float)Np, hNp = 0.5f / (float)Np;
  const double* VCb = VC + blk_off[bc] + part[ac] * Np;
  int ajs[2];
  const double* VCj[2];  // row pj of VC(aj -> ac): + pj dimc
#pragma unroll
  for (int t2 = 0; t2 < 2; t2++) {
    ajs[t2] = t2 < ncc ? cpl[cc0 + t2] : 0;
    VCj[t2] = VCb + (size_t)(t2 < ncc ? part[ajs[t2]] * Np : 0) * dimc;
  }
  for (int q0 = 0; q0 < Nq; q0 += QW) {
    const int qw = min(QW, Nq - q0), cw = qw * Np;  // columns of this chunk
    __syncthreads();
    // ---- T chunk, one warp per T row
    for (int rr = warp; rr < RT; rr += NWARP) {
      double* Trow = sT + (size_t)rr * LD;
      for (int c = lane; c < cw; c += 32) Trow[c] = 0.0;
      __syncwarp();
#pragma unroll
      for (int t2 = 0; t2 < 2; t2++) {
        if (t2 >= ncc) break;
        const int p = rr * 2 + t2;
        const int32_t cbase = ajs[t2] * NqNp + q0 * Np, lim = cbase + cw;
        int64_t base = sBase[p];
        const int64_t end = sEnd[p];
        int pos = sPos[p];
        int at = 0;  // q' of the sums in acc
        double acc[2] = {0.0, 0.0};
        auto put = [&](int qn) {
          if (lane < Np) Trow[at * Np + lane] += acc[0];
          if (MT > 4 && lane + 32 < Np) Trow[at * Np + lane + 32] += acc[1];
          acc[0] = acc[1] = 0.0;
          at = qn;
        };
        while (base < end) {
          const int32_t cj = sCol[p * AB_CAP + lane];
          const double vj = 2.0 * sVal[p * AB_CAP + lane];
          const int last = pos + __popc(__ballot_sync(0xffffffffu, lane >= pos && cj < lim));
          // rel / Np by a float reciprocal: rel < cw <= 4096, so the product's
          // error (< 2^-11 / Np) stays below the 0.5 / Np margin
          const int rel = cj - cbase, qj = (int)((float)rel * rNp + hNp), pj = rel - qj * Np;
          for (int i = pos; i < last; i += 4) {
            // four VC rows asked for at a time
            double v[4], w[4][2];
            int qi[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
              const int l = min(i + u, last - 1);
              qi[u] = __shfl_sync(0xffffffffu, qj, l);
              const int pu = __shfl_sync(0xffffffffu, pj, l);
              v[u] = __shfl_sync(0xffffffffu, vj, l);
              const double* row = VCj[t2] + (size_t)pu * dimc;
              w[u][0] = lane < Np ? __ldg(row + lane) : 0.0;
              w[u][1] = (MT > 4 && lane + 32 < Np) ? __ldg(row + lane + 32) : 0.0;
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
              if (i + u >= last) break;
              if (qi[u] != at) put(qi[u]);
              acc[0] += v[u] * w[u][0];
              if (MT > 4) acc[1] += v[u] * w[u][1];
            }
          }
          pos = last;
          if (pos < AB_CAP || base + AB_CAP >= end) break;
          // the window is used up: the next one of this range
          base += AB_CAP;
          pos = 0;
          __syncwarp();
          const int64_t e = base + lane;
          sCol[p * AB_CAP + lane] = e < end ? col[e] : INT_MAX;
          sVal[p * AB_CAP + lane] = e < end ? val[e] : 0.0;
          if (lane == 0) sBase[p] = base;
          __syncwarp();
        }
        put(0);
        if (lane == 0) sPos[p] = pos;
        __syncwarp();
      }
    }
    __syncthreads();
    // ---- A chunk: (Np x RT) Ct times (RT x cw) T as 8 x 8 tiles; NWARP / MT warps
    // share a row tile, each with four column tiles at a time
    {
      const int nt = (cw + 7) / 8;
      double* Arow = A + ((size_t)R * Np + prow) * n + (size_t)(ac * Nq + q0) * Np;
      for (int j0 = warp / MT * 4; j0 < nt; j0 += NWARP / MT * 4) {
        double acc[4][2];
#pragma unroll
        for (int j = 0; j < 4; j++) acc[j][0] = acc[j][1] = 0.0;
        const double* Tk = sT + (size_t)tig * LD + gid;
        __syncwarp();  // after the stores' branches: mma.sync.aligned
#pragma unroll
        for (int ks = 0; ks < KMAX; ks++) {
          if (ks >= KS) break;
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const double b = Tk[(size_t)ks * 4 * LD + min(j0 + j, nt - 1) * 8];
            asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                         : "+d"(acc[j][0]), "+d"(acc[j][1])
                         : "d"(ct[ks]), "d"(b));
          }
        }
        if (prow < Np) {
#pragma unroll
          for (int j = 0; j < 4; j++) {
            if (j0 + j >= nt) break;
            const int c = (j0 + j) * 8 + 2 * tig;
            double* p = Arow + c;
            if (c + 1 < cw && ((uintptr_t)p & 15) == 0) {
              __stcs(reinterpret_cast<double2*>(p), make_double2(acc[j][0], acc[j][1]));
            } else {
              if (c < cw) __stcs(p, acc[j][0]);
              if (c + 1 < cw) __stcs(p + 1, acc[j][1]);
            }
          }
        }
      }
    }
  }
}

}  // namespace

int alpha_offsets_device(const DeviceLayout& L, const DeviceCSR& P, int32_t* d_aoff, cudaStream_t st) {
  const size_t total = (size_t)L.n * (L.Nalpha + 1);
  if (total == 0) return TT_OK;
  k_alpha_offsets<<<ceil_div(total, 256), 256, 0, st>>>(L.n, L.Nalpha, L.Nq * L.Np, P.rowptr.ptr, P.col.ptr, d_aoff);
  count_launch();
  TT_CUDA_TRY(cudaGetLastError());
  return TT_OK;
}

int build_A_device(const DeviceLayout& L, const DeviceCSR& P, const int32_t* d_aoff, double* d_A, cudaStream_t st) {
  const int n = L.n;
  if (n == 0) return TT_OK;
  if (L.Np > 64) {
    set_error("Np_WP > 64 is not supported by the A-build kernel");
    return TT_ERR_UNSUPPORTED;
  }
  // dense contraction 2 k Np n^2 and sparse product 2 k Np nnz flops (k = mean
  // coupled partners); A written once, P123 read once per coupled column wave
  const double kcpl = L.Nalpha ? (double)L.cpl.count / L.Nalpha : 0.0;
  ProfScope prof(TT_PROF_A_BUILD, st, 2.0 * kcpl * L.Np * ((double)P.nnz + (double)n * n),
                 12.0 * kcpl * (double)P.nnz + 8.0 * (double)n * n);
  dim3 grid(L.Nalpha * L.Nq, L.Nalpha);
  const AbLayout ly1(L.Np, L.Nq, 1), ly2(L.Np, L.Nq, 2);
  const size_t smem = std::max(ly1.bytes, ly2.bytes);
  TT_TRY(smem_limit_once(L.Np <= 32 ? (const void*)k_abuild<4> : (const void*)k_abuild<8>, (int)smem));
  auto launch = [&](auto kernel) {
    kernel<<<grid, AB_THREADS, smem, st>>>(ly1, ly2, L.Nalpha, L.Nq, L.Np, P.rowptr.ptr, P.col.ptr, P.val.ptr, d_aoff,
                                               L.blk.ptr, L.part.ptr, L.cpl_off.ptr, L.cpl.ptr, L.blk_off.ptr,
                                               L.blk_dim.ptr, L.C.ptr, L.VC.ptr, d_A);
  };
  if (L.Np <= 32) launch(k_abuild<4>);
  else launch(k_abuild<8>);
  count_launch();
  TT_CUDA_TRY(cudaGetLastError());
  return TT_OK;
}

}  // namespace tt
