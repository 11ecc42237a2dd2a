// Host preparation of the per-channel tables the device P123 builder consumes.
// Everything that decides *which* permutation-matrix entries exist (meshes,
// sin/cos of the phi mesh, recoupling coefficients) is computed here in FP64
// with the reference's arithmetic; the device only does +,-,*,/,sqrt,min,max on
// these tables (compiled without FMA contraction), so the overlap decisions are
// bit-identical to the reference's host loops.
#pragma once
#include <cstdint>
#include <vector>

#include "tt_host.h"

namespace tt {

// The geometric function of a pair (alpha', alpha) (auxiliary.cpp:991-1061) depends on
// the partial waves' spins and isospins only through one factor per L_total:
//   Gtilde_{alpha' alpha} = norm(L12) sum_Lt 8 pi^2 Atilde(alpha', alpha, Lt) F_f,  f = (o', o, Lt),
//   F_f(phi, x) = sum_M CG(L12 l3 Lt; 0 M) (-1)^M Y_{l3 M}(x) B_{o Lt M}(phi, x),
//   B_{o Lt M}  = sum_M' CG(L12' l3' Lt; M' M-M') Y_{L12' M'}(theta1) Y_{l3' M-M'}(theta2),
// with the orbital pairs o' = (L12, l3) of alpha' and o = (L12', l3') of alpha.  A
// channel has tens of orbital pairs against up to 63^2 pairs of partial waves, so
// F is what the device tabulates and integrates; the pairs are sums of few F.
// In a channel of one parity the terms of M and -M are equal and M >= 0 is kept.
struct BTerm {  // c Y_{i2}(theta1) Y_{i3}(theta2), signs of negative m in c
  double c;
  int32_t i2, i3;
};
struct FTerm {  // c Y_{i1}(x) B, B the y-th of the phase
  double c;
  int32_t i1, y;
};

struct P123Tables {
  int Np = 0, Nq = 0, Nalpha = 0, Nphi = 0, Nx = 0;
  int two_J_3N = 0, P_3N = 0;
  bool production_run = true;
  std::vector<double> p_WP, q_WP;     // boundaries
  std::vector<double> x, wx;          // [Nx], gauss_legendre
  std::vector<double> phi, wphi;      // [Nq*Np*Nphi], per (q',p') mesh
  std::vector<double> sinphi, cosphi; // host libm values of the phi mesh
  int max_L12 = 0, max_l3 = 0, lenL = 0, lenl = 0;
  std::vector<double> plm1;           // [lenl][Nx] spharm(l3max, x)
  // active (alpha', alpha) pairs: those with at least one term; pair i is the
  // sum of pair_c[t] F[pair_f[t]] for pair_off[i] <= t < pair_off[i+1]
  std::vector<int32_t> pair_ap, pair_a;
  std::vector<int32_t> pair_off, pair_f;
  std::vector<double> pair_c;         // 8 pi^2 Atilde sqrt((2 L12 + 1)/(4 pi))
  // B and F in phases: a phase's F read only its own B (at most max_phase_b)
  int n_f = 0, max_phase_b = 0;
  std::vector<int32_t> phase_b, phase_f;  // [n_phases+1], first B and F of each phase
  std::vector<int32_t> b_off, f_off;      // [n_b+1], [n_f+1] into the terms
  std::vector<BTerm> b_terms;
  std::vector<FTerm> f_terms;
  std::vector<int32_t> L12, l3;       // per alpha, for the device Legendre indexing
};

// Builds all tables for one 3N channel (make_permutation_matrix.cpp:324-611).
bool p123_prepare(const RunParams& rp, const FWPStates& fwp, const PWChannel& ch, P123Tables& t,
                  std::string* err);

// Atilde(alpha, alpha', L_total), auxiliary.cpp:863-884.
double atilde(const PWChannel& ch, int a, int ap, int Ltot, int two_J, int two_T);

}  // namespace tt
