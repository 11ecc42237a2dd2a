"""What a user of this framework has it do: the cases whose time is followed.

Each case is one call, or the few calls that belong together, of the public
Python mirror of the C-ABI (tictac_b200): the three drop-in functions (P123,
resolvent, Faddeev solve) on host arrays, and the run handle, which keeps a
channel's P123 on the GPU and builds and solves the kernel matrix for every new
set of potential constants.  Sizes are those of the tests, of the bench
configurations and of runs between them:

    j<=1, N=8 .. 13      the tests' bases, n = 512 .. 1,900
    j<=2, N=24           the 64-energy scan, n = 10,944 .. 20,160
    j<=3, N=12, 16, 30   the basis of the headline metric, n = 3,888 .. 56,700

    listed()             the cases, smallest and largest of each kind among them
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  what a program holds before the call
    run(state)           one pass; its outputs, whole
    work(case)           bytes and operations that a pass cannot do without
    exact(case, seed)    the outputs in 64 bits, by plain torch

A seed moves the wave-packet grid's scale and, where the potential has them, its
low-energy constants by about a percent (the offsets of the gradient checks).
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tic-tac_b200", "python"))
import tictac_b200 as tt  # noqa: E402

M_P, M_N = 938.272, 939.565  # MeV
LECS = (-0.00112927, -0.0008734)  # C_1S0, C_3S1 of the LO potential
DENSITY = 0.025  # nonzeros of P123 over n^2, about, from N = 12 to 30
EXACT_N = 25_000  # largest order solved densely in complex128 in exact()


def listed():
    return [
        # the drop-in resolvent of one energy at the smallest configuration: launches and host work
        dict(name="resolvent_mt_n512", kind="resolvent", pot="mt", j=1, J=1, P=1, Np=16, Nq=16),
        # the resolvents of a whole scan for the largest channel, into the caller's device memory
        dict(name="resolvent_scan_n56700", kind="resolvent_dev", pot="lo", j=3, J=7, P=1, Np=30, Nq=30, nE=14),
        # P123 of a small channel, returned as the reference's COO arrays
        dict(name="p123_j1_n960", kind="p123", pot="lo", j=1, J=3, P=1, Np=8, Nq=8),
        # P123 of a channel of the scan
        dict(name="p123_j2_n17856", kind="p123", pot="lo", j=2, J=3, P=-1, Np=24, Nq=24),
        # a channel of the headline basis from nothing: P123, A, resolvents and the refined solve
        dict(name="channel_j3_n16128", kind="channel", pot="lo", j=3, J=7, P=1, Np=16, Nq=16, labs="10"),
        # solves for a new parameter set, P123 resident: A, resolvents, LU, refinement
        dict(name="solve_mt_n512", kind="solve", pot="mt", j=1, J=1, P=1, Np=16, Nq=16, labs="13"),
        # odd order, six energies (a group of four and one of two)
        dict(name="solve_odd_n1859", kind="solve", pot="lo", j=1, J=1, P=1, Np=13, Nq=13, labs="5,30,100"),
        # four energies of the scan factored together
        dict(name="scan4_j2_n20160", kind="scan", pot="lo", j=2, J=5, P=1, Np=24, Nq=24, labs="5,30,100", nE=4),
        # a channel of the headline configuration
        dict(name="solve_j3_n42300", kind="solve", pot="lo", j=3, J=3, P=1, Np=30, Nq=30, labs="10"),
        # the drop-in solve on host arrays, complex128 throughout
        dict(name="dropin_fp64_n8496", kind="dropin", pot="lo", j=3, J=5, P=1, Np=12, Nq=12, labs="10", fp64=True),
        # the reference's production solver with its breakup amplitudes
        dict(name="pade_breakup_n24300", kind="pade", pot="lo", j=3, J=1, P=1, Np=30, Nq=30, labs="10"),
        # U and its derivatives in the potential's constants
        dict(name="adjoint_j2_n10944", kind="adjoint", pot="lo", j=2, J=1, P=1, Np=24, Nq=24, labs="10"),
    ]


# partial waves of the channels (two-body j <= j, total 2J), either parity
NALPHA = {(1, 1): 11, (1, 3): 15, (2, 1): 19, (2, 3): 31, (2, 5): 35, (3, 1): 27, (3, 3): 47, (3, 5): 59, (3, 7): 63}
# largest order drawn of each kind
MOST_N = {"resolvent": 56_700, "resolvent_dev": 56_700, "p123": 17_856, "channel": 16_128, "solve": 30_000,
          "scan": 20_160, "dropin": 8_496, "pade": 24_300, "adjoint": 15_000}


def draw(rng):
    kind = rng.choice(["resolvent", "resolvent_dev", "p123", "p123", "channel", "solve", "solve", "solve", "scan",
                       "dropin", "pade", "adjoint"])
    while True:
        j, J = rng.choice(sorted(NALPHA))
        Np, Nq = (int(round(math.exp(rng.uniform(math.log(8), math.log(30.5))))) for _ in range(2))
        n = NALPHA[j, J] * Np * Nq
        if n <= MOST_N[kind]:
            break
    c = dict(kind=kind, pot="lo", j=j, J=J, P=rng.choice([1, -1]), Np=Np, Nq=Nq)
    if kind == "resolvent_dev":
        c["nE"] = rng.randint(1, 14)
    elif kind == "scan":
        c.update(labs="5,30,100", nE=rng.randint(2, 4))
    elif kind in ("channel", "solve", "dropin", "pade", "adjoint"):
        # away from the inelastic edges of the smallest grids
        c["labs"] = "%.1f" % rng.uniform(5, 60) if rng.random() < 0.7 else "5,30,100"
        if kind == "adjoint" or n > 16_000:
            c["labs"] = "%.1f" % rng.uniform(5, 60)
    if kind == "dropin":
        c["fp64"] = rng.random() < 0.5
    return c


# ---------------------------------------------------------------------------


def options(case, seed):
    """Run options of a case: the grid's scale and the constants moved by the seed."""
    rng = np.random.RandomState(seed % (1 << 31))
    scale, lecs = 200.0 * (1 + 0.01 * rng.uniform(-1, 1)), 0.01 * rng.uniform(-1, 1, 2) * LECS
    o = dict(J_2N_max=case["j"], two_J_3N_max=case["J"], Np_WP=case["Np"], Nq_WP=case["Nq"],
             chebyshev_s=repr(float(scale)), lab_energies=case.get("labs", "10"))
    if case["pot"] == "mt":
        return dict(o, potential_model="malfliet_tjon", swave_only="true", isospin_breaking_1S0="false",
                    tensor_force="false")
    return dict(o, potential_model="LO_internal", lec_offsets=",".join(repr(float(x)) for x in lecs))


def flags(case):
    lo = int(case["pot"] == "lo")
    return dict(tensor_force=lo, isospin_breaking_1S0=lo)


def channel_of(run, case):
    for c in range(run.num_channels):
        i = run.channel_info(c)
        if (i["two_J_3N"], i["P_3N"]) == (case["J"], case["P"]):
            return c
    raise ValueError("no channel 2J=%d P=%d" % (case["J"], case["P"]))


def swp_of(run, case):
    Np, Nq = case["Np"], case["Nq"]
    eu, ec = run.host_array(7), run.host_array(8)
    return tt.SWP(Np, Nq, len(eu) // (Np + 1), len(ec) // (2 * (Np + 1)), run.E_bound, eu, ec, run.host_array(5),
                  run.host_array(6), run.host_array(2))


def deuterons(pw):
    return [a for a in range(pw.shape[0]) if tuple(int(x) for x in pw[a, :4]) == (0, 1, 1, 0)]


def csc_of(run, c, nnz):
    """The channel's P123 in the reference's CSC form."""
    rowptr, col, val = run.P123_csr(c, nnz)
    n = len(rowptr) - 1
    row = np.repeat(np.arange(n, dtype=np.int32), np.diff(rowptr))
    order = np.argsort(col, kind="stable")
    colptr = np.concatenate([[0], np.cumsum(np.bincount(col, minlength=n))]).astype(np.uint64)
    return val[order], row[order], colptr


def prepare(case, seed):
    run = tt.Run(**options(case, seed))
    c = channel_of(run, case)
    pw = run.host_array(0, c).reshape(-1, 9)
    s = dict(case=case, run=run, c=c, n=run.channel_info(c)["n"])
    kind = case["kind"]
    if kind in ("resolvent", "resolvent_dev", "dropin"):
        s.update(swp=swp_of(run, case), pw=tt.PW(pw))
    if kind == "resolvent":
        s["E"] = float(run.energies()[1][0]) + run.E_bound
    elif kind == "resolvent_dev":
        s["E"] = np.linspace(3.0, 100.0, case["nE"]) + run.E_bound
        s["G"] = torch.empty((case["nE"], s["n"]), dtype=torch.complex128, device="cuda")
    elif kind == "p123":
        s.update(pw=tt.PW(pw), p=run.host_array(1), q=run.host_array(2))
    elif kind == "dropin":
        val, row, colptr = csc_of(run, c, run.build_P123(c))
        run.build_resolvent(c)
        s.update(G=run.G(c), val=val, row=row, colptr=colptr, Vu=run.host_array(3), Vc=run.host_array(4),
                 q_idx=run.energies()[2], deut=deuterons(pw))
        run.release(c)
    elif kind != "channel":
        run.build_P123(c)
        if kind == "adjoint":
            dV = [run.lec_derivative(k) for k in range(len(run.lecs()))]
            s.update(dVu=np.stack([d[0] for d in dV]), dVc=np.stack([d[1] for d in dV]))
        elif kind == "pade":
            run.breakup_cells(c)
    return s


def run(s):
    case, r, c = s["case"], s["run"], s["c"]
    kind = case["kind"]
    if kind == "resolvent":
        return tt.resolvent(s["E"], s["swp"], s["pw"], **flags(case))
    if kind == "resolvent_dev":
        tt.resolvent_noalloc(s["G"].data_ptr(), s["E"], s["swp"], s["pw"],
                             stream=torch.cuda.current_stream().cuda_stream, **flags(case))
        return s["G"]
    if kind == "p123":
        return tt.fill_P123_arrays(s["pw"], s["p"], s["q"])
    if kind == "dropin":
        prec = tt.PRECISION_FP64 if case["fp64"] else tt.PRECISION_MIXED
        return tt.solve_faddeev(s["G"], s["val"], s["row"], s["colptr"], s["Vu"], s["Vc"], s["swp"], s["q_idx"],
                                s["deut"], s["pw"], precision=prec, **flags(case))[0]
    if kind == "channel":
        r.build_P123(c)
    r.build_A(c)
    if kind == "scan":
        return r.solve_energies(c, np.arange(case["nE"]))[0]
    r.build_resolvent(c)
    if kind == "pade":
        return r.solve_breakup(c)[:2]
    if kind == "adjoint":
        return r.solve_adjoint(c, s["dVu"], s["dVc"])[:2]
    return r.solve(c)[0]


def work(case):
    """P123: its nonzeros written, each a sum over the 48 x 48 mesh.  Solves: P123
    read, and the LU of each energy (8/3 n^3); the Pade series reads A twice per
    order, about ten orders, four multiply-adds per element and on-shell row."""
    n = (2 if case["pot"] == "mt" else NALPHA[case["j"], case["J"]]) * case["Np"] * case["Nq"]
    nE = case.get("nE") or (2 * len(case["labs"].split(",")) if "labs" in case else 1)
    nnz, lu = DENSITY * n * n, 8.0 / 3.0 * n**3 * nE
    mesh = 2.0 * 48 * 48 * nnz
    kind = case["kind"]
    if kind in ("resolvent", "resolvent_dev"):
        return {"bytes": 16.0 * n * nE, "flops": 60.0 * n * nE}
    if kind == "p123":
        return {"bytes": 16.0 * nnz, "flops": mesh}
    if kind == "pade":
        return {"bytes": 12.0 * nnz + 8.0 * n * n * 21, "flops": 4.0 * n * n * 20 * 2 * nE}
    return {"bytes": 12.0 * nnz + 8.0 * n * n, "flops": lu + (mesh if kind == "channel" else 0.0)}


# ---------------------------------------------------------------------------
# 64-bit values, by plain torch


def blocks(pw, case):
    """Per partial wave: is its two-body block coupled, the block's index, the part in it."""
    lo = case["pot"] == "lo"
    out = []
    for L, S, J, T, _, _, _, tT, _ in (tuple(int(x) for x in r) for r in pw):
        s0 = S == 0 and J == 0 and L == 0
        if lo and L != J and J != 0:
            out.append((True, J, 0 if L < J else 1))
        elif lo and s0:
            out.append((True, 0, 0 if tT == 1 else 1))
        elif lo:
            out.append((False, 2 * J + S - 1, 0))
        else:
            out.append((False, J * (4 * (J > 1) + 2) + (S == 1) + (S == 1 and J != 0) * (J - L + 1), 0))
    return out


def exact_resolvent(run, pw, case, E):
    """[len(E)][n]: the bound-continuum and continuum-continuum bin averages of the free resolvent."""
    Np, Nq = case["Np"], case["Nq"]
    e_u, e_c, q = run.host_array(7), run.host_array(8), run.host_array(2)
    eb = np.stack([e_c[b * 2 * (Np + 1) + p * (Np + 1):][:Np + 1] if cpl else e_u[b * (Np + 1):][:Np + 1]
                   for cpl, b, p in blocks(pw, case)])
    lo, hi = eb[:, None, :-1], eb[:, None, 1:]  # [Na][1][Np]
    bound = lo < 0
    Eb = np.where(bound, lo, 0.0)
    mu = M_N * (M_N + M_P + Eb) / (2 * M_N + M_P + Eb)
    ql, qu = q[None, :-1, None] ** 2 / (2 * mu), q[None, 1:, None] ** 2 / (2 * mu)
    Dq, Dp = qu - ql, hi - lo
    out = []
    step = lambda v: np.where(v < 0, 0.0, 1.0)  # noqa: E731
    for En in np.atleast_1d(E):
        with np.errstate(all="ignore"):
            x, y = ql + Eb - En, qu + Eb - En
            re_b, im_b = np.log(np.abs(x / y)) / Dq, (step(y) - step(x)) * -np.pi / Dq
            d, m, p = 0.5 * (lo + hi) + 0.5 * (ql + qu) - En, 0.5 * (Dp - Dq), 0.5 * (Dp + Dq)
            f = lambda g: (g(d + m) + g(d - m) - g(d + p) - g(d - p)) / (Dp * Dq)  # noqa: E731
            re_c, im_c = f(lambda v: v * np.log(np.abs(v))), f(lambda v: v * step(v)) * np.pi
        out.append((np.where(bound, re_b, re_c) + 1j * np.where(bound, im_b, im_c)).reshape(-1))
    return np.stack(out)


def exact_A(run, c, pw, case):
    """A = C^T (2 P123) (V C), dense, on the GPU, from the run's P123, V and C."""
    Na, Np, Nq = len(pw), case["Np"], case["Nq"]
    n = Na * Np * Nq
    rowptr, col, val = run.P123_csr(c, run.build_P123(c))
    run.release(c)
    cuda = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    P = torch.zeros(n * n, dtype=torch.float64, device="cuda")
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), cuda(np.diff(rowptr)))
    P[rows * n + cuda(col).long()] = 2 * cuda(val)
    P = P.view(n, Na, Nq, Np)
    del rows
    V, C = (run.host_array(3), run.host_array(4)), (run.host_array(5), run.host_array(6))
    bl = blocks(pw, case)

    def block(X, a):
        cpl, b, _ = bl[a]
        d = (2 if cpl else 1) * Np
        return cuda(X[int(cpl)][b * d * d:(b + 1) * d * d]).view(d, d)

    def partners(a):
        same = [3, 2, 1, 4, 5] if case["pot"] == "lo" else [3, 2, 1, 4, 5, 0]
        return [b for b in range(Na) if all(pw[a, k] == pw[b, k] for k in same)
                and abs(int(pw[a, 0]) - int(pw[b, 0])) <= 2]

    def part(X, a, b):
        return X[bl[a][2] * Np:][:Np, bl[b][2] * Np:][:, :Np]

    T = torch.empty_like(P)
    for a in range(Na):
        VC = block(V, a) @ block(C, a)
        T[:, a] = sum(P[:, b] @ part(VC, b, a) for b in partners(a))
    T = T.view(Na, Nq, Np, n)
    A = P.view(Na, Nq, Np, n)  # reused
    for a in range(Na):
        A[a] = sum(part(block(C, a), b, a).T @ T[b] for b in partners(a))
    return A.view(n, n)


def exact_U(run, c, pw, case, nE=None):
    """U[d'][d][j] of (1 - A G_j) U = A, complex128 LU."""
    Np, Nq = case["Np"], case["Nq"]
    _, E, q_idx = run.energies()
    E, q_idx = E[:nE], q_idx[:nE]
    A, G = exact_A(run, c, pw, case), exact_resolvent(run, pw, case, E + run.E_bound)
    U = np.zeros((len(deuterons(pw)),) * 2 + (len(E),), dtype=np.complex128)
    for j in range(len(E)):
        rows = torch.tensor([d * Nq * Np + int(q_idx[j]) * Np for d in deuterons(pw)], device="cuda")
        L = -A * torch.from_numpy(G[j]).cuda()
        L.diagonal().add_(1)
        U[:, :, j] = torch.linalg.solve(L, A[:, rows].to(L.dtype))[rows].cpu().numpy()
        del L
    return U.reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "p123":  # a quadrature per nonzero and recoupling sums per mesh point: minutes in plain torch
        return None
    if kind == "pade":  # the approximants' determinants turn rounding into 1e-7: 64 bits leave no such value
        return None
    run = tt.Run(**options(case, seed))
    c = channel_of(run, case)
    pw = run.host_array(0, c).reshape(-1, 9)
    if kind == "resolvent":
        return exact_resolvent(run, pw, case, float(run.energies()[1][0]) + run.E_bound)[0]
    if kind == "resolvent_dev":
        return exact_resolvent(run, pw, case, np.linspace(3.0, 100.0, case["nE"]) + run.E_bound)
    if run.channel_info(c)["n"] > EXACT_N:
        return None
    U = exact_U(run, c, pw, case, case.get("nE"))
    return (U, None) if kind == "adjoint" else U  # the derivative's basis change has no plain-torch form here
