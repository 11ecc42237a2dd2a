"""Kernels at the edges of their tiles, against the CPU oracle."""
import numpy as np
import pytest

import harness as oracle
import tictac_b200 as tt
from conftest import rel

pytestmark = pytest.mark.gpu

# P123 values are sums of Nphi Nx positive weights times sums of a few dozen
# products of order one: rounding stays some 1e-15 of the largest value
P123_TOL = 1e-13


@pytest.mark.parametrize("j,J,Np,Nq,Nphi,Nx", [
    (1, 1, 8, 5, 7, 9),      # odd mesh of 63 points: scalar copies, ragged last block of points
    (1, 3, 5, 8, 2, 2),      # the smallest mesh: one partial block
    (2, 5, 6, 6, 16, 15),    # more than 64 orbital functions, several phases
    (1, 1, 12, 3, 33, 2),    # rows of more than 8 cells in tiles of 8
])
def test_p123_orbital_functions_at_tile_edges(j, J, Np, Nq, Nphi, Nx):
    run = tt.Run(potential_model="malfliet_tjon", isospin_breaking_1S0="false", J_2N_max=j, two_J_3N_max=J, Np_WP=16,
                 Nq_WP=16, lab_energies="13")
    p, q = (a[::16 // (N + 1)][:N + 1] for a, N in ((run.host_array(1), Np), (run.host_array(2), Nq)))
    for c in (run.num_channels - 2, run.num_channels - 1):
        pw = run.host_array(0, c).reshape(-1, 9)
        r, cc, v = tt.fill_P123_arrays(tt.PW(pw, j), p, q, Nphi=Nphi, Nx=Nx)
        r_o, c_o, v_o = oracle.p123(pw, p, q, Nphi, Nx)
        assert np.array_equal(r, r_o) and np.array_equal(cc, c_o), c
        assert rel(v, v_o) <= P123_TOL, c
    run.close()


def test_p123_of_waves_of_both_parities():
    # a table that mixes parities keeps the terms of negative M (in a channel of
    # one parity they equal those of positive M)
    run = tt.Run(potential_model="malfliet_tjon", isospin_breaking_1S0="false", J_2N_max=1, two_J_3N_max=1, Np_WP=6,
                 Nq_WP=5, lab_energies="13")
    pw = np.concatenate([run.host_array(0, c).reshape(-1, 9) for c in range(2)])
    p, q = run.host_array(1), run.host_array(2)
    n = pw.shape[0] * 30
    r, c, v = tt.fill_P123_arrays(tt.PW(pw), p, q, Nphi=12, Nx=12)
    r_o, c_o, v_o = oracle.p123(pw, p, q, 12, 12)
    A, B = np.zeros((n, n)), np.zeros((n, n))
    A[r, c], B[r_o, c_o] = v, v_o
    assert rel(A, B) <= P123_TOL
    run.close()


def run_and_oracle_U(c, run, Np, Nq):
    """Oracle U of a run's channel, from the oracle's own A and G on the run's P123."""
    T, E_com, q_idx = run.energies()
    pw = run.host_array(0, c).reshape(-1, 9)
    rowptr, col, val = run.P123_csr(c, run.build_P123(c))
    rows = np.repeat(np.arange(len(rowptr) - 1, dtype=np.int32), np.diff(rowptr))
    lay = oracle.layout(pw, Np, *[run.host_array(k) for k in range(3, 9)])
    G = np.stack([oracle.resolvent(lay, pw.shape[0], Nq, Np, run.host_array(2), e + run.E_bound) for e in E_com])
    A = oracle.build_A(lay, pw.shape[0], Nq, Np, rows, col, val)
    return oracle.dense_solve(A, G, q_idx, oracle.deuterons(pw), Nq, Np)


# the sub-panel kernel's layouts: one CTA up to 224 rows, a cluster up to 4,096,
# records in L2 beyond; the last sub-panel narrower than a register block.  U to the refinement's and the suite's 1e-10 per element.
@pytest.mark.parametrize("Np,Nq", [(7, 5),     # n = 385: a substitution block of one row
                                   (6, 6),     # n = 396: a cluster of two, last sub-panel 12 wide
                                   (9, 5),     # n = 495: a cluster of two, last 15 wide
                                   (15, 5),    # n = 825: a cluster of four, last 25 wide
                                   (19, 4),    # n = 836
                                   (17, 10)])  # n = 1,870: clusters of 8
@pytest.mark.parametrize("batch", [1, 4])
def test_subpanel_layouts(Np, Nq, batch):
    from conftest import rel_elem

    run = tt.Run(potential_model="LO_internal", J_2N_max=1, two_J_3N_max=1, Np_WP=Np, Nq_WP=Nq, Nphi=12, Nx=12,
                 lab_energies="5,30", energy_batch=batch, chebyshev_s=150)
    U_o = run_and_oracle_U(0, run, Np, Nq)
    for prec in (tt.PRECISION_FP64, tt.PRECISION_MIXED, tt.PRECISION_MIXED_SIMT):
        U, rep = run.solve(0, prec)
        assert rel_elem(U, U_o) <= 1e-10, (prec, rep)
    run.close()


@pytest.mark.parametrize("precision", [tt.PRECISION_FP64, tt.PRECISION_MIXED])
@pytest.mark.parametrize("i0", [0, 37, 511])
def test_zero_column_is_reported_singular(precision, i0):
    # A = diag(2 v), G = 1 / A in one element: column i0 of 1 - A G is exactly zero
    Np = Nq = 16
    n = 2 * Np * Nq
    pw = np.array([[0, 0, 0, 1, 0, 1, 1, 1, 1], [0, 1, 1, 0, 0, 1, 1, 1, 1]], dtype=np.int32)
    eye, e = np.tile(np.eye(Np).ravel(), 6), np.tile(np.linspace(-2, 100, Np + 1), 6)
    swp = tt.SWP(Np, Nq, 6, 0, -2.0, e, None, eye, None, np.linspace(0, 1000, Nq + 1))
    G = np.full(n, 0.125 + 0.25j)
    G[i0] = 0.5
    with pytest.raises(tt.TicTacError) as err:
        tt.solve_faddeev(G, np.ones(n), np.arange(n, dtype=np.int32), np.arange(n + 1, dtype=np.uint64), eye, None, swp,
                         [3], [1], tt.PW(pw), precision=precision, tensor_force=0, isospin_breaking_1S0=0)
    assert err.value.code == tt.TT_ERR_SINGULAR and f"column {i0 + 1} " in str(err.value)


def test_buffers_of_concurrent_threads():
    # every thread works on a stream of its own; buffers released on one stream
    # are reused on others, and each result must equal the single-threaded one
    import threading

    opts = [dict(potential_model="LO_internal", J_2N_max=1, two_J_3N_max=1, Np_WP=8 + k, Nq_WP=9, Nphi=12, Nx=12,
                 lab_energies="5,30") for k in range(3)]

    def work(k, out):
        run = tt.Run(**opts[k])
        for prec in (tt.PRECISION_MIXED, tt.PRECISION_FP64):
            out.append(run.solve(1, prec)[0])
        run.release(1)
        out.append(run.solve(1, tt.PRECISION_MIXED)[0])
        run.close()

    alone = [[] for _ in opts]
    for k in range(len(opts)):
        work(k, alone[k])
    together = [[] for _ in range(2 * len(opts))]
    threads = [threading.Thread(target=work, args=(i % len(opts), together[i])) for i in range(len(together))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for i, got in enumerate(together):
        for a, b in zip(alone[i % len(opts)], got, strict=True):
            assert np.array_equal(a, b), i
    tt.release_cached_device_memory()
    assert tt.cached_device_memory() == 0


@pytest.mark.parametrize("Np,Nq,labs", [
    (7, 5, "8"),          # n = 385: odd order, few slabs of rows
    (6, 7, "5,30,100"),   # n = 462: five energies, on-shell rows in groups of 8 and less
    (13, 11, "5,30"),     # n = 1,573: odd, more than one block of columns
])
def test_pade_series_and_transposed_products(Np, Nq, labs):
    # TT_PRECISION_PADE against the oracle's restatement on the oracle's A and G, at
    # the method's accuracy (its approximants differ by up to 1e-6 where they stop)
    run = tt.Run(potential_model="LO_internal", J_2N_max=1, two_J_3N_max=1, Np_WP=Np, Nq_WP=Nq, Nphi=12, Nx=12,
                 lab_energies=labs, chebyshev_s=150)
    pw = run.host_array(0, 1).reshape(-1, 9)
    T, E_com, q_idx = run.energies()
    rowptr, col, val = run.P123_csr(1, run.build_P123(1))
    rows = np.repeat(np.arange(len(rowptr) - 1, dtype=np.int32), np.diff(rowptr))
    lay = oracle.layout(pw, Np, *[run.host_array(k) for k in range(3, 9)])
    G = np.stack([oracle.resolvent(lay, pw.shape[0], Nq, Np, run.host_array(2), e + run.E_bound) for e in E_com])
    A = oracle.build_A(lay, pw.shape[0], Nq, Np, rows, col, val)
    U_o = oracle.pade_solve(A, G, q_idx, oracle.deuterons(pw), Nq, Np)
    U, rep = run.solve(1, tt.PRECISION_PADE)
    assert rel(U, U_o) <= 1e-5 and 1 <= rep["refine_iters"] <= 14
    U2, _ = run.solve(1, tt.PRECISION_PADE)
    assert np.array_equal(U, U2)  # no sum depends on the order of threads
    run.close()


@pytest.mark.parametrize("Np,Nq,j", [
    (33, 2, 1),   # two warps' worth of columns of VC, tiles of 8 rows up to 40
    (8, 33, 1),   # one chunk of all q', ranges longer than a staged window
    (7, 13, 2),   # odd rows: 8-byte stores, T rows padded to a k step
    (30, 6, 1),   # the headline grid's p bins
])
def test_A_build_chunks(Np, Nq, j):
    # FP64 sums of up to a few hundred terms of both signs, against the largest element
    run = tt.Run(potential_model="LO_internal", J_2N_max=j, two_J_3N_max=1, Np_WP=Np, Nq_WP=Nq, Nphi=10, Nx=10,
                 lab_energies="8", chebyshev_s=150)
    pw = run.host_array(0, 0).reshape(-1, 9)
    rowptr, col, val = run.P123_csr(0, run.build_P123(0))
    rows = np.repeat(np.arange(len(rowptr) - 1, dtype=np.int32), np.diff(rowptr))
    lay = oracle.layout(pw, Np, *[run.host_array(k) for k in range(3, 9)])
    A_o = oracle.build_A(lay, pw.shape[0], Nq, Np, rows, col, val)
    run.build_A(0)
    assert rel(run.A(0), A_o) <= 1e-12
    run.close()


def test_tall_subpanels_of_a_batch():
    # four matrices of order 18,207 share 148 CTAs, 37 each and two rows a thread;
    # one at a time they take 38 CTAs and a row a thread.  The same operations on
    # every element either way
    opts = dict(potential_model="LO_internal", J_2N_max=3, two_J_3N_max=7, Np_WP=17, Nq_WP=17, lab_energies="5,30",
                Nphi=12, Nx=12)
    U = []
    for batch in (1, 4):
        run = tt.Run(**opts, energy_batch=batch)
        c = run.num_channels - 1
        assert run.channel_info(c)["n"] == 18_207 and len(run.energies()[0]) == 4
        U.append(run.solve(c, tt.PRECISION_MIXED)[0])
        run.close()
    assert np.array_equal(U[0], U[1])


# where a sub-panel's pivots lie: on the diagonal, off it but in the 32 x 32 diagonal
# block, in a few columns below the block, or anywhere; each energy's matrix its own way.
# n = 512: a cluster, then one CTA; n = 4,608: records in L2 first
@pytest.mark.parametrize("Np,kinds", [(16, ("diagonal", "block", "below", "anywhere")), (16, ("anywhere", "anywhere")),
                                      (48, ("below", "block"))])
@pytest.mark.parametrize("precision", [tt.PRECISION_FP64, tt.PRECISION_MIXED, tt.PRECISION_MIXED_SIMT])
def test_pivots_in_and_below_the_diagonal_block(precision, Np, kinds):
    import torch

    n, rng = 2 * Np * Np, np.random.default_rng(5)
    pw = np.array([[0, 0, 0, 1, 0, 1, 1, 1, 1], [0, 1, 1, 0, 0, 1, 1, 1, 1]], dtype=np.int32)
    eye, e = np.tile(np.eye(Np).ravel(), 6), np.tile(np.linspace(-2, 100, Np + 1), 6)
    swp = tt.SWP(Np, Np, 6, 0, -2.0, e, None, eye, None, np.linspace(0, 1000, Np + 1))
    # A = 2 P, strong within the 32 x 32 diagonal blocks and in the columns j of `far` at row j + 300
    P = rng.standard_normal((n, n)) * (1e-2 / np.sqrt(n))
    block = np.arange(n) // 32
    P += np.where(block[:, None] == block[None, :], rng.standard_normal((n, n)), 0) * 2e-2
    far = np.arange(17, n - 300, 97)
    far = far[(far % 32 != 0) & (far % 7 != 0)]
    scale = {"diagonal": 0.1, "block": 100.0, "below": 0.1, "anywhere": 3e4}
    G = np.stack([scale[k] * np.exp(1j * rng.uniform(0, 2 * np.pi, n)) for k in kinds])
    P[far + 300, far] = 1.0
    for j, k in enumerate(kinds):
        G[j, far] = 40.0 if k == "below" else 0.01
    q_idx = np.arange(3, 3 + len(kinds))
    rows = np.tile(np.arange(n, dtype=np.int32), n)
    U, rep = tt.solve_faddeev(G, P.T.ravel(), rows, np.arange(0, n * n + 1, n, dtype=np.uint64), eye, None, swp, q_idx,
                              [1], tt.PW(pw), precision=precision, tensor_force=0, isospin_breaking_1S0=0)
    A = torch.from_numpy(2 * P).cuda()
    for j in range(len(kinds)):
        L = torch.eye(n, dtype=torch.complex128, device="cuda") - A * torch.from_numpy(G[j]).cuda()
        row = Np * Np + int(q_idx[j]) * Np
        want = torch.linalg.solve(L, A[:, row].to(L.dtype))[row].item()
        assert abs(U[j] - want) <= 1e-10 * abs(want), (kinds[j], U[j], want, rep)


@pytest.mark.parametrize("precision", [tt.PRECISION_FP64, tt.PRECISION_MIXED])
def test_drop_in_solve_uses_the_callers_resolvents(precision):
    # A = diag(a): U = a / (1 - a G) at the on-shell element.  Every call brings other
    # resolvents in pageable memory (147 KB), none of them the resolvent of the grid, whose
    # first element at E = 0 is 0 log 0
    Np = Nq = 48
    n, rng = 2 * Np * Nq, np.random.default_rng(11)
    pw = np.array([[0, 0, 0, 1, 0, 1, 1, 1, 1], [0, 1, 1, 0, 0, 1, 1, 1, 1]], dtype=np.int32)
    eye, e = np.tile(np.eye(Np).ravel(), 6), np.tile(np.linspace(0, 100, Np + 1), 6)
    swp = tt.SWP(Np, Nq, 6, 0, -2.0, e, None, eye, None, np.linspace(0, 1000, Nq + 1))
    v, q_idx = rng.uniform(0.5, 1.5, n), np.array([3, 40])
    at = Np * Nq + q_idx * Np
    for _ in range(8):
        G = rng.uniform(0.1, 0.3, (2, n)) * np.exp(1j * rng.uniform(0, 2 * np.pi, (2, n)))
        U, _ = tt.solve_faddeev(G, v, np.arange(n, dtype=np.int32), np.arange(n + 1, dtype=np.uint64), eye, None, swp,
                                q_idx, [1], tt.PW(pw), precision=precision, tensor_force=0, isospin_breaking_1S0=0)
        want = 2 * v[at] / (1 - 2 * v[at] * G[[0, 1], at])
        assert np.all(abs(U - want) <= 1e-10 * abs(want))


def test_pade_determinants_with_rows_exchanged():
    # coefficients that grow threefold an order: every column of the determinants has its
    # pivot in the last row.  Approximants stop 1e-7 apart on elements of 0.02 to 0.05, so
    # 5e-6 relative, and a few times that from the solution; a wrong pivot gives another value
    import torch

    Np = Nq = 8
    n, rng = 2 * Np * Nq, np.random.default_rng(3)
    pw = np.array([[0, 0, 0, 1, 0, 1, 1, 1, 1], [0, 1, 1, 0, 0, 1, 1, 1, 1]], dtype=np.int32)
    eye, e = np.tile(np.eye(Np).ravel(), 6), np.tile(np.linspace(-2, 100, Np + 1), 6)
    swp = tt.SWP(Np, Nq, 6, 0, -2.0, e, None, eye, None, np.linspace(0, 1000, Nq + 1))
    Q, _ = np.linalg.qr(rng.standard_normal((n, 8)))
    A = (Q * 3.0 * 0.4 ** np.arange(8)) @ Q.T
    q_idx, G = np.arange(8), np.exp(1j * np.linspace(0.5, 2.5, 8))[:, None] * np.ones(n)
    args = (G, (A / 2).T.ravel(), np.tile(np.arange(n, dtype=np.int32), n), np.arange(0, n * n + 1, n, dtype=np.uint64),
            eye, None, swp, q_idx, [1], tt.PW(pw))
    U = [tt.solve_faddeev(*args, precision=tt.PRECISION_PADE, tensor_force=0, isospin_breaking_1S0=0)[0]
         for _ in range(3)]
    at = Np * Nq + q_idx * Np
    want = np.array([torch.linalg.solve(torch.eye(n, dtype=torch.complex128) - torch.from_numpy(A * G[j]),
                                        torch.from_numpy(A[:, at[j]]).to(torch.complex128))[at[j]].item()
                     for j in range(8)])
    assert np.all(abs(U[0] - want) <= 1e-4 * abs(want).max())
    assert np.array_equal(U[0], U[1]) and np.array_equal(U[0], U[2])


@pytest.mark.parametrize("precision", [tt.PRECISION_FP64, tt.PRECISION_MIXED])
def test_pivots_found_in_two_trips(precision):
    # n = 8,192: 37 CTAs a matrix and so two trips through L2 for a search (records of one
    # element, then the winner's row) down to 7,168 rows; a fifth to a third of the sub-panels
    # have pivots below their block.  P has 80 nonzeros a column (the condition numbers are
    # 4e5 to 4e7, the elements come out to 1e-15 in 64 bits).
    import torch

    Np = 64
    n, rng = 2 * Np * Np, np.random.default_rng(7)
    pw = np.array([[0, 0, 0, 1, 0, 1, 1, 1, 1], [0, 1, 1, 0, 0, 1, 1, 1, 1]], dtype=np.int32)
    eye, e = np.tile(np.eye(Np).ravel(), 6), np.tile(np.linspace(-2, 100, Np + 1), 6)
    swp = tt.SWP(Np, Np, 6, 0, -2.0, e, None, eye, None, np.linspace(0, 1000, Np + 1))
    far = np.arange(17, n - 300, 97)
    far = far[(far % 32 != 0) & (far % 7 != 0)]
    i = np.arange(n)
    row = np.concatenate([np.repeat(i, 32), np.repeat(i, 48), far + 300])
    col = np.concatenate([(i[:, None] // 32 * 32 + np.arange(32)).ravel(), rng.integers(0, n, n * 48), far])
    val = np.concatenate([rng.standard_normal(n * 32) * 2e-2, rng.standard_normal(n * 48) * (1e-2 / np.sqrt(48)),
                          np.ones(len(far))])
    at, which = np.unique(col.astype(np.int64) * n + row, return_inverse=True)  # by column, then row
    val = np.bincount(which, weights=val)
    colptr = np.concatenate([[0], np.cumsum(np.bincount(at // n, minlength=n))]).astype(np.uint64)
    scale = {"below": 0.1, "block": 100.0, "anywhere": 3e4}
    G = np.stack([scale[k] * np.exp(1j * rng.uniform(0, 2 * np.pi, n)) for k in scale])
    G[:, far] = np.array([40.0, 0.01, 0.01])[:, None]
    q_idx = np.array([3, 20, 50])
    U, rep = tt.solve_faddeev(G, val, (at % n).astype(np.int32), colptr, eye, None, swp, q_idx, [1], tt.PW(pw),
                              precision=precision, tensor_force=0, isospin_breaking_1S0=0)
    A = torch.zeros(n * n, dtype=torch.float64, device="cuda")
    A[torch.from_numpy(at % n * n + at // n).cuda()] = torch.from_numpy(2 * val).cuda()
    A = A.view(n, n)
    for j in range(3):
        L = torch.eye(n, dtype=torch.complex128, device="cuda") - A * torch.from_numpy(G[j]).cuda()
        r = Np * Np + int(q_idx[j]) * Np
        want = torch.linalg.solve(L, A[:, r].to(L.dtype))[r].item()
        assert abs(U[j] - want) <= 1e-10 * abs(want), (j, U[j], want, rep)


@pytest.mark.parametrize("precision", [tt.PRECISION_FP64, tt.PRECISION_MIXED])
@pytest.mark.parametrize("Np", [16, 48])  # clusters and one CTA; records in L2
def test_resolvents_that_are_not_finite(precision, Np):
    # A = diag(2): a NaN in G makes its column of 1 - A G NaN, which has no pivot.  So does an
    # infinity (0 inf is NaN, and elimination carries the NaN above down onto the infinity),
    # except in the first column, where it is the pivot and makes everything behind it NaN.
    n = 2 * Np * Np
    pw = np.array([[0, 0, 0, 1, 0, 1, 1, 1, 1], [0, 1, 1, 0, 0, 1, 1, 1, 1]], dtype=np.int32)
    eye, e = np.tile(np.eye(Np).ravel(), 6), np.tile(np.linspace(-2, 100, Np + 1), 6)
    swp = tt.SWP(Np, Np, 6, 0, -2.0, e, None, eye, None, np.linspace(0, 1000, Np + 1))

    def solve(g, at):
        G = np.full(n, 0.125 + 0.25j)
        G[at] = g
        return tt.solve_faddeev(G, np.ones(n), np.arange(n, dtype=np.int32), np.arange(n + 1, dtype=np.uint64), eye,
                                None, swp, [3], [1], tt.PW(pw), precision=precision, tensor_force=0,
                                isospin_breaking_1S0=0)[0]

    for g, at, col in ((np.nan, 0, 1), (np.nan, 40, 41), (np.nan, n - 1, n), (np.inf, 0, 2), (np.inf, 31, 32),
                       (np.inf, n - 200, n - 199), (np.inf, n - 1, n)):
        with pytest.raises(tt.TicTacError) as err:
            solve(g, at)
        assert err.value.code == tt.TT_ERR_SINGULAR and f"column {col} " in str(err.value), (g, at, str(err.value))
    assert np.all(np.isfinite(solve(0.5j, 5)))
