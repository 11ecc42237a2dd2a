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
