"""Small FP64 tensor-core kernels at the edges of their tiles: the density matrix and purity (8 x 8
blocks, 32 trajectories per stage) against the oracle bit for bit, and the split tree's products
(32 x 32 tiles, 8 k per stage) against numpy."""
import numpy as np
import pytest

from oracle import oracle_py as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,n", [(2, 1), (8, 31), (9, 32), (97, 33), (104, 65), (105, 96), (201, 127), (401, 40)])
def test_density_matrix_bit_exact(d, n):
    import os_d_b200 as q

    rng = np.random.default_rng(d)
    psi = rng.normal(size=(n, d)) + 1j * rng.normal(size=(n, d))
    psi[:, d // 2] = 0.0
    eye = np.eye(d, dtype=complex)
    eng = q.Engine(eye[None, None], eye, [1.0], eye, None, 1.0, n)
    eng.set_states(psi)
    p, rho = eng.purity(want_rho=True)
    p_o, rho_o = O.purity(psi)
    assert np.array_equal(rho, rho_o) and p == p_o
    assert np.array_equal(eng.states()[0], psi)


@pytest.mark.parametrize("d", [2, 7, 8, 31, 32, 33, 65, 130])
def test_split_tree_products(d):
    import scipy.linalg as sl

    import os_d_b200 as q

    H, Hd, L, U = q.build_dimer_gpu(d - 1, 1.0, 0.5, 1.0, 1.5, 0.1, 1.0, 8)
    K = q.dimer_generators(d - 1, 1.0, 0.5, 1.0, 1.5, 0.1)
    for b in range(2):
        exact = sl.expm(K[b] * (2 * np.pi / 512))  # the finest level
        assert np.abs(U[b, 7] - exact).max() < 1e-12
        for lvl in range(7):  # each level the square of the next: n products of size <= 1, rounded once each
            sq = U[b, lvl + 1] @ U[b, lvl + 1]
            assert np.abs(U[b, lvl] - sq).max() < 8 * d * 2.0 ** -53
