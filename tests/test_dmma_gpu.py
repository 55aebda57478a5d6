"""FP64 tensor-core kernels at the edges of their tiles: the split tree's products (32 x 32 tiles, 8 k
per stage) against numpy."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


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
