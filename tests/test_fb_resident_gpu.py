"""The f-basis RK4's resident forms (one cluster; the whole grid) on systems with rows at the edges of
their row forms: 0 to 70 nonzeros (20 is the longest row held by a thread, 32 the lanes of the
canonical sum), drive rows of 0 to 3, sizes around the cluster sizes and past the largest.  Equal to
the oracle bit for bit with the sign drive."""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle import oracle_py as O

pytestmark = pytest.mark.gpu


def system(n, seed, drive_max):
    rng = np.random.default_rng(seed)

    def csr(lens):
        cols = [np.sort(rng.choice(n, size=k, replace=False)) for k in lens]
        M = sp.csr_matrix((rng.normal(size=int(lens.sum())) * 0.05, np.concatenate(cols).astype(np.int32),
                           np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)), shape=(n, n))
        return M

    lens = rng.choice([0, 1, 2, 7, 17, 18, 19, 20], size=n)
    lens[rng.choice(n, size=max(1, n // 40), replace=False)] = rng.choice([21, 31, 32, 33, 64, 70], size=max(1, n // 40))
    G, Q = csr(np.minimum(lens, n)), csr(np.minimum(rng.integers(0, drive_max + 1, size=n), n))
    return G, Q, rng.normal(size=n) * 0.01, rng.normal(size=n)


@pytest.mark.parametrize("n,drive_max,cluster", [(1, 1, 1), (3, 1, 1), (192, 1, 1), (193, 3, 2), (700, 1, 4),
                                                 (3000, 1, 16), (3100, 3, 16), (9000, 1, 0), (12001, 3, 0)])
def test_resident_forms_bit_exact(n, drive_max, cluster):
    import os_d_b200 as q

    G, Q, ks, x0 = system(n, n, drive_max)
    T, steps = 0.5, 40
    fb = q.FBasis(G, Q, ks, x0, 1.5, drv_type=0, drv_freq=9.0, T=T, num_steps=steps)
    assert fb.cluster_size() == cluster
    fb.run(0, 2)
    fb.run(2, 1)
    x = fb.get()[0]
    x_o = O.fb_rk4(G, Q, ks, x0, 1.5, freq=9.0, drv_type=0, T=T, num_steps=steps, period0=0, n_periods=3)
    assert np.all(np.isfinite(x_o)) and np.abs(x_o - x0).max() > 1e-3
    assert np.array_equal(x, x_o)
