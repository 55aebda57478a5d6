"""f-basis RK4 on systems whose CTAs have more long rows (over 20 nonzeros, or several of the drive) than
warps: slices of 32 rows, a thread each, in the cluster form and the grid form, with row lengths at the
edges of four and 32 nonzeros.  Equal to the oracle bit for bit."""
import numpy as np
import pytest
import scipy.sparse as sp

from oracle import oracle_py as O

pytestmark = pytest.mark.gpu


def csr(rng, n, lens):
    cols = [np.sort(rng.choice(n, size=k, replace=False)) for k in lens]
    return sp.csr_matrix((rng.normal(size=int(lens.sum())) * 0.05, np.concatenate(cols).astype(np.int32),
                          np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)), shape=(n, n))


# (rows, nonzeros per row, of the drive): one CTA with 17 long rows (one more than warps), 33 and 100; two
# CTAs; 16; the grid form with 9 to 61 a CTA; rows long for their drive alone
@pytest.mark.parametrize("n,lens,drive,cluster", [
    (100, [21], [0], 1), (17, [17], [2], 1), (33, [0, 3, 31], [1, 2, 4, 5], 1), (190, [20, 21, 24, 25], [1], 1),
    (300, [25, 32, 33, 64, 65], [0, 1, 2, 3], None), (2600, [0, 20, 21, 25], [1, 2], 16), (9000, [5, 18], [1, 2], 0),
    (9000, [33, 40], [0, 1, 2, 7], 0)])
def test_slices_bit_exact(n, lens, drive, cluster):
    import os_d_b200 as q

    rng = np.random.default_rng(n)
    G, Q = csr(rng, n, rng.choice(np.minimum(lens, n), size=n)), csr(rng, n, rng.choice(drive, size=n))
    ks, x0 = rng.normal(size=n) * 0.01, rng.normal(size=n)
    fb = q.FBasis(G, Q, ks, x0, 1.5, drv_type=0, drv_freq=9.0, T=0.5, num_steps=40)
    assert cluster is None or fb.cluster_size() == cluster
    fb.run(0, 2)
    x_o = O.fb_rk4(G, Q, ks, x0, 1.5, freq=9.0, drv_type=0, T=0.5, num_steps=40, period0=0, n_periods=2)
    assert np.abs(x_o - x0).max() > 1e-3
    assert np.array_equal(fb.get()[0], x_o)
