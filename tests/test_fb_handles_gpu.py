"""Two f-basis handles of different size alive at once: the larger, created first, still runs."""
import numpy as np
import pytest

from oracle import oracle_py as O
from tests.test_fb_resident_gpu import system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("large,small,clustered", [(3000, 700, True), (12001, 9000, False)])
def test_the_larger_of_two_handles_runs(large, small, clustered):
    import os_d_b200 as q

    handles = []
    for n in (large, small):
        G, Q, ks, x0 = system(n, n, 1)
        fb = q.FBasis(G, Q, ks, x0, 1.5, drv_type=0, drv_freq=9.0, T=0.5, num_steps=20)
        assert (fb.cluster_size() > 0) == clustered
        handles.append((fb, G, Q, ks, x0))
    for fb, G, Q, ks, x0 in handles:
        fb.run(0, 1)
        x_o = O.fb_rk4(G, Q, ks, x0, 1.5, freq=9.0, drv_type=0, T=0.5, num_steps=20, period0=0, n_periods=1)
        assert np.array_equal(fb.get()[0], x_o)
