"""The f-basis RK4's cluster form over many short stages, most of its warps without rows, equal to the
oracle bit for bit: a warp that the cluster gets ahead of must not lose count of the stages."""
import numpy as np
import pytest

from oracle import oracle_py as O
from tests.test_fb_resident_gpu import system

pytestmark = pytest.mark.gpu


# one row; rows for two warps of 16; two and four CTAs with 3 to 4 warps of rows; 16 CTAs with long rows
@pytest.mark.parametrize("n,drive_max,steps", [(1, 1, 30000), (48, 1, 30000), (200, 1, 10000), (400, 3, 5000), (3000, 3, 1000)])
def test_many_short_stages(n, drive_max, steps):
    import os_d_b200 as q

    G, Q, ks, x0 = system(n, n, drive_max)
    fb = q.FBasis(G, Q, ks, x0, 1.5, drv_type=0, drv_freq=9.0, T=0.5, num_steps=steps)
    assert fb.cluster_size() > 0
    fb.run(0, 2)
    x_o = O.fb_rk4(G, Q, ks, x0, 1.5, freq=9.0, drv_type=0, T=0.5, num_steps=steps, period0=0, n_periods=2)
    assert np.array_equal(fb.get()[0], x_o)
