"""An f-basis run whose waits give up (no poll allowed): the call says so, x is what it was before, and the
handle runs again."""
import numpy as np
import pytest

from oracle import oracle_py as O
from tests.test_fb_resident_gpu import system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,cluster", [(700, 4), (3000, 16), (9000, 0)])
def test_a_run_after_a_timeout(monkeypatch, n, cluster):
    import os_d_b200 as q

    G, Q, ks, x0 = system(n, n, 1)
    fb = q.FBasis(G, Q, ks, x0, 1.5, drv_type=0, drv_freq=9.0, T=0.5, num_steps=40)
    assert fb.cluster_size() == cluster
    monkeypatch.setenv("QJX_FB_POLLS", "0")
    with pytest.raises(q.QjxError, match="gave up"):
        fb.run(0, 3)
    assert np.array_equal(fb.get()[0], x0)
    monkeypatch.delenv("QJX_FB_POLLS")
    fb.run(0, 3)
    x_o = O.fb_rk4(G, Q, ks, x0, 1.5, freq=9.0, drv_type=0, T=0.5, num_steps=40, period0=0, n_periods=3)
    assert np.array_equal(fb.get()[0], x_o)
