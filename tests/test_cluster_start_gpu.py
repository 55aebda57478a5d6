"""One trajectory per cluster with more clusters than the chip holds, so that clusters start one after
another beside running ones: each stores into its CTAs' shared memory as soon as it starts.  GPU against
the oracle, bit for bit."""
import numpy as np
import pytest

from oracle import oracle_py as O
from tests.helpers import T2PI, start_states
from tests.test_large_dim_gpu import fast_problem

pytestmark = pytest.mark.gpu


# 2 and 4 CTAs per cluster, 348 and 274 trajectories: 696 CTAs of 160 threads and 1096 of 160
@pytest.mark.parametrize("d,n", [(257, 348), (513, 274)])
def test_clusters_in_waves(d, n):
    import os_d_b200 as q

    P = fast_problem(d - 1, 3, g=2.0 / d)
    ens = O.Ensemble(P["U"], P["L"], [1.0], P["HE"], None, T2PI, n, seed=4, record=1, rec_cap=2000)
    eng = q.Engine(P["U"], P["L"], [1.0], P["HE"], None, T2PI, n, seed=4, record=1, rec_cap=64)
    ens.init(1, 0)
    eng.set_states(start_states(n, d, 1))
    eng.init_thresholds()
    assert ens.run_periods(1) == 0
    eng.run_periods(1)
    psi, t, eta, _ = eng.states()
    assert np.array_equal(psi, ens.phi) and np.array_equal(t, ens.t) and np.array_equal(eta, ens.eta)
    assert ens.jumps_counts.sum() > 0
