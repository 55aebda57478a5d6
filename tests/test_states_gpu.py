"""The states read back on both sides of the size at which they are packed on the device (40 KB of both slots:
53 trajectories of d = 21), after a period that leaves trajectories in either slot."""
import numpy as np
import pytest

from oracle import oracle_py as O
from tests.helpers import T2PI, dimer_problem, start_states

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d,n", [(2, 1), (21, 53), (21, 54), (40, 32), (41, 32)])
def test_states_of_either_slot(d, n):
    import os_d_b200 as q

    P = dimer_problem(d - 1, g=2.0 / d, deep=6)
    ens = O.Ensemble(P["U"], P["L"], [1.0], P["HE"], None, T2PI, n, seed=9, record=0, rec_cap=2000)
    eng = q.Engine(P["U"], P["L"], [1.0], P["HE"], None, T2PI, n, seed=9)
    ens.init(1, 0)
    eng.set_states(start_states(n, d, 1))
    eng.init_thresholds()
    assert np.array_equal(eng.states()[0], start_states(n, d, 1))
    assert ens.run_periods(1) == 0
    eng.run_periods(1)
    psi, t, eta, _ = eng.states()
    assert np.array_equal(psi, ens.phi) and np.array_equal(t, ens.t) and np.array_equal(eta, ens.eta)
