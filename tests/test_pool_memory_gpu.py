"""A serving pool holds all its device memory from its creation on: loading slots, running and reading
states and observables back takes no more, so admission by the estimate stays right."""
import numpy as np
import pytest

from tests.helpers import T2PI, dimer_problem, start_states

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d_cap,n_cap", [(32, 256), (256, 1024)])
def test_a_pool_grows_by_nothing(d_cap, n_cap):
    import os_d_b200 as q
    from os_d_b200.serve import pool_footprint

    eng = q.Engine.slots(2, d_cap, n_cap, deep=4, max_dumps=1, rec_cap=16)
    created = eng.device_bytes()
    d = d_cap - 3
    P = dimer_problem(d - 1, g=2.0 / d, deep=4)
    eng.slot_load(1, dict(U=P["U"], L=P["L"], g=[1.0], HE=P["HE"], n_traj=n_cap - 1, T=T2PI, seed=1, tr_base=0))
    eng.run_periods(1, is_obs=1, dump_at=[1], dump_base=0)
    eng.observables(0, 1)
    psi = eng.states()[0]
    assert np.abs(np.linalg.norm(psi[n_cap:2 * n_cap - 1], axis=1)).min() > 0
    assert eng.device_bytes() == created
    assert abs(pool_footprint(2, d_cap, n_cap, 4) - created) < 0.1 * created + (1 << 20)
    eng.close()
