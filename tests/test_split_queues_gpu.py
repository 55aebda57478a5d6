"""The split form's tiles taken from queues against the same tiles in lock-step micro-steps, bit for
bit: one trajectory, tiles of eight rows up to the full 128, rechecks as rare and as frequent as
trajectories, and record buffers that pause the run."""
import numpy as np
import pytest

from tests.helpers import T2PI, dimer_problem, start_states

pytestmark = pytest.mark.gpu


def run(P, n, d, recheck, cap):
    import os_d_b200 as q

    eng = q.Engine(P["U"], P["L"], [1.0], P["HE"], None, T2PI, n, seed=5, record=2, rec_cap=cap, precision=1,
                   split_recheck=recheck, max_dumps=1)
    eng.set_states(start_states(n, d, 1))
    eng.init_thresholds()
    eng.run_periods(1, dump_at=[1])
    return eng.states(), eng.observables(0, 1), [eng.jumps(tr) for tr in range(0, n, 11)], eng.stats()


@pytest.mark.parametrize("d,n,recheck,cap", [(10, 1, 0.0, 50), (41, 7, 0.5, 2), (63, 1185, 0.0, 3), (41, 20000, 1e-3, 50),
                                             (201, 149, 0.2, 50), (256, 33, 0.0, 50)])
def test_queues_equal_lock_step(monkeypatch, d, n, recheck, cap):
    P = dimer_problem(d - 1, g=4.0 / d, deep=4)
    a = run(P, n, d, recheck, cap)
    monkeypatch.setenv("QJX_SPLIT_COOP", "0")
    b = run(P, n, d, recheck, cap)
    for x, y in zip(a[0], b[0]):
        assert np.array_equal(x, y)
    for k in ("norm", "mean", "energy"):
        assert np.array_equal(a[1][k], b[1][k]), k
    for x, y in zip(a[2], b[2]):
        assert all(np.array_equal(u, v) for u, v in zip(x, y))
    assert a[3]["rechecks"] == b[3]["rechecks"] and (recheck == 0.0 or a[3]["rechecks"] > 0)
    assert a[3]["matvecs"] == b[3]["matvecs"]
