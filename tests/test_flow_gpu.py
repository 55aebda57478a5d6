"""The plain form's two kernels at the edges of their ranges: shared sub-tiles (more trajectories than
run one to a CTA at their dimension: 250 + 6.5e6 / d^2) and one trajectory per CTA or cluster.  GPU
against the oracle, bit for bit."""
import numpy as np
import pytest

from oracle import oracle_py as O
from tests.helpers import T2PI, dimer_problem, random_observable, start_states
from tests.test_generic_gpu import generic_system
from tests.test_rk_gpu import problem

pytestmark = pytest.mark.gpu


def solo_max(d):
    return 250 + int(6.5e6 / d**2)


def check(eng, ens, n, d, jumps=()):
    psi, t, eta, jc = eng.states()
    assert np.array_equal(psi, ens.phi) and np.array_equal(t, ens.t) and np.array_equal(eta, ens.eta)
    for tr in jumps:
        for a, b in zip(eng.jumps(tr), ens.jumps(tr)):
            assert np.array_equal(a, b), tr
    return jc


# d at the edges of the sub-tile widths (32 columns to d = 128, two 256-thread CTAs per SM while 16
# columns and slabs of 6 k rows fit half of the shared memory, one CTA of 512 threads above), odd and
# even, and of the clusters (256 rows per CTA); n just past and just up to the switch
@pytest.mark.parametrize("d,over", [(61, 37), (128, 37), (129, 37), (201, 5), (225, 37), (233, 37), (256, 37), (257, 37),
                                    (401, 11), (129, 0), (257, -300), (513, -500)])
def test_kernels_by_dimension(d, over):
    import os_d_b200 as q

    n, deep = max(24, solo_max(d) + over), 5
    P = dimer_problem(d - 1, g=4.0 / d, deep=deep)
    R = random_observable(d, 5)[None] if d < 250 else None
    ens = O.Ensemble(P["U"], P["L"], [1.0], P["HE"], R, T2PI, n, seed=3, record=2, rec_cap=2000)
    eng = q.Engine(P["U"], P["L"], [1.0], P["HE"], R, T2PI, n, seed=3, record=2, rec_cap=3, keep_adr=1, max_dumps=1)
    ens.init(1, 0)
    eng.set_states(start_states(n, d, 1))
    eng.init_thresholds()
    assert ens.run_periods(1) == 0
    eng.run_periods(1, dump_at=[1])
    assert check(eng, ens, n, d, range(0, n, 7)).max() > 3  # the record buffers were drained and resumed
    o, g = ens.observables(), eng.observables(0, 1)
    for k in ("norm", "mean", "energy"):
        assert np.array_equal(g[k][0], o[k]), k
    if R is not None:
        assert np.array_equal(g["random_obs"][0], o["random_obs"])


def test_sub_tiles_with_several_channels():
    import os_d_b200 as q

    d = 140
    n = solo_max(d) + 20
    Ut, L, gs, HE = generic_system(d)
    ens = O.Ensemble(Ut, L, gs, HE, None, T2PI * 2.0 / 3.0, n, seed=13, record=2, rec_cap=2000)
    eng = q.Engine(Ut, L, gs, HE, None, T2PI * 2.0 / 3.0, n, seed=13, record=2, rec_cap=64)
    ens.init(0, 0)
    eng.set_states(start_states(n, d))
    eng.init_thresholds()
    assert ens.run_periods(1) == 0
    eng.run_periods(1)
    assert check(eng, ens, n, d, range(0, n, 11)).sum() > 20


def test_sub_tiles_with_the_rk_propagator():
    import os_d_b200 as q

    N, ns = 60, 24
    d, n = N + 1, solo_max(N + 1) + 9
    H, Hd, L, Heff = problem(N)
    Heff, Hd = 0.02 * Heff, 0.02 * Hd  # (a stable step)
    ens = O.Ensemble(np.zeros((2, 1, d, d), complex), L, [1.0], H, None, T2PI, n, seed=5, record=2, rec_cap=2000)
    eng = q.Engine.rk(Heff, Hd, L, [1.0], H, None, T2PI, n, E0=1.0, A=1.5, rk_ns=ns, seed=5, record=2, rec_cap=64)
    ens.init(0, 0)
    eng.set_states(start_states(n, d))
    eng.init_thresholds()
    assert ens.run_periods_rk(1, Heff, Hd, 1.0, 1.5, ns, period0=0) == 0
    eng.run_periods(1)
    check(eng, ens, n, d, range(0, n, 50))


def test_sub_tiles_of_an_uneven_batch_equal_the_ensembles_alone():
    import os_d_b200 as q

    deep, ens, psi = 6, [], []
    dims, n = (30, 97, 128, 261), 260
    for i, d in enumerate(dims):
        P = dimer_problem(d - 1, g=4.0 / d, deep=deep)
        ens.append(dict(U=P["U"], L=P["L"], g=[1.0], HE=P["HE"], n_traj=n, T=T2PI, seed=i, tr_base=10 * i))
    B = q.Engine.batch(ens, deep=deep)
    s = np.zeros((4 * n, max(dims)), complex)
    for i, d in enumerate(dims):
        s[i * n:(i + 1) * n, :d] = start_states(n, d, 1)
    B.set_states(s)
    B.init_thresholds()
    B.run_periods(1)
    psi_b, t_b, eta_b, _ = B.states()
    for i, (d, x) in enumerate(zip(dims, ens)):
        A = q.Engine(x["U"], x["L"], x["g"], x["HE"], None, T2PI, n, seed=i, tr_base=10 * i)
        A.set_states(start_states(n, d, 1))
        A.init_thresholds()
        A.run_periods(1)
        psi, t, eta, _ = A.states()
        r = B.ranges[i]
        assert np.array_equal(psi_b[r, :d], psi) and not psi_b[r, d:].any() and np.array_equal(eta_b[r], eta)
        A.close()
    B.close()
