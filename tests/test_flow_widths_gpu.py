"""The plain form's shared sub-tiles where no other test runs them: every instantiation by dimension up to
1024 (just past the trajectories that run one to a CTA: 250 + 6.5e6 / d^2) against the oracle, explicit
tile shapes, the deep tasks' dumps and serving slots, bit for bit.  (tests/test_large_dim_gpu.py and the
plain part of the autotuner test in tests/test_split_gpu.py, written for the sub-tiles, have fewer
trajectories and run one to a CTA.)"""
import numpy as np
import pytest

from oracle import oracle_py as O
from tests.helpers import T2PI, dimer_problem, start_states
from tests.test_flow_gpu import solo_max

pytestmark = pytest.mark.gpu


# 32-column sub-tiles of one row block per warp; 65 to 96 rows; 161 to 192; 321 to 384 and 449 to 512 (one CTA
# of 512 threads); 8 columns above 512, at the edges of the row blocks per warp
@pytest.mark.parametrize("d", [30, 90, 190, 350, 500, 513, 640, 641, 768, 769, 896, 897, 1024])
def test_sub_tiles_by_dimension(d):
    import os_d_b200 as q

    n, deep = solo_max(d) + 13, 3
    H, Hd, L, U = q.build_dimer_gpu(d - 1, 1.0, 0.5, 1.0, 1.5, 1.5 / d, 1.0, deep)
    HE = H + Hd
    ens = O.Ensemble(U, L, [1.0], HE, None, T2PI, n, seed=3, record=2, rec_cap=2000)
    eng = q.Engine(U, L, [1.0], HE, None, T2PI, n, seed=3, record=2, rec_cap=2, max_dumps=1)
    ens.init(1, 0)
    eng.set_states(start_states(n, d, 1))
    eng.init_thresholds()
    assert ens.run_periods(1) == 0
    eng.run_periods(1, dump_at=[1])
    psi, t, eta, _ = eng.states()
    assert np.array_equal(psi, ens.phi) and np.array_equal(t, ens.t) and np.array_equal(eta, ens.eta)
    o, g = ens.observables(), eng.observables(0, 1)
    for k in ("norm", "mean", "energy"):
        assert np.array_equal(g[k][0], o[k]), k
    assert ens.jumps_counts.max() > 2  # the record buffers were drained and resumed


def thresholds(q, P, n, d):
    eng = q.Engine(P["U"], P["L"], [1.0], P["HE"], None, T2PI, n, seed=8)
    eng.set_states(start_states(n, d, 1))
    eng.init_thresholds()
    eta = eng.states()[2]
    eng.close()
    return eta


@pytest.mark.parametrize("d,shapes", [(41, [(8, 2), (8, 16), (16, 6), (32, 2), (32, 14)]), (130, [(8, 4), (16, 10), (32, 16), (32, 2)]),
                                      (201, [(8, 16), (16, 2), (32, 8)]), (300, [(8, 16), (16, 4)]), (600, [(8, 2), (8, 6)])])
def test_explicit_shapes_give_the_same_bits(d, shapes):
    import os_d_b200 as q

    n = solo_max(d) + 60
    P = dimer_problem(d - 1, g=3.0 / d, deep=3) if d < 250 else None
    if P is None:
        H, Hd, L, U = q.build_dimer_gpu(d - 1, 1.0, 0.5, 1.0, 1.5, 3.0 / d, 1.0, 3)
        P = dict(U=U, L=L, HE=H + Hd)

    def run(**kw):
        eng = q.Engine(P["U"], P["L"], [1.0], P["HE"], None, T2PI, n, seed=8, **kw)
        eng.set_states(start_states(n, d, 1))
        eng.init_thresholds()
        eng.run_periods(1)
        s = eng.states()
        eng.close()
        return s

    a = run()
    assert (a[2] != thresholds(q, P, n, d)).any()  # there were jumps
    for nc, kb in shapes:
        b = run(tiles=dict(nc=nc, kb=kb))
        assert all(np.array_equal(x, y) for x, y in zip(a[:3], b[:3])), (nc, kb)


def test_deep_task_dumps_of_sub_tiles_equal_those_of_lone_trajectories():
    import os_d_b200 as q

    d, steps, deep = 61, 3, 5
    n = solo_max(d) + 40
    H, Hd, L, U = q.build_dimer_deep(d - 1, 1.0, 0.5, 1.0, 1.5, 3.0 / d, 1.0, deep, steps)

    def run(tr0, tr1):
        m = tr1 - tr0
        eng = q.Engine(U, L, [1.0], H + Hd, None, T2PI, m, seed=2, tr_base=tr0, deep_num_steps=steps, max_dumps=4 * steps)
        eng.set_states(start_states(m, d, 1))
        eng.init_thresholds()
        eng.observe(0, is_start=True)
        eng.run_periods(2, is_obs=1)
        o = eng.observables(0, 4 * steps)
        s = eng.states()
        eng.close()
        return o, s

    o, s = run(0, n)
    for tr0, tr1 in ((0, 700), (700, 1400), (n - 300, n)):
        o1, s1 = run(tr0, tr1)
        for k in ("norm", "mean", "dispersion", "m2", "energy"):
            assert np.array_equal(o[k][:, tr0:tr1], o1[k]), k
        assert all(np.array_equal(x[tr0:tr1], y) for x, y in zip(s[:3], s1[:3]))


def test_serving_slots_in_sub_tiles_equal_the_ensembles_alone():
    import os_d_b200 as q

    n_cap, deep = 700, 5
    eng = q.Engine.slots(4, 64, n_cap, deep=deep, max_dumps=1, rec_cap=16)  # 2100 loaded, of 64: 1836 run one to a CTA

    def ens(d, n, seed):
        P = dimer_problem(d - 1, g=3.0 / d, deep=deep)
        return dict(U=P["U"], L=P["L"], g=[1.0], HE=P["HE"], n_traj=n, T=T2PI, seed=seed, tr_base=5 * seed)

    loaded = {0: ens(64, 700, 1), 2: ens(33, 699, 2), 3: ens(50, 700, 3)}
    for s, e in loaded.items():
        eng.slot_load(s, e)
    eng.run_periods(2, is_obs=1, dump_at=[2], dump_base=0)
    eng.slot_release(2)
    loaded[2] = ens(57, 700, 4)  # joins the others' run
    eng.slot_load(2, loaded[2])
    eng.run_periods(1, is_obs=1, dump_at=[1], dump_base=0)
    psi, t, eta, _ = eng.states()
    mean = eng.observables(0, 1)["mean"][0]
    eng.close()
    for s, e in loaded.items():
        d, n = e["U"].shape[-1], e["n_traj"]
        A = q.Engine(e["U"], e["L"], e["g"], e["HE"], None, T2PI, n, seed=e["seed"], tr_base=e["tr_base"], max_dumps=1)
        A.set_states(start_states(n, d))
        A.init_thresholds()
        A.run_periods(1 if s == 2 else 3, is_obs=1, dump_at=[1 if s == 2 else 3])
        p, ta, ea, _ = A.states()
        r = slice(s * n_cap, s * n_cap + n)
        assert np.array_equal(psi[r, :d], p) and np.array_equal(t[r], ta) and np.array_equal(eta[r], ea), s
        assert np.array_equal(mean[r], A.observables(0, 1)["mean"][0])
        A.close()
