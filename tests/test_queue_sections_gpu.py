"""Batches whose queues are looked over in several sections (256 queues at most): many ensembles, more
sections than the 64 whose progress is looked at, ensembles that end long before others, and ensembles
with more than 256 queues each.  Every ensemble equals its run in an engine of its own, bit for bit."""
import numpy as np
import pytest

from tests.helpers import T2PI, dimer_problem, start_states

pytestmark = pytest.mark.gpu


def channels(d, nd, deep, seed, k):
    """A dimer's split tree with nd random jump channels that conserve the norm's decay (weights only)."""
    P = dimer_problem(d - 1, g=k / d, deep=deep)
    rng = np.random.default_rng(seed)
    L = rng.normal(size=(nd, d, d)) + 1j * rng.normal(size=(nd, d, d))
    return P["U"], L, rng.uniform(0.5, 1.0, nd), P["HE"]


# (ensembles, dimensions, trajectories each, channels, split levels, precision): sections of 7 ensembles in
# sub-tiles (2080 trajectories of d <= 61), one trajectory per CTA and split precision; 70 sections; two parts each
CASES = [(16, (50, 61), 130, 1, 16, 0), (20, (6, 30), 9, 1, 16, 0), (20, (17, 80), 30, 1, 16, 1), (70, (3, 5), 3, 200, 2, 0),
         (70, (17, 20), 2, 200, 2, 1), (3, (8, 20), 50, 300, 4, 0), (3, (17, 33), 50, 300, 4, 1)]


@pytest.mark.parametrize("E,dims,n,nd,deep,precision", CASES)
def test_sections(E, dims, n, nd, deep, precision):
    import os_d_b200 as q

    ens, dmax = [], dims[1]
    psi = np.zeros((E * n, dmax), complex)
    for i in range(E):
        d = dims[0] + (dims[1] - dims[0]) * i // (E - 1)
        k = 0.5 if i % 3 else 6.0  # a third of the ensembles jump twelve times as often
        if nd == 1:
            P = dimer_problem(d - 1, g=k / d, deep=deep)
            U, L, g, HE = P["U"], P["L"], [1.0], P["HE"]
        else:
            U, L, g, HE = channels(d, nd, deep, i, k)
        ens.append(dict(U=U, L=L, g=g, HE=HE, n_traj=n, T=T2PI, seed=i, tr_base=7 * i))
        psi[i * n:(i + 1) * n, :d] = start_states(n, d, 1) * (1 - 1e-9)
    B = q.Engine.batch(ens, deep=deep, max_dumps=1, precision=precision)
    B.set_states(psi)
    B.init_thresholds()
    B.run_periods(2, dump_at=[2])
    psi_b, t_b, eta_b, _ = B.states()
    mean_b = B.observables(0, 1)["mean"][0]
    B.close()
    drawn = 0
    for i, x in enumerate(ens):
        d, r = x["U"].shape[-1], slice(i * n, (i + 1) * n)
        A = q.Engine(x["U"], x["L"], x["g"], x["HE"], None, T2PI, n, seed=i, tr_base=7 * i, max_dumps=1, precision=precision)
        A.set_states(psi[r, :d])
        A.init_thresholds()
        eta0 = A.states()[2]
        A.run_periods(2, dump_at=[2])
        p, t, eta, _ = A.states()
        assert np.array_equal(psi_b[r, :d], p) and np.array_equal(t_b[r], t) and np.array_equal(eta_b[r], eta)
        assert np.array_equal(mean_b[r], A.observables(0, 1)["mean"][0])
        drawn += (eta != eta0).sum()
        A.close()
    assert drawn > 0  # there were jumps
