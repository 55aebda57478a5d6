"""Timed cases of the engine's public entry points.

Every case is one call, or one short chain of calls, that a program using os_d_b200 makes: solve an
ensemble for a period or two and read it back, advance an uneven batch, take a Lyapunov step of a
parameter sweep, integrate the f-basis Lindblad equation, take the ensemble purity, build a split
tree.  `run` starts from the same inputs each time it is called (the f-basis integrator goes on from
where it stands, at the same cost), so passes of one state do the same work.

Start states are spin-coherent states of the dimer, cos(theta/2)^(N-k) sin(theta/2)^k e^(i k phi) with
binomial weights: a condensate with a given imbalance and phase, drawn per trajectory.
"""
import math

import numpy as np
import torch

import os_d_b200 as q

T2PI = 2.0 * 3.1415926535897932384626433832795
DEEP = 16                  # split levels (the reference's ex_deep default)
J, U0, E0, A = 1.0, 0.5, 1.0, 1.5


def listed():
    return [
        # the smallest call: a quick look at a small ensemble, all latency
        dict(name="qj_d21_n64", kind="qj", N=20, n=64, periods=2, g=0.1, precision=0, record=1),
        # the ordinary ensemble: N = 100 bosons, 1000 trajectories, observables after the period
        dict(name="qj_d101_n1000", kind="qj", N=100, n=1000, periods=2, g=0.1, precision=0, record=0),
        # the headline ensemble in the plain FP64 form
        dict(name="qj_d201_n10000", kind="qj", N=200, n=10000, periods=1, g=0.1, precision=0, record=0),
        # a large Hilbert space with few trajectories
        dict(name="qj_d401_n100", kind="qj", N=400, n=100, periods=1, g=0.1, precision=0, record=0),
        # the headline ensemble in split precision
        dict(name="split_d201_n10000", kind="qj", N=200, n=10000, periods=2, g=0.1, precision=1, record=0),
        # ensembles of uneven dimension in one engine (N from 50 to 400)
        dict(name="batch_8x200", kind="batch", M=8, lo=50, hi=400, n=200, precision=0),
        # the production sweep: Lyapunov pairs at N = 500, 20 trajectories per value of U
        dict(name="lpn_d501_4x20", kind="lpn", N=500, M=4, n=20),
        # the RK propagator, with a step at which a period's jump times keep some digits
        dict(name="rk_d61_n300", kind="rk", N=60, n=300, ns=4000, g=0.2, drv_type=0),
        # the density-matrix oracle at the sizes it is used at: N = 50, dt = 1e-3, and twice that
        dict(name="fbasis_N50", kind="fbasis", N=50, steps=6284, drv_type=0),
        dict(name="fbasis_N100", kind="fbasis", N=100, steps=6284, drv_type=1),
        # purity and density matrix of the headline ensemble (taken after every period)
        dict(name="purity_d201_n10000", kind="purity", N=200, n=10000),
        # the split trees a serving loop builds for each request
        dict(name="tree_d512", kind="tree", N=511),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["qj", "qj", "qj", "split", "split", "batch", "batch", "lpn", "rk", "fbasis", "fbasis", "purity",
                       "tree"])
    if kind == "qj":
        N = _log(rng, 15, 400)
        most = min(10000, int(0.8 * 10000 * (201.0 / (N + 1)) ** 3))
        n = _log(rng, 20, max(100, most))
        return dict(kind="qj", N=N, n=n, periods=1, g=rng.choice([0.05, 0.1]), precision=0, record=rng.randrange(2))
    if kind == "split":
        N = _log(rng, 31, 255)
        return dict(kind="qj", N=N, n=_log(rng, 300, 9000), periods=1, g=rng.choice([0.05, 0.1]), precision=1, record=0)
    if kind == "batch":
        precision = rng.randrange(2)
        lo = rng.randrange(20, 80)
        hi = rng.randrange(lo + 40, 256 if precision else 380)
        return dict(kind="batch", M=rng.randrange(3, 9), lo=lo, hi=hi, n=_log(rng, 30, 180), precision=precision)
    if kind == "lpn":
        return dict(kind="lpn", N=_log(rng, 40, 450), M=rng.randrange(1, 5), n=2 * rng.randrange(3, 11))
    if kind == "rk":
        return dict(kind="rk", N=_log(rng, 12, 40), n=_log(rng, 40, 300), ns=rng.randrange(2500, 3900), g=0.1,
                    drv_type=rng.randrange(2))
    if kind == "fbasis":
        return dict(kind="fbasis", N=_log(rng, 6, 98), steps=rng.randrange(3000, 6000), drv_type=rng.randrange(2))
    if kind == "purity":
        return dict(kind="purity", N=_log(rng, 15, 400), n=_log(rng, 100, 10000))
    return dict(kind="tree", N=_log(rng, 63, 500))


# ---------------------------------------------------------------- inputs
def _dimer(N, U, E, g):
    """H, Hd, L and the split tree (on the GPU where the host exponentials take longest)."""
    build = q.build_dimer_gpu if N >= 128 else q.build_dimer
    return build(N, J, U, E, A, g, 1.0, DEEP)


def _coherent(N, n, rng):
    """[n][N + 1] spin-coherent states, norm a hair below 1 (a norm above 1 is an error of the path)."""
    k = np.arange(N + 1)
    lg = torch.lgamma(torch.arange(1, N + 2, dtype=torch.float64)).numpy()
    logw = 0.5 * (lg[N] - lg[k] - lg[N - k])
    z, phi = rng.uniform(-0.95, 0.95, n), rng.uniform(0.0, T2PI, n)
    lc, ls = 0.5 * np.log((1 + z) / 2), 0.5 * np.log((1 - z) / 2)
    a = np.exp(logw[None, :] + lc[:, None] * (N - k)[None, :] + ls[:, None] * k[None, :])
    psi = a * np.exp(1j * phi[:, None] * k[None, :])
    return psi * ((1.0 - 1e-10) / np.sqrt((np.abs(psi) ** 2).sum(1, keepdims=True)))


def _batch_dims(case):
    """(N, E0, g) per ensemble, spread over the case's range."""
    M = case["M"]
    out = []
    for i in range(M):
        x = i / max(1, M - 1)
        N = int(round(case["lo"] + (case["hi"] - case["lo"]) * x))
        out.append((N, 2.0 * ((i * 5) % M) / M, 0.02 * 5.0 ** ((3 * i % M) / M)))
    return out


def _rk_ops(case):
    N, g = case["N"], case["g"]
    H, Hd, L, _ = q.build_dimer(N, J, U0, E0, A, g, 1.0, 1)
    L = np.asarray(L).reshape(N + 1, N + 1)
    return H - 0.5j * (g / N) * (L.conj().T @ L), Hd, L, H + E0 * Hd


def _weights(N, rng):
    return rng.dirichlet(np.ones(N + 1))


def _mixture(N, rng):
    """f-vector of a random mixture of Fock states (a density matrix)."""
    p = _weights(N, rng)
    return sum(p[k] * q.fbasis_pure_state(N, k) for k in range(N + 1))


def _tree_args(case, seed):
    rng = np.random.default_rng(seed)
    return case["N"], J, rng.uniform(0.1, 0.7), rng.uniform(0.0, 2.0), A, 10.0 ** rng.uniform(-1.5, -0.5), 1.0, DEEP


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind, N = case["kind"], case.get("N")
    if kind == "qj":
        H, Hd, L, Ut = _dimer(N, U0, E0, case["g"])
        eng = q.Engine(Ut, L, [1.0], H + E0 * Hd, None, T2PI, case["n"], seed=seed, max_dumps=1 + case["periods"],
                       precision=case["precision"], record=case["record"], rec_cap=256)
        return dict(kind=kind, eng=eng, psi=_coherent(N, case["n"], rng), periods=case["periods"])
    if kind == "batch":
        ens, dims, n = [], _batch_dims(case), case["n"]
        dmax = max(N_ for N_, _, _ in dims) + 1
        psi = np.zeros((len(dims) * n, dmax), np.complex128)
        for i, (N_, E, g) in enumerate(dims):
            H, Hd, L, Ut = _dimer(N_, U0, E, g)
            ens.append(dict(U=Ut, L=L, g=[1.0], HE=H + E * Hd, n_traj=n, T=T2PI, seed=seed, tr_base=i * n))
            psi[i * n:(i + 1) * n, :N_ + 1] = _coherent(N_, n, rng)
        eng = q.Engine.batch(ens, deep=DEEP, max_dumps=2, precision=case["precision"])
        return dict(kind="qj", eng=eng, psi=psi, periods=1)
    if kind == "lpn":
        ens, n = [], case["n"]
        for i in range(case["M"]):
            H, Hd, L, Ut = _dimer(N, 0.01 * (i + 1), E0, 0.1)
            R = np.diag(np.linspace(-1.0, 1.0, N + 1)).astype(np.complex128)[None]
            ens.append(dict(U=Ut, L=L, g=[1.0], HE=H + E0 * Hd, R=R, n_traj=n, T=T2PI, seed=seed, tr_base=i * n))
        eng = q.Engine.batch(ens, deep=DEEP, max_dumps=1)
        return dict(kind=kind, eng=eng, psi=_coherent(N, n * case["M"], rng))
    if kind == "rk":
        He, Hd, L, HE = _rk_ops(case)
        eng = q.Engine.rk(He, Hd, L, [1.0], HE, None, T2PI, case["n"], E0=E0, A=A, rk_ns=case["ns"],
                          drv_type=case["drv_type"], seed=seed, max_dumps=2)
        return dict(kind="qj", eng=eng, psi=_coherent(N, case["n"], rng), periods=1)
    if kind == "fbasis":
        from scipy.sparse import csr_matrix

        (gr, gc, gv), (qr, qc, qv), ks = q.fb_build_dimer(N, J, U0, E0, 0.1)
        m = len(ks)
        fb = q.FBasis(csr_matrix((gv, gc, gr), (m, m)), csr_matrix((qv, qc, qr), (m, m)), ks, _mixture(N, rng), A,
                      drv_type=case["drv_type"], T=T2PI, num_steps=case["steps"])
        return dict(kind=kind, fb=fb)
    if kind == "purity":
        eye = np.eye(N + 1, dtype=np.complex128)
        eng = q.Engine(eye[None, None], eye, [1.0], eye, None, T2PI, case["n"], seed=seed)
        eng.set_states(_coherent(N, case["n"], rng))
        return dict(kind=kind, eng=eng)
    return dict(kind=kind, args=_tree_args(case, seed))


# ---------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind == "qj":  # an ensemble from given states: start values, the periods with their dumps, read back
        eng, P = state["eng"], state["periods"]
        eng.set_states(state["psi"])
        eng.init_thresholds()
        eng.reset_times()
        eng.observe(0, is_start=True)
        eng.run_periods(P, is_obs=1, dump_at=list(range(1, P + 1)), dump_base=1)
        obs = eng.observables(0, 1 + P)
        psi, t, eta, jumps = eng.states()
        return [obs["norm"], obs["mean"], obs["dispersion"], obs["m2"], obs["energy"], psi, t, eta]
    if kind == "lpn":  # perturb the variations, one period, the Lyapunov update
        eng = state["eng"]
        eng.set_states(state["psi"])
        eng.init_thresholds()
        eng.lpn_start(lpn_type=0)
        eng.reset_times()
        eng.run_periods(1)
        eng.lpn_period(T2PI)
        v = eng.lpn_values()
        return [v["lambda"], v["delta_s"], v["mean_lpn"], v["energy_lpn"], v["robs_lpn"], v["num_renorms"],
                eng.states()[0]]
    if kind == "fbasis":
        state["fb"].run(0, 1)
        return state["fb"].get()[0]
    if kind == "purity":
        p, rho = state["eng"].purity(want_rho=True)
        return [p, rho]
    H, Hd, L, Ut = q.build_dimer_gpu(*state["args"])
    return [H, Hd, L, Ut]


# ---------------------------------------------------------------- work that a pass cannot do without
def _matvecs(N, g):
    """Matrix-vector products per trajectory and period: the jump rate (about 0.5 N g / 0.1 jumps a period)
    times the split levels a located jump walks through and back (about 22 products)."""
    return 4.0 + 22.0 * 5.0 * g * N


def work(case):
    kind, N = case["kind"], case.get("N")
    if kind == "qj":
        d, n, P = N + 1, case["n"], case["periods"]
        return {"bytes": 16.0 * ((2 * DEEP + 2) * d * d + 2 * n * d), "flops": 8.0 * d * d * n * P * _matvecs(N, case["g"])}
    if kind == "batch":
        n, b, f = case["n"], 0.0, 0.0
        for N_, _, g in _batch_dims(case):
            d = N_ + 1
            b += 16.0 * ((2 * DEEP + 2) * d * d + 2 * n * d)
            f += 8.0 * d * d * n * _matvecs(N_, g)
        return {"bytes": b, "flops": f}
    if kind == "lpn":
        d, n, M = N + 1, case["n"], case["M"]
        return {"bytes": 16.0 * M * ((2 * DEEP + 3) * d * d + 2 * n * d),
                "flops": 8.0 * d * d * n * M * (_matvecs(N, 0.1) + 40.0)}
    if kind == "rk":
        d, n = N + 1, case["n"]
        return {"bytes": 16.0 * (4 * d * d + 2 * n * d), "flops": 8.0 * d * d * n * 8.0 * case["ns"]}
    if kind == "fbasis":
        m = (N + 1) ** 2 - 1
        nnz = 18.0 * (N + 1) ** 2
        return {"bytes": 12.0 * nnz + 24.0 * m, "flops": 8.0 * case["steps"] * (nnz + 4.0 * m)}
    if kind == "purity":
        d, n = N + 1, case["n"]
        return {"bytes": 16.0 * (n * d + d * d), "flops": 8.0 * d * d * n}
    d = N + 1
    return {"bytes": 16.0 * 2 * (1 + DEEP) * d * d, "flops": 2.0 * (14 + DEEP) * 8.0 * d ** 3}


# ---------------------------------------------------------------- plain 64-bit values
def _philox(seed, stream, draws):
    """[len(stream)][draws] uniforms in (0, 1]: Philox4x32-10 under key `seed`, two draws per block."""
    m32 = np.uint64(0xFFFFFFFF)
    nb = (draws + 1) // 2
    st = np.asarray(stream, np.uint64)[:, None]
    blk = np.arange(nb, dtype=np.uint64)[None, :]
    c = [np.broadcast_to(x, (len(stream), nb)).copy() for x in (blk & m32, blk >> np.uint64(32), st & m32,
                                                              st >> np.uint64(32))]
    k0, k1 = seed & 0xFFFFFFFF, (seed >> 32) & 0xFFFFFFFF
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ np.uint64(k0), p1 & m32, (p0 >> np.uint64(32)) ^ c[3] ^ np.uint64(k1), p0 & m32]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    u = np.empty((len(stream), nb, 2))
    for j in range(2):
        u[:, :, j] = (((c[2 * j] >> np.uint64(5)) << np.uint64(26) | (c[2 * j + 1] >> np.uint64(6))) + np.uint64(1)) * 2.0 ** -53
    return torch.from_numpy(u.reshape(len(stream), 2 * nb)[:, :draws]).cuda()


def _plain_ops(N, U):
    """H, H_drv and L of the dimer, from their definition (row k: k bosons on one site, N - k on the other)."""
    k = np.arange(N + 1.0)
    s = np.sqrt((N - k[:N]) * (k[:N] + 1.0))
    H = np.diag(2.0 * U / N * (k * (k - 1.0) + (N - k) * (N - k - 1.0)))
    H = H - J * (np.diag(s, 1) + np.diag(s, -1))
    L = np.diag(2.0 * k - N) + np.diag(s, 1) - np.diag(s, -1)
    return tuple(x.astype(np.complex128) for x in (H, np.diag(N - 2.0 * k), L))


def _plain_tree(N, U, E, drive, g):
    """[2][deep] matrix exponentials of -i (H + (E +- drive) H_drv) - (g / 2 N) L^+ L."""
    H, Hd, L = (torch.from_numpy(x).cuda() for x in _plain_ops(N, U))
    K = [-1j * (H + e * Hd) - 0.5 * (g / N) * (L.conj().T @ L) for e in (E + drive, E - drive)]
    return torch.stack([torch.stack([torch.linalg.matrix_exp(k * (T2PI * 2.0 ** -(l + 2))) for l in range(DEEP)])
                        for k in K])


class _Observer:
    """norm, mean, dispersion, m2 and energy of the states, one column per trajectory."""

    def __init__(self, HE, n, dumps):
        self.HE = HE  # [ensembles][d][d], transposed
        self.v = torch.zeros(5, dumps, n, dtype=torch.float64, device="cuda")
        self.start = torch.zeros(n, dtype=torch.float64, device="cuda")

    def take(self, dump, psi, ens, rows):
        if rows.numel() == 0:
            return
        x = psi[rows]
        k = torch.arange(x.shape[1], dtype=torch.float64, device="cuda")
        p = x.real ** 2 + x.imag ** 2
        nrm = p.sum(1)
        p = p / nrm[:, None]
        mean = (p * k).sum(1)
        en = torch.empty_like(mean)
        for e in range(self.HE.shape[0]):
            at = ens[rows] == e
            y = x[at] @ self.HE[e]
            en[at] = (x[at].conj() * y).sum(1).real / nrm[at]
        if not torch.is_tensor(dump):  # the start
            self.start[rows] = mean
            dump = torch.full_like(rows, dump)
        m2 = (p * (k[None, :] - mean[:, None]) ** 2).sum(1)
        for i, w in enumerate((nrm, mean, (mean - self.start[rows]) ** 2, m2, en)):
            self.v[i, dump, rows] = w


def _solve(ensembles, psi, n, seed, periods):
    """The quantum-jump path of every ensemble (N, E, g) from psi, all trajectories in
    lock step: the split tree's bisection with the time inside a branch counted in finest steps.  One
    matrix product per step over all matrices, the trajectories gathered by matrix."""
    E, dmax = len(ensembles), psi.shape[1]
    G = 2 * DEEP + 1
    MT = torch.zeros(E * G, dmax, dmax, dtype=torch.complex128, device="cuda")
    HE = torch.zeros(E, dmax, dmax, dtype=torch.complex128, device="cuda")
    for e, (N, drive0, g) in enumerate(ensembles):
        d = N + 1
        H, Hd, L = _plain_ops(N, U0)
        MT[e * G:e * G + 2 * DEEP, :d, :d] = _plain_tree(N, U0, drive0, A, g).reshape(2 * DEEP, d, d).transpose(1, 2)
        MT[e * G + 2 * DEEP, :d, :d] = torch.from_numpy(L).cuda().T
        HE[e, :d, :d] = torch.from_numpy(H + drive0 * Hd).cuda().T
    nt = psi.shape[0]
    ar = torch.arange(nt, device="cuda")
    ens = torch.repeat_interleave(torch.arange(E, device="cuda"), n)
    psi = torch.from_numpy(psi).cuda()
    draws = 2048
    u = _philox(seed, np.arange(nt), draws)
    pos = torch.ones_like(ar)
    eta = u[:, 0].clone()
    zero = torch.zeros_like(ar)
    b, lvl, tau, pc, rec = zero.clone(), zero.clone(), zero.clone(), zero.clone(), zero.bool()
    ctz = torch.zeros(2 ** DEEP + 1, dtype=torch.int64)
    for s in range(1, DEEP + 1):
        ctz[:: 2 ** s] = s
    ctz = ctz.cuda()
    obs = _Observer(HE, nt, 1 + periods)
    obs.take(0, psi, ens, ar)
    step = 0
    while True:
        live = pc < periods
        g = ens * G + torch.where(rec, 2 * DEEP, b * DEEP + lvl)
        g = torch.where(live, g, E * G)
        order = torch.argsort(g)
        gs = g[order]
        counts = torch.bincount(gs, minlength=E * G + 1)
        c = int(counts[:-1].max())
        if c == 0:
            break
        first = torch.cumsum(counts, 0) - counts
        rank = ar - first[gs]
        keep = gs < E * G
        gi, ri, oi = gs[keep], rank[keep], order[keep]
        X = torch.zeros(E * G, -(-c // 4) * 4, dmax, dtype=torch.complex128, device="cuda")
        X[gi, ri] = psi[oi]
        y = psi.clone()
        y[oi] = torch.bmm(X, MT)[gi, ri]
        nrm = (y.real ** 2 + y.imag ** 2).sum(1)
        cross = live & ~rec & (nrm <= eta)
        jump = cross & (lvl == DEEP - 1)
        done = live & (rec | (~rec & ~cross))  # a step of its level completed
        scale = torch.where(jump | (live & rec), 1.0 / torch.sqrt(nrm), torch.ones_like(nrm))
        psi = torch.where((live & ~cross | jump)[:, None], y * scale[:, None], psi)
        # the jump's two draws: its channel (one channel: unused), then the new threshold
        fin = live & rec
        eta = torch.where(fin, u[ar, (pos + 1).clamp(max=draws - 1)], eta)
        pos = pos + 2 * fin
        tau = tau + torch.where(done, 2 ** (DEEP - 1 - lvl), zero)
        lvl = torch.where(done, DEEP - 1 - ctz[tau].clamp(max=DEEP - 1), lvl + (cross & ~jump).long())
        rec = jump
        end = tau == 2 ** DEEP
        tau, lvl = torch.where(end, zero, tau), torch.where(end, zero, lvl)
        b = b + end
        per = b == 2
        b, pc = torch.where(per, zero, b), pc + per
        step += 1
        rows = torch.nonzero(per).flatten()
        obs.take(pc[rows], psi, ens, rows)
    if int(pos.max()) >= draws:
        return None
    return [obs.v[i].cpu().numpy() for i in range(5)] + [psi.cpu().numpy(), np.full(nt, T2PI * periods), eta.cpu().numpy()]


def _solve_rk(case, psi, seed):
    """RK4 of dpsi/dt = -i (H_eff + E(t) H_drv) psi with the located jumps of the RK propagator (the stage
    arguments use the whole step also inside a part of one)."""
    H, Hd, L = _plain_ops(case["N"], U0)
    He = H - 0.5j * (case["g"] / case["N"]) * (L.conj().T @ L)
    He, Hd, L, HE = (torch.from_numpy(x).cuda().T.contiguous() for x in (He, Hd, L, H + E0 * Hd))
    n, ns = psi.shape[0], case["ns"]
    h0 = T2PI / ns
    psi = torch.from_numpy(psi).cuda()
    draws = 1024
    u = _philox(seed, np.arange(n), draws)
    ar = torch.arange(n, device="cuda")
    pos = torch.ones_like(ar)
    eta = u[:, 0].clone()
    obs = _Observer(HE[None], n, 2)
    ens = torch.zeros_like(ar)
    obs.take(0, psi, ens, ar)

    def drive(t):
        if case["drv_type"] == 1:
            return E0 + A * torch.sin(t)
        return torch.where(torch.fmod(t, T2PI) < T2PI * 0.5, E0 + A, E0 - A)

    def step(x, t, h):
        """The step's result (h: per row) and the time after it."""
        def f(a, s):
            return -1j * (a @ He + drive(s)[:, None] * (a @ Hd))

        k1 = f(x, t)
        k2 = f(x + 0.5 * h0 * k1, t + 0.5 * h)
        k3 = f(x + 0.5 * h0 * k2, t + 0.5 * h)
        k4 = f(x + h0 * k3, t + h)
        return x + (k1 + 2 * k2 + 2 * k3 + k4) * (h / 6.0)[:, None], t + h

    def square(x):
        return (x.real ** 2 + x.imag ** 2).sum(1)

    for s in range(ns):
        rows, x = ar, psi
        t = torch.full((n,), s * h0, dtype=torch.float64, device="cuda")
        h = torch.full_like(t, h0)
        prev = square(x)
        while True:
            y, _ = step(x, t, h)
            nrm = square(y)
            ok = nrm > eta[rows]
            psi[rows[ok]] = y[ok]
            bad = ~ok
            if not bool(bad.any()):
                break
            rows, x, t, h, prev, nrm = rows[bad], x[bad], t[bad], h[bad], prev[bad], nrm[bad]
            part = (prev - eta[rows]) / (prev - nrm)
            x, t = step(x, t, h * part)
            x = x @ L
            x = x / torch.sqrt(square(x))[:, None]
            eta[rows] = u[rows, pos[rows] + 1]
            pos[rows] += 2
            h, prev = h * (1.0 - part), square(x)
    obs.take(torch.ones_like(ar), psi, ens, ar)
    # states and thresholds of the trajectories that decay slowest keep no digit: a jump time is the
    # interpolated crossing of a nearly constant norm, and each jump multiplies its rounding
    return [obs.v[i].cpu().numpy() for i in range(5)] + [None, None, None]


def _solve_fbasis(case, seed):
    """The same Lindblad equation on the density matrix: RK4 of d rho/dt, then its Gell-Mann coordinates."""
    N, d = case["N"], case["N"] + 1
    H, Hd, L = (torch.from_numpy(x).cuda() for x in _plain_ops(N, U0))
    H = H + E0 * Hd
    gamma, LdL = 0.1 / N, L.conj().T @ L
    rho = torch.diag(torch.from_numpy(_weights(N, np.random.default_rng(seed)))).to(torch.complex128).cuda()
    h = T2PI / case["steps"]

    def f(r, t):
        s = math.sin(t)
        e = A * (s if case["drv_type"] == 1 else (-1.0 if s < 0.0 else 1.0))
        K = -1j * (H + e * Hd) - 0.5 * gamma * LdL
        return (K @ r + r @ K.conj().T + gamma * (L @ r @ L.conj().T)) * h

    for i in range(case["steps"]):
        t = i * h
        k1 = f(rho, t)
        k2 = f(rho + k1 / 2, t + h / 2)
        k3 = f(rho + k2 / 2, t + h / 2)
        k4 = f(rho + k3, t + h)
        rho = rho + (k1 + 2 * k2 + 2 * k3 + k4) / 6
    r = rho.cpu().numpy()
    up = r[np.triu_indices(d, 1)] * math.sqrt(2.0)
    p, m = np.diag(r).real, np.arange(N)
    diag = (np.cumsum(p)[:N] - (m + 1) * p[1:]) / np.sqrt((m + 1.0) * (m + 2.0))
    return np.concatenate([np.stack([up.real, up.imag], 1).reshape(-1), diag])


def exact(case, seed):
    rng = np.random.default_rng(seed)
    kind, N = case["kind"], case.get("N")
    if kind in ("qj", "batch"):
        # split precision leaves the 64-bit path at the first decision its rounding flips, a period at most
        if case["precision"]:
            return None
        dims = _batch_dims(case) if kind == "batch" else [(N, E0, case["g"])]
        n = case["n"]
        dmax = max(N_ for N_, _, _ in dims) + 1
        psi = np.zeros((len(dims) * n, dmax), np.complex128)
        for i, (N_, _, _) in enumerate(dims):
            psi[i * n:(i + 1) * n, :N_ + 1] = _coherent(N_, n, rng)
        return _solve(dims, psi, n, seed, case["periods"] if kind == "qj" else 1)
    if kind == "lpn":  # the perturbation's size is searched to a tolerance: it has no 64-bit value
        return None
    if kind == "rk":
        return _solve_rk(case, _coherent(N, case["n"], rng), seed)
    if kind == "fbasis":
        return _solve_fbasis(case, seed)
    if kind == "purity":
        x = torch.from_numpy(_coherent(N, case["n"], rng)).cuda()
        x = x / torch.sqrt((x.real ** 2 + x.imag ** 2).sum(1))[:, None]
        rho = (x.T @ x.conj()) / case["n"]
        return [float((rho.real ** 2 + rho.imag ** 2).sum()), rho.cpu().numpy()]
    _, _, U, E, drive, g, _, _ = _tree_args(case, seed)
    return [*_plain_ops(N, U), _plain_tree(N, U, E, drive, g).cpu().numpy()]
