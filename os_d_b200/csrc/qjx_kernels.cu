// qjx_kernels.cu -- sm_100a kernels of the QJ trajectory engine.
//
// The reference advances one trajectory at a time through a recursive bisection over
// split levels (qj_proc.cpp:271-343): every step is one dense complex matvec with the
// propagator U[b][level] of its branch and level, followed by a norm test against the
// trajectory's threshold.  Jumps are frequent (about 50 per period at N = 100 and 110 at
// N = 200), so the bisection, not the jump-free stroboscopic step, is the hot path.
//
// B200 design: every active trajectory needs one matvec at a time, with one of G matrices (2 x
// ex_deep propagators, the jump operators, the energy operator, the random observables).  The
// trajectories wait in one queue per matrix, and the CTAs of a persistent kernel are independent
// workers: a CTA takes up to 32 trajectories from the fullest queue, multiplies them by that
// queue's matrix, runs the state machine on each, appends each to the queue of its next matrix
// and takes the next batch.  No CTA waits for another, so there is no lock-step, no grid barrier
// and no plan:
//   * a sub-tile is one matrix x 8, 16 or 32 trajectory columns, full height (all d rows), so the
//     column norm needed by the jump test stays inside the CTA;
//   * the gathered state columns and the propagator K-slabs are copied to shared memory with cp.async,
//     two slabs in turn, so the tensor pipe is fed while the next slab streams from L2;
//   * the epilogue is the whole trajectory state machine: norm test, descend / accept,
//     jump record, renormalisation, channel choice, threshold redraw, time bookkeeping,
//     period and dump accounting and the observables.
// FP64 has no tcgen05 kind, so the plain form's contraction runs on the FP64 tensor core
// (mma.sync m8n8k4 f64), laid out so that every output keeps the oracle's k-ascending fma
// chain (bit-identical results).  The split-precision form (qjx_split.cuh, included at the
// end) runs the same queues with bf16x3 products on the tcgen05 tensor cores.
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "qjx_device.cuh"

namespace qjx {

constexpr long long kWaitLimit = 1ll << 24;  // bounded mbarrier polls before giving up

__device__ __forceinline__ double2 *slot_ptr(const Params &P, int slot, int tr)
{
    return P.psi + ((size_t)slot * P.n + tr) * P.MD;
}

// What the state machine needs of a trajectory's ensemble: dimension, first group, split-level steps
// [nb][deep] and jump rates.
struct Ens {
    int d, g0;
    const double *dt, *rate;
};

__device__ __forceinline__ Ens global_ens(const Params &P, int e)
{
    return Ens{P.e_d[e], e * P.Ge, P.e_dt + (size_t)e * P.nb * P.deep, P.e_rate + (size_t)e * P.nd};
}

// The state slots of one trajectory: in P.psi, or a copy in shared memory.
struct Slots {
    double2 *base;
    size_t stride;
    __device__ __forceinline__ double2 *operator()(int slot) const { return base + slot * stride; }
};

__device__ __forceinline__ Slots global_slots(const Params &P, int tr)
{
    return Slots{slot_ptr(P, 0, tr), (size_t)P.n * P.MD};
}

// Whether run calls advance trajectory tr.
__device__ __forceinline__ bool runs(const Params &P, int tr)
{
    return tr < P.n_active && (!P.active || P.active[tr]);
}

// Bucket (global group) of a trajectory's next matvec, or -1.
__device__ __forceinline__ int group_of(const Params &P, const TrajState &s)
{
    int g;
    switch (s.phase) {
    case PH_STEP: g = s.b * P.deep + s.lvl; break;
    case PH_REC_W:
    case PH_REC_A: g = P.gL0 + s.sub; break;
    case PH_OBS_E: g = P.gHE; break;
    case PH_OBS_R: g = P.gR0 + s.sub; break;
    case PH_RK: g = s.rk_part; break;  // group 0 H_eff, group 1 H_drv
    default: return -1;
    }
    return P.e_g0[s.ens] + g;
}

// Slot holding the input vector of a trajectory's next matvec: psi, the normalised copy for
// the observables, or the RK stage argument.
__device__ __forceinline__ int src_slot(int phase, int cur, int rk_stage)
{
    if (phase == PH_RK) return rk_stage == 1 ? cur : kSlotArgs;
    return (phase == PH_OBS_E || phase == PH_OBS_R) ? (cur ^ 1) : cur;
}

// ---------------------------------------------------------------- RK propagator helpers
// E(t) of rk_right_part_dimer (core.cpp:11073-11103)
__device__ __forceinline__ double rk_drive(const Params &P, double t)
{
    if (P.drv_type == 1)
        return __dadd_rn(P.E0, __dmul_rn(P.A, sin(__dadd_rn(__dmul_rn(P.drv_freq, t), P.drv_phase))));
    const double mod_time = fmod(t, P.T), half_T = __dmul_rn(P.T, 0.5);
    return (mod_time < half_T) ? __dadd_rn(P.E0, P.A) : __dsub_rn(P.E0, P.A);
}

// Start time of step rk_sid of the current period (rk_period, core.cpp:446)
__device__ __forceinline__ double rk_step_time(const Params &P, const TrajState &s)
{
    return __dadd_rn(__dmul_rn((double)(P.period0 + s.pc), P.T), __dmul_rn((double)s.rk_sid, P.rk_step));
}

// Begin an RK step of size h from psi (slot cur) with norm prev; returns its first matvec's group.
__device__ __forceinline__ int rk_begin(TrajState &s, double h, double prev, int ctx)
{
    s.phase = PH_RK;
    s.rk_h = h;
    s.rk_prev = prev;
    s.rk_stage = 1;
    s.rk_part = 0;
    s.rk_ctx = ctx;
    return 0;
}

// Queue entry of a trajectory: its index and the slot of its next matvec's input, so that the copy
// of the input need not wait for the trajectory's record.
__device__ __forceinline__ unsigned entry_of(int tr, const TrajState &s)
{
    return ((unsigned)tr << 3) | (unsigned)src_slot(s.phase, s.cur, s.rk_stage);
}

// Appends trajectory tr to bucket g before a run: to its queue (whose entries past the tail are
// free), or the lock-step lists of step 0.
__device__ __forceinline__ void enqueue(const Params &P, int g, int tr)
{
    if (!P.flow) {
        const int pos = atomicAdd(&P.cnt[g], 1);
        P.lists[P.g_loff[g] + pos] = tr;
    } else {
        const unsigned pos = atomicAdd(&P.q[g].tail, 1u);
        P.ring[P.gd[g].roff + (pos & P.gd[g].rmask())] = entry_of(tr, P.st[tr]);
        atomicAdd(&P.q[g].avail, 1);
        atomicAdd(P.ctrl + kLive, 1);
        atomicAdd(P.left + P.st[tr].ens / P.sect_ens, 1);
    }
}

__device__ __forceinline__ void report_error(const Params &P, int tr, int code)
{
    if (atomicAdd(&P.ctrl[0], 1) == 0) {
        P.ctrl[1] = tr;
        P.ctrl[3] = code;
    }
}

// Counter bookkeeping after a completed step at level s.lvl (qj_proc.cpp:317-320, 330-338):
// advance the level's counter; a level that finished both steps returns to its parent,
// which undoes and redoes its own time advance (t -= dt; t += dt) and counts its step.
// Returns 0 inside a unit (two level-0 steps), 1 when a unit finished, 2 when the last unit
// of the last branch of a period finished.  A branch has brep units (1, or 2 deep_num_steps
// for the deep tasks, whose sub-period is two units: one_sub_period_deep, qj_proc.cpp:345-359).
__device__ __forceinline__ int advance(TrajState &s, const double *dt, int nb, int brep)
{
    int l = s.lvl;
    unsigned long long m = s.mask;
    while (true) {
        if (!((m >> l) & 1ull)) {
            m |= (1ull << l);
            s.lvl = l;
            s.mask = m;
            return 0;
        }
        m &= ~(1ull << l);
        if (l == 0) {
            s.mask = m;
            s.lvl = 0;
            if (++s.rk_sid < brep) return 1;
            s.rk_sid = 0;
            s.b += 1;
            if (s.b == nb) {
                s.b = 0;
                return 2;
            }
            return 1;
        }
        l -= 1;
        s.t = __dadd_rn(__dsub_rn(s.t, dt[l]), dt[l]);
    }
}

// |psi_k|^2 / norm as mult_scalar_double(mult_scalar_complex(phi, phi, 1), 1/norm).real
// (core.cpp:665-725), recomputed wherever it is needed (no scratch array)
__device__ __forceinline__ double adr_of(double2 v, double inv)
{
    return __dmul_rn(__dadd_rn(0.0, __dadd_rn(__dmul_rn(v.x, v.x), __dmul_rn(v.y, v.y))), inv);
}

// Observables of the state held in `col` (calc_chars_std[_start], core.cpp:665-725) and
// the normalised state psi / sqrt(norm) written to the spare slot for the energy and
// random-observable matvecs.  Warp-cooperative; every lane computes the sequential
// sums identically.
__device__ void obs_prep(const Params &P, const TrajState &s, int tr, const Ens &sys, const Slots &slots, const double2 *col, int lane,
                         int dump, int is_start)
{
    const int d = sys.d;
    const double nrm = warp_norm(col, d, lane);
    const double sq = __dsqrt_rn(nrm);
    const double inv = __ddiv_rn(1.0, nrm);
    double2 *hat = slots(s.cur ^ 1);
    double *adr_out = !P.o_adr ? nullptr
                      : (P.keep_adr ? P.o_adr + ((size_t)dump * P.n + tr) * P.d : P.o_adr + (size_t)tr * P.d);
    for (int k = lane; k < d; k += 32) {
        const double2 v = col[k];
        hat[k] = make_double2(__ddiv_rn(v.x, sq), __ddiv_rn(v.y, sq));
        if (adr_out) adr_out[k] = adr_of(v, inv);
    }
    double mean = 0.0;
    for (int k = lane; k < d; k += 32) mean = __dadd_rn(mean, __dmul_rn((double)k, adr_of(col[k], inv)));
    mean = warp_allsum(mean);
    const double ms = is_start ? mean : P.mean_start[tr];
    const double disp = __dmul_rn(__dsub_rn(mean, ms), __dsub_rn(mean, ms));
    double m2 = 0.0;
    for (int k = lane; k < d; k += 32) {
        const double dk = __dsub_rn((double)k, mean);
        m2 = __dadd_rn(m2, __dmul_rn(__dmul_rn(dk, dk), adr_of(col[k], inv)));
    }
    m2 = warp_allsum(m2);
    if (lane == 0) {
        const size_t o = (size_t)dump * P.n + tr;
        if (is_start) P.mean_start[tr] = mean;
        P.o_norm[o] = nrm;
        P.o_mean[o] = mean;
        P.o_disp[o] = disp;
        P.o_m2[o] = m2;
    }
    __syncwarp();
}

// Continue after a completed split step: period / dump / target bookkeeping.  Returns the
// next group, or -1 when the trajectory is done for this call.
__device__ int after_step(const Params &P, TrajState &s, int tr, const Ens &sys, const Slots &slots, const double2 *col, int lane)
{
    const int a = advance(s, (sys.dt + s.b * P.deep), P.nb, P.brep);
    if (a == 2) s.pc += 1;
    if (a >= 1 && P.subdump && (s.rk_sid & 1) == 0) {  // deep task: a sub-period ended
        obs_prep(P, s, tr, sys, slots, col, lane, P.dump_base + s.di, 0);
        s.phase = PH_OBS_E;
        return P.gHE;
    }
    if (a == 2) {
        if (s.di < P.n_dumps && s.pc == P.dump_at[s.di]) {
            obs_prep(P, s, tr, sys, slots, col, lane, P.dump_base + s.di, 0);
            s.phase = PH_OBS_E;
            return P.gHE;
        }
        if (s.pc >= P.target) {
            s.phase = PH_DONE;
            return -1;
        }
    }
    return s.b * P.deep + s.lvl;
}

__device__ int finish_obs(const Params &P, TrajState &s)
{
    s.di += 1;
    if (s.pc >= P.target || (P.sub_target > 0 && s.di >= P.sub_target)) {
        s.phase = PH_DONE;
        return -1;
    }
    if (P.prop == 1) {  // next RK step of the period
        s.t = rk_step_time(P, s);
        return rk_begin(s, P.rk_step, s.rk_prev, 0);
    }
    s.phase = PH_STEP;
    return s.b * P.deep + s.lvl;
}

// An RK step finished without crossing (rk_period, core.cpp:443-449): next step, period and dump
// bookkeeping.  `col` holds psi, nrm its norm.
__device__ int rk_after_step(const Params &P, TrajState &s, int tr, const Ens &sys, const Slots &slots, const double2 *col, int lane,
                             double nrm)
{
    s.rk_prev = nrm;
    s.rk_sid += 1;
    if (s.rk_sid == P.rk_ns) {
        s.rk_sid = 0;
        s.pc += 1;
        if (s.di < P.n_dumps && s.pc == P.dump_at[s.di]) {
            obs_prep(P, s, tr, sys, slots, col, lane, P.dump_base + s.di, 0);
            s.phase = PH_OBS_E;
            return P.gHE;
        }
        if (s.pc >= P.target) {
            s.phase = PH_DONE;
            return -1;
        }
    }
    s.t = rk_step_time(P, s);
    return rk_begin(s, P.rk_step, nrm, 0);
}

// Apply the chosen jump channel: psi = (L_idx psi_hat) / sqrt(w_idx / g_idx)
// (experiment.cpp:1346-1369), record the channel, redraw eta (qj_proc.cpp:310-314) and
// count the finest-level step.
__device__ int apply_jump(const Params &P, TrajState &s, int tr, const Ens &sys, const Slots &slots, double2 *col, int lane, int idx,
                          double w_idx, int *err)
{
    const int d = sys.d;
    const double q = __dsqrt_rn(__ddiv_rn(w_idx, sys.rate[idx]));
    double2 *dst = slots(s.cur ^ 1);
    for (int k = lane; k < d; k += 32) {
        const double2 v = col[k];
        const double2 r = make_double2(__ddiv_rn(v.x, q), __ddiv_rn(v.y, q));
        dst[k] = r;
        col[k] = r;
    }
    __syncwarp();
    s.cur ^= 1;
    if (P.record && lane == 0) P.r_type[(size_t)(s.nrec - 1) * P.n + tr] = idx;
    s.eta = draw(P, tr, s, err);
    while (s.eta == 0.0 && *err == 0) s.eta = draw(P, tr, s, err);
    if (*err) return -1;
    if (P.prop == 1) {  // the end part of the interrupted RK step (rk_step_dimer, core.cpp:11946)
        const double nrm = warp_norm(col, d, lane);
        return rk_begin(s, s.rk_end, nrm, 0);
    }
    s.phase = PH_STEP;
    s.t = __dadd_rn(s.t, (sys.dt + s.b * P.deep)[P.deep - 1]);
    return after_step(P, s, tr, sys, slots, col, lane);
}

// Warp-cooperative epilogue of one trajectory column: `col` holds M_g * psi in shared memory,
// `s_in` the trajectory's state record (loaded by the caller), `sys` its ensemble, `slots` its states; the new record
// goes to `out`.  Returns the bucket of the trajectory's next micro-step, or -1 (done, paused or
// failed), and its queue entry in `entry`; the caller appends it.  `lead` is false in all but one of
// several CTAs that run the same column.
__device__ int column_epilogue(const Params &P, double2 *col, int tr, const TrajState &s_in, int lane, unsigned &entry,
                               const Ens &sys, const Slots &slots, TrajState *out, bool lead)
{
    const int d = sys.d;
    TrajState s = s_in;
    int g2 = -1;
    int err = 0;
    bool paused = false;

    switch (s.phase) {
    case PH_STEP: {
        const double nrm = warp_norm(col, d, lane);
        // is_norm_crossed throws (experiment.cpp:1247-1251); the split-precision form allows its
        // matvec rounding (a few 1e-6 of the norm) above 1 before calling it an error
        if (nrm > (P.split ? 1.0 + kSplitNormSlack : 1.0)) {
            err = ERR_NORM;
            break;
        }
        // split form: a norm within the split error of the threshold is not decided here; the
        // same step is computed again in FP64 and decides (the recheck itself clears the flag)
        const bool rechecked = s.rechk != 0;
        s.rechk = 0;
        if (P.split && P.recheck_tol > 0.0 && !rechecked && fabs(nrm - s.eta) <= P.recheck_tol * nrm) {
            s.rechk = 1;
            g2 = kRecheck;
            break;
        }
        const double dt = (sys.dt + s.b * P.deep)[s.lvl];
        if (nrm > s.eta) {  // not crossed: accept psi' (qj_proc.cpp:317, 335)
            double2 *dst = slots(s.cur ^ 1);
            for (int k = lane; k < d; k += 32) dst[k] = col[k];
            s.cur ^= 1;
            s.t = __dadd_rn(s.t, dt);
            g2 = after_step(P, s, tr, sys, slots, col, lane);
        } else if (s.lvl < P.deep - 1) {  // crossed on a coarse level: bisect from psi (qj_proc.cpp:328-331)
            s.lvl += 1;
            g2 = s.b * P.deep + s.lvl;
        } else {  // crossed on the finest level: jump (qj_proc.cpp:294-315)
            if (P.record) {
                if (s.nrec >= P.rec_cap) {  // record buffer full: hold here, host drains and resumes
                    paused = true;
                    break;
                }
                if (lane == 0) {
                    const size_t o = (size_t)s.nrec * P.n + tr;
                    P.r_time[o] = __dadd_rn(s.t, dt);
                    P.r_norm[o] = nrm;
                    P.r_eta[o] = s.eta;
                    P.r_type[o] = -1;
                }
                s.nrec += 1;
                s.jumps += 1;
            }
            // recovery: psi' /= sqrt(norm_square(psi'))  (experiment.cpp:1291-1296)
            const double sq = __dsqrt_rn(nrm);
            double2 *dst = slots(s.cur ^ 1);
            for (int k = lane; k < d; k += 32) {
                const double2 v = col[k];
                dst[k] = make_double2(__ddiv_rn(v.x, sq), __ddiv_rn(v.y, sq));
            }
            s.cur ^= 1;
            s.ran = draw(P, tr, s, &err);
            if (err) break;
            s.tmpw = 0.0;
            s.phase = PH_REC_W;
            s.sub = 0;
            g2 = P.gL0;
        }
    } break;

    case PH_REC_W: {  // gnorms[i] = norm_square(L_i psi_hat) * g[i]  (experiment.cpp:1301-1322)
        double w = warp_norm(col, d, lane);
        w = __dmul_rn(w, sys.rate[s.sub]);
        if (lane == 0) P.gn[(size_t)tr * P.nd + s.sub] = w;
        s.tmpw = __dadd_rn(s.tmpw, w);
        if (s.sub + 1 < P.nd) {
            s.sub += 1;
            g2 = P.gL0 + s.sub;
            break;
        }
        __syncwarp();
        // channel choice (experiment.cpp:1324-1344)
        const double *gn = P.gn + (size_t)tr * P.nd;
        double ran = __dmul_rn(s.ran, s.tmpw);
        // the index never passes nd - 1 (the reference's loop reads past the end when
        // nd == 1 and ran > gnorms[0], which its own draws cannot produce)
        int index = 0;
        while (index < P.nd - 1 && __dsub_rn(ran, gn[index]) > 0.0) {
            ran = __dsub_rn(ran, gn[index]);
            index++;
        }
        if (s.tmpw == 0.0) {
            err = ERR_ZERO_W;
            break;
        }
        for (int it = 0; gn[index] == 0.0; it++) {
            if (it > 2 * P.nd) { err = ERR_ZERO_W; break; }
            index = (index == 0) ? index + 1 : index - 1;
            if (index >= P.nd) { err = ERR_ZERO_W; break; }
        }
        if (err) break;
        if (P.nd == 1) {
            g2 = apply_jump(P, s, tr, sys, slots, col, lane, index, w, &err);
        } else {
            s.phase = PH_REC_A;
            s.sub = index;
            g2 = P.gL0 + index;
        }
    } break;

    case PH_REC_A: {
        const double w = P.gn[(size_t)tr * P.nd + s.sub];
        g2 = apply_jump(P, s, tr, sys, slots, col, lane, s.sub, w, &err);
    } break;

    case PH_RK: {  // one right-hand side of rk_int_dimer (core.cpp:11592-11619), col = M arg
        if (s.rk_part == 0) {  // H_eff arg, kept for the drive part
            double2 *dst = slots(kSlotND);
            for (int k = lane; k < d; k += 32) dst[k] = col[k];
            s.rk_part = 1;
            g2 = 1;
            break;
        }
        // k = -i (H_eff arg + E H_drv arg)  (core.cpp:11106-11112)
        const double E = rk_drive(P, s.t);
        const double2 *nd = slots(kSlotND);
        const double2 *phi = slots(s.cur);
        const double h = s.rk_h;
        if (s.rk_stage < 4) {
            // arg_upd (rk_proc.cpp:146-185) uses the full rk_step, also inside a begin or end part
            const double c = (s.rk_stage == 3) ? __dmul_rn(1.0, P.rk_step) : __dmul_rn(0.5, P.rk_step);
            double2 *kd = slots(kSlotK1 + s.rk_stage - 1);
            double2 *args = slots(kSlotArgs);
            for (int k = lane; k < d; k += 32) {
                const double2 a = nd[k], b = col[k], x = phi[k];
                const double kr = __dadd_rn(a.y, __dmul_rn(E, b.y)), ki = -__dadd_rn(a.x, __dmul_rn(E, b.x));
                kd[k] = make_double2(kr, ki);
                args[k] = make_double2(__dadd_rn(x.x, __dmul_rn(c, kr)), __dadd_rn(x.y, __dmul_rn(c, ki)));
            }
            if (s.rk_stage != 2) s.t = __dadd_rn(s.t, __dmul_rn(h, 0.5));
            s.rk_stage += 1;
            s.rk_part = 0;
            g2 = 0;
            break;
        }
        if (s.rk_ctx == 1 && P.record && s.nrec >= P.rec_cap) {  // record buffer full: hold here
            paused = true;
            break;
        }
        // rk_final (rk_proc.cpp:187-196): psi + (k1 + 2 k2 + 2 k3 + k4) h / 6, into col
        const double2 *k1 = slots(kSlotK1), *k2 = slots(kSlotK1 + 1);
        const double2 *k3 = slots(kSlotK1 + 2);
        for (int k = lane; k < d; k += 32) {
            const double2 a = nd[k], b = col[k], x = phi[k], p1 = k1[k], p2 = k2[k], p3 = k3[k];
            const double kr = __dadd_rn(a.y, __dmul_rn(E, b.y)), ki = -__dadd_rn(a.x, __dmul_rn(E, b.x));
            const double sr = __dadd_rn(__dadd_rn(__dadd_rn(p1.x, __dmul_rn(2.0, p2.x)), __dmul_rn(2.0, p3.x)), kr);
            const double si = __dadd_rn(__dadd_rn(__dadd_rn(p1.y, __dmul_rn(2.0, p2.y)), __dmul_rn(2.0, p3.y)), ki);
            col[k] = make_double2(__dadd_rn(x.x, __ddiv_rn(__dmul_rn(sr, h), 6.0)),
                                  __dadd_rn(x.y, __ddiv_rn(__dmul_rn(si, h), 6.0)));
        }
        __syncwarp();
        const double nrm = warp_norm(col, d, lane);
        if (s.rk_ctx == 0) {
            if (nrm > 1.0) {  // is_norm_crossed throws (experiment.cpp:1247-1251)
                err = ERR_NORM;
                break;
            }
            if (nrm > s.eta) {  // not crossed: accept psi in place
                double2 *dst = slots(s.cur);
                for (int k = lane; k < d; k += 32) dst[k] = col[k];
                g2 = rk_after_step(P, s, tr, sys, slots, col, lane, nrm);
            } else {  // crossed: integrate the begin part from psi, still in its slot (core.cpp:11913-11922)
                const double norm_diff = __dsub_rn(s.rk_prev, nrm);
                const double begin_part = __ddiv_rn(__dsub_rn(s.rk_prev, s.eta), norm_diff);
                const double end_part = __dsub_rn(1.0, begin_part);
                s.rk_end = __dmul_rn(h, end_part);
                s.t = __dsub_rn(s.t, h);
                g2 = rk_begin(s, __dmul_rn(h, begin_part), s.rk_prev, 1);
            }
        } else {  // begin part done: record the jump, rk_recovery (rk_proc.cpp:198-305)
            if (P.record) {
                if (lane == 0) {
                    const size_t o = (size_t)s.nrec * P.n + tr;
                    P.r_time[o] = s.t;
                    P.r_norm[o] = nrm;
                    P.r_eta[o] = s.eta;
                    P.r_type[o] = -1;
                }
                s.nrec += 1;
                s.jumps += 1;
            }
            const double sq = __dsqrt_rn(nrm);
            double2 *dst = slots(s.cur ^ 1);
            for (int k = lane; k < d; k += 32) {
                const double2 v = col[k];
                dst[k] = make_double2(__ddiv_rn(v.x, sq), __ddiv_rn(v.y, sq));
            }
            s.cur ^= 1;
            s.ran = draw(P, tr, s, &err);
            if (err) break;
            s.tmpw = 0.0;
            s.phase = PH_REC_W;
            s.sub = 0;
            g2 = P.gL0;
        }
    } break;

    case PH_OBS_E: {  // energy <psi_hat| H + E0 Hd |psi_hat>  (experiment.cpp:1423-1469)
        const double2 *hat = slots(s.cur ^ 1);
        double e = 0.0;
        for (int k = lane; k < d; k += 32) {
            const double2 h = hat[k], m = col[k];
            e = __dadd_rn(e, __dadd_rn(__dmul_rn(h.x, m.x), __dmul_rn(h.y, m.y)));
        }
        e = warp_allsum(e);
        if (lane == 0) P.o_energy[(size_t)(P.dump_base + s.di) * P.n + tr] = e;
        __syncwarp();
        if (P.nr > 0) {
            s.phase = PH_OBS_R;
            s.sub = 0;
            g2 = P.gR0;
        } else {
            g2 = finish_obs(P, s);
        }
    } break;

    case PH_OBS_R: {  // <psi_hat| R |psi_hat>  (experiment.cpp:2037-2068)
        const double2 *hat = slots(s.cur ^ 1);
        double rr = 0.0, ri = 0.0;
        for (int k = lane; k < d; k += 32) {
            const double2 h = hat[k], m = col[k];
            const double cr = h.x, ci = -h.y;
            rr = __dadd_rn(rr, __dsub_rn(__dmul_rn(cr, m.x), __dmul_rn(ci, m.y)));
            ri = __dadd_rn(ri, __dadd_rn(__dmul_rn(ci, m.x), __dmul_rn(cr, m.y)));
        }
        rr = warp_allsum(rr);
        ri = warp_allsum(ri);
        if (lane == 0) P.o_robs[((size_t)(P.dump_base + s.di) * P.n + tr) * P.nr + s.sub] = make_double2(rr, ri);
        __syncwarp();
        if (s.sub + 1 < P.nr) {
            s.sub += 1;
            g2 = P.gR0 + s.sub;
        } else {
            g2 = finish_obs(P, s);
        }
    } break;

    default: break;
    }

    if (err || paused) g2 = -1;
    const bool to_recheck = (g2 == kRecheck);
    if (to_recheck) g2 = -1;
    if (lane == 0) {
        if (err) {
            s.err = err;
            s.phase = PH_ERROR;
            if (lead) report_error(P, tr, err);
        } else if (paused) {
            s.paused = 1;
            if (lead) atomicAdd(&P.ctrl[2], 1);
        }
        *out = s;
    }
    __syncwarp();
    entry = entry_of(tr, s);
    if (to_recheck) return kRecheck;
    return g2 >= 0 ? sys.g0 + g2 : -1;  // local group -> the ensemble's bucket
}

// Copies a 144-byte trajectory record with 16-byte accesses.
__device__ __forceinline__ void load_state(TrajState *dst, const TrajState *src)
{
    const uint4 *s = reinterpret_cast<const uint4 *>(src);
    uint4 *t = reinterpret_cast<uint4 *>(dst);
#pragma unroll
    for (int i = 0; i < (int)(sizeof(TrajState) / 16); i++) t[i] = s[i];
}

__device__ __forceinline__ double neg(double x)
{
    return __longlong_as_double(__double_as_longlong(x) ^ (long long)0x8000000000000000ull);
}

// FP64 tensor-core MMA D = A(8x4) B(4x8) + D.  On sm_100a its accumulation equals the
// sequential chain fma(a3,b3, fma(a2,b2, fma(a1,b1, fma(a0,b0,c)))) bit for bit (checked on
// the device against that chain, the reverse chain and a single rounding), which is the
// oracle's per-output k-ascending order.
__device__ __forceinline__ void dmma(double &c0, double &c1, double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
        : "+d"(c0), "+d"(c1)
        : "d"(a), "d"(b));
}

// 16 bytes global -> shared (past L1), asynchronously; zeros where !valid (the address is not read then).
__device__ __forceinline__ void cp16(double2 *dst, const double2 *src, bool valid)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(valid ? 16 : 0)
                 : "memory");
}

__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

template <int N>
__device__ __forceinline__ void cp_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Starts the copy of slab `sl` (KS k rows from KS sl on; nothing past the last) into its half of the
// slab buffer, as one group of this thread.
template <int NT>
__device__ __forceinline__ void load_slab(const double2 *mat, double2 *Us, int sl, int kp, int KS, int MD)
{
    const int n = min(KS, kp - sl * KS) * MD;
    double2 *dst = Us + (sl & 1) * KS * MD;
    const double2 *src = mat + (size_t)sl * KS * MD;
#pragma unroll 4
    for (int i = threadIdx.x; i < n; i += NT) cp16(dst + i, src + i, true);
    cp_commit();
}

// Complex sub-tile product on the FP64 tensor core.  Rows are in 8-row blocks (RB of them,
// MD = 8 RB), columns in 8-column blocks.  For one pair of complex k the real parts use
// A = [Mr_k, Mi_k, Mr_k+1, Mi_k+1] against B = [xr_k; -xi_k; xr_k+1; -xi_k+1] and the imaginary
// parts the same A against B = [xi_k; xr_k; ...]; that is the k-ascending chain re += Mr xr;
// re -= Mi xi; im += Mr xi; im += Mi xr of the contract (the sign of a product is exact).  With
// the matrix as [k / 2][row][k % 2], lane l's A operand of row block rb is double 32 rb + l of the
// k pair: one conflict-free 256-byte read per warp and row block, no sign or select on the A side.
// (The layout [k][row] before it put the two k of a pair on the same banks: 4 shared-memory
// wavefronts a read instead of 2, about half of the pipe at d = 201.)
// The K-slabs (KS rows each, even) come through two buffers by cp.async; the caller has started the
// first.
// WPC warps share one column block; warp `sub` of them owns row blocks sub, sub + WPC, ...
//
// tile_rows: the share of a warp with exactly N row blocks, two k pairs at a time, their operands read
// together ahead of the MMAs.  With only two to four warps on a scheduler it is the instructions
// between the MMAs that cost: a test of the row block around each MMA, a slab of two k pairs with its
// barrier or mbarrier, a counter of warps per stage.  (A lone 8-column sub-tile of d = 201 took 56k
// cycles with those, now 36k, against 21k of tensor pipe.)
template <int N, int WPC, int NT>
__device__ __forceinline__ void tile_rows(const double2 *mat, double2 *Bt, double2 *Us, int d, int kp, int KS, int MD,
                                          int S16, int cb, int sub, int lane)
{
    constexpr int NA = N > 0 ? N : 1;
    const int g = lane >> 2, t = lane & 3, todd = t & 1;
    double re[NA][2], im[NA][2];
#pragma unroll
    for (int i = 0; i < NA; i++) re[i][0] = re[i][1] = im[i][0] = im[i][1] = 0.0;
    auto mma = [&](const double (&v)[NA], const double2 &x) {
        const double bre = todd ? neg(x.y) : x.x, bim = todd ? x.x : x.y;
#pragma unroll
        for (int i = 0; i < N; i++) {
            dmma(re[i][0], re[i][1], v[i], bre);
            dmma(im[i][0], im[i][1], v[i], bim);
        }
    };
    const double2 *b = Bt + (8 * cb + g) * S16 + (t >> 1);
    const size_t astep = 4 * (size_t)MD;
    const int nslab = (kp + KS - 1) / KS;
#pragma unroll 1
    for (int sl = 0; sl < nslab; sl++) {
        cp_wait<0>();
        __syncthreads();  // slab sl (and the columns) has landed for every thread, and no one reads the other buffer
        const int nk = min(KS, kp - sl * KS) / 2;
        const double *a = reinterpret_cast<const double *>(Us + (sl & 1) * KS * MD) + 32 * sub + lane;
        auto pairs = [&](int k0, int k1) {  // k pairs k0 .. k1 of the slab
            if constexpr (N > 0) {
                int k = k0;
#pragma unroll 1
                for (; k + 2 <= k1; k += 2, a += 2 * astep, b += 4) {
                    const double2 x0 = b[0], x1 = b[2];
                    double v0[NA], v1[NA];
#pragma unroll
                    for (int i = 0; i < N; i++) v0[i] = a[32 * WPC * i];
#pragma unroll
                    for (int i = 0; i < N; i++) v1[i] = a[astep + 32 * WPC * i];
                    mma(v0, x0);
                    mma(v1, x1);
                }
                if (k < k1) {
                    const double2 x0 = b[0];
                    double v0[NA];
#pragma unroll
                    for (int i = 0; i < N; i++) v0[i] = a[32 * WPC * i];
                    mma(v0, x0);
                    b += 2;
                }
            }
        };
        // the next slab's copies are issued while the first k pair's MMAs run
        const int first = min(nk, 1);
        pairs(0, first);
        a = reinterpret_cast<const double *>(Us + (sl & 1) * KS * MD) + 32 * sub + lane + first * astep;
        load_slab<NT>(mat, Us, sl + 1, kp, KS, MD);
        pairs(first, nk);
    }
    __syncthreads();
    // stage: thread (g, t) of row block rb holds rows 8 rb + g, columns 8 cb + 2t, 8 cb + 2t + 1
#pragma unroll
    for (int i = 0; i < N; i++) {
        const int row = 8 * (sub + WPC * i) + g;
        if (row < d) {
            Bt[(8 * cb + 2 * t) * S16 + row] = make_double2(re[i][0], im[i][0]);
            Bt[(8 * cb + 2 * t + 1) * S16 + row] = make_double2(re[i][1], im[i][1]);
        }
    }
}

template <int NRB, int WPC, int NT>
__device__ __forceinline__ void tile_dmma(const double2 *mat, double2 *Bt, double2 *Us, int d, int kp, int KS, int RB,
                                          int S16, int warp, int lane)
{
    // warp w runs on scheduler w % 4; rotating the row-block index by column block gives each
    // scheduler the same number of row blocks (two column blocks of four warps: by half a turn)
    const int cb = warp / WPC, sub = (warp % WPC + cb * WPC / (NT == 256 && WPC == 4 ? 2 : 4)) % WPC;
    const int nr = RB > sub ? (RB - sub + WPC - 1) / WPC : 0;  // this warp's row blocks (at most NRB)
    auto rows = [&](auto count) {
        constexpr int N = decltype(count)::value;
        if constexpr (N <= NRB) tile_rows<N, WPC, NT>(mat, Bt, Us, d, kp, KS, 8 * RB, S16, cb, sub, lane);
    };
    switch (nr) {
    case 1: rows(std::integral_constant<int, 1>()); break;
    case 2: rows(std::integral_constant<int, 2>()); break;
    case 3: rows(std::integral_constant<int, 3>()); break;
    case 4: rows(std::integral_constant<int, 4>()); break;
    case 5: rows(std::integral_constant<int, 5>()); break;
    case 6: rows(std::integral_constant<int, 6>()); break;
    case 7: rows(std::integral_constant<int, 7>()); break;
    case 8: rows(std::integral_constant<int, 8>()); break;
    default: rows(std::integral_constant<int, 0>()); break;
    }
}

// Starts the copies of column c of a sub-tile (trajectory and slot of entry `en`) and its record (one
// warp; no group is committed).
__device__ __forceinline__ void stage_column(const Params &P, unsigned en, int kp, double2 *col, TrajState *st, int lane)
{
    const int tr = (int)(en >> 3);
    const double2 *src = slot_ptr(P, (int)(en & 7u), tr);
    for (int k = lane; k < kp; k += 32) cp16(col + k, src + k, true);
    if (lane < (int)(sizeof(TrajState) / 16))
        cp16(reinterpret_cast<double2 *>(st) + lane, reinterpret_cast<const double2 *>(&P.st[tr]) + lane, true);
}

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// What a CTA has done, kept in shared memory by one thread: matvecs, sub-tiles and (for
// qjx_set_trace) clock64 cycles per part.
struct Tally {
    long long begin, work, subtiles, blocks, setup, claim, loop, epi;
    __device__ void reset()
    {
        begin = clock64();
        work = subtiles = blocks = setup = claim = loop = epi = 0;
    }
    // a sub-tile of n columns in nb 8-column blocks: taken at t0, staged at t1, product done at t2,
    // epilogue at t3
    __device__ void add(int n, int nb, long long t0, long long t1, long long t2, long long t3)
    {
        work += n;
        subtiles += 1;
        blocks += nb;
        setup += t1 - t0;
        loop += t2 - t1;
        epi += t3 - t2;
    }
    __device__ void flush(const Params &P) const
    {
        if (work) {
            atomicAdd((unsigned long long *)P.work, (unsigned long long)work);
            atomicAdd((unsigned long long *)(P.work + 3), (unsigned long long)subtiles);
        }
        if (!P.trace) return;
        const long long v[kTraceFields] = {clock64() - begin, setup, claim, loop, epi, subtiles, blocks, work};
        long long *t = P.trace + (size_t)(blockIdx.x % P.grid) * kTraceFields;
        for (int i = 0; i < kTraceFields; i++) atomicAdd((unsigned long long *)(t + i), (unsigned long long)v[i]);
    }
};

// A queue to take from and how many trajectories: 0 when all are empty, -1 when the call is done
// (at most stop_live trajectories left).
struct Pick {
    int n, g;
};

// Looks over at most 256 queues, base to end - 1 (one warp, converged).  A claim is at most NCM trajectories
// and an equal share of the `live` unfinished ones in whole 8-column blocks, or `least` if that is more
// (NCM = 1: one trajectory).  Any queue that has the share waiting will do (a different one for each CTA
// and attempt, so that claims spread), else the fullest; MANY: any with `goal` waiting and half of the
// fullest's.  Leaves `pick` as it is when that has as many.
template <int NCM, bool MANY>
__device__ __forceinline__ void look_over(const Params &P, int base, int end, int live, int least, int goal, unsigned turn, int lane,
                                          Pick &pick)
{
    int av[8], cap[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int gi = base + 32 * i + lane;
        av[i] = cap[i] = 0;
        if (gi < end) {
            const int4 v = __ldcg(reinterpret_cast<const int4 *>(P.q) + gi);
            av[i] = v.x;
            cap[i] = v.w;
        }
    }
    const int share = min(NCM, max(least, 8 * ((live + 8 * (int)gridDim.x - 1) / (8 * (int)gridDim.x))));
    int b = 0, bi = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int a = min(av[i], min(share, cap[i]));
        if (a > b) {
            b = a;
            bi = base + 32 * i + lane;
        }
    }
    const int m = __reduce_max_sync(0xffffffffu, b);
    if (m > pick.n) {
        // 128 rows: any lane's queue with more than half as many, so that CTAs spread over short queues, and
        // more tries (18 ensembles of 1000, d 60 to 240: 174 ms a period; in lock-step 217)
        const unsigned who =
            __ballot_sync(0xffffffffu, NCM == 128 ? 2 * b > m : (MANY ? b >= max(min(m, goal), (m + 1) / 2) : b == m));
        const int r = turn & 31, from = (__ffs(__funnelshift_r(who, who, r)) - 1 + r) & 31;
        pick.n = __shfl_sync(0xffffffffu, b, from);
        pick.g = __shfl_sync(0xffffffffu, bi, from);
    }
}

// The queue to take from: -1 when at most stop_live trajectories are left.  More than 256 queues are looked over
// by sections (see Params), from one that differs by CTA.  Most queues of many ensembles never hold a
// share, and CTAs that all look for the fullest take it from each other: the scan ends at the first
// section with more waiting in one queue than in the mean queue, and sections whose ensembles are done are
// passed over.  ms a period, looking for a share everywhere / now / in lock-step: 64 ensembles of 200 (d 21 to 121)
// 216 / 52 / 206, in split precision 168 / 102 / 135; 128 of 30 (d 21 to 201) 434 / 90 / 431; 128 of 100
// in split precision 383 / 136 / 205; 8 of 200 (d 51 to 401) 159 / 152 / 365.
template <int NCM>
__device__ __forceinline__ Pick scan(const Params &P, int stop_live, int least, unsigned &turn, int lane)
{
    turn += 7u;
    const int live = __ldcg(P.ctrl + kLive);
    Pick pick{0, 0};
    if (P.sections == 1) {
        look_over<NCM, false>(P, 0, P.G, live, least, 0, turn, lane, pick);
    } else {
        const int sections = P.sections, per = P.sect_ens * P.Ge, goal = min(NCM, live / P.G + 1);
        int at = (int)(turn % (unsigned)sections);
        for (int c = 0; c < sections && pick.n < goal;) {
            if (P.sect_parts == 1) {  // the next section with trajectories left
                const int s = at + lane;
                const unsigned left =
                    __ballot_sync(0xffffffffu, lane < sections - c && __ldcg(P.left + (s < sections ? s : s - sections)) > 0);
                const int skip = left ? __ffs(left) - 1 : 32;
                c += skip;
                at += skip;
                if (at >= sections) at -= sections;
                if (!left) continue;
            }
            const int block = at / P.sect_parts;
            look_over<NCM, true>(P, block * per + 256 * (at - block * P.sect_parts), min(P.G, (block + 1) * per), live, least, goal,
                                 turn, lane, pick);
            c++;
            at = at + 1 < sections ? at + 1 : 0;
        }
    }
    if (live <= stop_live) pick.n = -1;
    return pick;
}

// A claim (one warp, converged): from `pick` first if that has any, else from what look() returns.
// Returns how many trajectories it got, 0 when the call's work is done, the slice is over, or
// nothing turned up for kIdleNs; gd is the queue's descriptor, pos the first entry's position.
// A claim is two atomics that cannot fail (a claim by compare-and-swap of the head, before, was lost
// to another CTA four times in five at d = 51): what the count of available entries grants, then as
// many positions.
template <int NCM, class Look>
__device__ __forceinline__ int grant(const Params &P, unsigned long long t_end, const Look &look, Pick pick, int lane,
                                     GroupDesc &gd, unsigned &pos)
{
    // a queue that others have nearly emptied since it was looked at is passed over this many times:
    // a sub-tile of a few columns costs as much tensor time as a full block of eight
    constexpr int kTries = NCM == 128 ? 8 : 2;
    unsigned long long t_idle = 0;
    int n = 0, tries = 0;
    while (true) {
        if (pick.n == 0) pick = look();
        const unsigned long long now = __shfl_sync(0xffffffffu, global_ns(), 0);
        if (pick.n < 0 || now >= t_end) return 0;
        if (pick.n > 0) {
            gd = load_desc(P.gd + pick.g);
            if (lane == 0) {
                Queue *q = P.q + pick.g;
                auto whole = [](int m) { return NCM == 32 && m > 16 && m <= 24 ? 16 : m; };  // no 3 column blocks
                const int want = whole(pick.n);
                n = whole(max(0, min(want, atomicSub(&q->avail, want))));
                if (4 * n < 3 * want && tries < kTries) n = 0;
                if (n < want) atomicAdd(&q->avail, want - n);
                if (n > 0) pos = atomicAdd(&q->head, (unsigned)n);
            }
            n = __shfl_sync(0xffffffffu, n, 0);
            if (n > 0) break;
            pick.n = 0;  // other CTAs took them: look again
            tries++;
            continue;
        }
        if (t_idle == 0) t_idle = now + kIdleNs;
        else if (now >= t_idle) return 0;
        __nanosleep(50);
    }
    pos = __shfl_sync(0xffffffffu, pos, 0);
    return n;
}

// The entry at a claimed position (kFree when it was never published: the bounded wait gave up).
__device__ __forceinline__ unsigned take_entry(const Params &P, const GroupDesc &gd, unsigned pos)
{
    unsigned en = kFree;
    unsigned *entry = P.ring + gd.roff + (pos & gd.rmask());
    for (long long i = 0; i < kWaitLimit && en == kFree; i++) en = atomicExch(entry, kFree);
    return en;
}

// A claim of up to NCM <= 32 trajectories with its entries: lane i < n gets the i-th in `en`.  What
// was written about the trajectories before their entries is visible to this SM afterwards.
template <int NCM>
__device__ __forceinline__ int take(const Params &P, unsigned long long t_end, int stop_live, Pick pick, unsigned &turn,
                                    int lane, GroupDesc &gd, unsigned &en)
{
    unsigned pos = 0;
    const int n = grant<NCM>(P, t_end, [&] { return scan<NCM>(P, stop_live, 0, turn, lane); }, pick, lane, gd, pos);
    en = lane < n ? take_entry(P, gd, pos + (unsigned)lane) : kFree;
    __threadfence();  // acquire
    if (__any_sync(0xffffffffu, lane < n && en == kFree)) {  // never published: report and stop
        if (lane == 0) {
            atomicAdd(&P.ctrl[4], 1);
            report_error(P, -1, ERR_TIMEOUT);
        }
        return 0;
    }
    return n;
}

// Appends trajectories to their next queues (one warp, converged): lanes with `has` have the bucket
// g2 and the entry `en` of one, -1 when it is finished, paused or failed.  Lanes with the same bucket
// find each other, the lowest reserves the run.  All are of one ensemble.
__device__ void append_lanes(const Params &P, bool has, int g2, unsigned en, int lane)
{
    __threadfence();  // release: what the CTA wrote, before the entries
    const int key = has ? g2 : -2;
    const unsigned m = __match_any_sync(0xffffffffu, key);
    const int leader = __ffs(m) - 1;
    GroupDesc gd{};
    if (key >= 0) gd = load_desc(P.gd + key);
    unsigned base = 0;
    if (lane == leader) {
        if (key >= 0) {
            base = atomicAdd(&P.q[key].tail, (unsigned)__popc(m));
            atomicAdd(&P.q[key].avail, __popc(m));
        } else if (key == -1) {
            atomicSub(P.left + P.st[en >> 3].ens / P.sect_ens, __popc(m));
            atomicSub(P.ctrl + kLive, __popc(m));
        }
    }
    base = __shfl_sync(0xffffffffu, base, leader);
    bool put = key < 0;
    unsigned *entry = P.ring + gd.roff + ((base + (unsigned)__popc(m & ((1u << lane) - 1u))) & gd.rmask());
    for (long long i = 0; i < kWaitLimit && !put; i++) put = atomicCAS(entry, kFree, en) == kFree;
    if (!put) {
        atomicAdd(&P.ctrl[4], 1);
        report_error(P, -1, ERR_TIMEOUT);
    }
    __syncwarp();
}

// The plain form's persistent kernel: every CTA takes sub-tiles from the queues until the call's
// trajectories are done, its time slice ends or it finds nothing to do for a while.  A CTA never
// waits for work of another (a trajectory that is neither queued nor finished is in a running
// CTA's sub-tile, and that CTA scans the queues again after appending it), so CTAs need not be
// co-resident and may leave at any time; the host launches again while trajectories are left.
// The only waits are for an entry that a running CTA has reserved and is about to write or take
// (bounded).  A queue is a ring of entries with a head and a tail count; it never holds
// more than the ensemble's trajectories, and a trajectory is in one place at a time.
// Results do not depend on which trajectories share a sub-tile: a column's arithmetic involves
// that column only.
//
// What bounds it: the FP64 tensor pipe (8 d^2 flop per column).  Two CTAs of 256 threads per SM
// while both fit the shared memory (16-column sub-tiles, d <= 232), so one CTA's scan, gather and
// epilogue overlap the other's products; one CTA of 512 threads (32, 16 or 8 columns) above that.
// R4, R2, R1: row blocks per warp of the sub-tiles whose column blocks are shared by 4 warps, by
// 8 and by 16 (512 threads) or 2 (256 threads, 32-column sub-tiles; 0: none wider than 16).
template <int NT, int R4, int R2, int R1>
__global__ void __launch_bounds__(NT, NT == 256 ? 2 : 1) flow_kernel(const Params P, int stop_live)
{
    constexpr int NW = NT / 32, NCM = (NT == 512 || R1 > 0) ? 32 : 16;
    extern __shared__ __align__(128) unsigned char smem[];
    double2 *Bt = reinterpret_cast<double2 *>(smem);
    __shared__ __align__(16) TrajState s_st[NCM];
    __shared__ int s_g2[NCM];
    __shared__ unsigned s_in[NCM], s_entry[NCM];
    __shared__ __align__(16) GroupDesc s_gd;
    __shared__ int s_n;
    __shared__ double s_dt[kMaxDt];
    __shared__ Tally tally;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) tally.reset();
    const unsigned long long t_end = global_ns() + kSliceNs;
    unsigned turn = blockIdx.x;
    Pick hint{0, 0};  // (warp 0) the next claim, looked for while the sub-tile before was being staged
    while (true) {
        const long long t0 = clock64();
        if (warp == 0) {
            GroupDesc gd{};
            unsigned en = kFree;
            const int n = take<NCM>(P, t_end, stop_live, hint, turn, lane, gd, en);
            if (lane < NCM) s_in[lane] = en;
            if (lane == 0) {
                tally.claim += clock64() - t0;
                s_gd = gd;
                s_n = n;
            }
        }
        __syncthreads();
        const int ncol = s_n;
        if (ncol <= 0) break;
        // the group's matrix: its ensemble's dimension, padded rows, k rows and tiling
        const int dg = s_gd.d, MD = 8 * ((dg + 7) / 8), RB = MD / 8, kp = (dg + 1) & ~1, S16 = MD + kColPad;
        const int KS = s_gd.kb;
        double2 *Us = Bt + s_gd.nc * S16;
        const double2 *mat = P.mats + s_gd.moff;
        const int ncb = (ncol + 7) / 8;
        for (int c = warp; c < ncol; c += NW) stage_column(P, s_in[c], kp, Bt + c * S16, &s_st[c], lane);
        load_slab<NT>(mat, Us, 0, kp, KS, MD);
        const int nbd = P.nb * P.deep;
        const Ens sys{dg, s_gd.ens * P.Ge, nbd <= kMaxDt ? s_dt : P.e_dt + (size_t)s_gd.ens * nbd,
                    P.e_rate + (size_t)s_gd.ens * P.nd};
        if (warp == 0) hint = scan<NCM>(P, stop_live, 0, turn, lane);
        else if (nbd <= kMaxDt && tid >= 32 && tid < 32 + nbd) s_dt[tid - 32] = __ldg(P.e_dt + (size_t)s_gd.ens * nbd + tid - 32);
        const long long t1 = clock64();
        if constexpr (NT == 256) {
            if (ncb == 1) tile_dmma<R2, 8, NT>(mat, Bt, Us, dg, kp, KS, RB, S16, warp, lane);
            else if (R1 == 0 || ncb == 2) tile_dmma<R4, 4, NT>(mat, Bt, Us, dg, kp, KS, RB, S16, warp, lane);
            else tile_dmma<R1, 2, NT>(mat, Bt, Us, dg, kp, KS, RB, S16, warp, lane);
        } else {
            if (ncb == 1) tile_dmma<R1, 16, NT>(mat, Bt, Us, dg, kp, KS, RB, S16, warp, lane);
            else if (ncb == 2) tile_dmma<R2, 8, NT>(mat, Bt, Us, dg, kp, KS, RB, S16, warp, lane);
            else tile_dmma<R4, 4, NT>(mat, Bt, Us, dg, kp, KS, RB, S16, warp, lane);
        }
        __syncthreads();
        const long long t2 = clock64();
        for (int c = warp; c < ncol; c += NW) {
            unsigned entry;
            const int tr = (int)(s_in[c] >> 3);
            const int g2 = column_epilogue(P, Bt + c * S16, tr, s_st[c], lane, entry, sys, global_slots(P, tr), &P.st[tr],
                                           true);
            if (lane == 0) {
                s_g2[c] = g2;
                s_entry[c] = entry;
            }
        }
        __syncthreads();
        // warp 1 appends while warp 0 takes the next sub-tile (s_g2 and s_entry are rewritten after that
        // sub-tile's products)
        if (warp == 1) append_lanes(P, lane < ncol, lane < ncol ? s_g2[lane] : -1, lane < ncol ? s_entry[lane] : kFree, lane);
        if (tid == 0) tally.add(ncol, (ncb == 3) ? 4 : ncb, t0, t1, t2, clock64());
    }
    if (tid == 0) tally.flush(P);
}

// ---------------------------------------------------------------- few trajectories: one per CTA or cluster
__device__ __forceinline__ void cluster_sync()
{
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ unsigned cluster_rank()
{
    unsigned r;
    asm volatile("mov.u32 %0, %cluster_ctarank;" : "=r"(r));
    return r;
}

// Address of `p` (this CTA's shared memory) in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t map_rank(const void *p, unsigned rank)
{
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    return a;
}

__device__ __forceinline__ void st_cluster(uint32_t addr, double2 v)
{
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(addr), "d"(v.x), "d"(v.y) : "memory");
}

__device__ __forceinline__ void st_cluster(uint32_t addr, int v)
{
    asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}

// Row `row` of two complex matrix columns k, k + 1 (32 bytes).
__device__ __forceinline__ void ld_kpair(const double2 *p, double2 &a, double2 &b)
{
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(a.x), "=d"(a.y), "=d"(b.x), "=d"(b.y) : "l"(p));
}

// y[row] = sum_k M[row][k] x[k] with the contract's k-ascending fma chain: `m` points at the row in
// k pair 0, a k pair is `step` components further.  Blocks of kPre k pairs, the next block's loads
// in flight behind the current one's fmas; no branch stands between the loads of a block (a test
// per load made the compiler wait for each: 390 cycles per k pair instead of 110 at d = 201, where
// one SM's L2 bandwidth, 64 bytes a cycle, gives 104).
template <int kPre>
__device__ __forceinline__ double2 row_matvec(const double2 *m, const double2 *x, int kp2, size_t step)
{
    double re = 0.0, im = 0.0;
    auto fmas = [&](const double2 &u, const double2 &v, const double2 &x0, const double2 &x1) {
        re = __fma_rn(u.x, x0.x, re);
        im = __fma_rn(u.x, x0.y, im);
        re = __fma_rn(-u.y, x0.y, re);
        im = __fma_rn(u.y, x0.x, im);
        re = __fma_rn(v.x, x1.x, re);
        im = __fma_rn(v.x, x1.y, im);
        re = __fma_rn(-v.y, x1.y, re);
        im = __fma_rn(v.y, x1.x, im);
    };
    // block k0 .. (past the end it reads the last pair again)
    auto load = [&](double2 (&u)[kPre], double2 (&v)[kPre], int k0) {
        if (k0 + kPre <= kp2) {
            const double2 *p = m + k0 * step;
#pragma unroll
            for (int j = 0; j < kPre; j++) ld_kpair(p + j * step, u[j], v[j]);
        } else if (k0 < kp2) {
#pragma unroll
            for (int j = 0; j < kPre; j++) ld_kpair(m + min(k0 + j, kp2 - 1) * step, u[j], v[j]);
        }
    };
    auto block = [&](const double2 (&u)[kPre], const double2 (&v)[kPre], int k0) {
        if (k0 + kPre <= kp2) {
#pragma unroll
            for (int j = 0; j < kPre; j++) fmas(u[j], v[j], x[2 * (k0 + j)], x[2 * (k0 + j) + 1]);
        } else {
#pragma unroll
            for (int j = 0; j < kPre; j++)
                if (k0 + j < kp2) fmas(u[j], v[j], x[2 * (k0 + j)], x[2 * (k0 + j) + 1]);
        }
    };
    double2 a[kPre], b[kPre], c[kPre], d[kPre];
    load(a, b, 0);
#pragma unroll 1
    for (int k = 0; k < kp2; k += 2 * kPre) {
        load(c, d, k + kPre);
        block(a, b, k);
        load(a, b, k + 2 * kPre);
        block(c, d, k + kPre);
    }
    return make_double2(re, im);
}

constexpr int kStint = 128;  // matvecs between two looks at the clock

// The plain form for few trajectories: a cluster of C CTAs takes one trajectory from the queues and
// runs its whole chain of matvecs (split tree, jumps, observables) until its work of this call is
// done or the slice is over, with the states and the record in shared memory.  Each CTA computes
// its share of the rows, a thread per row with the matrix straight from L2 (or L1, for small d),
// and stores them into every CTA's copy of the product; after one cluster barrier all CTAs run the
// same epilogue on their own copies, so a step has no global round trip, no queue and no second
// barrier (the product is double-buffered).
// What bounds it: the chain of 2 d dependent FP64 fmas per row and the epilogue's latency, or the
// L2 reads of a whole matrix per trajectory and step (16 d^2 bytes; the sub-tiles of flow_kernel
// share them over up to 32 trajectories), which is why it takes few trajectories only.
template <int C, int kPre>
__global__ void __launch_bounds__(kSoloThreads, kPre > 4 ? 1 : 2) solo_kernel(const Params P, int rows)
{
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(16) TrajState s_st;
    __shared__ int s_go, s_tr, s_group, s_next;
    __shared__ unsigned s_entry;
    __shared__ double s_dt[kMaxDt];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int rank = C > 1 ? (int)cluster_rank() : 0;
    const bool lead = rank == 0;
    const int nslots = P.prop == 1 ? kRkSlots : 2, SD = P.MD + 2;
    double2 *const sl = reinterpret_cast<double2 *>(smem);
    double2 *const yb = sl + (size_t)nslots * SD;  // [2][SD]
    const Slots slots{sl, (size_t)SD};
    const unsigned long long t_end = global_ns() + kSliceNs;
    unsigned turn = blockIdx.x;
    __shared__ Tally tally;
    if (tid == 0) tally.reset();
    if (C > 1) cluster_sync();  // every CTA of the cluster has started: its shared memory may be written
    auto sync = [&] {
        if (C > 1) cluster_sync();
        else __syncthreads();
    };

    while (true) {
        const long long t0 = clock64();
        // the lead takes a trajectory and tells the others: 0 none, 1 run
        if (lead && warp == 0) {
            GroupDesc gd{};
            unsigned en;
            const int n = take<1>(P, t_end, 0, Pick{0, 0}, turn, lane, gd, en);
            en = __shfl_sync(0xffffffffu, en, 0);
            const int tr = (int)(en >> 3), g = gd.group;
            if (lane < C) {
                if (C > 1) {
                    st_cluster(map_rank(&s_go, lane), n);
                    st_cluster(map_rank(&s_tr, lane), tr);
                    st_cluster(map_rank(&s_group, lane), g);
                    st_cluster(map_rank(&s_next, lane), (int)(en & 7u));
                } else {
                    s_go = n;
                    s_tr = tr;
                    s_group = g;
                    s_next = (int)(en & 7u);
                }
            }
        }
        sync();
        if (s_go <= 0) break;
        const int tr = s_tr;
        int g = s_group, in = s_next;
        if (C > 1) __threadfence();  // the lead's acquire, for this CTA's reads of the trajectory
        if (tid < (int)(sizeof(TrajState) / 16))
            reinterpret_cast<uint4 *>(&s_st)[tid] = __ldcg(reinterpret_cast<const uint4 *>(&P.st[tr]) + tid);
        for (int i = 0; i < nslots; i++) {
            const double2 *src = slot_ptr(P, i, tr);
            for (int k = tid; k < P.MD; k += blockDim.x) sl[i * SD + k] = __ldcg(src + k);
        }
        __syncthreads();
        const int e = s_st.ens, nbd = P.nb * P.deep;
        Ens E = global_ens(P, e);
        if (nbd <= kMaxDt) {
            if (tid < 32)
                for (int i = tid; i < nbd; i += 32) s_dt[i] = E.dt[i];
            E.dt = s_dt;
        }
        const int d = E.d, MD = 8 * ((d + 7) / 8), kp2 = (d + 1) / 2;
        // the ensemble's matrices are equally far apart
        const int g0 = E.g0;
        const long long m0 = P.g_off[g0], mstep = P.g_off[g0 + 1] - m0;
        const int row = rank * rows + tid;
        const bool mine = tid < rows && row < d;
        const double2 *mrow = P.mats + m0 + 2 * row;
        int steps = 0, buf = 0, g2 = g;
        long long t1 = clock64();
        if (tid == 0) tally.setup += t1 - t0;
        while (true) {
            double2 *y = yb + buf * SD;
            if (mine) {
                const double2 v = row_matvec<kPre>(mrow + (g2 - g0) * mstep, sl + in * SD, kp2, 2 * (size_t)MD);
                if (C > 1) {
#pragma unroll
                    for (int r = 0; r < C; r++) st_cluster(map_rank(y + row, r), v);
                } else {
                    y[row] = v;
                }
            }
            sync();
            const long long t2 = clock64();
            if (warp == 0) {
                unsigned entry;
                const int next = column_epilogue(P, y, tr, s_st, lane, entry, E, slots, &s_st, lead);
                if (lane == 0) {
                    s_group = next;
                    s_entry = entry;
                }
            }
            __syncthreads();
            if (tid == 0) tally.add(1, 1, t1, t1, t2, clock64());
            t1 = clock64();
            steps++;
            buf ^= 1;
            g2 = s_group;
            in = (int)(s_entry & 7u);
            if (g2 < 0) break;
            if (steps % kStint == 0) {  // the lead's clock decides for all
                if (lead && tid < C) {
                    const int go = global_ns() < t_end ? 1 : 0;
                    if (C > 1) st_cluster(map_rank(&s_go, tid), go);
                    else s_go = go;
                }
                sync();
                if (s_go == 0) break;
            }
        }
        if (lead) {  // back to global memory, then to the queue of its next matrix (or done)
            for (int i = 0; i < nslots; i++) {
                double2 *dst = slot_ptr(P, i, tr);
                for (int k = tid; k < d; k += blockDim.x) dst[k] = sl[i * SD + k];
            }
            if (tid < (int)(sizeof(TrajState) / 16))
                reinterpret_cast<uint4 *>(&P.st[tr])[tid] = reinterpret_cast<const uint4 *>(&s_st)[tid];
            __syncthreads();
            if (tid == 0) {
                __threadfence();  // release
                if (g2 >= 0) {
                    const GroupDesc gd = load_desc(P.gd + g2);
                    const unsigned pos = atomicAdd(&P.q[g2].tail, 1u);
                    atomicAdd(&P.q[g2].avail, 1);
                    unsigned *entry = P.ring + gd.roff + (pos & gd.rmask());
                    bool put = false;
                    for (long long i = 0; i < kWaitLimit && !put; i++) put = atomicCAS(entry, kFree, s_entry) == kFree;
                    if (!put) {
                        atomicAdd(&P.ctrl[4], 1);
                        report_error(P, -1, ERR_TIMEOUT);
                    }
                } else {
                    atomicSub(P.left + e / P.sect_ens, 1);
                    atomicSub(P.ctrl + kLive, 1);
                }
            }
        }
        sync();  // no CTA's shared memory is rewritten or left while another still uses it
    }
    if (C > 1) cluster_sync();
    if (lead && tid == 0) tally.flush(P);
}

// Bucket trajectories for step 0 of a call.  mode 0: start of a run of P.target periods;
// mode 1: resume trajectories paused on a full record buffer; mode 2: continue a deep task from
// where the previous call stopped (a sub-period boundary: branch, unit and period count kept).
__global__ void schedule_kernel(const Params P, int mode)
{
    const int tr = blockIdx.x * blockDim.x + threadIdx.x;
    if (tr >= P.n) return;
    TrajState s = P.st[tr];
    if (s.phase == PH_ERROR) return;
    if (mode == 0) {
        s.pc = 0;
        s.di = 0;
        s.b = 0;
        s.lvl = 0;
        s.mask = 0;
        s.rk_sid = 0;
        s.paused = 0;
        s.phase = (P.target > 0 && runs(P, tr)) ? PH_STEP : PH_DONE;
    } else if (mode == 2) {
        s.di = 0;
        s.paused = 0;
        s.phase = (P.sub_target > 0 && runs(P, tr)) ? PH_STEP : PH_DONE;
    } else {
        if (!s.paused) return;
        s.paused = 0;
    }
    P.st[tr] = s;
    const int g = group_of(P, s);
    if (g >= 0) enqueue(P, g, tr);
}

// Host-initiated observables of the current states (one warp per trajectory); the energy
// and random-observable matvecs follow from the queues.
__global__ void observe_kernel(const Params P, int dump, int is_start)
{
    extern __shared__ __align__(128) unsigned char smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tr = blockIdx.x * (blockDim.x / 32) + warp;
    if (tr >= P.n || (P.active && !P.active[tr])) return;
    double2 *col = reinterpret_cast<double2 *>(smem) + (size_t)warp * P.MD;
    TrajState s = P.st[tr];
    if (s.phase == PH_ERROR) return;
    const double2 *src = slot_ptr(P, s.cur, tr);
    for (int k = lane; k < P.e_d[s.ens]; k += 32) col[k] = src[k];
    __syncwarp();
    obs_prep(P, s, tr, global_ens(P, s.ens), global_slots(P, tr), col, lane, dump, is_start);
    if (lane == 0) {
        s.pc = 0;
        s.di = 0;
        s.phase = PH_OBS_E;
        P.st[tr] = s;
        enqueue(P, P.e_g0[s.ens] + P.gHE, tr);
    }
}

// ---------------------------------------------------------------- ensemble purity
// rho = (1/n) sum_tr psi_hat psi_hat^dagger over the current states, purity = ||rho||_F^2 (the
// formula of calc_purity, source/cpp/CQdiss/CQdiss/CalcTraseRO2.cpp:57-75, applied to the
// trajectory ensemble).  Canonical order, shared bit-for-bit with the CPU oracle: psi_hat =
// psi / sqrt(p) with the canonical 32-lane norm p; rho_ij accumulates trajectories in ascending
// order with fma (re += a_r b_r, re += a_i b_i, im += a_i b_r, im += -a_r b_i) and is divided by n;
// the purity is the canonical 32-lane squared norm of rho flattened row-major.
__global__ void normalize_kernel(const Params P, double2 *hat)
{
    const int lane = threadIdx.x & 31;
    const int tr = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (tr >= P.n) return;
    const double2 *src = slot_ptr(P, P.st[tr].cur, tr);
    const double q = __dsqrt_rn(warp_norm(src, P.d, lane));
    double2 *dst = hat + (size_t)tr * P.MD;
    for (int k = lane; k < P.d; k += 32) {
        const double2 v = src[k];
        dst[k] = make_double2(__ddiv_rn(v.x, q), __ddiv_rn(v.y, q));
    }
}

constexpr int kRhoBlocks = 5;       // most 8 x 8 blocks of rho per CTA
constexpr int kRhoT = 32;           // trajectories per stage
constexpr int kRhoLoaders = 128;   // threads that load
constexpr int kRhoStages = 5;
constexpr int kRhoStride = 12;      // components between trajectories of a staged block of 8 (192 bytes: the
                                    // two trajectories of an MMA fall on different banks)

size_t rho_smem_bytes(int per) { return (size_t)kRhoStages * (per + 2) * kRhoT * kRhoStride * sizeof(double2); }

// rho_ij = (1/n) sum_t hat_t[i] conj(hat_t[j]) on the FP64 tensor core.  One warp per part (re or
// im) of an 8 x 8 block: two trajectories are one MMA, A = [xr, xi] (re) or [xi, -xr] (im) of two
// trajectories against B = [yr; yi], which is the canonical chain re += xr yr; re += xi yi;
// im += xi yr; im -= xr yi with trajectories ascending, bit for bit.  The chain over n cannot be
// split, so the work is spread over chains: a CTA takes `per` consecutive blocks (row-major), at
// d = 201 676 blocks in 136 CTAs, 10 warps on each of 136 SMs at most 3 to a scheduler.  Four more
// warps load: with the MMA warps loading too, all of them put their copies before the MMAs of a
// stage at the same time (ncu: 283 us, with the loaders 262; in a running program 255 us, and 246
// with five stages instead of three).
// Bound: the MMA pipe would need 3 chains x n / 2 MMAs of 16 cycles = 123 us at d = 201, n = 10^4;
// an MMA's two operand loads and the copies take about as many cycles of shared memory.  246 us; two
// fma chains per thread on 16 x 16 tiles before: the purity took 1.01 ms in all, now 0.445 ms.
__global__ void __launch_bounds__(64 * kRhoBlocks + kRhoLoaders) rho_kernel(const Params P, const double2 *hat, double2 *rho, int per)
{
    extern __shared__ __align__(128) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int RB = (P.d + 7) / 8, b0 = blockIdx.x * per, nb = min(per, RB * RB - b0);
    const int part = warp & 1, mine = warp >> 1;
    const bool loads = tid >= 64 * per, mma = mine < nb && !loads;
    const int g = lane >> 2, t = lane & 3, th = t >> 1, todd = t & 1;
    const int nst = (P.n + kRhoT - 1) / kRhoT;
    // staged sets of 8 components per trajectory: 0 and 1 the row blocks of the run (two at most:
    // per > 1 needs RB > 12), 2 + b the column block of its block b
    const int ib0 = b0 / RB, sets = 2 + nb;
    const bool two = (b0 + nb - 1) / RB > ib0;
    auto at = [&](int it, int set) {
        return reinterpret_cast<double2 *>(smem) + (size_t)((it % kRhoStages) * (per + 2) + set) * kRhoT * kRhoStride;
    };
    // a stage is sets x kRhoT x 8 components; a loading thread copies component tid % 8 of every
    // 16th trajectory of every set (the addresses are worked out once: doing it in each stage took
    // most of the kernel's time)
    const int k = tid & 7, t0 = (tid - 64 * per) >> 3;
    int comp[kRhoBlocks + 2];
#pragma unroll
    for (int set = 0; set < kRhoBlocks + 2; set++) {
        const int c = 8 * (set < 2 ? ib0 + set : (b0 + set - 2) % RB) + k;
        comp[set] = (set < sets && (set != 1 || two)) ? (c < P.d ? c : -1) : -2;  // -1: zeros, -2: not staged
    }
    auto load = [&](int it) {
        if (it < nst) {
            double2 *dst = at(it, 0) + k;
            for (int tt = t0; tt < kRhoT; tt += kRhoLoaders / 8) {
                const int tr = it * kRhoT + tt;
                const double2 *src = hat + (size_t)min(tr, P.n - 1) * P.MD;
#pragma unroll
                for (int set = 0; set < kRhoBlocks + 2; set++)
                    if (comp[set] > -2)
                        cp16(dst + (set * kRhoT + tt) * kRhoStride, src + max(comp[set], 0), comp[set] >= 0 && tr < P.n);
            }
        }
        cp_commit();
    };
    const int blk = b0 + mine, aset = blk / RB - ib0, bset = 2 + mine;
    double c0 = 0.0, c1 = 0.0;
    for (int i = 0; loads && i < kRhoStages - 1; i++) load(i);
    for (int it = 0; it < nst; it++) {
        if (loads) cp_wait<kRhoStages - 2>();
        __syncthreads();  // stage `it` has landed, and nobody reads the one refilled next
        if (loads) load(it + kRhoStages - 1);
        if (!mma) continue;
        const double *a = reinterpret_cast<const double *>(at(it, aset) + th * kRhoStride + g) + (part ? 1 - todd : todd);
        const double *b = reinterpret_cast<const double *>(at(it, bset) + th * kRhoStride + g) + todd;
#pragma unroll
        for (int k = 0; k < kRhoT; k += 2) {
            const double x = a[2 * k * kRhoStride];
            dmma(c0, c1, (part && todd) ? neg(x) : x, b[2 * k * kRhoStride]);
        }
    }
    if (!mma) return;
    const int i = 8 * (blk / RB) + g, j = 8 * (blk % RB) + 2 * t;
    double *out = reinterpret_cast<double *>(rho) + part;
    if (i < P.d && j < P.d) out[2 * ((size_t)i * P.d + j)] = __ddiv_rn(c0, (double)P.n);
    if (i < P.d && j + 1 < P.d) out[2 * ((size_t)i * P.d + j + 1)] = __ddiv_rn(c1, (double)P.n);
}

constexpr int kPurityThreads = 1024, kPurityTile = 2 * kPurityThreads;

// Canonical 32-lane squared norm of rho.  Its 32 chains of d^2 / 32 additions are one warp's; all
// warps read rho and square it a tile ahead of them (one warp doing both spent its time on the loads).
__global__ void __launch_bounds__(kPurityThreads) purity_kernel(const double2 *rho, int dd, double *out)
{
    __shared__ double sq[2][kPurityTile];
    const int tid = threadIdx.x, nt = (dd + kPurityTile - 1) / kPurityTile;
    double2 v0 = make_double2(0.0, 0.0), v1 = v0;
    auto fetch = [&](int it) {
        const int i = it * kPurityTile + tid;
        if (i < dd) v0 = rho[i];
        if (i + kPurityThreads < dd) v1 = rho[i + kPurityThreads];
    };
    fetch(0);
    double s = 0.0;
    for (int it = 0; it < nt; it++) {
        double *p = sq[it & 1];
        p[tid] = __dadd_rn(__dmul_rn(v0.x, v0.x), __dmul_rn(v0.y, v0.y));
        p[tid + kPurityThreads] = __dadd_rn(__dmul_rn(v1.x, v1.x), __dmul_rn(v1.y, v1.y));
        fetch(it + 1);
        __syncthreads();  // (the tile before last, whose buffer is written next, has been added)
        if (tid < 32) {
            const int m = min(kPurityTile, dd - it * kPurityTile);
#pragma unroll 8
            for (int e = tid; e < m; e += 32) s = __dadd_rn(s, p[e]);
        }
    }
    if (tid < 32) s = warp_allsum(s);
    if (tid == 0) *out = s;
}

// The current states of trajectories tr0 .. tr0 + count - 1, packed [count][d] (one warp each).
__global__ void gather_states_kernel(const Params P, int tr0, int count, double2 *out)
{
    const int lane = threadIdx.x & 31, i = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (i >= count) return;
    const int tr = tr0 + i;
    const double2 *src = slot_ptr(P, P.st[tr].cur, tr);
    for (int k = lane; k < P.d; k += 32) out[(size_t)i * P.d + k] = src[k];
}

cudaError_t launch_gather_states(const Params &P, int tr0, int count, double2 *out, cudaStream_t st)
{
    gather_states_kernel<<<(count + 7) / 8, 256, 0, st>>>(P, tr0, count, out);
    return cudaGetLastError();
}

__global__ void init_state_kernel(const Params P, int tr0, int tr1)
{
    const int tr = tr0 + blockIdx.x * blockDim.x + threadIdx.x;
    if (tr >= tr1) return;
    TrajState s;
    s.t = 0.0;
    s.eta = 0.0;
    s.ran = 0.0;
    s.tmpw = 0.0;
    s.rng_pos = 0;
    s.mask = 0;
    s.lvl = 0;
    s.b = 0;
    s.phase = PH_DONE;
    s.cur = 0;
    s.sub = 0;
    s.pc = 0;
    s.di = 0;
    s.jumps = 0;
    s.nrec = 0;
    s.err = 0;
    s.paused = 0;
    s.rng_src = tr;
    s.rk_h = 0.0;
    s.rk_prev = 0.0;
    s.rk_end = 0.0;
    s.rk_sid = 0;
    s.rk_stage = 0;
    s.rk_part = 0;
    s.rk_ctx = 0;
    int lo = 0, hi = P.E;  // ensemble e with e_tr0[e] <= tr < e_tr0[e + 1]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (P.e_tr0[mid] <= tr) lo = mid;
        else hi = mid;
    }
    s.ens = lo;
    s.rechk = 0;
    // rows past the ensemble's dimension stay zero (they meet the zero rows of its matrices)
    double2 *psi0 = P.psi + (size_t)tr * P.MD;
    for (int k = P.e_d[lo]; k < P.MD; k++) psi0[k] = make_double2(0.0, 0.0);
    P.st[tr] = s;
}

// eta_0 draw of trans_process_single (experiment.cpp:3260-3265)
__global__ void thresholds_kernel(const Params P, int tr0, int tr1)
{
    const int tr = tr0 + blockIdx.x * blockDim.x + threadIdx.x;
    if (tr >= tr1) return;
    TrajState s = P.st[tr];
    int err = 0;
    s.eta = 0.0;
    while (s.eta == 0.0 && err == 0) s.eta = draw(P, tr, s, &err);
    if (err) {
        s.err = err;
        s.phase = PH_ERROR;
        report_error(P, tr, err);
    }
    P.st[tr] = s;
}

__global__ void reset_times_kernel(const Params P)
{
    const int tr = blockIdx.x * blockDim.x + threadIdx.x;
    if (tr < P.n) P.st[tr].t = 0.0;
}

__global__ void clear_records_kernel(const Params P)
{
    const int tr = blockIdx.x * blockDim.x + threadIdx.x;
    if (tr < P.n) P.st[tr].nrec = 0;
}

// ---------------------------------------------------------------- host-side launchers
// Lets a kernel take all the shared memory the current device gives a CTA, once per device (the same
// value whoever asks, so engines on several threads do not disturb each other).
template <class Kernel>
static cudaError_t allow_smem(Kernel *kernel, std::atomic<unsigned long long> &done)
{
    int dev = 0, optin = 0;
    cudaError_t e = cudaGetDevice(&dev);
    const unsigned long long bit = 1ull << (dev & 63);
    if (e != cudaSuccess || (done.load() & bit)) return e;
    cudaFuncAttributes a{};
    e = cudaFuncGetAttributes(&a, kernel);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)a.sharedSizeBytes);
    if (e == cudaSuccess) done.fetch_or(bit);
    return e;
}

template <int NT, int R4, int R2, int R1>
static cudaError_t launch_flow_t(const Params &P, int stop_live, int grid, cudaStream_t st)
{
    static std::atomic<unsigned long long> done{0};
    const cudaError_t e = allow_smem(flow_kernel<NT, R4, R2, R1>, done);
    if (e != cudaSuccess) return e;
    flow_kernel<NT, R4, R2, R1><<<grid, NT, P.step_smem, st>>>(P, stop_live);
    return cudaGetLastError();
}

// Instantiation for the threads per CTA (nt) and the largest padded rows MD.  256 threads (two
// CTAs per SM): 16-column sub-tiles have 4 warps per column block, 8-column ones 8.  512 threads:
// up to 256 rows every sub-tile width may occur (R4 = ceil(RB / 4)); up to 512 the 32-column
// sub-tiles belong to ensembles of at most 256 rows (R4 = 8) and R2 = ceil(RB / 8); up to 1024
// also R2 = 8 and R1 = ceil(RB / 16).
cudaError_t launch_flow(const Params &P, int nt, int stop_live, int grid, cudaStream_t st)
{
    const int RB = P.MD / 8;
    if (nt == 256) {
        switch ((RB + 3) / 4) {
        case 1: return launch_flow_t<256, 1, 1, 2>(P, stop_live, grid, st);
        case 2: return launch_flow_t<256, 2, 1, 4>(P, stop_live, grid, st);
        case 3: return launch_flow_t<256, 3, 2, 6>(P, stop_live, grid, st);
        case 4: return launch_flow_t<256, 4, 2, 8>(P, stop_live, grid, st);
        case 5: return launch_flow_t<256, 5, 3, 0>(P, stop_live, grid, st);
        case 6: return launch_flow_t<256, 6, 3, 0>(P, stop_live, grid, st);
        case 7: return launch_flow_t<256, 7, 4, 0>(P, stop_live, grid, st);
        case 8: return launch_flow_t<256, 8, 4, 0>(P, stop_live, grid, st);
        default: return cudaErrorInvalidValue;
        }
    }
    if (RB <= 32) return launch_flow_t<512, 8, 4, 2>(P, stop_live, grid, st);
    if (RB <= 64) {
        switch ((RB + 7) / 8) {
        case 5: return launch_flow_t<512, 8, 5, 3>(P, stop_live, grid, st);
        case 6: return launch_flow_t<512, 8, 6, 3>(P, stop_live, grid, st);
        case 7: return launch_flow_t<512, 8, 7, 4>(P, stop_live, grid, st);
        default: return launch_flow_t<512, 8, 8, 4>(P, stop_live, grid, st);
        }
    }
    switch ((RB + 15) / 16) {
    case 5: return launch_flow_t<512, 8, 8, 5>(P, stop_live, grid, st);
    case 6: return launch_flow_t<512, 8, 8, 6>(P, stop_live, grid, st);
    case 7: return launch_flow_t<512, 8, 8, 7>(P, stop_live, grid, st);
    case 8: return launch_flow_t<512, 8, 8, 8>(P, stop_live, grid, st);
    default: return cudaErrorInvalidValue;
    }
}

size_t solo_smem_bytes(const Params &P)
{
    return (size_t)((P.prop == 1 ? kRkSlots : 2) + 2) * (P.MD + 2) * sizeof(double2);
}

// Rows per CTA when C CTAs share a matrix of at most d rows (whole 8-row blocks).
static int solo_rows(int d, int C) { return 8 * ((d + 8 * C - 1) / (8 * C)); }

template <int C, int kPre>
static cudaError_t launch_solo_t(const Params &P, int workers, cudaStream_t st)
{
    const size_t smem = solo_smem_bytes(P);
    static std::atomic<unsigned long long> done{0};
    const cudaError_t e = allow_smem(solo_kernel<C, kPre>, done);
    if (e != cudaSuccess) return e;
    const int rows = solo_rows(P.d, C);
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(workers * C);
    lc.blockDim = dim3(32 * ((rows + 31) / 32));
    lc.dynamicSmemBytes = smem;
    lc.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    lc.attrs = at;
    lc.numAttrs = C > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&lc, solo_kernel<C, kPre>, P, rows);
}

// Eight k pairs in flight per thread where every CTA of the launch is resident with the registers
// that takes (a lone CTA's matvec at d = 201: 110 cycles per k pair against 137), else four.  (Four with two
// CTAs per SM leave 128 registers: with C > 1 the compiler spills about 24 of them, 400 bytes of stores and 456 of
// loads per thread, with C = 1 two.)
template <int C>
static cudaError_t launch_solo_c(const Params &P, int workers, cudaStream_t st)
{
    const int threads = 32 * ((solo_rows(P.d, C) + 31) / 32), per_sm = (workers * C + P.grid - 1) / P.grid;
    return per_sm * threads * 256 <= 65536 ? launch_solo_t<C, 8>(P, workers, st) : launch_solo_t<C, 4>(P, workers, st);
}

// `workers` clusters of C CTAs (C a power of two up to 8, at least d / kSoloThreads).
cudaError_t launch_solo(const Params &P, int C, int workers, cudaStream_t st)
{
    switch (C) {
    case 1: return launch_solo_c<1>(P, workers, st);
    case 2: return launch_solo_c<2>(P, workers, st);
    case 4: return launch_solo_c<4>(P, workers, st);
    case 8: return launch_solo_c<8>(P, workers, st);
    default: return cudaErrorInvalidValue;
    }
}

// Padded rows for dimension d: whole 8-row blocks (the m8n8k4 row block).
int pick_layout(int d, int *rows_per_block)
{
    *rows_per_block = 8;
    return 8 * ((d + 7) / 8);
}

// Shared memory of the plain kernel: nc staged columns of MD + kColPad components (columns 32
// bytes apart modulo the banks: conflict-free B operand reads) and two slabs of kb k rows.
size_t step_smem_bytes(int MD, int nc, int kb)
{
    return (size_t)(nc * (MD + kColPad) + 2 * kb * MD) * sizeof(double2);
}

// Static shared memory of the plain kernel with nt threads (the same for every instantiation).
size_t step_static_smem(int nt)
{
    cudaFuncAttributes a{};
    const cudaError_t e = nt == 256 ? cudaFuncGetAttributes(&a, flow_kernel<256, 1, 1, 2>)
                                    : cudaFuncGetAttributes(&a, flow_kernel<512, 8, 4, 2>);
    if (e != cudaSuccess) return 16384;
    return a.sharedSizeBytes;
}

// Widest sub-tile (at most nc_max: 32, 16 or 8 columns) whose staged columns leave room for slabs
// of at least 8 k rows (at most 16, even) in `budget` bytes of dynamic shared memory, with at most
// 8 row blocks per warp; failing that, the widest with 2-row slabs.  Returns false when none fits.
bool pick_step_tiles(int MD, size_t budget, int nt, int nc_max, int *nc, int *kb)
{
    const int RB = MD / 8;
    for (int min_kb = 8; min_kb >= 2; min_kb -= 6) {
        for (int c = nc_max; c >= 8; c /= 2) {
            const int W1 = nt / 32 / (c / 8);  // warps per column block
            if ((RB + W1 - 1) / W1 > 8) continue;
            const size_t bt = (size_t)c * (MD + kColPad) * sizeof(double2);
            if (bt >= budget) continue;
            int k = (int)((budget - bt) / ((size_t)2 * MD * sizeof(double2)));
            k = std::min(k, kKB) & ~1;
            if (k < min_kb) continue;
            *nc = c;
            *kb = k;
            return true;
        }
    }
    return false;
}

// The first lock-step micro-step after a host-side enqueue needs its plan.
cudaError_t launch_split_plan(const Params &P, cudaStream_t st);

static cudaError_t launch_plan(const Params &P, cudaStream_t st)
{
    return P.flow ? cudaGetLastError() : launch_split_plan(P, st);
}

cudaError_t launch_schedule(const Params &P, int mode, cudaStream_t st)
{
    schedule_kernel<<<(P.n + 255) / 256, 256, 0, st>>>(P, mode);
    return launch_plan(P, st);
}

cudaError_t launch_observe(const Params &P, int dump, int is_start, cudaStream_t st)
{
    const size_t smem = (size_t)8 * P.MD * sizeof(double2);
    static bool attr_set = false;
    if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(observe_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)(8 * kMaxMD * sizeof(double2)));
        if (e != cudaSuccess) return e;
        attr_set = true;
    }
    observe_kernel<<<(P.n + 7) / 8, 256, smem, st>>>(P, dump, is_start);
    return launch_plan(P, st);
}

cudaError_t launch_purity(const Params &P, double2 *hat, double2 *rho, double *out, cudaStream_t st)
{
    normalize_kernel<<<(P.n + 7) / 8, 256, 0, st>>>(P, hat);
    const int RB = (P.d + 7) / 8, blocks = RB * RB;
    // output blocks per CTA: all CTAs on the chip at once where there are few, at most kRhoBlocks
    const int per = std::max(1, std::min(kRhoBlocks, (blocks + P.grid - 1) / P.grid));
    static std::atomic<unsigned long long> done{0};
    const cudaError_t e = allow_smem(rho_kernel, done);
    if (e != cudaSuccess) return e;
    rho_kernel<<<(blocks + per - 1) / per, 64 * per + kRhoLoaders, rho_smem_bytes(per), st>>>(P, hat, rho, per);
    purity_kernel<<<1, kPurityThreads, 0, st>>>(rho, P.d * P.d, out);
    return cudaGetLastError();
}

// Start of a run with the RK propagator: step 0 of the first period from psi (warp per trajectory).
__global__ void rk_schedule_kernel(const Params P)
{
    const int lane = threadIdx.x & 31;
    const int tr = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (tr >= P.n) return;
    TrajState s = P.st[tr];
    if (s.phase == PH_ERROR) return;
    const double nrm = warp_norm(slot_ptr(P, s.cur, tr), P.d, lane);
    s.pc = 0;
    s.di = 0;
    s.paused = 0;
    s.rk_sid = 0;
    if (P.target > 0 && runs(P, tr)) {
        s.t = rk_step_time(P, s);
        rk_begin(s, P.rk_step, nrm, 0);
    } else {
        s.phase = PH_DONE;
    }
    if (lane == 0) {
        P.st[tr] = s;
        if (s.phase == PH_RK) enqueue(P, P.e_g0[s.ens], tr);
    }
}

cudaError_t launch_rk_schedule(const Params &P, cudaStream_t st)
{
    rk_schedule_kernel<<<(P.n + 7) / 8, 256, 0, st>>>(P);
    return launch_plan(P, st);
}

cudaError_t launch_init_state(const Params &P, cudaStream_t st, int tr0, int tr1)
{
    if (tr1 < 0) tr1 = P.n;
    if (tr1 <= tr0) return cudaSuccess;
    init_state_kernel<<<(tr1 - tr0 + 255) / 256, 256, 0, st>>>(P, tr0, tr1);
    return cudaGetLastError();
}

cudaError_t launch_thresholds(const Params &P, cudaStream_t st, int tr0, int tr1)
{
    if (tr1 < 0) tr1 = P.n;
    if (tr1 <= tr0) return cudaSuccess;
    thresholds_kernel<<<(tr1 - tr0 + 255) / 256, 256, 0, st>>>(P, tr0, tr1);
    return cudaGetLastError();
}

cudaError_t launch_reset_times(const Params &P, cudaStream_t st)
{
    reset_times_kernel<<<(P.n + 255) / 256, 256, 0, st>>>(P);
    return cudaGetLastError();
}

// FP64 FMA throughput microbenchmark: 8 independent fma chains per thread.
__global__ void fp64_peak_kernel(double *out, int iters, double a, double b)
{
    double x[8];
#pragma unroll
    for (int i = 0; i < 8; i++) x[i] = threadIdx.x * 1e-9 + i;
    for (int it = 0; it < iters; it++) {
#pragma unroll
        for (int i = 0; i < 8; i++) x[i] = __fma_rn(x[i], a, b);
    }
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < 8; i++) s += x[i];
    if (s == 12345.678) out[0] = s;  // keeps the chains live
}

// FP64 tensor-core throughput microbenchmark: 8 independent m8n8k4 accumulator chains per warp.
__global__ void dmma_peak_kernel(double *out, int iters, double a, double b)
{
    double c[8][2];
#pragma unroll
    for (int i = 0; i < 8; i++) c[i][0] = c[i][1] = threadIdx.x * 1e-9 + i;
    for (int it = 0; it < iters; it++) {
#pragma unroll
        for (int i = 0; i < 8; i++) dmma(c[i][0], c[i][1], a, b);
    }
    double s = 0.0;
#pragma unroll
    for (int i = 0; i < 8; i++) s += c[i][0] + c[i][1];
    if (s == 12345.678) out[0] = s;
}

cudaError_t launch_dmma_peak(double *out, int blocks, int iters, cudaStream_t st)
{
    dmma_peak_kernel<<<blocks, 256, 0, st>>>(out, iters, 1e-3, 1e-3);
    return cudaGetLastError();
}

cudaError_t launch_fp64_peak(double *out, int blocks, int iters, cudaStream_t st)
{
    fp64_peak_kernel<<<blocks, 256, 0, st>>>(out, iters, 0.9999999, 1e-7);
    return cudaGetLastError();
}

cudaError_t launch_clear_records(const Params &P, cudaStream_t st)
{
    clear_records_kernel<<<(P.n + 255) / 256, 256, 0, st>>>(P);
    return cudaGetLastError();
}

// ---------------------------------------------------------------- split-precision form
#include "qjx_split.cuh"

cudaError_t launch_split_plan(const Params &P, cudaStream_t st)
{
    split_plan_kernel<<<1, 512, 0, st>>>(P, P.grid);
    return cudaGetLastError();
}

// Static shared memory of the split kernel (the same in both modes).
size_t split_static_smem()
{
    cudaFuncAttributes a{}, b{};
    if (cudaFuncGetAttributes(&a, split_kernel<true>) != cudaSuccess ||
        cudaFuncGetAttributes(&b, split_kernel<false>) != cudaSuccess)
        return 32768;
    return std::max(a.sharedSizeBytes, b.sharedSizeBytes);
}

template <bool FLOW>
static cudaError_t launch_split(const Params &P, int s, int grid, cudaStream_t st)
{
    static std::atomic<unsigned long long> done{0};
    const cudaError_t e = allow_smem(split_kernel<FLOW>, done);
    if (e != cudaSuccess) return e;
    split_kernel<FLOW><<<grid, kThreads, split_smem_bytes(P.MDs, P.MD, P.sstages), st>>>(P, s);
    return cudaGetLastError();
}

// One time slice of the split form, or its lock-step micro-step s.
cudaError_t launch_split_flow(const Params &P, int grid, cudaStream_t st) { return launch_split<true>(P, 0, grid, st); }
cudaError_t launch_split_step(const Params &P, int s, int grid, cudaStream_t st) { return launch_split<false>(P, s, grid, st); }

// The most matvecs (rechecks included) of one trajectory since the counts were cleared, into P.sdone.
__global__ void __launch_bounds__(1024) longest_chain_kernel(const Params P)
{
    __shared__ int s_max;
    if (threadIdx.x == 0) s_max = 0;
    __syncthreads();
    int m = 0;
    for (int i = threadIdx.x; i < P.n; i += 1024) m = max(m, P.chain[i]);
    atomicMax(&s_max, m);
    __syncthreads();
    if (threadIdx.x == 0) *P.sdone = s_max;
}

cudaError_t launch_longest_chain(const Params &P, cudaStream_t st)
{
    longest_chain_kernel<<<1, 1024, 0, st>>>(P);
    return cudaGetLastError();
}

}  // namespace qjx
