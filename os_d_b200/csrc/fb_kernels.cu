// fb_kernels.cu -- f-basis Lindblad RK4 on the GPU (density-matrix oracle of the QJ ensemble).
//
// The reference integrates dx/dt = Gs x + E(t) Qs_drv x - Ks with classic RK4
// (source/cpp/CQdiss_os_dimer/CQdiss/calcODE.cpp:75-118 calcVectValue_real, :249-389
// calcODE_trans/std), two mkl_dcsrgemv per stage.  GPU paths:
//   * resident forms, one launch per period: rk4_cluster holds the whole system in the shared memory
//     of one thread-block cluster, rk4_grid spreads a larger one over every SM;
//   * rk_stage: one launch per RK stage (four per step) computes both CSR row products, the
//     stage vector k = (Gs x + drv Qs x - Ks) h and the next stage argument, or in stage 4 the
//     RK4 update of x.  The stage arguments are double-buffered (stage s reads one buffer and
//     writes the other), as the reference keeps x, tmp and k1..k4 apart (calcODE.cpp:249-309):
//     a row may read any other row's argument, and rows of one launch run in no fixed order.
//
// Canonical row sum (shared bit-for-bit with the CPU oracle): lane l of a warp accumulates
// the row's nonzeros l, l+32, l+64, ... in CSR order with fma, then the 32 partial sums are
// combined by an xor butterfly (offsets 16, 8, 4, 2, 1).  All other arithmetic is literal
// (-fmad=false).  The drive uses sin() of the stage time (CUDA libdevice), so drv_type 1
// matches the CPU within rounding, not bit-for-bit.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "../../include/qjx_b200.h"

namespace fb {

struct FbParams {
    int n;
    const int *gr, *gc;
    const double *gv;
    const int *qr, *qc;
    const double *qv;
    const double *Ks;
    double drv_ampl;  // -A (calcODE.cpp:91)
    double drv_freq, drv_phase;
    int drv_type;
    double *x;
    double *va, *vb;     // stage arguments: stage 1 writes va, 2 writes vb, 3 writes va
    double *k1, *k2, *k3;
};

__device__ __forceinline__ double warp_row_sum(const int *rp, const int *ci, const double *v, const double *x, int row,
                                               int lane)
{
    double s = 0.0;
    const int b = rp[row], e = rp[row + 1];
    for (int j = b + lane; j < e; j += 32) s = __fma_rn(v[j], x[ci[j]], s);
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) s = __dadd_rn(s, __shfl_xor_sync(0xffffffffu, s, off));
    return s;
}

// Stage 1..4 of one RK4 step at time t (calcODE.cpp:278-302), one warp per row.  Stage s reads
// its argument (x, va, vb, va) and writes only a buffer no row of this launch reads (va, vb, va,
// and in stage 4 the row's own x: x += (k1 + 2 k2 + 2 k3 + k4) / 6, calcODE.cpp:299-302).
__global__ void rk_stage(const FbParams P, int stage, double t, double h)
{
    const int warps = blockDim.x >> 5;
    const int row = blockIdx.x * warps + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= P.n) return;
    const double *arg = (stage == 1) ? P.x : ((stage == 3) ? P.vb : P.va);
    const double tt = (stage == 1) ? t : ((stage == 4) ? __dadd_rn(t, h) : __dadd_rn(t, __ddiv_rn(h, 2.0)));
    const double t1 = warp_row_sum(P.gr, P.gc, P.gv, arg, row, lane);
    const double t2 = warp_row_sum(P.qr, P.qc, P.qv, arg, row, lane);
    if (lane != 0) return;
    double drv;
    const double sn = sin(__dadd_rn(__dmul_rn(P.drv_freq, tt), P.drv_phase));
    if (P.drv_type == 1) drv = __dmul_rn(P.drv_ampl, sn);
    else drv = __dmul_rn(P.drv_ampl, (sn < 0.0) ? -1.0 : 1.0);
    const double k = __dmul_rn(__dsub_rn(__dadd_rn(t1, __dmul_rn(drv, t2)), P.Ks[row]), h);
    const double x = P.x[row];
    if (stage == 1) {
        P.k1[row] = k;
        P.va[row] = __dadd_rn(x, __ddiv_rn(k, 2.0));
    } else if (stage == 2) {
        P.k2[row] = k;
        P.vb[row] = __dadd_rn(x, __ddiv_rn(k, 2.0));
    } else if (stage == 3) {
        P.k3[row] = k;
        P.va[row] = __dadd_rn(x, k);
    } else {
        const double sum =
            __dadd_rn(__dadd_rn(__dadd_rn(P.k1[row], __dmul_rn(2.0, P.k2[row])), __dmul_rn(2.0, P.k3[row])), k);
        P.x[row] = __dadd_rn(x, __ddiv_rn(sum, 6.0));
    }
}

// Queues the four stage launches of every RK4 step of n_periods periods from period0 on `st`;
// returns the first launch error (cudaLaunchKernelEx reports the launch's own status).
static cudaError_t queue_rk_stages(const FbParams &P, double T, int num_steps, int period0, int n_periods,
                                   cudaStream_t st)
{
    const double step = T / double(num_steps);  // data.cpp:10
    const int warps = 8;
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((P.n + warps - 1) / warps);
    lc.blockDim = dim3(warps * 32);
    lc.stream = st;
    for (int p = period0; p < period0 + n_periods; p++)
        for (int s = 0; s < num_steps; s++) {
            const double t = double(p) * T + double(s) * step;  // calcODE.cpp:280
            for (int stage = 1; stage <= 4; stage++) {
                const cudaError_t e = cudaLaunchKernelEx(&lc, rk_stage, P, stage, t, step);
                if (e != cudaSuccess) return e;
            }
        }
    return cudaSuccess;
}

// ---------------------------------------------------------------- resident RK4
// Both resident forms keep each CTA's rows in shared memory for a whole launch (a period).  Short rows
// (at most kW nonzeros and one of the drive, all but about N of the dimer's N^2) are held thread-per-row, nonzero l of
// consecutive rows side by side (no bank conflicts), padded with a zero value and a column that holds
// zero; long rows are done by a warp each, or (MANY) in slices of 32 rows, a thread each, where a CTA has more
// of them than warps.  Thread-per-row keeps the canonical order (lane partial
// sums over nonzeros l, l + 32, ..., then the butterfly tree): with at most kW <= 32 nonzeros each
// lane holds one product, and a level of the tree that pairs a product with an absent lane's +0.0
// changes nothing but a -0 into +0, which one addition at the end does for all.
constexpr int kW = 20;
constexpr long long kFbWait = 1ll << 24;  // polls of a wait before it gives up (default of QJX_FB_POLLS)

// Rows of one CTA: S short rows, then L long ones; row i of the CTA is entry base + i of the vectors.
struct FbRows {
    int base, S, L, ln;  // first entry, short rows, long rows, their nonzeros
};

struct FbResParams {
    int n;
    const FbRows *rows;                      // [CTAs]
    const double *ev;                        // short rows: [kW][RS] values per CTA (RS = maxS)
    const unsigned short *ec16;              // and columns (entry numbers; n: the zero)
    const int *ec32;                         // the same for the grid form
    const double *lv;                        // long rows: nonzeros, each row's (MANY: each slice's) of Gs, then of Qs
    const int *lc, *lp;                      // columns, starts [CTA][2 maxL + 1]: Gs of row or slice j at 2 j, Qs at 2 j + 1
    const double *ks, *qv;                   // per entry: constant term; short rows: drive value (0: none)
    const int *qc;                           // and column (n: none)
    const int *perm;                         // entry -> row of the caller's vectors
    double *x;
    double *buf;                             // grid form: two arguments [2][n + 1]
    unsigned *arrived;                       // grid form: CTAs that have passed a stage
    int *fail;                               // a wait that gave up (the launch's result is not valid then)
    long long polls;                         // polls of a wait before it gives up
    int maxS, maxL, maxN;                    // strides of the per-CTA arrays
    double drv_ampl, drv_freq, drv_phase;
    int drv_type;
    double T, h;
    int num_steps, period;
};

__device__ __forceinline__ double short_row(const double *val, int stride, const double (&x)[kW])
{
    double p[kW];
#pragma unroll
    for (int l = 0; l < kW; l++) p[l] = __fma_rn(val[l * stride], x[l], 0.0);
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1)
#pragma unroll
        for (int l = 0; l < off; l++)
            if (l + off < kW && (off == 16 || l + off < 2 * off)) p[l] = __dadd_rn(p[l], p[l + off]);
    return __dadd_rn(p[0], 0.0);
}

// Row sum of a long row by a warp (the canonical order itself).
template <class Load>
__device__ __forceinline__ double long_row(const double *v, const int *c, int b, int e, int lane, const Load &arg)
{
    double s = 0.0;
    for (int j = b + lane; j < e; j += 32) s = __fma_rn(v[j], arg(c[j]), s);
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) s = __dadd_rn(s, __shfl_xor_sync(0xffffffffu, s, off));
    return s;
}

// Row sum of a long row by a thread: its nonzero l at v[32 l], a multiple of four of them (zero values of the zero
// column past the row's).
template <class Load>
__device__ __forceinline__ double slice_row(const double *v, const int *c, int len, const Load &arg)
{
    double p[32];
#pragma unroll
    for (int l = 0; l < 32; l++) p[l] = 0.0;
    for (int j = 0; j < len; j += 32) {
#pragma unroll
        for (int l = 0; l < 32; l += 4) {
            if (j + l >= len) break;
#pragma unroll
            for (int i = l; i < l + 4; i++) p[i] = __fma_rn(v[32 * (j + i)], arg(c[32 * (j + i)]), p[i]);
        }
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1)
#pragma unroll
        for (int l = 0; l < off; l++) p[l] = __dadd_rn(p[l], p[l + off]);
    return p[0];
}

// The long rows of a CTA in a stage: emit(i, t1, t2) gets entry i and its two row sums, from one thread.
template <bool MANY, class Load, class Emit>
__device__ __forceinline__ void long_rows(const FbRows &r, const double *lv, const int *lc, const int *lp, int warp, int nw, int lane,
                                          const Load &arg, const Emit &emit)
{
    if (MANY) {
        for (int j = nw - 1 - warp; 32 * j < r.L; j += nw) {
            const int g = lp[2 * j], q = lp[2 * j + 1], e = lp[2 * j + 2];
            const double t1 = slice_row(lv + g + lane, lc + g + lane, (q - g) >> 5, arg);
            const double t2 = slice_row(lv + q + lane, lc + q + lane, (e - q) >> 5, arg);
            if (32 * j + lane < r.L) emit(r.S + 32 * j + lane, t1, t2);
        }
    } else {
        for (int j = nw - 1 - warp; j < r.L; j += nw) {
            const double t1 = long_row(lv, lc, lp[2 * j], lp[2 * j + 1], lane, arg);
            const double t2 = long_row(lv, lc, lp[2 * j + 1], lp[2 * j + 2], lane, arg);
            if (lane == 0) emit(r.S + j, t1, t2);
        }
    }
}

// drv of stage 1 (j = 0), 2 and 3 (j = 1) or 4 (j = 2) of step s (calcODE.cpp:84-94, 278-302)
__device__ __forceinline__ double stage_drive(const FbResParams &P, int s, int j)
{
    const double t = __dadd_rn(__dmul_rn((double)P.period, P.T), __dmul_rn((double)s, P.h));
    const double tt = j == 0 ? t : (j == 2 ? __dadd_rn(t, P.h) : __dadd_rn(t, __ddiv_rn(P.h, 2.0)));
    const double sn = sin(__dadd_rn(__dmul_rn(P.drv_freq, tt), P.drv_phase));
    return P.drv_type == 1 ? __dmul_rn(P.drv_ampl, sn) : __dmul_rn(P.drv_ampl, (sn < 0.0) ? -1.0 : 1.0);
}

// Shared memory of a CTA's rows (both forms): per-row vectors, short-row values, long-row values, then
// the integers.
struct FbSmem {
    double *x, *k1, *k2, *k3, *ks, *qv, *ev, *lv, *drv;
    int *qc, *lc, *lp;
};

__host__ __device__ inline size_t fb_rows_bytes(int maxS, int maxL, int maxN)
{
    return sizeof(double) * (6 * (size_t)(maxS + maxL) + (size_t)kW * maxS + maxN + 6) +
           sizeof(int) * ((size_t)(maxS + maxL) + maxN + 2 * (size_t)maxL + 2);
}

__device__ __forceinline__ FbSmem fb_carve(const FbResParams &P, unsigned char *smem)
{
    FbSmem m;
    const int R = P.maxS + P.maxL;
    m.x = reinterpret_cast<double *>(smem);
    m.k1 = m.x + R;
    m.k2 = m.k1 + R;
    m.k3 = m.k2 + R;
    m.ks = m.k3 + R;
    m.qv = m.ks + R;
    m.ev = m.qv + R;
    m.lv = m.ev + (size_t)kW * P.maxS;
    m.drv = m.lv + P.maxN;  // [2][3]
    m.qc = reinterpret_cast<int *>(m.drv + 6);
    m.lc = m.qc + R;
    m.lp = m.lc + P.maxN;
    return m;
}

// Whether a wait of this run has given up.
__device__ __forceinline__ bool fb_failed(const FbResParams &P)
{
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(P.fail) : "memory");
    return v != 0;
}

// Loads a CTA's rows and the first step's drive (CTA-wide; the caller synchronises).
__device__ __forceinline__ void fb_load_rows(const FbResParams &P, int cta, const FbRows &r, const FbSmem &m)
{
    const int tid = threadIdx.x, nt = blockDim.x;
    for (int i = tid; i < r.S + r.L; i += nt) {
        m.x[i] = P.x[P.perm[r.base + i]];
        m.ks[i] = P.ks[r.base + i];
        m.qv[i] = P.qv[r.base + i];
        m.qc[i] = P.qc[r.base + i];
    }
    for (int i = tid; i < kW * P.maxS; i += nt) m.ev[i] = P.ev[(size_t)cta * kW * P.maxS + i];
    for (int i = tid; i < r.ln; i += nt) {
        m.lv[i] = P.lv[(size_t)cta * P.maxN + i];
        m.lc[i] = P.lc[(size_t)cta * P.maxN + i];
    }
    for (int i = tid; i <= 2 * r.L; i += nt) m.lp[i] = P.lp[(size_t)cta * (2 * P.maxL + 1) + i];
    if (tid < 3) m.drv[tid] = stage_drive(P, 0, tid);
}

// Row i of a stage from its two row sums: k = (Gs x + drv Qs x - Ks) h and the entry of the next
// stage's argument, or in stage 4 of the new x (calcODE.cpp:95-117, 278-302).
__device__ __forceinline__ double fb_finish(const FbResParams &P, const FbSmem &m, int stage, int i, double t1, double t2,
                                            double drv)
{
    const double k = __dmul_rn(__dsub_rn(__dadd_rn(t1, __dmul_rn(drv, t2)), m.ks[i]), P.h);
    const double x = m.x[i];
    if (stage == 1) {
        m.k1[i] = k;
        return __dadd_rn(x, __ddiv_rn(k, 2.0));
    }
    if (stage == 2) {
        m.k2[i] = k;
        return __dadd_rn(x, __ddiv_rn(k, 2.0));
    }
    if (stage == 3) {
        m.k3[i] = k;
        return __dadd_rn(x, k);
    }
    const double sum = __dadd_rn(__dadd_rn(__dadd_rn(m.k1[i], __dmul_rn(2.0, m.k2[i])), __dmul_rn(2.0, m.k3[i])), k);
    const double v = __dadd_rn(x, __ddiv_rn(sum, 6.0));
    m.x[i] = v;
    return v;
}

// ---- cluster form: the whole system in the shared memory of one cluster of at most 16 CTAs
constexpr int kMaxCluster = 16, kClusterThreads = 512, kClusterRows = 192;

__device__ __forceinline__ uint32_t fb_smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint32_t fb_map(uint32_t addr, int rank)
{
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    return a;
}

__device__ __forceinline__ bool fb_wait(uint32_t bar, uint32_t parity, long long polls)
{
    for (long long i = 0; i < polls; i++) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// Every CTA holds full copies of two arguments, used in turn; a stage's entries are stored into every
// CTA with st.async, whose bytes complete the receiver's mbarrier of that stage: a CTA goes on when
// all n entries have arrived, with no cluster barrier (two round trips) and no wait for stores to be
// acknowledged.  Two mbarriers and two arguments are enough: a CTA can send entries of stage s + 1
// only after it has all of stage s, so after every CTA has finished reading the argument of stage s
// (the one that stage s + 1 overwrites is that of stage s - 1).  That holds for warps with rows, whose
// entries the next stage needs, and for the two that arrive at the mbarrier; the others (about half
// at N = 50) skip the stages: nothing would keep the cluster from getting two stages ahead of one, whose
// mbarrier would then show the old parity again.  One warp works out the next step's drive values
// meanwhile.  A thread whose wait gives up runs on to the end without waiting, sending or arriving (its
// mbarriers may not take more than a stage brings), so every other wait ends too.
// Bound: the latency of a stage (gather, row sum, st.async, mbarrier),
// 1.5 us at N = 50.  Before (cluster barriers, thread-per-row CSR with a 32-lane pass, every thread
// its own sine): 2.9 us.
template <bool MANY>
__global__ void __launch_bounds__(kClusterThreads, 1) rk4_cluster(const FbResParams P, int cs)
{
    extern __shared__ __align__(16) unsigned char fsm[];
    __shared__ __align__(8) uint64_t bar[2];
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
    const int n = P.n;
    if (fb_failed(P)) return;  // (in an earlier period: the same for every CTA)
    int rank;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    double *buf = reinterpret_cast<double *>(fsm);  // [2][n + 1]
    const FbSmem m = fb_carve(P, fsm + sizeof(double) * 2 * (size_t)(n + 1));
    unsigned short *ec = reinterpret_cast<unsigned short *>(m.lp + 2 * P.maxL + 2);  // [kW][maxS]
    const FbRows r = P.rows[rank];
    fb_load_rows(P, rank, r, m);
    for (int i = tid; i < kW * P.maxS; i += nt) ec[i] = P.ec16[(size_t)rank * kW * P.maxS + i];
    for (int i = tid; i <= n; i += nt) {
        buf[i] = i < n ? P.x[P.perm[i]] : 0.0;
        if (i == n) buf[n + 1 + n] = 0.0;
    }
    const uint32_t bar0 = fb_smem_u32(bar);
    if (tid == 0) {
        for (int q = 0; q < 2; q++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 2;" ::"r"(bar0 + 8 * q) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    const bool works = warp == 0 || warp == nw - 1 || 32 * warp < r.S || (MANY ? 32 : 1) * (nw - 1 - warp) < r.L;
    int to = cs;      // CTAs that this thread sends to (0: its wait gave up)
    uint32_t it = 0;  // stages done
    for (int s = 0; works && s < P.num_steps; s++) {
#pragma unroll 1
        for (int stage = 1; stage <= 4; stage++, it++) {
            const double *arg = buf + (it & 1) * (size_t)(n + 1);
            const uint32_t out = fb_smem_u32(buf + ((it & 1) ^ 1) * (size_t)(n + 1) + r.base);
            const uint32_t mb = bar0 + 8 * (it & 1);
            const double drv = m.drv[3 * (s & 1) + (stage == 1 ? 0 : (stage == 4 ? 2 : 1))];
            auto send = [&](int i, double v) {
                for (int c = 0; c < to; c++)
                    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(
                                     fb_map(out + 8 * i, c)),
                                 "l"(__double_as_longlong(v)), "r"(fb_map(mb, c))
                                 : "memory");
            };
            auto drive_sum = [&](int i) { return __dadd_rn(__fma_rn(m.qv[i], arg[m.qc[i]], 0.0), 0.0); };
            for (int i = tid; i < r.S; i += nt) {
                double x[kW];
#pragma unroll
                for (int l = 0; l < kW; l++) x[l] = arg[ec[l * P.maxS + i]];
                const double t1 = short_row(m.ev + i, P.maxS, x);
                send(i, fb_finish(P, m, stage, i, t1, drive_sum(i), drv));
            }
            long_rows<MANY>(r, m.lv, m.lc, m.lp, warp, nw, lane, [&](int c) { return arg[c]; },
                            [&](int i, double t1, double t2) { send(i, fb_finish(P, m, stage, i, t1, t2, drv)); });
            if (warp == nw - 1) {
                if (stage == 1 && lane < 3) m.drv[3 * ((s + 1) & 1) + lane] = stage_drive(P, s + 1, lane);
                __syncwarp();
                if (lane == 0 && to) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mb) : "memory");
            }
            if (tid == 0 && to)
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mb), "r"(8 * n) : "memory");
            if (to && !fb_wait(mb, (it >> 1) & 1, P.polls)) {
                to = 0;
                atomicExch(P.fail, 1);
            }
            __syncwarp();  // (no lane starts a stage while another still waits for the one before)
        }
    }
    // every thread is past its last stage, so all stores into this CTA have arrived, unless a wait gave up:
    // then they get 100 us to
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (fb_failed(P)) {
        for (int i = 0; i < 100; i++) __nanosleep(1000);
        return;
    }
    for (int i = tid; i < r.S + r.L; i += nt) P.x[P.perm[r.base + i]] = m.x[i];
}

// ---- grid form: systems too large for a cluster, on every SM
// The rows of the system over all CTAs of one cooperative launch, the two arguments in global memory
// (L2), a bounded grid barrier per stage.  Bound: the latency of a stage (L2 gather, row sum, barrier),
// 3.3 us at N = 100; one launch per stage before this took 8.2 us.
constexpr int kGridThreads = 256;

template <bool MANY>
__global__ void __launch_bounds__(kGridThreads, 1) rk4_grid(const FbResParams P)
{
    extern __shared__ __align__(16) unsigned char fsm[];
    __shared__ int s_ok;
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
    const int n = P.n, cta = blockIdx.x;
    if (fb_failed(P)) return;  // (in an earlier period; in this one the other CTAs' waits give up too)
    const FbSmem m = fb_carve(P, fsm);
    int *ec = m.lp + 2 * P.maxL + 2;  // [kW][maxS]
    const FbRows r = P.rows[cta];
    fb_load_rows(P, cta, r, m);
    for (int i = tid; i < kW * P.maxS; i += nt) ec[i] = P.ec32[(size_t)cta * kW * P.maxS + i];
    if (tid == 0) s_ok = 1;
    __syncthreads();
    uint32_t it = 0;  // barriers passed
    auto sync = [&] {
        __syncthreads();
        it++;
        if (tid == 0) {
            __threadfence();
            atomicAdd(P.arrived, 1u);
            const unsigned want = it * gridDim.x;
            long long i = 0;
            unsigned v;
            do {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(P.arrived) : "memory");
            } while ((int)(v - want) < 0 && ++i < P.polls);
            if ((int)(v - want) < 0) {
                s_ok = 0;
                atomicExch(P.fail, 1);
            }
            __threadfence();
        }
        __syncthreads();
        return s_ok != 0;
    };
    for (int i = tid; i < r.S + r.L; i += nt) __stcg(P.buf + r.base + i, m.x[i]);
    if (cta == 0 && tid < 2) __stcg(P.buf + tid * (size_t)(n + 1) + n, 0.0);
    bool ok = sync();
    uint32_t q = 0;  // argument in use
    for (int s = 0; s < P.num_steps && ok; s++) {
#pragma unroll 1
        for (int stage = 1; stage <= 4 && ok; stage++) {
            const double *arg = P.buf + q * (size_t)(n + 1);
            double *out = P.buf + (q ^ 1) * (size_t)(n + 1) + r.base;
            const double drv = m.drv[3 * (s & 1) + (stage == 1 ? 0 : (stage == 4 ? 2 : 1))];
            auto drive_sum = [&](int i) { return __dadd_rn(__fma_rn(m.qv[i], __ldcg(arg + m.qc[i]), 0.0), 0.0); };
            for (int i = tid; i < r.S; i += nt) {
                double x[kW];
#pragma unroll
                for (int l = 0; l < kW; l++) x[l] = __ldcg(arg + ec[l * P.maxS + i]);
                const double t2 = drive_sum(i);
                const double t1 = short_row(m.ev + i, P.maxS, x);
                __stcg(out + i, fb_finish(P, m, stage, i, t1, t2, drv));
            }
            long_rows<MANY>(r, m.lv, m.lc, m.lp, warp, nw, lane, [&](int c) { return __ldcg(arg + c); },
                            [&](int i, double t1, double t2) { __stcg(out + i, fb_finish(P, m, stage, i, t1, t2, drv)); });
            if (stage == 1 && warp == nw - 1 && lane < 3) m.drv[3 * ((s + 1) & 1) + lane] = stage_drive(P, s + 1, lane);
            q ^= 1;
            ok = sync();
        }
    }
    if (ok)
        for (int i = tid; i < r.S + r.L; i += nt) P.x[P.perm[r.base + i]] = m.x[i];
}

}  // namespace fb

struct qjx_fb {
    fb::FbParams P{};
    // resident forms: cs CTAs of one cluster, or `grid` CTAs of a cooperative launch (neither: stage kernels)
    int cs = 0, grid = 0;
    bool many = false;  // long rows in slices
    size_t smem = 0;
    fb::FbResParams R{};
    double *x0 = nullptr;   // x before the call, for a call in which a wait gives up
    int device = 0;
    double T = 0.0;
    int num_steps = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    std::vector<void *> allocs;
    double last_ms = 0.0;
};

static void *fb_alloc(qjx_fb *h, size_t bytes)
{
    void *p = nullptr;
    if (cudaMalloc(&p, bytes ? bytes : 16) != cudaSuccess) return nullptr;
    h->allocs.push_back(p);
    return p;
}

// The caller's system (host CSR).
struct FbSystem {
    int n;
    const int *gr, *gc;
    const double *gv;
    const int *qr, *qc;
    const double *qv;
    const double *ks;
};

// The rows dealt to `nc` CTAs and their shared-memory form: the rows of each nonzero count, in their
// natural order (neighbours read neighbouring columns), cut into nc equal runs, so every CTA gets the
// same mix.  Entries of the vectors are numbered CTA after CTA, short rows first.
struct FbDeal {
    std::vector<fb::FbRows> rows;
    std::vector<int> perm, pos;  // entry -> row, row -> entry
    int maxS = 0, maxL = 0, maxN = 0;
    bool many = false;  // a CTA has more long rows than warps: slices of 32
};

static int fb_pad4(int k) { return (k + 3) & ~3; }

// Nonzeros of Gs and Qs (each a multiple of four) that slice j of a CTA's long rows holds per row.
static void fb_slice(const FbSystem &y, const FbDeal &d, const fb::FbRows &r, int j, int &g, int &q)
{
    g = q = 0;
    for (int i = 32 * j; i < std::min(r.L, 32 * j + 32); i++) {
        const int row = d.perm[r.base + r.S + i];
        g = std::max(g, fb_pad4(y.gr[row + 1] - y.gr[row]));
        q = std::max(q, fb_pad4(y.qr[row + 1] - y.qr[row]));
    }
}

static void fb_deal(const FbSystem &y, int nc, int warps, FbDeal &d)
{
    const int n = y.n;
    // a row's nonzeros; past kW (long) also when its drive has several
    std::vector<int> nnz(n), order(n), first;
    int most = 0;
    for (int i = 0; i < n; i++) {
        const int g = y.gr[i + 1] - y.gr[i], q = y.qr[i + 1] - y.qr[i];
        nnz[i] = q > 1 ? fb::kW + 1 + g + q : g;
        most = std::max(most, nnz[i]);
    }
    first.assign(most + 2, 0);
    for (int i = 0; i < n; i++) first[nnz[i] + 1]++;
    for (int k = 0; k <= most; k++) first[k + 1] += first[k];
    const std::vector<int> runs = first;  // rows of k nonzeros: order[runs[k]] .. order[runs[k + 1] - 1]
    for (int i = 0; i < n; i++) order[first[nnz[i]]++] = i;
    std::vector<std::vector<int>> mine(nc);
    for (auto &m : mine) m.reserve(n / nc + 64);
    int turn = 0;  // where the remainders of a count go next
    for (int k = 0; k <= most; k++) {
        const int i = runs[k], j = runs[k + 1];
        const int per = (j - i) / nc;
        for (int c = 0; c < nc; c++) mine[c].insert(mine[c].end(), order.begin() + i + c * per, order.begin() + i + (c + 1) * per);
        for (int l = i + nc * per; l < j; l++, turn++) mine[turn % nc].push_back(order[l]);
    }
    d = FbDeal();
    d.perm.reserve(n);
    d.pos.assign(n, 0);
    for (int c = 0; c < nc; c++) {
        fb::FbRows r{(int)d.perm.size(), 0, 0, 0};
        for (int i : mine[c]) {  // ascending counts: the long rows are last
            if (nnz[i] <= fb::kW) {
                r.S++;
            } else {
                r.L++;
                r.ln += y.gr[i + 1] - y.gr[i] + y.qr[i + 1] - y.qr[i];
            }
            d.pos[i] = (int)d.perm.size();
            d.perm.push_back(i);
        }
        d.rows.push_back(r);
        d.maxS = std::max(d.maxS, r.S);
        d.maxL = std::max(d.maxL, r.L);
    }
    // Where the line lies: a warp takes about 1.1 us per long row, one after the other, a slice about as long as
    // one or two of them (2600 rows of 25 nonzeros in a cluster, us a stage: 11.8 by warps, 2.1 in slices, 2.9 before
    // both as CSR rows between cluster barriers; 40,000 of 40 in the grid form: 42.7, 7.6, stage kernels 16.9).
    d.many = d.maxL > warps;
    for (fb::FbRows &r : d.rows) {
        if (d.many) {
            r.ln = 0;
            for (int j = 0; 32 * j < r.L; j++) {
                int g, q;
                fb_slice(y, d, r, j, g, q);
                r.ln += 32 * (g + q);
            }
        }
        d.maxN = std::max(d.maxN, r.ln);
    }
    d.maxS = std::max(32, (d.maxS + 31) & ~31);
}

// One device allocation for several arrays: room() for each, then alloc(), then at().
struct FbArena {
    size_t bytes = 0;
    unsigned char *dev = nullptr;
    template <class V>
    size_t room(size_t n)
    {
        const size_t at = bytes;
        bytes += (n * sizeof(V) + 15) & ~(size_t)15;
        return at;
    }
    bool alloc(qjx_fb *h) { return (dev = (unsigned char *)fb_alloc(h, bytes)) != nullptr; }
    template <class V>
    V *at(size_t off) const
    {
        return (V *)(dev + off);
    }
    template <class V>
    V *put(size_t off, const V *v, size_t n) const
    {
        if (n) cudaMemcpy(dev + off, v, n * sizeof(V), cudaMemcpyHostToDevice);
        return at<V>(off);
    }
};

static bool fb_upload_deal(qjx_fb *h, const FbSystem &y, const FbDeal &d, bool cluster)
{
    const int n = y.n, nc = (int)d.rows.size();
    const size_t nev = (size_t)nc * fb::kW * d.maxS, nlv = (size_t)nc * d.maxN, nlp = (size_t)nc * (2 * d.maxL + 1);
    FbArena a;
    const size_t orows = a.room<fb::FbRows>(nc), oev = a.room<double>(nev), olv = a.room<double>(nlv), oks = a.room<double>(n);
    const size_t oqv = a.room<double>(n), olc = a.room<int>(nlv), olp = a.room<int>(nlp), oqc = a.room<int>(n);
    const size_t operm = a.room<int>(n), oec = cluster ? a.room<unsigned short>(nev) : a.room<int>(nev);
    const size_t filled = a.bytes;
    const size_t ofail = a.room<int>(1), ox0 = a.room<double>(n), oarrived = a.room<unsigned>(1);
    const size_t obuf = a.room<double>(cluster ? 0 : 2 * ((size_t)n + 1));
    std::unique_ptr<unsigned char[]> host(new (std::nothrow) unsigned char[filled]);
    if (!host || !a.alloc(h)) return false;
    unsigned char *const at0 = host.get();
    double *const ev = (double *)(at0 + oev), *const lv = (double *)(at0 + olv), *const ks = (double *)(at0 + oks);
    double *const qv = (double *)(at0 + oqv);
    int *const lc = (int *)(at0 + olc), *const lp = (int *)(at0 + olp), *const qc = (int *)(at0 + oqc);
    std::memcpy(at0 + orows, d.rows.data(), nc * sizeof(fb::FbRows));
    std::memcpy(at0 + operm, d.perm.data(), n * sizeof(int));
    std::fill(ev, ev + nev, 0.0);
    std::fill(lv, lv + nlv, 0.0);
    std::fill(qv, qv + n, 0.0);
    std::fill(lc, lc + nlv, n);
    std::fill(lp, lp + nlp, 0);
    std::fill(qc, qc + n, n);
    if (cluster) std::fill((unsigned short *)(at0 + oec), (unsigned short *)(at0 + oec) + nev, (unsigned short)n);
    else std::fill((int *)(at0 + oec), (int *)(at0 + oec) + nev, n);
    for (int c = 0; c < nc; c++) {
        const fb::FbRows &r = d.rows[c];
        int *const start = lp + (size_t)c * (2 * d.maxL + 1);
        double *const v = lv + (size_t)c * d.maxN;
        int *const col = lc + (size_t)c * d.maxN;
        for (int i = 0; i < r.S + r.L; i++) ks[r.base + i] = y.ks[d.perm[r.base + i]];
        for (int i = 0; i < r.S; i++) {
            const int row = d.perm[r.base + i], b = y.gr[row], len = y.gr[row + 1] - b;
            for (int l = 0; l < len; l++) {
                const size_t e = ((size_t)c * fb::kW + l) * d.maxS + i;
                ev[e] = y.gv[b + l];
                if (cluster) ((unsigned short *)(at0 + oec))[e] = (unsigned short)d.pos[y.gc[b + l]];
                else ((int *)(at0 + oec))[e] = d.pos[y.gc[b + l]];
            }
            if (y.qr[row + 1] > y.qr[row]) {
                qv[r.base + i] = y.qv[y.qr[row]];
                qc[r.base + i] = d.pos[y.qc[y.qr[row]]];
            }
        }
        // the nonzeros of long row i from `at` on, `step` apart
        auto put = [&](int i, const int *rp, const int *ci, const double *val, int at, int step) {
            const int row = d.perm[r.base + r.S + i];
            for (int l = rp[row]; l < rp[row + 1]; l++, at += step) {
                v[at] = val[l];
                col[at] = d.pos[ci[l]];
            }
            return at;
        };
        int at = 0;
        for (int j = 0; d.many && 32 * j < r.L; j++) {
            int g, q;
            fb_slice(y, d, r, j, g, q);
            start[2 * j + 1] = at + 32 * g;
            start[2 * j + 2] = at + 32 * (g + q);
            for (int i = 32 * j; i < std::min(r.L, 32 * j + 32); i++) {
                put(i, y.gr, y.gc, y.gv, at + i - 32 * j, 32);
                put(i, y.qr, y.qc, y.qv, start[2 * j + 1] + i - 32 * j, 32);
            }
            at = start[2 * j + 2];
        }
        for (int j = 0; !d.many && j < r.L; j++) {
            start[2 * j + 1] = put(j, y.gr, y.gc, y.gv, at, 1);
            start[2 * j + 2] = at = put(j, y.qr, y.qc, y.qv, start[2 * j + 1], 1);
        }
    }
    if (cudaMemcpy(a.dev, at0, filled, cudaMemcpyHostToDevice) != cudaSuccess) return false;
    fb::FbResParams &R = h->R;
    R.n = n;
    R.rows = a.at<fb::FbRows>(orows);
    R.ev = a.at<double>(oev);
    if (cluster) R.ec16 = a.at<unsigned short>(oec);
    else R.ec32 = a.at<int>(oec);
    R.lv = a.at<double>(olv);
    R.lc = a.at<int>(olc);
    R.lp = a.at<int>(olp);
    R.ks = a.at<double>(oks);
    R.qv = a.at<double>(oqv);
    R.qc = a.at<int>(oqc);
    R.perm = a.at<int>(operm);
    R.x = h->P.x;
    R.fail = a.at<int>(ofail);
    h->x0 = a.at<double>(ox0);
    R.arrived = a.at<unsigned>(oarrived);
    R.buf = a.at<double>(obuf);
    R.maxS = d.maxS;
    R.maxL = d.maxL;
    R.maxN = d.maxN;
    R.drv_ampl = h->P.drv_ampl;
    R.drv_freq = h->P.drv_freq;
    R.drv_phase = h->P.drv_phase;
    R.drv_type = h->P.drv_type;
    R.T = h->T;
    R.h = h->T / double(h->num_steps);
    R.num_steps = h->num_steps;
    h->many = d.many;
    return true;
}

// Lets a kernel take all the shared memory that the device gives a CTA.  The limit belongs to the kernel,
// not to a handle: set to what one handle needs, a smaller handle's creation would take it from a larger.
template <class Kernel>
static bool fb_allow_smem(Kernel *kernel, int optin)
{
    cudaFuncAttributes a{};
    return cudaFuncGetAttributes(&a, kernel) == cudaSuccess &&
           cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, optin - (int)a.sharedSizeBytes) ==
               cudaSuccess;
}

// The cluster form: the smallest cluster (a power of two up to 16) with at most kClusterRows rows a
// CTA, or 16, when its shared memory holds the system.
static bool fb_setup_cluster(qjx_fb *h, const FbSystem &y)
{
    if (y.n >= 65535) return false;  // 16-bit columns
    int optin = 0;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, h->device);
    int cs = 1;
    while (cs < fb::kMaxCluster && (y.n + cs - 1) / cs > fb::kClusterRows) cs *= 2;
    for (; cs <= fb::kMaxCluster; cs *= 2) {
        FbDeal d;
        fb_deal(y, cs, fb::kClusterThreads / 32, d);
        auto *const kernel = d.many ? fb::rk4_cluster<true> : fb::rk4_cluster<false>;
        const size_t bytes = sizeof(double) * 2 * ((size_t)y.n + 1) + fb::fb_rows_bytes(d.maxS, d.maxL, d.maxN) +
                             sizeof(unsigned short) * fb::kW * d.maxS + 16;
        if (bytes + 1024 > (size_t)optin) continue;
        if (!fb_allow_smem(kernel, optin) ||
            (cs > 8 && cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)) {
            cudaGetLastError();
            continue;
        }
        cudaLaunchConfig_t lc = {};
        lc.gridDim = dim3(cs);
        lc.blockDim = dim3(fb::kClusterThreads);
        lc.dynamicSmemBytes = bytes;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = cs;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        lc.attrs = at;
        lc.numAttrs = 1;
        int nclusters = 0;
        if (cudaOccupancyMaxActiveClusters(&nclusters, kernel, &lc) != cudaSuccess || nclusters < 1) {
            cudaGetLastError();
            continue;
        }
        if (!fb_upload_deal(h, y, d, true)) return false;
        h->cs = cs;
        h->smem = bytes;
        return true;
    }
    return false;
}

// The grid form: one CTA on every SM, when the shared memory holds each CTA's rows.
static bool fb_setup_grid(qjx_fb *h, const FbSystem &y)
{
    int optin = 0, sms = 0, coop = 0, per = 0;
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, h->device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, h->device);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, h->device);
    if (!coop || sms < 1) return false;
    FbDeal d;
    fb_deal(y, sms, fb::kGridThreads / 32, d);
    auto *const kernel = d.many ? fb::rk4_grid<true> : fb::rk4_grid<false>;
    const size_t bytes = fb::fb_rows_bytes(d.maxS, d.maxL, d.maxN) + sizeof(int) * fb::kW * d.maxS + 16;
    if (bytes + 1024 > (size_t)optin ||
        !fb_allow_smem(kernel, optin) ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, fb::kGridThreads, bytes) != cudaSuccess || per < 1) {
        cudaGetLastError();
        return false;
    }
    if (!fb_upload_deal(h, y, d, false)) return false;
    h->grid = sms;
    h->smem = bytes;
    return true;
}

extern "C" qjx_status qjx_fb_create(int n, const int *gs_rowptr, const int *gs_col, const double *gs_val,
                                    const int *qs_rowptr, const int *qs_col, const double *qs_val, const double *Ks,
                                    const double *x0, double drv_ampl, double drv_freq, double drv_phase, int drv_type,
                                    double T, int num_steps, int device, qjx_fb **out)
{
    if (n < 1 || !gs_rowptr || !gs_col || !gs_val || !qs_rowptr || !qs_col || !qs_val || !Ks || !x0 || !out ||
        num_steps < 1 || !(T > 0.0) || (drv_type != 0 && drv_type != 1))
        return QJX_ERR_INVALID_ARG;
    *out = nullptr;
    qjx_fb *h = new (std::nothrow) qjx_fb();
    if (!h) return QJX_ERR_OOM;
    h->device = device;
    h->T = T;
    h->num_steps = num_steps;
    if (cudaSetDevice(device) != cudaSuccess) {
        delete h;
        return QJX_ERR_CUDA;
    }
    cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking);
    cudaEventCreate(&h->e0);
    cudaEventCreate(&h->e1);
    fb::FbParams &P = h->P;
    P.n = n;
    P.drv_ampl = -drv_ampl;
    P.drv_freq = drv_freq;
    P.drv_phase = drv_phase;
    P.drv_type = drv_type;
    P.x = (double *)fb_alloc(h, sizeof(double) * n);
    if (!P.x) {
        qjx_fb_destroy(h);
        return QJX_ERR_OOM;
    }
    cudaMemcpy(P.x, x0, sizeof(double) * n, cudaMemcpyHostToDevice);
    // resident forms; QJX_FB_PATH=stages forces the per-stage kernels
    const char *path = std::getenv("QJX_FB_PATH");
    const bool stages = path && std::string(path) == "stages";
    const FbSystem sys{n, gs_rowptr, gs_col, gs_val, qs_rowptr, qs_col, qs_val, Ks};
    if (stages || !fb_setup_cluster(h, sys)) {
        // the stage kernels' system and vectors (for the grid form: where its CTAs cannot all be resident)
        const size_t gnz = gs_rowptr[n], qnz = qs_rowptr[n];
        FbArena a;
        const size_t gr = a.room<int>(n + 1), gc = a.room<int>(gnz), gv = a.room<double>(gnz), qr = a.room<int>(n + 1);
        const size_t qc = a.room<int>(qnz), qv = a.room<double>(qnz), ks = a.room<double>(n), v = a.room<double>(5 * (size_t)n);
        if (!a.alloc(h)) {
            qjx_fb_destroy(h);
            return QJX_ERR_OOM;
        }
        P.gr = a.put(gr, gs_rowptr, n + 1);
        P.gc = a.put(gc, gs_col, gnz);
        P.gv = a.put(gv, gs_val, gnz);
        P.qr = a.put(qr, qs_rowptr, n + 1);
        P.qc = a.put(qc, qs_col, qnz);
        P.qv = a.put(qv, qs_val, qnz);
        P.Ks = a.put(ks, Ks, n);
        P.va = a.at<double>(v);
        P.vb = P.va + n;
        P.k1 = P.vb + n;
        P.k2 = P.k1 + n;
        P.k3 = P.k2 + n;
        if (!stages) fb_setup_grid(h, sys);
    }
    if (cudaDeviceSynchronize() != cudaSuccess) {
        qjx_fb_destroy(h);
        return QJX_ERR_CUDA;
    }
    cudaGetLastError();
    *out = h;
    return QJX_OK;
}

extern "C" qjx_status qjx_fb_run(qjx_fb *h, int period0, int n_periods)
{
    if (!h || period0 < 0 || n_periods < 0) return QJX_ERR_INVALID_ARG;
    if (cudaSetDevice(h->device) != cudaSuccess) return QJX_ERR_CUDA;
    const fb::FbParams &P = h->P;
    cudaEventRecord(h->e0, h->stream);
    const bool resident = h->cs || h->grid;
    if (resident) {  // one launch per period
        cudaLaunchConfig_t lc = {};
        lc.gridDim = dim3(h->cs ? h->cs : h->grid);
        lc.blockDim = dim3(h->cs ? fb::kClusterThreads : fb::kGridThreads);
        lc.dynamicSmemBytes = h->smem;
        lc.stream = h->stream;
        cudaLaunchAttribute at[1];
        if (h->cs) {
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = h->cs;
            at[0].val.clusterDim.y = 1;
            at[0].val.clusterDim.z = 1;
        } else {
            at[0].id = cudaLaunchAttributeCooperative;
            at[0].val.cooperative = 1;
        }
        lc.attrs = at;
        lc.numAttrs = 1;
        const size_t xbytes = sizeof(double) * P.n;
        cudaMemsetAsync(h->R.fail, 0, sizeof(int), h->stream);
        cudaMemcpyAsync(h->x0, P.x, xbytes, cudaMemcpyDeviceToDevice, h->stream);
        const char *polls = std::getenv("QJX_FB_POLLS");
        for (int p = period0; p < period0 + n_periods; p++) {
            fb::FbResParams C = h->R;
            C.polls = polls ? std::atoll(polls) : fb::kFbWait;
            C.period = p;
            if (!h->cs) cudaMemsetAsync(C.arrived, 0, sizeof(unsigned), h->stream);
            const cudaError_t e =
                h->cs ? cudaLaunchKernelEx(&lc, h->many ? fb::rk4_cluster<true> : fb::rk4_cluster<false>, C, h->cs)
                      : cudaLaunchKernelEx(&lc, h->many ? fb::rk4_grid<true> : fb::rk4_grid<false>, C);
            if (e == cudaErrorCooperativeLaunchTooLarge && !h->cs) {
                // not every CTA can be resident (another context holds SMs): the stage kernels
                cudaGetLastError();
                h->grid = 0;
                if (fb::queue_rk_stages(P, h->T, h->num_steps, p, period0 + n_periods - p, h->stream) != cudaSuccess)
                    return QJX_ERR_CUDA;
                break;
            }
            if (e != cudaSuccess) return QJX_ERR_CUDA;
        }
    } else if (fb::queue_rk_stages(P, h->T, h->num_steps, period0, n_periods, h->stream) != cudaSuccess) {
        return QJX_ERR_CUDA;
    }
    cudaEventRecord(h->e1, h->stream);
    if (cudaEventSynchronize(h->e1) != cudaSuccess) return QJX_ERR_CUDA;
    float ms = 0.f;
    cudaEventElapsedTime(&ms, h->e0, h->e1);
    h->last_ms = ms;
    int failed = 0;
    if (resident && cudaMemcpy(&failed, h->R.fail, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return QJX_ERR_CUDA;
    if (failed) {  // the states of before the call; the handle can be run again
        if (cudaMemcpyAsync(P.x, h->x0, sizeof(double) * P.n, cudaMemcpyDeviceToDevice, h->stream) != cudaSuccess ||
            cudaStreamSynchronize(h->stream) != cudaSuccess)
            return QJX_ERR_CUDA;
        return QJX_ERR_TIMEOUT;
    }
    return QJX_OK;
}

extern "C" qjx_status qjx_fb_info(qjx_fb *h, int *cluster_size)
{
    if (!h || !cluster_size) return QJX_ERR_INVALID_ARG;
    *cluster_size = h->cs;
    return QJX_OK;
}

extern "C" qjx_status qjx_fb_get(qjx_fb *h, double *x, double *last_period_ms)
{
    if (!h) return QJX_ERR_INVALID_ARG;
    if (cudaSetDevice(h->device) != cudaSuccess) return QJX_ERR_CUDA;
    if (x && cudaMemcpy(x, h->P.x, sizeof(double) * h->P.n, cudaMemcpyDeviceToHost) != cudaSuccess)
        return QJX_ERR_CUDA;
    if (last_period_ms) *last_period_ms = h->last_ms;
    return QJX_OK;
}

// ---------------------------------------------------------------- allocation-free variant
// Stage vectors va, vb, k1, k2, k3 of the allocation-free entry point, one static array shared by
// all its calls on a device.  In host code this name is only a stand-in for the symbol; its
// device address comes from cudaGetSymbolAddress.
static __device__ __align__(256) double g_fb_noalloc_scratch[5 * QJX_FB_NOALLOC_MAX_N];

static double *fb_noalloc_scratch_ptr(int device)
{
    constexpr int kMaxDevices = 64;
    static std::mutex mu;
    static double *ptr[kMaxDevices] = {nullptr};
    if (device < 0 || device >= kMaxDevices) return nullptr;
    std::lock_guard<std::mutex> lock(mu);
    if (!ptr[device]) {
        void *p = nullptr;
        if (cudaGetSymbolAddress(&p, g_fb_noalloc_scratch) != cudaSuccess) return nullptr;
        ptr[device] = static_cast<double *>(p);
    }
    return ptr[device];
}

extern "C" qjx_status qjx_fb_rk4_noalloc(int n, const int *gs_rowptr, const int *gs_col, const double *gs_val,
                                         const int *qs_rowptr, const int *qs_col, const double *qs_val,
                                         const double *Ks, double *x, double drv_ampl, double drv_freq,
                                         double drv_phase, int drv_type, double T, int num_steps, int period0,
                                         int n_periods, int device, void *stream)
{
    if (n < 1 || !gs_rowptr || !gs_col || !gs_val || !qs_rowptr || !qs_col || !qs_val || !Ks || !x ||
        num_steps < 1 || !(T > 0.0) || (drv_type != 0 && drv_type != 1) || period0 < 0 || n_periods < 0)
        return QJX_ERR_INVALID_ARG;
    if (n > QJX_FB_NOALLOC_MAX_N) return QJX_ERR_UNSUPPORTED;
    if (cudaSetDevice(device) != cudaSuccess) return QJX_ERR_CUDA;
    double *scratch = fb_noalloc_scratch_ptr(device);
    if (!scratch) return QJX_ERR_CUDA;
    fb::FbParams P{};
    P.n = n;
    P.gr = gs_rowptr;
    P.gc = gs_col;
    P.gv = gs_val;
    P.qr = qs_rowptr;
    P.qc = qs_col;
    P.qv = qs_val;
    P.Ks = Ks;
    P.drv_ampl = -drv_ampl;
    P.drv_freq = drv_freq;
    P.drv_phase = drv_phase;
    P.drv_type = drv_type;
    P.x = x;
    P.va = scratch;
    P.vb = scratch + QJX_FB_NOALLOC_MAX_N;
    P.k1 = scratch + 2 * QJX_FB_NOALLOC_MAX_N;
    P.k2 = scratch + 3 * QJX_FB_NOALLOC_MAX_N;
    P.k3 = scratch + 4 * QJX_FB_NOALLOC_MAX_N;
    // only the status of this call's own launches is reported; an error left by other code
    // stays where the caller can still read it
    const cudaError_t e =
        fb::queue_rk_stages(P, T, num_steps, period0, n_periods, static_cast<cudaStream_t>(stream));
    return e == cudaSuccess ? QJX_OK : QJX_ERR_CUDA;
}

extern "C" void qjx_fb_destroy(qjx_fb *h)
{
    if (!h) return;
    cudaSetDevice(h->device);
    if (h->stream) cudaStreamSynchronize(h->stream);
    for (void *p : h->allocs) cudaFree(p);
    if (h->e0) cudaEventDestroy(h->e0);
    if (h->e1) cudaEventDestroy(h->e1);
    if (h->stream) cudaStreamDestroy(h->stream);
    delete h;
}
