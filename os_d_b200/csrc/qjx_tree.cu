// qjx_tree.cu -- split trees (the QJ propagators U_{b,l} = exp(K_b dt_{b,l})) built on the GPU.
//
// The reference exponentiates every level of every branch on the host (Eigen exp(),
// QJX/qj_proc.cpp:55,98), and so does qjx_build_dimer (Higham's Pade scaling and squaring, one
// level at a time).  At d = 1024 that is about a minute of host time per ensemble, which a
// serving loop cannot spend per request.  Here the levels are related as the tree is: dt halves
// from one level to the next, so U_l = U_{l+1}^2.  The finest level is a Taylor series of the
// scaled generator X = K dt / 2^s with ||X||_1 <= 1/4 (degree 14: remainder below 1e-19 of ||e^X||),
// squared s times; every coarser level is one squaring.  All products are FP64 complex GEMMs on the
// FP64 tensor core.
#include <algorithm>
#include <cmath>
#include <utility>
#include <vector>

#include "../../include/qjx_b200.h"

namespace tree {

constexpr int BM = 32, BN = 32, BK = 8, kStages = 4;   // 256 threads
constexpr int kAStride = BK + 2, kBStride = BN + 2;    // components; both 32 bytes modulo the banks

__device__ __forceinline__ void dmma(double &c0, double &c1, double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
                 : "+d"(c0), "+d"(c1)
                 : "d"(a), "d"(b));
}

// 16 bytes global -> shared, zeros where !valid (the address is not read then).
__device__ __forceinline__ void cp16(double2 *dst, const double2 *src, bool valid)
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

// C = A B for n x n complex row-major matrices, or with div != 0 a Horner step of the Taylor
// series, C = I + (A B) / div.  FP64 tensor-core MMA, per output the k-ascending chain
// c.x += a.x b.x; c.x -= a.y b.y; c.y += a.x b.y; c.y += a.y b.x (A = [ar, ai] of two k against
// B = [br; -bi] and [bi; br]: the MMA's accumulation is that chain, see qjx_kernels.cu), so the
// results are those of a plain fma loop bit for bit.
// Bound: the FP64 tensor pipe (8 n^3 flop).  32 x 32 tiles, because n = 256 .. 512 has too few
// 64 x 64 tiles for 148 SMs (64 at n = 512); a warp owns one 8-row block and two 8-column blocks
// (four independent chains), and a four-stage cp.async ring of 8 k feeds the CTA.
__global__ void __launch_bounds__(256) zgemm_kernel(int n, const double2 *A, const double2 *B, double2 *C, double div)
{
    __shared__ __align__(16) double2 As[kStages][BM * kAStride];
    __shared__ __align__(16) double2 Bs[kStages][BK * kBStride];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3, th = t >> 1, todd = t & 1;
    const int row0 = blockIdx.y * BM, col0 = blockIdx.x * BN;
    const int rb = warp & 3, cb = 2 * (warp >> 2);
    const int nk = (n + BK - 1) / BK;
    auto load = [&](int it) {
        if (it < nk) {
            double2 *as = As[it % kStages], *bs = Bs[it % kStages];
            for (int e = tid; e < BM * BK; e += 256) {
                const int m = e / BK, k = e % BK, r = row0 + m, kk = it * BK + k;
                const bool v = r < n && kk < n;
                cp16(as + m * kAStride + k, A + (v ? (size_t)r * n + kk : 0), v);
            }
            for (int e = tid; e < BK * BN; e += 256) {
                const int k = e / BN, c = e % BN, kk = it * BK + k, cc = col0 + c;
                const bool v = kk < n && cc < n;
                cp16(bs + k * kBStride + c, B + (v ? (size_t)kk * n + cc : 0), v);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    double re[2][2], im[2][2];
#pragma unroll
    for (int j = 0; j < 2; j++) re[j][0] = re[j][1] = im[j][0] = im[j][1] = 0.0;
    for (int i = 0; i < kStages - 1; i++) load(i);
    for (int it = 0; it < nk; it++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
        __syncthreads();  // stage `it` has landed for every thread, and nobody reads the one refilled next
        load(it + kStages - 1);
        const double *as = reinterpret_cast<const double *>(As[it % kStages] + (8 * rb + g) * kAStride) + t;
        const double2 *bs = Bs[it % kStages] + th * kBStride + 8 * cb + g;
#pragma unroll
        for (int k = 0; k < BK; k += 2) {
            const double a = as[2 * k];
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const double2 b = bs[k * kBStride + 8 * j];
                dmma(re[j][0], re[j][1], a, todd ? -b.y : b.x);
                dmma(im[j][0], im[j][1], a, todd ? b.x : b.y);
            }
        }
    }
    const int r = row0 + 8 * rb + g;
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int c = col0 + 8 * (cb + j) + 2 * t + i;
            if (r >= n || c >= n) continue;
            double2 v = make_double2(re[j][i], im[j][i]);
            if (div != 0.0) v = make_double2(__dadd_rn(r == c ? 1.0 : 0.0, __ddiv_rn(v.x, div)), __ddiv_rn(v.y, div));
            C[(size_t)r * n + c] = v;
        }
}

// T = I
__global__ void identity_kernel(int n, double2 *T)
{
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e < (size_t)n * n) T[e] = make_double2((e / n) == (e % n) ? 1.0 : 0.0, 0.0);
}

// X = s K (complex K, real s)
__global__ void scale_kernel(int n, const double2 *K, double s, double2 *X)
{
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (size_t)n * n) return;
    X[e] = make_double2(__dmul_rn(K[e].x, s), __dmul_rn(K[e].y, s));
}

static cudaError_t gemm(int n, const double2 *A, const double2 *B, double2 *C, double div, cudaStream_t st)
{
    const dim3 grid((n + BN - 1) / BN, (n + BM - 1) / BM);
    zgemm_kernel<<<grid, 256, 0, st>>>(n, A, B, C, div);
    return cudaGetLastError();
}

}  // namespace tree

extern "C" qjx_status qjx_expm_tree(int d, int nb, const double *K, const double *head, int deep, int device,
                                    double *Utree)
{
    using namespace tree;
    if (d < 1 || nb < 1 || deep < 1 || deep > 62 || !K || !head || !Utree) return QJX_ERR_INVALID_ARG;
    for (int b = 0; b < nb; b++)
        if (!(head[b] > 0.0)) return QJX_ERR_INVALID_ARG;
    if (cudaSetDevice(device) != cudaSuccess) return QJX_ERR_CUDA;
    // a private stream and stream-ordered allocations: no device-wide synchronisation, so trees can
    // be built while engines run on the same device
    cudaStream_t st = nullptr;
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) return QJX_ERR_CUDA;
    const size_t dd = (size_t)d * d, bytes = dd * sizeof(double2);
    double2 *dK = nullptr, *X = nullptr, *T = nullptr, *P = nullptr;
    qjx_status status = QJX_OK;
    if (cudaMallocAsync(&dK, bytes, st) != cudaSuccess || cudaMallocAsync(&X, bytes, st) != cudaSuccess ||
        cudaMallocAsync(&T, bytes, st) != cudaSuccess || cudaMallocAsync(&P, bytes, st) != cudaSuccess)
        status = QJX_ERR_OOM;
    const int eb = 256, eg = (int)((dd + eb - 1) / eb);
    for (int b = 0; b < nb && status == QJX_OK; b++) {
        const double *Kb = K + 2 * dd * b;
        // the finest level's step and the 1-norm of K dt (largest column sum of |K_ij|), on the host
        const double dt = std::ldexp(head[b], -(deep + 1));
        double norm1 = 0.0;
        for (int j = 0; j < d; j++) {
            double s = 0.0;
            for (int i = 0; i < d; i++) s += std::hypot(Kb[2 * ((size_t)i * d + j)], Kb[2 * ((size_t)i * d + j) + 1]);
            norm1 = std::max(norm1, s);
        }
        norm1 *= dt;
        int sq = 0;
        while (std::ldexp(norm1, -sq) > 0.25) sq++;
        if (cudaMemcpyAsync(dK, Kb, bytes, cudaMemcpyHostToDevice, st) != cudaSuccess) {
            status = QJX_ERR_CUDA;
            break;
        }
        scale_kernel<<<eg, eb, 0, st>>>(d, dK, std::ldexp(dt, -sq), X);
        // Horner: T = I; T = I + X T / k for k = 14 .. 1
        identity_kernel<<<eg, eb, 0, st>>>(d, T);
        for (int k = 14; k >= 1; k--) {
            if (gemm(d, X, T, P, (double)k, st) != cudaSuccess) status = QJX_ERR_CUDA;
            std::swap(T, P);
        }
        for (int i = 0; i < sq; i++) {  // (e^X)^(2^sq)
            if (gemm(d, T, T, P, 0.0, st) != cudaSuccess) status = QJX_ERR_CUDA;
            std::swap(T, P);
        }
        // levels deep-1 .. 0: each the square of the next finer one
        for (int l = deep - 1; l >= 0 && status == QJX_OK; l--) {
            if (l < deep - 1) {
                if (gemm(d, T, T, P, 0.0, st) != cudaSuccess) status = QJX_ERR_CUDA;
                std::swap(T, P);
            }
            if (cudaMemcpyAsync(Utree + 2 * dd * ((size_t)b * deep + l), T, bytes, cudaMemcpyDeviceToHost, st) !=
                cudaSuccess)
                status = QJX_ERR_CUDA;
        }
    }
    cudaFreeAsync(dK, st);
    cudaFreeAsync(X, st);
    cudaFreeAsync(T, st);
    cudaFreeAsync(P, st);
    if (cudaStreamSynchronize(st) != cudaSuccess) status = QJX_ERR_CUDA;
    cudaStreamDestroy(st);
    return status;
}
