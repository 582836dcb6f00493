// Linear least-squares (LLS) detector and the APSM llsInitialization.
//
// Reference: cpp/lib/noma/lls_detector.cu:136-218.  Training solves
//   min_w || A w - y ||,  A = Dedup real rows of the pilots (2P x 2N),
//   y = interleaved (Re, Im) pilot symbols,
// which the reference hands to cuBLAS (cublasSgelsBatched, FP32 Householder
// QR, :163-179).  Here the solve runs in this file's kernels, in double
// precision through the normal equations: the Gram matrix A^T A and the
// right-hand sides A^T y are summed over blocks of 64 rows (each block's
// partial in FP64, the blocks added in a fixed order), then one CTA factors
// A^T A = L L^T (Cholesky, in shared memory) and solves for every user.  With
// FP64 the squared condition number costs nothing at these sizes (2N <= 128
// features, kappa(A)^2 * 1e-16 far below FP32 rounding), so the weights are
// the exact least-squares solution rounded to FP32 -- at least as accurate as
// the reference's FP32 QR.  Several users are several right-hand sides of one
// solve.  Detection is est = A_data w (the reference's cublasSgemm,
// :207-218), a small kernel over the packed data rows.  llsInitialization
// copies w / linearKernelWeight into the APSM linear weights before training
// (copyWeightMat, cpp/lib/apsm/apsm_noma_detector.cu:321-346).
#include "apsm_host.hpp"
#include "apsm_kernels.cuh"
#include "apsm_gram.cuh"
#include "apsm_lls.cuh"

#include <algorithm>
#include <string>

namespace apsm {

struct LlsWorkspace {
    DevBuf<double> part; // [blocks][D][D + users] per-block sums (upper triangle of A^T A, then A^T y)
    DevBuf<int> err;     // set when A^T A is not positive definite (rank-deficient pilots)
    DevBuf<float> w;     // users x 2N solution
};

void lls_workspace_free(LlsWorkspace* l) { delete l; }

namespace {

constexpr int kLlsRows = 64;      // pilot rows per Gram block
constexpr int kLlsThreads = 256;
constexpr int kSolveThreads = 1024;

// Per-block sums over rows [blk * kLlsRows, ...): part[blk][i][j] = sum_r x_r[i] z_r[j] with
// z = (features, targets), for j >= i among the features and every target j >= D.
__global__ void __launch_bounds__(kLlsThreads)
    lls_gram_kernel(const float* __restrict__ rows, int n, int Dp, int D, const float* __restrict__ y,
                    size_t y_stride, int row0, int users, double* __restrict__ part)
{
    extern __shared__ float xz[]; // [kLlsRows][D + users]
    const int W = D + users;
    const int r0 = blockIdx.x * kLlsRows;
    const int nr = min(kLlsRows, n - r0);
    for (int idx = threadIdx.x; idx < kLlsRows * W; idx += kLlsThreads) {
        const int r = idx / W, j = idx % W;
        float v = 0.f;
        if (r < nr) v = j < D ? rows[size_t(r0 + r) * Dp + j] : y[size_t(j - D) * y_stride + row0 + r0 + r];
        xz[idx] = v;
    }
    __syncthreads();
    // a thread sums 2 x 2 entries: one conversion to FP64 per product (they bound the kernel), not two
    double* out = part + size_t(blockIdx.x) * D * W;
    const int ti = (D + 1) / 2, tj = (W + 1) / 2;
    for (int e = threadIdx.x; e < ti * tj; e += kLlsThreads) {
        const int i = 2 * (e / tj), j = 2 * (e % tj);
        if (j + 1 < i) continue; // below the diagonal: never read
        const int i1 = min(i + 1, D - 1), j1 = min(j + 1, W - 1);
        double a00 = 0.0, a01 = 0.0, a10 = 0.0, a11 = 0.0;
#pragma unroll 4
        for (int r = 0; r < nr; ++r) {
            const float* x = xz + r * W;
            const double p = x[i], q = x[i1], u = x[j], v = x[j1];
            a00 = fma(p, u, a00);
            a01 = fma(p, v, a01);
            a10 = fma(q, u, a10);
            a11 = fma(q, v, a11);
        }
        out[i * W + j] = a00;
        if (j + 1 < W) out[i * W + j + 1] = a01;
        if (i + 1 < D) out[(i + 1) * W + j] = a10;
        if (i + 1 < D && j + 1 < W) out[(i + 1) * W + j + 1] = a11;
    }
}

// One CTA: G = sum of the blocks' partials (fixed order), G = L D L^T, then
// L D L^T w_u = c_u for every user; w[u][d] = w_u[d] / divide_by.
// Bound: the chain of D pivots.  The factorization runs on the upper triangle
// with the right-hand sides as further columns, so L z = c comes with it; there
// is no square root, one division and one barrier per pivot, and rows are read
// along the lanes.  The back substitution goes by columns, one warp per user with
// its solution in registers (a shuffle and a product per step, no sum over
// lanes).  32 features, 8 users, 32 blocks: 55 us with L L^T, three barriers a
// pivot and dot products by shuffles, now 25 us.
__global__ void __launch_bounds__(kSolveThreads)
    lls_solve_kernel(const double* __restrict__ part, int blocks, int D, int users, float divide_by,
                     float* __restrict__ w, int* __restrict__ err)
{
    extern __shared__ double g[]; // [D][W]: upper triangle of G, then the right-hand sides
    const int W = D + users;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    for (int e = threadIdx.x; e < D * W; e += blockDim.x) {
        if (e % W < e / W) continue;
        double acc = 0.0;
#pragma unroll 8
        for (int b = 0; b < blocks; ++b) acc += part[size_t(b) * D * W + e];
        g[e] = acc;
    }
    __syncthreads();
    // after step k, row k holds d_k L(., k) and, from column D, (L^-1 c)(k)
    for (int k = 0; k < D; ++k) {
        const double* const gk = g + k * W;
        if (!(gk[k] > 0.0)) { // uniform: every thread reads the same value
            if (threadIdx.x == 0) *err = 1;
            return;
        }
        const double inv = 1.0 / gk[k];
        for (int i = k + 1 + warp; i < D; i += warps) {
            const double l = gk[i] * inv;
            for (int j = i + lane; j < W; j += 32) g[i * W + j] = fma(-l, gk[j], g[i * W + j]);
        }
        __syncthreads();
    }
    // D L^T x = z: x_i = z_i / d_i once every later x_j has been taken out of it
    constexpr int kT = kMaxFeatures / 32;
    double inv[kT];
#pragma unroll
    for (int t = 0; t < kT; ++t) inv[t] = 32 * t + lane < D ? 1.0 / g[(32 * t + lane) * (W + 1)] : 0.0;
    for (int u = warp; u < users; u += warps) {
        double x[kT];
#pragma unroll
        for (int t = 0; t < kT; ++t) x[t] = 32 * t + lane < D ? g[(32 * t + lane) * W + D + u] * inv[t] : 0.0;
#pragma unroll
        for (int t = kT - 1; t >= 0; --t)
            for (int i = min(D, 32 * (t + 1)) - 1; i >= 32 * t; --i) {
                const double xi = __shfl_sync(0xffffffffu, x[t], i & 31);
#pragma unroll
                for (int v = 0; v <= t; ++v) {
                    const int j = 32 * v + lane;
                    if (j < i) x[v] = fma(-(g[j * W + i] * inv[v]), xi, x[v]);
                }
            }
#pragma unroll
        for (int t = 0; t < kT; ++t)
            if (32 * t + lane < D) w[size_t(u) * D + 32 * t + lane] = float(x[t] / double(divide_by));
    }
}

} // namespace

// Solve for every user's linear weights from the packed pilot rows
// (rows: n = 2P rows of pitch Dp; targets y rows [row0, row0 + n)).
// On success h->lls->w holds users x 2N weights divided by `divide_by`.
apsm_status lls_solve(apsm_detector* h, const float* rows, int n, const float* y, size_t y_stride, int row0,
                      float divide_by, cudaStream_t s)
{
    const int D = int(h->D), U = int(h->U);
    if (!h->lls) h->lls = new LlsWorkspace();
    LlsWorkspace* l = h->lls;
    if (n < D) {
        h->last_error = "LLS needs at least as many real pilot rows as features (2P >= 2N)";
        return APSM_ERR_INVALID_ARGUMENT;
    }
    cudaError_t e;
#define LL_CK(x)                                              \
    do {                                                      \
        e = (x);                                              \
        if (e != cudaSuccess) return h->cuda_fail(e, #x);     \
    } while (0)
    const int W = D + U;
    const int blocks = (n + kLlsRows - 1) / kLlsRows;
    LL_CK(l->part.ensure(size_t(blocks) * D * W));
    LL_CK(l->err.ensure(1));
    LL_CK(l->w.ensure(size_t(U) * D));
    LL_CK(cudaMemsetAsync(l->err.p, 0, sizeof(int), s));
    lls_gram_kernel<<<blocks, kLlsThreads, sizeof(float) * kLlsRows * W, s>>>(rows, n, int(h->Dp), D, y, y_stride,
                                                                             row0, U, l->part.p);
    LL_CK(cudaGetLastError());
    const size_t smem = sizeof(double) * size_t(D) * W;
    if (smem > kMaxSmem) {
        h->last_error = "LLS: " + std::to_string(U) + " users with " + std::to_string(D) +
                        " features exceed the solver's shared memory";
        return APSM_ERR_UNSUPPORTED;
    }
    LL_CK(allow_smem(lls_solve_kernel));
    // a pivot's barrier and division cost more than its update of a 32-feature triangle: eight warps there
    lls_solve_kernel<<<1, D <= 32 ? 256 : kSolveThreads, smem, s>>>(l->part.p, blocks, D, U, divide_by, l->w.p, l->err.p);
    LL_CK(cudaGetLastError());
    int bad = 0;
    LL_CK(cudaMemcpyAsync(&bad, l->err.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    LL_CK(cudaStreamSynchronize(s));
#undef LL_CK
    if (bad) {
        h->last_error = "LLS: the pilots' feature matrix is rank-deficient (A^T A not positive definite)";
        return APSM_ERR_INVALID_ARGUMENT;
    }
    return APSM_OK;
}

apsm_status lls_detect(apsm_detector* h, int ns, float* d_out, cudaStream_t s)
{
    if (!h->lls || h->used == 0) {
        // untrained: the reference's weight matrix is uninitialised device memory;
        // here an untrained LLS detector outputs zeros
        cudaError_t e = cudaMemsetAsync(d_out, 0, sizeof(float) * size_t(h->U) * ns, s);
        return e == cudaSuccess ? APSM_OK : h->cuda_fail(e, "cudaMemsetAsync");
    }
    const int U = int(h->U);
    cudaError_t e = cudaSuccess;
    const int D = int(h->D);
    for (int u = 0; u < U && e == cudaSuccess; u += kLinearUsers) // est = A_data w
        e = launch_linear_part(h->xs.p, int(h->Dp), D, h->lls->w.p + size_t(u) * D, 1.f, nullptr, 0,
                               std::min(U - u, kLinearUsers), ns, d_out + size_t(u) * ns, size_t(ns), s);
    return e == cudaSuccess ? APSM_OK : h->cuda_fail(e, "lls_detect");
}

const float* lls_weights(apsm_detector* h) { return h->lls ? h->lls->w.p : nullptr; }

} // namespace apsm
