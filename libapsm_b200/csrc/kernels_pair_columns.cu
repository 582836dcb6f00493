// Kernel columns of the single detector's training sweep, in pair form.
//
// For every pair n that enters a window, column n holds against every visible
// pair b <= n the three distinct values of the 2 x 2 block of Dedup rows
// (A, Bp, Bm; see apsm_batch.cuh), each from its own squared distance -- the
// difference form of the reference's loop (cpp/lib/apsm/apsm_detect.cu:131-152)
// -- and expf.  With y_b = (p, q) and y_n = (r, s) per antenna the distances are
//   A:  (p - r)^2 + (q - s)^2,  Bp: (p - s)^2 + (q + r)^2,  Bm: (p + s)^2 + (q - r)^2,
// three packed additions and three packed fma on (p, q), (r, s) and (s, -r).
// Entries of the sweep's window (b >= max(n_first, n - 1 - qP)) are combined
// with the linear kernel, wL r + i m = wL y_b^H y_n.
//
// Bound: the FP32 pipe, 12 N operations per pair of pairs (16 N for the four
// row values that the reference evaluates; half the instructions by packing).
// Tiles that no column reaches (b > n, or evicted) are skipped: 8192 pilots of
// 64 antennas write 537 MB instead of 1.07 GB of row-form columns.
#include "apsm_batch.cuh"
#include "packed_f32.cuh"

namespace apsm {

namespace {

constexpr int kTb = 64;  // pairs b per block (16 threads x 4)
constexpr int kTn = 32;  // columns n per block (16 threads x 2)
constexpr int kTk = 16;  // antennas per shared-memory chunk

struct PairColumnsArgs {
    const float* X; // nU x Dp Dedup rows (row 2b = [Re y_b; Im y_b])
    int N, Dp, nP, n_first, capP, qP;
    long long base;
    float ew, wG, wL;
    float4* K;
};

template <bool BAND>
__device__ __forceinline__ void columns_tile(const PairColumnsArgs& g, int b0, int n0, f32x2 (*sb)[kTb],
                                             f32x2 (*sn)[kTn])
{
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    f32x2 dA[4][2], dP[4][2], dM[4][2];
    float lr[BAND ? 4 : 1][2], li[BAND ? 4 : 1][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            dA[i][j] = dP[i][j] = dM[i][j] = 0ull;
            if constexpr (BAND) lr[i][j] = li[i][j] = 0.f;
        }
    for (int k0 = 0; k0 < g.N; k0 += kTk) {
        __syncthreads();
        // features of the chunk as (Re, Im); antennas past N are zero in both operands
        for (int i = threadIdx.x; i < kTk * (kTb + kTn); i += 256) {
            const int k = i % kTk, r = i / kTk, p = r < kTb ? b0 + r : n0 + r - kTb;
            f32x2 v = 0ull;
            if (p < g.nP && k0 + k < g.N) {
                const float* row = g.X + size_t(2 * p) * g.Dp + k0 + k;
                v = pack2(__ldg(row), __ldg(row + g.N));
            }
            if (r < kTb) sb[k][r] = v;
            else sn[k][r - kTb] = v;
        }
        __syncthreads();
#pragma unroll 4
        for (int k = 0; k < kTk; ++k) {
            f32x2 nA[2], nP[2], nM[2];
            float2 nf[2];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                nf[j] = unpack2(sn[k][2 * ty + j]);
                nA[j] = pack2(-nf[j].x, -nf[j].y); // y_b - (r, s)
                nP[j] = pack2(-nf[j].y, nf[j].x);  // y_b - (s, -r)
                nM[j] = pack2(nf[j].y, -nf[j].x);  // y_b + (s, -r)
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const f32x2 b = sb[k][tx + 16 * i];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    f32x2 d = add2(b, nA[j]);
                    dA[i][j] = fma2(d, d, dA[i][j]);
                    d = add2(b, nP[j]);
                    dP[i][j] = fma2(d, d, dP[i][j]);
                    d = add2(b, nM[j]);
                    dM[i][j] = fma2(d, d, dM[i][j]);
                    if constexpr (BAND) {
                        const float2 bf = unpack2(b);
                        lr[i][j] = fmaf(bf.x, nf[j].x, fmaf(bf.y, nf[j].y, lr[i][j]));
                        li[i][j] = fmaf(bf.x, nf[j].y, fmaf(-bf.y, nf[j].x, li[i][j]));
                    }
                }
            }
        }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int n = n0 + 2 * ty + j;
        if (n >= g.nP) continue;
        const int lo = col_begin(n, g.capP), band = max(g.n_first, n - 1 - g.qP);
        float4* col = g.K + (column_prefix(n, 1, g.nP, g.capP) - g.base) - lo;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int b = b0 + tx + 16 * i;
            if (b < lo || b > n) continue;
            const float2 a = unpack2(dA[i][j]), p = unpack2(dP[i][j]), m = unpack2(dM[i][j]);
            float4 v = make_float4(__fmul_rn(g.wG, expf(__fmul_rn(g.ew, a.x + a.y))),
                                   __fmul_rn(g.wG, expf(__fmul_rn(g.ew, p.x + p.y))),
                                   __fmul_rn(g.wG, expf(__fmul_rn(g.ew, m.x + m.y))), 0.f);
            if constexpr (BAND)
                if (b >= band) {
                    v.x = fmaf(g.wL, lr[i][j], v.x);
                    v.y = fmaf(g.wL, li[i][j], v.y);
                    v.z = fmaf(-g.wL, li[i][j], v.z);
                }
            col[b] = v;
        }
    }
}

__global__ void __launch_bounds__(256, 2) pair_columns_kernel(PairColumnsArgs g)
{
    __shared__ __align__(16) f32x2 sb[kTk][kTb];
    __shared__ __align__(16) f32x2 sn[kTk][kTn];
    const int n0 = g.n_first + blockIdx.y * kTn, n1 = min(n0 + kTn, g.nP) - 1;
    const int b0 = blockIdx.x * kTb;
    if (b0 > n1 || b0 + kTb - 1 < col_begin(n0, g.capP)) return;
    if (b0 + kTb - 1 >= max(g.n_first, n0 - 1 - g.qP)) columns_tile<true>(g, b0, n0, sb, sn);
    else columns_tile<false>(g, b0, n0, sb, sn);
}

// Old-pair sums of columns [n_first, n_first + n_cols) for every user: sum over the pairs b < n_first
// that pair n meets (b >= lo_min: visible at the call's first step) of a_b K(b, n), in `splits` parts ([user][n - n_first][part]).  A block takes kSumCols
// columns x kSumUsers users x one part of the pairs: 128 fma per 12 loads of a thread, the columns
// (from DRAM) read once for 8 users, the coefficients (from L2) once for 4 columns.
constexpr int kSumCols = 4, kSumUsers = 8, kSumThreads = 128;

__global__ void __launch_bounds__(kSumThreads)
    old_pair_sums_kernel(const float4* __restrict__ K, long long base, int nP, int n_first, int n_cols, int capP, int lo_min,
                         const float* __restrict__ a, size_t a_stride, int users, int splits, float2* __restrict__ out)
{
    __shared__ float2 part[kSumThreads / 32][kSumCols * kSumUsers];
    const int c0 = blockIdx.x * kSumCols, u0 = blockIdx.y * kSumUsers, sp = blockIdx.z;
    const float4* col[kSumCols];
    int lo[kSumCols];
#pragma unroll
    for (int c = 0; c < kSumCols; ++c) {
        const int n = n_first + min(c0 + c, n_cols - 1);
        lo[c] = max(col_begin(n, capP), lo_min);
        col[c] = K + (column_prefix(n, 1, nP, capP) - base) - col_begin(n, capP);
    }
    float2 g[kSumCols][kSumUsers];
#pragma unroll
    for (int c = 0; c < kSumCols; ++c)
#pragma unroll
        for (int u = 0; u < kSumUsers; ++u) g[c][u] = make_float2(0.f, 0.f);
    const int len = (n_first - lo[0] + splits - 1) / splits;
    const int b_end = min(n_first, lo[0] + (sp + 1) * len);
    for (int b = lo[0] + sp * len + int(threadIdx.x); b < b_end; b += kSumThreads) {
        float4 k[kSumCols];
#pragma unroll
        for (int c = 0; c < kSumCols; ++c) k[c] = b >= lo[c] ? __ldg(col[c] + b) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int u = 0; u < kSumUsers; ++u) {
            const float2 ab = u0 + u < users ? *reinterpret_cast<const float2*>(a + size_t(u0 + u) * a_stride + 2 * b)
                                             : make_float2(0.f, 0.f);
#pragma unroll
            for (int c = 0; c < kSumCols; ++c) {
                g[c][u].x = fmaf(ab.x, k[c].x, fmaf(ab.y, k[c].z, g[c][u].x));
                g[c][u].y = fmaf(ab.x, k[c].y, fmaf(ab.y, k[c].x, g[c][u].y));
            }
        }
    }
#pragma unroll
    for (int c = 0; c < kSumCols; ++c)
#pragma unroll
        for (int u = 0; u < kSumUsers; ++u) {
            float2 v = g[c][u];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
                v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
            }
            if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5][c * kSumUsers + u] = v;
        }
    __syncthreads();
    if (threadIdx.x < kSumCols * kSumUsers) {
        const int c = threadIdx.x / kSumUsers, u = threadIdx.x % kSumUsers;
        float2 v = part[0][threadIdx.x];
#pragma unroll
        for (int w = 1; w < kSumThreads / 32; ++w) {
            v.x += part[w][threadIdx.x].x;
            v.y += part[w][threadIdx.x].y;
        }
        if (c0 + c < n_cols && u0 + u < users) out[(size_t(u0 + u) * n_cols + c0 + c) * splits + sp] = v;
    }
}

} // namespace

cudaError_t launch_old_pair_sums(const float4* K, int nP, int n_first, int n_cols, int capP, int lo_min, const float* a,
                                 size_t a_stride, int users, int splits, float2* out, cudaStream_t s)
{
    if (n_cols <= 0) return cudaSuccess;
    old_pair_sums_kernel<<<dim3((n_cols + kSumCols - 1) / kSumCols, (users + kSumUsers - 1) / kSumUsers, splits),
                           kSumThreads, 0, s>>>(K, column_prefix(n_first, 1, nP, capP), nP, n_first, n_cols, capP,
                                                lo_min, a, a_stride, users, splits, out);
    return cudaGetLastError();
}

cudaError_t launch_pair_columns(const float* X, int N, int Dp, int nP, int n_first, int capP, int qP, float ew,
                                float wG, float wL, float4* K, cudaStream_t s)
{
    if (nP <= n_first) return cudaSuccess;
    PairColumnsArgs g{X, N, Dp, nP, n_first, capP, qP, column_prefix(n_first, 1, nP, capP), ew, wG, wL, K};
    pair_columns_kernel<<<dim3((nP + kTb - 1) / kTb, (nP - n_first + kTn - 1) / kTn), 256, 0, s>>>(g);
    return cudaGetLastError();
}

} // namespace apsm
