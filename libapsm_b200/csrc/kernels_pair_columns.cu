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

namespace apsm {

namespace {

constexpr int kTb = 64;  // pairs b per block (16 threads x 4)
constexpr int kTn = 32;  // columns n per block (16 threads x 2)
constexpr int kTk = 16;  // antennas per shared-memory chunk

using f32x2 = unsigned long long;

__device__ __forceinline__ f32x2 pack2(float lo, float hi)
{
    f32x2 v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ float2 unpack2(f32x2 v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

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
            v.w = v.x;
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

} // namespace

cudaError_t launch_pair_columns(const float* X, int N, int Dp, int nP, int n_first, int capP, int qP, float ew,
                                float wG, float wL, float4* K, cudaStream_t s)
{
    if (nP <= n_first) return cudaSuccess;
    PairColumnsArgs g{X, N, Dp, nP, n_first, capP, qP, column_prefix(n_first, 1, nP, capP), ew, wG, wL, K};
    pair_columns_kernel<<<dim3((nP + kTb - 1) / kTb, (nP - n_first + kTn - 1) / kTn), 256, 0, s>>>(g);
    return cudaGetLastError();
}

} // namespace apsm
