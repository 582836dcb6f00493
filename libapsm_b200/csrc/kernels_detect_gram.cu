// Tensor-core Gram detection on B200 (tcgen05 / TMEM / bulk async copies).
//
// The detection model (cpp/lib/apsm/apsm_detect.cu:690-876)
//   f_u(x_s) = wL <w_u, x_s> + sum_b (a_ub wG) exp(ew ||d_b - x_s||^2)
// is recast with ||d - x||^2 = ||x||^2 + ||d||^2 - 2 x.d: the cross terms of a
// 128-sample tile against a 256-row dictionary chunk are one UMMA
// (tcgen05.mma, M=128, N=256, FP32 accumulators in tensor memory), the norms
// stay FP32, and the epilogue warps read the accumulator tile (tcgen05.ld),
// form the squared distance, exponentiate on the SFU (ex2.approx) and
// contract with every user's coefficients.  Operand precision:
//   gram_bf16    x.d from BF16 operands (1 product)
//   gram_bf16x3  compensated: x = xh + xl, d = dh + dl (BF16 each);
//                x.d ~ xh.dh + xh.dl + xl.dh (3 products, ~2^-16 relative)
//   gram_tf32    TF32 operands (1 product)
//   gram_tf32x3  compensated TF32 split (3 products, ~FP32 accuracy;
//                kernels_gram_tmem.cu)
// The squared distance is clamped at 0.  Compensated cross terms (the
// single-product forms bf16 / tf32): rounding both operands to the format's
// unit u moves x.d by at most 2u |x||d|, the base-2 exponent
// ew log2(e) (|x|^2 + |d|^2 - 2 x.d) by at most 2u |es| (es = ew log2(e)
// (|x|^2 + |d|^2)), and a kernel value's contribution to user u's output by at
// most |a_u wG| k ln2 2u |es|.  Where cancellation bites (near-duplicate
// points: x.d ~ (|x|^2 + |d|^2) / 2 with k near 1) the epilogue flags the
// entries whose bound, with the largest coefficient of the row over the
// users, exceeds kFixEps, and recomputes their squared distance exactly as
// sum (x - d)^2 in FP32 from the rows themselves.  Each CTA owns one tile of
// data rows and a contiguous range of dictionary chunks; partial sums per
// range are combined in a fixed order by gram_finish_kernel, so results are
// deterministic.
//
// Roles (320 threads): warps 0-7 epilogue (warp w reads TMEM lanes
// 32*(w%4).., columns of half w/4 of each chunk), warp 8 producer (bulk copies
// of dictionary chunks into a 3-stage ring), warp 9 TMEM allocator and MMA
// issuer.  Every mbarrier wait is bounded; on expiry the kernel records an
// error, stops issuing work, still releases its tensor memory and returns.
#include "apsm_gram.cuh"
#include "apsm_kernels.cuh"
#include "apsm_tc.cuh"
#include "packed_f32.cuh"

#include <cuda_bf16.h>

#include <algorithm>
#include <cstdint>
#include <string>

namespace apsm {

constexpr int kTileM = 128;       // data rows per CTA tile (UMMA M)
constexpr int kMaxStages = 3;     // dictionary chunk ring
constexpr int kEpiWarps = 8;
constexpr int kThreads = (kEpiWarps + 2) * 32;
constexpr int kMaxUsers = kLinearUsers;

struct GramWorkspace {
    DevBuf<uint8_t> a_ops, b_ops, w_ops; // operand tiles in the UMMA canonical K-major layout
    DevBuf<float> xn, dn, aw, part, fw, gate, xd;
    DevBuf<int> err;
    int* h_err = nullptr;
};

void gram_workspace_free(GramWorkspace* g)
{
    if (!g) return;
    if (g->h_err) cudaFreeHost(g->h_err);
    delete g;
}

namespace {

using namespace tc;

// ------------------------------------------------------ operand packing --

// rows: n x Dp fp32.  Writes tiles of R rows: element (r, k) of tile t at byte
// t*R*KE*elem + (k/kc)*(R*16) + (r/8)*128 + (r%8)*16 + (k%kc)*elem, where the
// K extent KE = Kp (hi part) [+ Kp (lo part) for split modes]; rows >= n and
// features >= D are zero.  Also the FP32 squared norms.
template <int MODE>
__global__ void gram_pack_kernel(const float* __restrict__ rows, int n, int Dp, int D, int Kp, int R, int n_tiles,
                                 uint8_t* __restrict__ ops, float* __restrict__ norms)
{
    using T = OpTraits<MODE>;
    const int KE = T::kSplit ? 2 * Kp : Kp;
    const size_t total = size_t(n_tiles) * R * Kp;
    for (size_t idx = blockIdx.x * size_t(blockDim.x) + threadIdx.x; idx < total; idx += size_t(gridDim.x) * blockDim.x) {
        const int k = int(idx % Kp);
        const size_t rr = idx / Kp;
        const int r = int(rr % R), t = int(rr / R);
        const int row = t * R + r;
        const float x = (row < n && k < D) ? rows[size_t(row) * Dp + k] : 0.f;
        float hi, lo;
        split_operand<MODE>(x, &hi, &lo);
        uint8_t* tile = ops + size_t(t) * R * KE * T::kElem;
        put_operand<MODE>(tile, R, r, k, hi);
        if constexpr (T::kSplit) put_operand<MODE>(tile, R, r, Kp + k, lo);
    }
    if (norms) {
        for (int row = blockIdx.x * blockDim.x + threadIdx.x; row < n; row += gridDim.x * blockDim.x) {
            float acc = 0.f;
            for (int k = 0; k < D; ++k) {
                const float v = rows[size_t(row) * Dp + k];
                acc = fmaf(v, v, acc);
            }
            norms[row] = acc;
        }
    }
}

// per-entry error a flagged entry would exceed (soft-output units) in the single-product forms
constexpr float kFixEps = 1.0f / 8192.0f;

// ln 2 * 2u / kFixEps of a mode's operand rounding unit u (0: split forms, no correction)
template <int MODE> __host__ __device__ constexpr float fix_scale()
{
    return MODE == kBF16 ? 0.69314718f * (2.0f / 256.0f) / kFixEps
                         : (MODE == kTF32 ? 0.69314718f * (2.0f / 2048.0f) / kFixEps : 0.0f);
}

// Fix weights of the compensated forms: fw[b] = max_u |a_u[b] wG| ln2 2u / kFixEps (0 past M)
// and per chunk of N dictionary rows gate[c] = (max fw, max fw |ewl2 dn[b]|, 0, 0).
template <int MODE>
__global__ void __launch_bounds__(256) gram_fix_kernel(const float* __restrict__ a, size_t a_stride, int users, int M,
                                                       int N, float wG, float ewl2, const float* __restrict__ dn,
                                                       float* __restrict__ fw, float* __restrict__ gate)
{
    __shared__ float red[2][8];
    const int c = blockIdx.x;
    float g0 = 0.f, g1 = 0.f;
    for (int k = threadIdx.x; k < N; k += blockDim.x) {
        const int b = c * N + k;
        float v = 0.f;
        if (b < M) {
            for (int u = 0; u < users; ++u) v = fmaxf(v, fabsf(__fmul_rn(a[size_t(u) * a_stride + b], wG)));
            v *= fix_scale<MODE>();
        }
        fw[b] = v;
        g0 = fmaxf(g0, v);
        g1 = fmaxf(g1, v * fabsf(ewl2 * dn[b]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        g0 = fmaxf(g0, __shfl_xor_sync(0xffffffffu, g0, o));
        g1 = fmaxf(g1, __shfl_xor_sync(0xffffffffu, g1, o));
    }
    if ((threadIdx.x & 31) == 0) {
        red[0][threadIdx.x >> 5] = g0;
        red[1][threadIdx.x >> 5] = g1;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < int(blockDim.x >> 5); ++w) {
            g0 = fmaxf(g0, red[0][w]);
            g1 = fmaxf(g1, red[1][w]);
        }
        gate[4 * c] = g0;
        gate[4 * c + 1] = g1;
        gate[4 * c + 2] = 0.f;
        gate[4 * c + 3] = 0.f;
    }
}

// Exact squared distance of two FP32 rows (16-byte aligned, D features), in feature order.
__device__ __forceinline__ float row_distance(const float* __restrict__ x, const float* __restrict__ d, int D)
{
    float acc = 0.f;
    int k = 0;
    for (; k + 4 <= D; k += 4) {
        const float4 xv = *reinterpret_cast<const float4*>(x + k);
        const float4 dv = *reinterpret_cast<const float4*>(d + k);
        acc = fmaf(xv.x - dv.x, xv.x - dv.x, acc);
        acc = fmaf(xv.y - dv.y, xv.y - dv.y, acc);
        acc = fmaf(xv.z - dv.z, xv.z - dv.z, acc);
        acc = fmaf(xv.w - dv.w, xv.w - dv.w, acc);
    }
    for (; k < D; ++k) acc = fmaf(x[k] - d[k], x[k] - d[k], acc);
    return acc;
}

// aw[u][b] = a_u[b] * wG (the reference's coeff * gaussianKernelWeight), 0 past M.
__global__ void gram_coeff_kernel(const float* __restrict__ a, size_t a_stride, int users, int M, int Mpad, float wG,
                                  float* __restrict__ aw)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= users * Mpad) return;
    const int u = i / Mpad, b = i % Mpad;
    aw[i] = b < M ? __fmul_rn(a[size_t(u) * a_stride + b], wG) : 0.f;
}

struct GramArgs {
    const uint8_t* a_ops; // data tiles (kTileM rows)
    const uint8_t* b_ops; // dictionary chunks (N rows)
    const float* xn;      // data norms
    const float* dn;      // dictionary norms (Mpad)
    const float* aw;      // users x Mpad
    const float* fw;      // fix weights (Mpad)
    const float* gate;    // per chunk: max fw, max fw |ewl2 dn|, 0, 0
    const float* xrows;   // data rows (n_samples x Dp, FP32) for the exact recompute
    const float* drows;   // dictionary rows (M x Dp, FP32)
    float* part;          // splits x users x n_samples partial sums
    int* err;
    int n_samples, Mpad, users, Kp, N, Dp, D;
    int chunks_per_split, n_chunks;
    int stages; // dictionary chunks in flight (<= kMaxStages)
    float ewl2; // ew * log2(e)
    unsigned long long wait_ns; // limit of the bounded waits
};

// NC accumulator columns of one data row: squared distance from the cross term
// and the norms, Gaussian value, contraction with every user's coefficients.
// xs: the stage's norms (xs[0 .. NC)), coefficient rows (xs[(1 + u) N + ...]) and
// fix weights (xs[(1 + users) N + ...]).  CHECK: entries whose error bound exceeds
// kFixEps are left out and returned as bits of the mask (column j -> bit j).
template <int NC, int NU, bool CHECK>
__device__ __forceinline__ uint32_t epilogue_columns(const float* gv, const float* xs, int N, float xn, float ewl2,
                                                     int users, float* acc)
{
    uint32_t mask = 0u;
#pragma unroll
    for (int j = 0; j < NC; j += 4) {
        const float4 dn4 = *reinterpret_cast<const float4*>(xs + j);
        const float t[4] = {xn + dn4.x, xn + dn4.y, xn + dn4.z, xn + dn4.w};
        float kv[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) kv[e] = ex2(ewl2 * fmaxf(fmaf(-2.f, gv[j + e], t[e]), 0.f));
        if constexpr (CHECK) {
            const float4 fw4 = *reinterpret_cast<const float4*>(xs + (1 + users) * N + j);
            const float fw[4] = {fw4.x, fw4.y, fw4.z, fw4.w};
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (kv[e] * (ewl2 * t[e]) * fw[e] < -1.f) {
                    mask |= 1u << (j + e);
                    kv[e] = 0.f;
                }
        }
#pragma unroll
        for (int u = 0; u < NU; ++u) {
            if (u < users) {
                const float4 a4 = *reinterpret_cast<const float4*>(xs + (1 + u) * N + j);
                acc[u] = fmaf(a4.x, kv[0], acc[u]);
                acc[u] = fmaf(a4.y, kv[1], acc[u]);
                acc[u] = fmaf(a4.z, kv[2], acc[u]);
                acc[u] = fmaf(a4.w, kv[3], acc[u]);
            }
        }
    }
    return mask;
}

// Largest |ewl2 xn| of the warp's rows.
__device__ __forceinline__ float warp_exn_max(float ewl2, float xn)
{
    float v = fabsf(ewl2 * xn);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

template <int MODE, int NU>
__global__ void __launch_bounds__(kThreads, 1) gram_detect_kernel(GramArgs g)
{
    using T = OpTraits<MODE>;
    extern __shared__ __align__(1024) uint8_t smem[];
    const int KE = T::kSplit ? 2 * g.Kp : g.Kp;
    const uint32_t a_bytes = uint32_t(kTileM) * KE * T::kElem;
    const uint32_t b_bytes = uint32_t(g.N) * KE * T::kElem;
    const uint32_t x_bytes = uint32_t(g.N) * 4 * (2 + g.users) + 16; // dn, aw rows, fw, chunk gate
    uint8_t* sA = smem;
    uint8_t* sB = sA + a_bytes;
    const int NS = g.stages;
    float* sX = reinterpret_cast<float*>(sB + size_t(NS) * b_bytes); // [stage][1 + users][N]
    uint64_t* bars = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(sX) + size_t(NS) * x_bytes);
    uint64_t* full = bars;            // [NS]
    uint64_t* empty = bars + NS;      // [NS]
    uint64_t* tfull = bars + 2 * NS;  // [2]
    uint64_t* tempty = tfull + 2;          // [2]
    uint64_t* afull = tempty + 2;          // [1]
    uint64_t* done = afull + 1;            // [1] all MMAs of the CTA completed
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    float* red = reinterpret_cast<float*>(tmem_slot + 4); // [4 warps][32][users] second-half partials

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x, split = blockIdx.y;
    const int c0 = split * g.chunks_per_split;
    const int c1 = min(g.n_chunks, c0 + g.chunks_per_split);
    const int nch = max(0, c1 - c0);
    const int N = g.N;
    const uint32_t ncols = uint32_t(2 * N);

    if (threadIdx.x == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1 + kEpiWarps);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&tfull[s], 1);
            mbar_init(&tempty[s], kEpiWarps);
        }
        mbar_init(afull, 1);
        mbar_init(done, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kEpiWarps + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(ncols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == kEpiWarps) {
        // ---------------- producer: data tile once, then dictionary chunks ----------------
        if (lane == 0) {
            mbar_expect_tx(afull, a_bytes);
            bulk_g2s(sA, g.a_ops + size_t(tile) * a_bytes, a_bytes, afull);
            int issued = 0;
            for (int i = 0; i < nch; ++i) {
                const int s = i % NS;
                if (i >= NS && !mbar_wait(&empty[s], ((i / NS) - 1) & 1, abort_flag, g.wait_ns)) break;
                ++issued;
                const int c = c0 + i;
                mbar_expect_tx(&full[s], b_bytes + x_bytes);
                bulk_g2s(sB + size_t(s) * b_bytes, g.b_ops + size_t(c) * b_bytes, b_bytes, &full[s]);
                float* xs = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(sX) + size_t(s) * x_bytes);
                bulk_g2s(xs, g.dn + size_t(c) * N, N * 4, &full[s]);
                for (int u = 0; u < g.users; ++u)
                    bulk_g2s(xs + (1 + u) * N, g.aw + size_t(u) * g.Mpad + size_t(c) * N, N * 4, &full[s]);
                bulk_g2s(xs + (1 + g.users) * N, g.fw + size_t(c) * N, N * 4, &full[s]);
                bulk_g2s(xs + (2 + g.users) * N, g.gate + size_t(c) * 4, 16, &full[s]);
            }
            // no bulk copy may still be writing shared memory when the CTA exits
            mbar_drain(afull, 0);
            for (int i = max(0, issued - NS); i < issued; ++i) mbar_drain(&full[i % NS], (i / NS) & 1);
        }
    } else if (warp == kEpiWarps + 1) {
        // ---------------- MMA issuer ----------------
        if (lane == 0 && mbar_wait(afull, 0, abort_flag, g.wait_ns)) {
            const uint32_t idesc = instr_desc<MODE>(kTileM, N);
            const uint32_t lbo_a = kTileM * 16, lbo_b = uint32_t(N) * 16;
            const int ksteps = g.Kp / T::kStepK;
            const int lo_off = g.Kp / T::kChunk; // K chunks to the lo half
            for (int i = 0; i < nch; ++i) {
                const int s = i % NS, buf = i & 1;
                if (!mbar_wait(&full[s], (i / NS) & 1, abort_flag, g.wait_ns)) break;
                if (i >= 2 && !mbar_wait(&tempty[buf], ((i >> 1) - 1) & 1, abort_flag, g.wait_ns)) break;
                tc_fence_after();
                const uint8_t* b = sB + size_t(s) * b_bytes;
                const uint32_t d = tmem + uint32_t(buf * N);
                uint32_t acc = 0;
                for (int kk = 0; kk < ksteps; ++kk) {
                    const uint64_t ah = smem_desc(sA + size_t(2 * kk) * lbo_a, lbo_a, 128);
                    const uint64_t bh = smem_desc(b + size_t(2 * kk) * lbo_b, lbo_b, 128);
                    umma<MODE>(d, ah, bh, idesc, acc);
                    acc = 1;
                    if constexpr (T::kSplit) {
                        const uint64_t al = smem_desc(sA + size_t(lo_off + 2 * kk) * lbo_a, lbo_a, 128);
                        const uint64_t bl = smem_desc(b + size_t(lo_off + 2 * kk) * lbo_b, lbo_b, 128);
                        umma<MODE>(d, ah, bl, idesc, 1);
                        umma<MODE>(d, al, bh, idesc, 1);
                    }
                }
                umma_commit(&tfull[buf]); // accumulator ready for the epilogue
                umma_commit(&empty[s]);   // operand stage free once these MMAs completed
            }
        }
        if (lane == 0) {
            // every MMA of this CTA has completed before tensor memory is released
            umma_commit(done);
            mbar_drain(done, 0);
        }
    } else {
        // ---------------- epilogue: 8 warps ----------------
        const int q = warp & 3, h = warp >> 2;
        const int row = tile * kTileM + q * 32 + lane;
        const bool valid = row < g.n_samples;
        const float xn = valid ? g.xn[row] : 0.f;
        const float exn_max = fix_scale<MODE>() > 0.f ? warp_exn_max(g.ewl2, xn) : 0.f;
        float acc[NU];
#pragma unroll
        for (int u = 0; u < NU; ++u) acc[u] = 0.f;
        const int half = N / 2;
        // flagged entries of one batch of columns: exact squared distance from the FP32 rows
        auto fix = [&](uint32_t mask, const float* xs, int col, int c) {
            if (!valid) return;
            while (mask) {
                const int j = __ffs(mask) - 1;
                mask &= mask - 1u;
                const float d2 = row_distance(g.xrows + size_t(row) * g.Dp, g.drows + size_t(c * N + col + j) * g.Dp, g.D);
                const float kv = ex2(g.ewl2 * d2);
#pragma unroll
                for (int u = 0; u < NU; ++u)
                    if (u < g.users) acc[u] = fmaf(xs[(1 + u) * N + col + j], kv, acc[u]);
            }
        };
        for (int i = 0; i < nch; ++i) {
            const int s = i % NS, buf = i & 1;
            // the stage's norms / coefficients (bulk copies) and the accumulator
            const bool ready = mbar_wait(&full[s], (i / NS) & 1, abort_flag, g.wait_ns) &&
                               mbar_wait(&tfull[buf], (i >> 1) & 1, abort_flag, g.wait_ns);
            if (!__all_sync(0xffffffffu, ready)) break; // (the loads below are warp-wide)
            tc_fence_after();
            const float* xs = reinterpret_cast<const float*>(reinterpret_cast<const uint8_t*>(sX) + size_t(s) * x_bytes);
            const uint32_t trow = tmem + (uint32_t(q * 32) << 16) + uint32_t(buf * N);
            // can any entry of this chunk exceed the bound for a row of this warp?  (warp-uniform)
            const float* gate = xs + (2 + g.users) * N;
            const bool check = fix_scale<MODE>() > 0.f && fmaf(exn_max, gate[0], gate[1]) > 1.f;
            for (int cb = 0; cb < half; cb += 32) {
                const int col = h * half + cb;
                float gv[32];
                __syncwarp(); // (lanes recompute different numbers of entries)
                tmem_ld32(trow + uint32_t(col), gv);
                if (check) fix(epilogue_columns<32, NU, true>(gv, xs + col, N, xn, g.ewl2, g.users, acc), xs, col, c0 + i);
                else epilogue_columns<32, NU, false>(gv, xs + col, N, xn, g.ewl2, g.users, acc);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&tempty[buf]);
                mbar_arrive(&empty[s]);
            }
        }
        // combine the two column halves: warps 4-7 hand their sums to warps 0-3
        asm volatile("bar.sync 1, %0;" ::"r"(kEpiWarps * 32) : "memory");
        if (h == 1) {
#pragma unroll
            for (int u = 0; u < NU; ++u)
                if (u < g.users) red[(q * 32 + lane) * g.users + u] = acc[u];
        }
        asm volatile("bar.sync 1, %0;" ::"r"(kEpiWarps * 32) : "memory");
        if (h == 0 && row < g.n_samples) {
#pragma unroll
            for (int u = 0; u < NU; ++u)
                if (u < g.users)
                    g.part[(size_t(split) * g.users + u) * g.n_samples + row] =
                        acc[u] + red[(q * 32 + lane) * g.users + u];
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == kEpiWarps + 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols));
    }
    if (threadIdx.x == 0 && *abort_flag) atomicExch(g.err, 1);
}

// out[u][s] = wL <w_u, x_s> + sum_split part[split][u][s] (fixed order; each linear
// term's d in order).  Bound: HBM (131072 rows of 128 features, 16 users: 84 MB, 13
// us).  A thread takes two samples (rows of the block's tile in shared memory) and
// four users, so 8 fma take 2 + 4 floats of shared memory instead of one each from
// there and from L1: 77 before, 43 us now.
constexpr int kFinSamples = 64;
constexpr int kFinPer = kFinSamples / 32;
constexpr int kFinThreads = 128; // warp: samples lane + 32 k, users 4 warp ..
constexpr int kFinPitch = kMaxUsers + 4;

size_t finish_smem(int Dp) // at most 44032 bytes
{
    return sizeof(float) * (size_t(kFinSamples) * (Dp + 4) + size_t(Dp) * kFinPitch);
}

__global__ void __launch_bounds__(kFinThreads)
    gram_finish_kernel(const float* __restrict__ xs, int Dp, int D, const float* __restrict__ w, float wL,
                       const float* __restrict__ part, int splits, int users, int n_samples, float* __restrict__ out,
                       size_t out_stride)
{
    extern __shared__ __align__(16) float fsm[];
    const int P = Dp + 4, q = Dp >> 2, tid = threadIdx.x, lane = tid & 31, u0 = 4 * (tid >> 5);
    float* const xt = fsm;                    // [kFinSamples][P]
    float* const wt = xt + kFinSamples * P;   // [Dp][kFinPitch]
    const int s0 = blockIdx.x * kFinSamples, n = min(kFinSamples, n_samples - s0);
    {
        const float4* const src = reinterpret_cast<const float4*>(xs + size_t(s0) * Dp);
        int r = tid / q, c = tid - r * q;
        const int dr = kFinThreads / q, dc = kFinThreads - dr * q;
#pragma unroll 8
        for (int idx = tid; idx < n * q; idx += kFinThreads) {
            *reinterpret_cast<float4*>(xt + r * P + 4 * c) = __ldg(src + idx);
            r += dr;
            c += dc;
            if (c >= q) {
                c -= q;
                ++r;
            }
        }
        for (int idx = tid; idx < Dp * kMaxUsers; idx += kFinThreads) {
            const int u = idx / Dp, d = idx - u * Dp;
            wt[d * kFinPitch + u] = u < users && d < D ? __ldg(w + size_t(u) * D + d) : 0.f;
        }
    }
    __syncthreads();
    if (u0 >= users) return;
    float lin[kFinPer][4];
#pragma unroll
    for (int k = 0; k < kFinPer; ++k)
#pragma unroll
        for (int u = 0; u < 4; ++u) lin[k][u] = 0.f;
#pragma unroll 2
    for (int d = 0; d < Dp; d += 4) {
        float4 x[kFinPer];
#pragma unroll
        for (int k = 0; k < kFinPer; ++k) x[k] = *reinterpret_cast<const float4*>(xt + (lane + 32 * k) * P + d);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float4 w4 = *reinterpret_cast<const float4*>(wt + (d + j) * kFinPitch + u0);
#pragma unroll
            for (int k = 0; k < kFinPer; ++k) {
                const float v = j == 0 ? x[k].x : j == 1 ? x[k].y : j == 2 ? x[k].z : x[k].w;
                lin[k][0] = fmaf(w4.x, v, lin[k][0]);
                lin[k][1] = fmaf(w4.y, v, lin[k][1]);
                lin[k][2] = fmaf(w4.z, v, lin[k][2]);
                lin[k][3] = fmaf(w4.w, v, lin[k][3]);
            }
        }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
        if (u0 + u < users)
#pragma unroll
            for (int k = 0; k < kFinPer; ++k) {
                const int s = s0 + lane + 32 * k;
                if (s >= n_samples) continue;
                float gsum = 0.f;
                for (int sp = 0; sp < splits; ++sp) gsum += part[(size_t(sp) * users + u0 + u) * n_samples + s];
                out[size_t(u0 + u) * out_stride + s] = fmaf(wL, lin[k][u], gsum);
            }
}

// ------------------------------------------------ two-product form (users >= 4) --
// The users' contraction on the tensor cores too (BF16 form): the Gram tile of a
// chunk of 128 dictionary rows becomes kernel values, and these as BF16 times the
// chunk's coefficients a * wG (BF16, padded with zero users to 16) add to the
// users' sums.  The epilogue then costs one exponential and half a conversion
// per kernel value instead of one FMA per user; the second product rounds kernel
// values and coefficients to BF16.  Used with 4 or more users: the soft outputs
// move from 1.4e-6 to 5.2e-5 of the largest output away from the float64 model
// (decisions unchanged, 64 antennas, 16 users); the TF32 form would gain 2 % for
// a 10x larger error, so the other forms keep the one-product kernel.
//
// Bound: the special function unit (131072 x 16384 exponentials: 0.47 ms) and the
// Gram tiles (0.33 ms).  With data tile, kernel values and norms in shared memory
// the products, stores and broadcasts took 1900 cycles a chunk against 1024 of
// exponentials; with the kernel values in tensor memory the second UMMA (16
// columns wide, between two Gram tiles) held the tensor pipe for as long as the
// Gram tile.  So the data tile (converted from the packed rows) is a
// tensor-memory operand, and the second product is made of warp-level MMAs: an
// accumulator loaded in the 16x256b shape, exponentiated and converted in place
// is their operand fragment, with no store, barrier or second pass.  Even and odd
// chunks have their own eight epilogue warps; three Gram buffers.
constexpr int kUsers2 = 16; // users of the second product
constexpr int kN2 = 128;    // dictionary rows per chunk
constexpr int kStages2 = 4; // chunks' rows in flight
constexpr int kXStages2 = 4; // chunks' coefficients and norms in flight
constexpr int kEpiWarps2 = 16;
constexpr int kGroup2 = kEpiWarps2 / 2; // warps of an even or odd chunk
constexpr int kThreads2 = (kEpiWarps2 + 2) * 32;
constexpr int kXd2 = 2 * kN2 + 4; // chunk norms, fix weights, gate

struct Gram2Args {
    const float* rows;    // data rows (n_samples x Dp, FP32)
    const uint8_t* b_ops; // dictionary chunks (kN2 rows)
    const uint8_t* w_ops; // per chunk: coefficient fragments (gram_pack_w_kernel)
    const float* dn;      // dictionary norms (Mpad)
    const float* fw;      // fix weights (Mpad)
    const float* gate;    // per chunk: max fw, max fw |ewl2 dn|, 0, 0
    const float* drows;   // dictionary rows (M x Dp, FP32) for the exact recompute
    float* part;          // splits x users x n_samples partial sums
    int* err;
    int n_samples, users, Kp, Dp, D;
    int chunks_per_split, n_chunks;
    float ewl2; // ew * log2(e)
    unsigned long long wait_ns; // limit of the bounded waits
};

// Tensor memory columns: three Gram buffers, the data tile (BF16 pairs)
constexpr int kBufs2 = 3;
constexpr uint32_t kTmA = kBufs2 * kN2;

// acc (16 rows x 8 users) += a (16 rows x 16 BF16) b (16 x 8 users)
__device__ __forceinline__ void warp_mma(float (&acc)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1)
{
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(acc[0]), "+f"(acc[1]), "+f"(acc[2]), "+f"(acc[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// 32 columns (sd: their norms, fix weights kN2 further) of four rows: thread t's columns 8 e + 2 (t % 4) + {0, 1}
// of rows t / 4 + 8 m, Gram values v as loaded, kernel values as BF16 pairs into p[m / 2][2 e + m % 2].  CHECK:
// entries whose error bound exceeds kFixEps are returned as bits 8 m + 2 e + {0, 1} of the mask (p is rewritten).
template <bool CHECK>
__device__ __forceinline__ uint32_t kernel_values(const uint32_t (&v)[2][16], const float* sd, const f32x2 (&xn)[4],
                                                  float ewl2, uint32_t (&p)[2][8])
{
    uint32_t mask = 0u;
    const f32x2 minus2 = pack2(-2.f, -2.f), ew2 = pack2(ewl2, ewl2);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const f32x2 dn = *reinterpret_cast<const f32x2*>(sd + 8 * e);
        f32x2 fw = 0ull;
        if constexpr (CHECK) fw = *reinterpret_cast<const f32x2*>(sd + kN2 + 8 * e);
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const uint32_t* const g = v[m >> 1] + 4 * e + 2 * (m & 1);
            const f32x2 t = add2(xn[m], dn);
            const float2 d2 = unpack2(fma2(minus2, pack2(__uint_as_float(g[0]), __uint_as_float(g[1])), t));
            const float2 x = unpack2(mul2(ew2, pack2(fmaxf(d2.x, 0.f), fmaxf(d2.y, 0.f))));
            const float k0 = ex2(x.x), k1 = ex2(x.y);
            if constexpr (CHECK) {
                const float2 b = unpack2(mul2(pack2(k0, k1), mul2(mul2(ew2, t), fw)));
                if (b.x < -1.f) mask |= 1u << (8 * m + 2 * e);
                if (b.y < -1.f) mask |= 2u << (8 * m + 2 * e);
            }
            const __nv_bfloat162 k2 = __floats2bfloat162_rn(k0, k1); // (round to nearest)
            p[m >> 1][2 * e + (m & 1)] = *reinterpret_cast<const uint32_t*>(&k2);
        }
    }
    return mask;
}

// Coefficients a[u][b] * wG as BF16 (0 past M and for u >= users) in the fragment order of warp_mma: 16 bytes per 16
// dictionary rows and lane t, word j holding rows 8 (j % 2) + 2 (t % 4) + {0, 1} of user 8 (j / 2) + t / 4.
__global__ void gram_pack_w_kernel(const float* __restrict__ a, size_t a_stride, int users, int M, int n_chunks, float wG,
                                   uint32_t* __restrict__ w_ops)
{
    const int total = n_chunks * (kN2 / 16) * 128;
    for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += gridDim.x * blockDim.x) {
        const int j = idx % 4, t = idx / 4 % 32, u = 8 * (j / 2) + t / 4, b = idx / 128 * 16 + 8 * (j % 2) + 2 * (t % 4);
        const float* const c = a + size_t(u) * a_stride + b;
        const __nv_bfloat162 v = __floats2bfloat162_rn(u < users && b < M ? __fmul_rn(c[0], wG) : 0.f,
                                                       u < users && b + 1 < M ? __fmul_rn(c[1], wG) : 0.f);
        w_ops[idx] = *reinterpret_cast<const uint32_t*>(&v);
    }
}

__global__ void __launch_bounds__(kThreads2, 1) gram_detect2_kernel(Gram2Args g)
{
    constexpr int MODE = kBF16, N = kN2, NS = kStages2, NX = kXStages2;
    using T = OpTraits<MODE>;
    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t b_bytes = uint32_t(N) * g.Kp * T::kElem;
    constexpr uint32_t w_bytes = kUsers2 * N * T::kElem;
    constexpr int kParts = kEpiWarps2 / 4; // warps that share a row: column halves of even and odd chunks
    uint8_t* const sB = smem;                           // [NS] chunk rows
    uint8_t* const sW = sB + size_t(NS) * b_bytes;      // [NX] chunk coefficients
    float* const sD = reinterpret_cast<float*>(sW + size_t(NX) * w_bytes); // [NX][kXd2]
    float* const sxn = sD + NX * kXd2;                  // [kTileM] data norms
    float* const red = sxn + kTileM;                    // [kParts][kTileM][kUsers2]
    uint64_t* const bars = reinterpret_cast<uint64_t*>(red + kParts * kTileM * kUsers2);
    uint64_t* const full = bars;             // [NS]
    uint64_t* const empty = full + NS;       // [NS]
    uint64_t* const xfull = empty + NS;      // [NX]
    uint64_t* const xempty = xfull + NX;     // [NX]
    uint64_t* const tfull = xempty + NX;     // [kBufs2] Gram tile
    uint64_t* const tempty = tfull + kBufs2; // [kBufs2]
    uint64_t* const afull = tempty + kBufs2; // [1]
    uint64_t* const done = afull + 1;        // [1] every product of the CTA completed
    uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    volatile int* const abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x, split = blockIdx.y;
    const int c0 = split * g.chunks_per_split;
    const int c1 = min(g.n_chunks, c0 + g.chunks_per_split);
    const int nch = max(0, c1 - c0);
    constexpr uint32_t ncols = 512;

    if (threadIdx.x == 0) {
        for (int s = 0; s < NS; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int s = 0; s < NX; ++s) {
            mbar_init(&xfull[s], 1);
            mbar_init(&xempty[s], kGroup2);
        }
        for (int s = 0; s < kBufs2; ++s) {
            mbar_init(&tfull[s], 1);
            mbar_init(&tempty[s], kGroup2);
        }
        mbar_init(afull, kEpiWarps2);
        mbar_init(done, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kEpiWarps2 + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(ncols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == kEpiWarps2) {
        // ---------------- producer: dictionary chunks with their W and norms ----------------
        if (lane == 0) {
            int issued = 0, xissued = 0;
            for (int i = 0; i < nch; ++i) {
                const int s = i % NS, x = i % NX, c = c0 + i;
                if (i >= NS && !mbar_wait(&empty[s], ((i / NS) - 1) & 1, abort_flag, g.wait_ns)) break;
                ++issued;
                mbar_expect_tx(&full[s], b_bytes);
                bulk_g2s(sB + size_t(s) * b_bytes, g.b_ops + size_t(c) * b_bytes, b_bytes, &full[s]);
                if (i >= NX && !mbar_wait(&xempty[x], ((i / NX) - 1) & 1, abort_flag, g.wait_ns)) break;
                ++xissued;
                mbar_expect_tx(&xfull[x], w_bytes + kXd2 * 4);
                bulk_g2s(sW + size_t(x) * w_bytes, g.w_ops + size_t(c) * w_bytes, w_bytes, &xfull[x]);
                float* sd = sD + size_t(x) * kXd2;
                bulk_g2s(sd, g.dn + size_t(c) * N, uint32_t(N) * 4, &xfull[x]);
                bulk_g2s(sd + N, g.fw + size_t(c) * N, uint32_t(N) * 4, &xfull[x]);
                bulk_g2s(sd + 2 * N, g.gate + size_t(c) * 4, 16, &xfull[x]);
            }
            for (int i = max(0, issued - NS); i < issued; ++i) mbar_drain(&full[i % NS], (i / NS) & 1);
            for (int i = max(0, xissued - NX); i < xissued; ++i) mbar_drain(&xfull[i % NX], (i / NX) & 1);
        }
    } else if (warp == kEpiWarps2 + 1) {
        // ---------------- MMA issuer ----------------
        if (lane == 0 && mbar_wait(afull, 0, abort_flag, g.wait_ns)) {
            const uint32_t idesc = instr_desc<MODE>(kTileM, N);
            constexpr uint32_t lbo = N * 16;
            const int ksteps = g.Kp / T::kStepK;
            // One thread issues everything: the descriptor is built once, a K step or a stage is an addition to its
            // address field (units of 16 bytes).  Building one for every product took 100 cycles each, more than
            // the product.
            constexpr uint64_t kStep = 2 * lbo / 16;
            constexpr uint32_t kStepA = T::kStepK / 2; // tensor-memory columns of a K step
            const uint64_t db = smem_desc(sB, lbo, 128);
            for (int i = 0; i < nch; ++i) {
                const int s = i % NS, buf = i % kBufs2;
                if (!mbar_wait(&full[s], (i / NS) & 1, abort_flag, g.wait_ns)) break;
                if (i >= kBufs2 && !mbar_wait(&tempty[buf], ((i / kBufs2) - 1) & 1, abort_flag, g.wait_ns)) break;
                tc_fence_after();
                const uint64_t b = db + uint64_t(s) * (b_bytes / 16);
                const uint32_t d = tmem + uint32_t(buf * N);
                umma_ts<MODE>(d, tmem + kTmA, b, idesc, 0u);
#pragma unroll
                for (int kk = 1; kk < kMaxFeatures / T::kStepK; ++kk)
                    if (kk < ksteps) umma_ts<MODE>(d, tmem + kTmA + kk * kStepA, b + kk * kStep, idesc, 1u);
                umma_commit(&tfull[buf]); // Gram tile ready for the epilogue
                umma_commit(&empty[s]);   // the chunk's rows are free
            }
        }
        if (lane == 0) {
            umma_commit(done);
            mbar_drain(done, 0);
        }
    } else {
        // ---------------- epilogue: kernel values of each chunk, times the coefficients ----------------
        const int q = warp & 3, group = warp >> 3, half = (warp >> 2 & 1) * (N / 2); // this warp's columns of its chunks
        const uint32_t tlane = tmem + (uint32_t(q * 32) << 16);
        const int row = tile * kTileM + q * 32 + lane; // of this thread's tensor-memory lane
        {
            // the data tile: K steps warp / 4, + 4, ... of this row; the first warps also the norms
            const float* const xr = g.rows + size_t(row) * g.Dp;
            auto load4 = [&](int k) {
                return row < g.n_samples && k < g.Dp ? __ldg(reinterpret_cast<const float4*>(xr + k))
                                                     : make_float4(0.f, 0.f, 0.f, 0.f);
            };
#pragma unroll 2
            for (int k = 16 * (warp >> 2); k < g.Kp; k += 64) {
                uint32_t w[8];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float4 v = load4(k + 4 * j);
                    const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
                    w[2 * j] = *reinterpret_cast<const uint32_t*>(&lo);
                    w[2 * j + 1] = *reinterpret_cast<const uint32_t*>(&hi);
                }
                tmem_st8(tlane + kTmA + uint32_t(k / 2), w);
            }
            if (warp < 4) {
                float acc = 0.f;
#pragma unroll 8
                for (int k = 0; k < g.Dp; k += 4) {
                    const float4 v = load4(k);
                    acc = fmaf(v.x, v.x, acc);
                    acc = fmaf(v.y, v.y, acc);
                    acc = fmaf(v.z, v.z, acc);
                    acc = fmaf(v.w, v.w, acc);
                }
                sxn[q * 32 + lane] = acc;
            }
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(afull);
            asm volatile("bar.sync 1, %0;" ::"n"(kEpiWarps2 * 32) : "memory");
        }
        const int r0 = q * 32 + (lane >> 2), cp = 2 * (lane & 3); // rows r0 + 8 m, columns cp, cp + 1 of each eight
        f32x2 xn[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) xn[m] = pack2(sxn[r0 + 8 * m], sxn[r0 + 8 * m]);
        const float exn_max = warp_exn_max(g.ewl2, sxn[q * 32 + lane]);
        float acc[2][2][4]; // rows 16 m .., users 8 n ..
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[m][n][j] = 0.f;
        for (int i = group; i < nch; i += 2) {
            const int x = i % NX, buf = i % kBufs2;
            bool ok = mbar_wait(&xfull[x], (i / NX) & 1, abort_flag, g.wait_ns) &&
                 mbar_wait(&tfull[buf], (i / kBufs2) & 1, abort_flag, g.wait_ns);
            ok = __all_sync(0xffffffffu, ok); // (the loads below are warp-wide)
            if (!ok) break;
            tc_fence_after();
            const float* sd = sD + size_t(x) * kXd2;
            // can any entry of this chunk exceed the bound for a row of this warp?  (warp-uniform)
            const bool check = fmaf(exn_max, sd[2 * N], sd[2 * N + 1]) > 1.f;
#pragma unroll 1
            for (int col = half; col < half + N / 2; col += 32) {
                uint32_t v[2][16], p[2][8];
                tmem_ld_16x32(tlane + uint32_t(buf * N + col), v[0]);
                tmem_ld_16x32(tlane + (16u << 16) + uint32_t(buf * N + col), v[1]);
                tmem_ld_wait(v[0], v[1]);
                if (col != half) { // the accumulators are in registers
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&tempty[buf]);
                }
                if (!check) {
                    kernel_values<false>(v, sd + col + cp, xn, g.ewl2, p);
                } else {
                    uint32_t mask = kernel_values<true>(v, sd + col + cp, xn, g.ewl2, p);
                    // flagged entries: exact squared distance from the FP32 rows, the value replaced
                    while (mask) {
                        const int j = __ffs(mask) - 1, fr = tile * kTileM + r0 + 8 * (j >> 3);
                        mask &= mask - 1u;
                        if (fr >= g.n_samples) continue;
                        const float d2 = row_distance(
                            g.rows + size_t(fr) * g.Dp,
                            g.drows + size_t((c0 + i) * N + col + cp + 8 * (j >> 1 & 3) + (j & 1)) * g.Dp, g.D);
                        const uint32_t k = __bfloat16_as_ushort(__float2bfloat16_rn(ex2(g.ewl2 * d2)));
#pragma unroll
                        for (int m = 0; m < 4; ++m)
#pragma unroll
                            for (int e = 0; e < 4; ++e)
                                if ((j >> 1) == 4 * m + e) {
                                    uint32_t& t = p[m >> 1][2 * e + (m & 1)];
                                    t = (j & 1) ? (t & 0xffffu) | k << 16 : (t & 0xffff0000u) | k;
                                }
                    }
                }
                __syncwarp();
                const uint4* const w = reinterpret_cast<const uint4*>(sW + size_t(x) * w_bytes) + (col / 16) * 32 + lane;
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const uint4 b = w[32 * k];
#pragma unroll
                    for (int m = 0; m < 2; ++m) {
                        warp_mma(acc[m][0], p[m][4 * k], p[m][4 * k + 1], p[m][4 * k + 2], p[m][4 * k + 3], b.x, b.y);
                        warp_mma(acc[m][1], p[m][4 * k], p[m][4 * k + 1], p[m][4 * k + 2], p[m][4 * k + 3], b.z, b.w);
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&xempty[x]);
        }
        // a row's sums from the four warps that share it, in a fixed order
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int j = 0; j < 4; j += 2)
                    *reinterpret_cast<float2*>(red + (size_t(warp >> 2) * kTileM + r0 + 16 * m + 4 * j) * kUsers2 + 8 * n +
                                               cp) = make_float2(acc[m][n][j], acc[m][n][j + 1]);
        asm volatile("bar.sync 1, %0;" ::"n"(kEpiWarps2 * 32) : "memory");
        for (int u = warp >> 2; u < g.users; u += kParts) {
            if (row >= g.n_samples) break;
            float sum = 0.f;
#pragma unroll
            for (int k = 0; k < kParts; ++k) sum += red[(size_t(k) * kTileM + q * 32 + lane) * kUsers2 + u];
            g.part[(size_t(split) * g.users + u) * g.n_samples + row] = sum;
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == kEpiWarps2 + 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(ncols));
    }
    if (threadIdx.x == 0 && *abort_flag) atomicExch(g.err, 1);
}

size_t gram2_smem(int Kp)
{
    return size_t(kStages2) * kN2 * Kp * 2 + size_t(kXStages2) * kUsers2 * kN2 * 2 +
           sizeof(float) * (kXStages2 * kXd2 + kTileM + kEpiWarps2 / 4 * kTileM * kUsers2) +
           (2 * kStages2 + 2 * kXStages2 + 2 * kBufs2 + 2) * 8 + 16;
}

template <int MODE, int NU> void launch_gram(const GramArgs& ga, int n_tiles, int splits, size_t smem, cudaStream_t s,
                                             cudaError_t* e)
{
    *e = allow_smem(gram_detect_kernel<MODE, NU>);
    if (*e != cudaSuccess) return;
    gram_detect_kernel<MODE, NU><<<dim3(n_tiles, splits), kThreads, smem, s>>>(ga);
    *e = cudaGetLastError();
}

apsm_status run_gram2(apsm_detector* h, uint32_t S, float* d_out, cudaStream_t s, int Kp)
{
    constexpr int MODE = kBF16, N = kN2;
    GramWorkspace* gw = h->gram;
    const int ns = int(2 * S);
    const int M = int(h->used);
    const int D = int(h->D), Dp = int(h->Dp), U = int(h->U);
    const int n_tiles = (ns + kTileM - 1) / kTileM;
    const int n_chunks = std::max(1, (M + N - 1) / N);
    const int Mpad = n_chunks * N;
    int splits = std::max(1, std::min(n_chunks, (148 + n_tiles - 1) / n_tiles)); // one CTA per SM
    const int cps = (n_chunks + splits - 1) / splits;
    splits = (n_chunks + cps - 1) / cps;

    cudaError_t e;
#define GR_CK(x)                                                   \
    do {                                                           \
        e = (x);                                                   \
        if (e != cudaSuccess) return h->cuda_fail(e, #x);          \
    } while (0)
    GR_CK(gw->b_ops.ensure(size_t(n_chunks) * N * Kp * 2));
    GR_CK(gw->w_ops.ensure(size_t(n_chunks) * kUsers2 * N * 2));
    GR_CK(gw->dn.ensure(Mpad));
    GR_CK(gw->fw.ensure(Mpad));
    GR_CK(gw->gate.ensure(size_t(4) * n_chunks));
    GR_CK(gw->part.ensure(size_t(splits) * U * ns));
    GR_CK(gw->err.ensure(1));
    GR_CK(cudaMemsetAsync(gw->err.p, 0, sizeof(int), s));
    GR_CK(cudaMemsetAsync(gw->dn.p, 0, sizeof(float) * Mpad, s));
    const float ewl2 = h->model_params().ew * 1.4426950408889634f;

    const int threads = 256;
    gram_pack_kernel<MODE><<<std::min(4096, (n_chunks * N * Kp + threads - 1) / threads), threads, 0, s>>>(
        h->dict_X.p, M, Dp, D, Kp, N, n_chunks, gw->b_ops.p, gw->dn.p);
    GR_CK(cudaGetLastError());
    gram_fix_kernel<MODE><<<n_chunks, 256, 0, s>>>(h->dict_a.p, h->cap, U, M, N, h->cfg.wG, ewl2, gw->dn.p, gw->fw.p,
                                                   gw->gate.p);
    GR_CK(cudaGetLastError());
    gram_pack_w_kernel<<<std::min(4096, (n_chunks * kUsers2 * N / 2 + threads - 1) / threads), threads, 0, s>>>(
        h->dict_a.p, h->cap, U, M, n_chunks, h->cfg.wG, reinterpret_cast<uint32_t*>(gw->w_ops.p));
    GR_CK(cudaGetLastError());

    Gram2Args ga;
    ga.rows = h->xs.p;
    ga.b_ops = gw->b_ops.p;
    ga.w_ops = gw->w_ops.p;
    ga.dn = gw->dn.p;
    ga.fw = gw->fw.p;
    ga.gate = gw->gate.p;
    ga.drows = h->dict_X.p;
    ga.part = gw->part.p;
    ga.err = gw->err.p;
    ga.n_samples = ns;
    ga.users = U;
    ga.Kp = Kp;
    ga.Dp = Dp;
    ga.D = D;
    ga.chunks_per_split = cps;
    ga.n_chunks = n_chunks;
    ga.ewl2 = ewl2;
    ga.wait_ns = wait_limit_ns();
    // >= 120 KB keeps one CTA per SM: its tensor memory (512 columns) is never contended
    const size_t smem = std::max<size_t>(gram2_smem(Kp) + 1024, 120 * 1024);
    GR_CK(allow_smem(gram_detect2_kernel));
    gram_detect2_kernel<<<dim3(n_tiles, splits), kThreads2, smem, s>>>(ga);
    GR_CK(cudaGetLastError());
    GR_CK(launch_linear_part(h->xs.p, Dp, D, h->w.p, h->cfg.wL, gw->part.p, splits, U, ns, d_out, size_t(ns), s));
    GR_CK(cudaMemcpyAsync(gw->h_err, gw->err.p, sizeof(int), cudaMemcpyDeviceToHost, s));
#undef GR_CK
    return APSM_OK;
}

// TF32 split form: the data tile in tensor memory (kernels_gram_tmem.cu).
apsm_status run_gram_tmem(apsm_detector* h, uint32_t S, float* d_out, cudaStream_t s)
{
    constexpr int MODE = kTF32x3;
    using T = OpTraits<MODE>;
    GramWorkspace* gw = h->gram;
    const int ns = int(2 * S);
    const int M = int(h->used);
    const int D = int(h->D), Dp = int(h->Dp), U = int(h->U);
    if (U > kMaxUsers) {
        h->last_error = "Gram detection supports at most " + std::to_string(kMaxUsers) + " users per detector";
        return APSM_ERR_UNSUPPORTED;
    }
    const int Kp = int(round_up(uint32_t(D), uint32_t(T::kStepK)));
    const int N = kGramTmemChunk;
    const int n_tiles = (ns + kTileM - 1) / kTileM;
    const int n_chunks = std::max(1, (M + N - 1) / N);
    int splits = std::max(1, std::min(n_chunks, (2 * 148 + n_tiles - 1) / n_tiles));
    const int cps = (n_chunks + splits - 1) / splits;
    splits = (n_chunks + cps - 1) / cps;

    cudaError_t e;
#define GR_CK(x)                                                   \
    do {                                                           \
        e = (x);                                                   \
        if (e != cudaSuccess) return h->cuda_fail(e, #x);          \
    } while (0)
    GR_CK(gw->b_ops.ensure(size_t(n_chunks) * N * 2 * Kp * T::kElem));
    GR_CK(gw->dn.ensure(size_t(n_chunks) * N));
    GR_CK(gw->xd.ensure(gram_tmem_data_floats(U) * n_chunks));
    GR_CK(gw->part.ensure(size_t(splits) * U * ns));
    GR_CK(gw->err.ensure(1));
    GR_CK(cudaMemsetAsync(gw->err.p, 0, sizeof(int), s));

    const int threads = 256;
    gram_pack_kernel<MODE><<<std::min(4096, (n_chunks * N * Kp + threads - 1) / threads), threads, 0, s>>>(
        h->dict_X.p, M, Dp, D, Kp, N, n_chunks, gw->b_ops.p, gw->dn.p);
    GR_CK(cudaGetLastError());

    GramTmemArgs ga;
    ga.rows = h->xs.p;
    ga.b_ops = gw->b_ops.p;
    ga.xd = gw->xd.p;
    ga.part = gw->part.p;
    ga.err = gw->err.p;
    ga.n_samples = ns;
    ga.users = U;
    ga.Kp = Kp;
    ga.Dp = Dp;
    ga.chunks_per_split = cps;
    ga.n_chunks = n_chunks;
    ga.ewl2 = h->model_params().ew * 1.4426950408889634f;
    ga.wait_ns = wait_limit_ns();
    GR_CK(launch_gram_tmem(ga, gw->dn.p, h->dict_a.p, h->cap, M, h->cfg.wG, gw->xd.p, n_tiles, splits, s));
    GR_CK(launch_linear_part(h->xs.p, Dp, D, h->w.p, h->cfg.wL, gw->part.p, splits, U, ns, d_out, size_t(ns), s));
    GR_CK(cudaMemcpyAsync(gw->h_err, gw->err.p, sizeof(int), cudaMemcpyDeviceToHost, s));
#undef GR_CK
    return APSM_OK;
}

template <int MODE>
apsm_status run_gram(apsm_detector* h, uint32_t S, float* d_out, cudaStream_t s)
{
    using T = OpTraits<MODE>;
    GramWorkspace* gw = h->gram;
    const int ns = int(2 * S);
    const int M = int(h->used);
    const int D = int(h->D), Dp = int(h->Dp), U = int(h->U);
    if (U > kMaxUsers) {
        h->last_error = "Gram detection supports at most " + std::to_string(kMaxUsers) + " users per detector";
        return APSM_ERR_UNSUPPORTED;
    }
    const int Kp = int(round_up(uint32_t(D), uint32_t(T::kStepK)));
    const int KE = T::kSplit ? 2 * Kp : Kp;
    // the users' contraction on the tensor cores; only in the BF16 form, whose kernel values and
    // coefficients may be BF16 too (in the other forms the second product's rounding would cost
    // more accuracy than its time saves)
    if constexpr (MODE == kBF16)
        if (U >= 4 && !h->gram_one_product) return run_gram2(h, S, d_out, s, Kp);
    // dictionary chunk width: the data tile and the chunk ring within shared memory (chunks of 256 down
    // to 64 columns; 64 fit at 128 features of every form that runs here)
    int N = 256;
    const int stages = kMaxStages;
    auto smem_for = [&](int n, int st) {
        return size_t(kTileM) * KE * T::kElem + size_t(st) * (size_t(n) * KE * T::kElem + size_t(n) * 4 * (2 + U) + 16) +
               (2 * st + 6) * 8 + 16 + size_t(4 * 32) * U * 4;
    };
    const size_t limit = 220 * 1024;
    while (N > 64 && smem_for(N, stages) > limit) N /= 2;
    if (smem_for(N, stages) > limit) {
        h->last_error = "Gram detection operands do not fit shared memory";
        return APSM_ERR_UNSUPPORTED;
    }
    const int n_tiles = (ns + kTileM - 1) / kTileM;
    const int n_chunks = std::max(1, (M + N - 1) / N);
    const int Mpad = n_chunks * N;
    int splits = std::max(1, std::min(n_chunks, (2 * 148 + n_tiles - 1) / n_tiles));
    const int cps = (n_chunks + splits - 1) / splits;
    splits = (n_chunks + cps - 1) / cps;

    cudaError_t e;
#define GR_CK(x)                                                   \
    do {                                                           \
        e = (x);                                                   \
        if (e != cudaSuccess) return h->cuda_fail(e, #x);          \
    } while (0)
    GR_CK(gw->a_ops.ensure(size_t(n_tiles) * kTileM * KE * T::kElem));
    GR_CK(gw->b_ops.ensure(size_t(n_chunks) * N * KE * T::kElem));
    GR_CK(gw->xn.ensure(size_t(n_tiles) * kTileM));
    GR_CK(gw->dn.ensure(Mpad));
    GR_CK(gw->aw.ensure(size_t(U) * Mpad));
    GR_CK(gw->fw.ensure(Mpad));
    GR_CK(gw->gate.ensure(size_t(4) * n_chunks));
    GR_CK(gw->part.ensure(size_t(splits) * U * ns));
    GR_CK(gw->err.ensure(1));
    GR_CK(cudaMemsetAsync(gw->err.p, 0, sizeof(int), s));
    GR_CK(cudaMemsetAsync(gw->dn.p, 0, sizeof(float) * Mpad, s));
    const float ewl2 = h->model_params().ew * 1.4426950408889634f;

    const int threads = 256;
    gram_pack_kernel<MODE><<<std::min(4096, (n_tiles * kTileM * Kp + threads - 1) / threads), threads, 0, s>>>(
        h->xs.p, ns, Dp, D, Kp, kTileM, n_tiles, gw->a_ops.p, gw->xn.p);
    GR_CK(cudaGetLastError());
    gram_pack_kernel<MODE><<<std::min(4096, (n_chunks * N * Kp + threads - 1) / threads), threads, 0, s>>>(
        h->dict_X.p, M, Dp, D, Kp, N, n_chunks, gw->b_ops.p, gw->dn.p);
    GR_CK(cudaGetLastError());
    gram_coeff_kernel<<<(U * Mpad + 255) / 256, 256, 0, s>>>(h->dict_a.p, h->cap, U, M, Mpad, h->cfg.wG, gw->aw.p);
    GR_CK(cudaGetLastError());
    gram_fix_kernel<MODE><<<n_chunks, 256, 0, s>>>(h->dict_a.p, h->cap, U, M, N, h->cfg.wG, ewl2, gw->dn.p, gw->fw.p,
                                                   gw->gate.p);
    GR_CK(cudaGetLastError());

    GramArgs ga;
    ga.a_ops = gw->a_ops.p;
    ga.b_ops = gw->b_ops.p;
    ga.xn = gw->xn.p;
    ga.dn = gw->dn.p;
    ga.aw = gw->aw.p;
    ga.fw = gw->fw.p;
    ga.gate = gw->gate.p;
    ga.xrows = h->xs.p;
    ga.drows = h->dict_X.p;
    ga.part = gw->part.p;
    ga.err = gw->err.p;
    ga.n_samples = ns;
    ga.Mpad = Mpad;
    ga.users = U;
    ga.Kp = Kp;
    ga.N = N;
    ga.Dp = Dp;
    ga.D = D;
    ga.chunks_per_split = cps;
    ga.n_chunks = n_chunks;
    ga.stages = stages;
    ga.ewl2 = ewl2;
    ga.wait_ns = wait_limit_ns();
    // >= 120 KB keeps one CTA per SM, so the 2N tensor-memory columns of a CTA never wait for another's
    const size_t smem = std::max<size_t>(smem_for(N, stages) + 1024, 120 * 1024);
    if (U <= 1) launch_gram<MODE, 1>(ga, n_tiles, splits, smem, s, &e);
    else if (U <= 2) launch_gram<MODE, 2>(ga, n_tiles, splits, smem, s, &e);
    else if (U <= 4) launch_gram<MODE, 4>(ga, n_tiles, splits, smem, s, &e);
    else if (U <= 8) launch_gram<MODE, 8>(ga, n_tiles, splits, smem, s, &e);
    else launch_gram<MODE, 16>(ga, n_tiles, splits, smem, s, &e);
    if (e != cudaSuccess) return h->cuda_fail(e, "gram_detect_kernel launch");
    GR_CK(launch_linear_part(h->xs.p, Dp, D, h->w.p, h->cfg.wL, gw->part.p, splits, U, ns, d_out, size_t(ns), s));
    GR_CK(cudaMemcpyAsync(gw->h_err, gw->err.p, sizeof(int), cudaMemcpyDeviceToHost, s));
#undef GR_CK
    return APSM_OK;
}

} // namespace

cudaError_t launch_linear_part(const float* xs, int Dp, int D, const float* w, float wL, const float* part, int splits,
                               int users, int n_samples, float* out, size_t out_stride, cudaStream_t s)
{
    gram_finish_kernel<<<(n_samples + kFinSamples - 1) / kFinSamples, kFinThreads, finish_smem(Dp), s>>>(
        xs, Dp, D, w, wL, part, splits, users, n_samples, out, out_stride);
    return cudaGetLastError();
}

} // namespace apsm

using namespace apsm;

// Expiry of a bounded wait in the last Gram detection, read after its stream
// synchronised (host calls): reported once, then cleared.
apsm_status detect_gram_check(apsm_detector* h)
{
    if (!h->gram || !h->gram->h_err || !*h->gram->h_err) return APSM_OK;
    *h->gram->h_err = 0;
    h->last_error = "Gram detection gave up waiting on the GPU (bounded wait expired); its estimates are invalid";
    return APSM_ERR_CUDA;
}

apsm_status detect_gram(apsm_detector* h, uint32_t S, float* d_out, cudaStream_t s)
{
    if (!h->gram) {
        h->gram = new GramWorkspace();
        if (cudaMallocHost(&h->gram->h_err, sizeof(int)) != cudaSuccess) {
            cudaGetLastError();
            h->last_error = "pinned allocation failed";
            return APSM_ERR_OUT_OF_MEMORY;
        }
        *h->gram->h_err = 0;
    }
    if (*h->gram->h_err) { // an earlier call on this stream (device mode) gave up: reported once
        *h->gram->h_err = 0;
        h->last_error = "a previous Gram detection gave up waiting on the GPU (bounded wait expired)";
        return APSM_ERR_CUDA;
    }
    switch (h->cfg.detect_mode) {
    case DetectMode::GramBF16: return run_gram<kBF16>(h, S, d_out, s);
    case DetectMode::GramBF16x3: return run_gram<kBF16x3>(h, S, d_out, s);
    case DetectMode::GramTF32: return run_gram<kTF32>(h, S, d_out, s);
    case DetectMode::GramTF32x3: return run_gram_tmem(h, S, d_out, s);
    default: break;
    }
    h->last_error = "not a Gram detection mode";
    return APSM_ERR_INVALID_ARGUMENT;
}
