// Gram detection in the TF32 split form (gram_tf32x3) with the data tile in
// tensor memory.
//
// Cross terms of a 128-row data tile against chunks of 128 dictionary rows:
// x.d ~ xh.dh + xh.dl + xl.dh (tcgen05.mma, FP32 accumulators), then per entry
// the squared distance with FP32 norms, one exponential and the contraction
// with every user's coefficients, all as in kernels_detect_gram.cu.
//
// What bounds it, at 131072 x 16384 rows of 128 features and 16 users: the three
// products (1.65e12 flop, 2.0 ms at half the measured BF16 rate) and the users'
// 16 fma per entry (1.0 ms).  Before, shared memory: a split data tile of 128
// features was 128 KB, read again for each chunk of 32 dictionary rows that
// fitted beside it, and a coefficient was fetched for one row per thread (9.19
// ms; now 2.92 ms).  At 1 user and 16 features (8000 x 2000 rows) a call takes 60
// us (77 us before), so every size of this form runs here.
//  - the data tile is split once into tensor memory (2 Kp of the 512 columns,
//    128 lanes); the UMMAs read only the dictionary from shared memory, and a
//    chunk is 128 rows wide whatever the feature count;
//  - dictionary chunks stream through a ring of K slices (32 features hi | lo,
//    32 KB), so the ring is as deep for 128 features as for 32;
//  - the epilogue loads accumulators in the 16x256b shape: a thread holds two
//    neighbouring columns of four rows, so a coefficient serves four rows, and
//    the users' sums run in packed FP32 pairs;
//  - the tile's rows and norms come straight from the packed FP32 rows (no
//    operand copy of the data in HBM).
//
// Roles (320 threads): warps 0-7 epilogue (warp w: TMEM lanes 32*(w%4).., columns
// of half w/4 of each chunk), warp 8 producer, warp 9 TMEM allocator and MMA
// issuer.  Every mbarrier wait is bounded; on expiry the CTA records an error,
// still waits for its own copies and MMAs, releases tensor memory and returns.
#include "apsm_gram.cuh"
#include "apsm_tc.cuh"
#include "packed_f32.cuh"

#include <algorithm>

namespace apsm {

namespace {

using namespace tc;

constexpr int kTileM = 128;  // data rows per CTA (UMMA M)
constexpr int kN = kGramTmemChunk;
constexpr int kSliceK = 32;  // features per ring slice
constexpr int kStages = 6;   // slices in flight
constexpr int kXStages = 2;  // chunk data (norms, coefficients) in flight
constexpr int kEpiWarps = 8;
constexpr int kThreads = (kEpiWarps + 2) * 32;
constexpr uint32_t kCols = 512;        // tensor memory: accumulators 0-255, data tile from 256
constexpr uint32_t kAcol = 2 * kN;

// chunk data: norms [kN], coefficients [kN][pitch]; the pitch puts the four column pairs that a warp
// reads at once on distinct banks
__host__ __device__ constexpr int coef_pitch(int nu) { return nu >= 8 ? nu + 4 : nu; }

template <int NU> struct ChunkData {
    static constexpr int kPitch = coef_pitch(NU);
    static constexpr int kFloats = kN * (1 + kPitch);
};

int user_class(int users) { return users <= 1 ? 1 : users <= 2 ? 2 : users <= 4 ? 4 : users <= 8 ? 8 : 16; }

__global__ void chunk_data_kernel(const float* __restrict__ dn, const float* __restrict__ a, size_t a_stride, int users,
                                  int M, int n_chunks, int pitch, float wG, float* __restrict__ xd)
{
    const int per = kN * pitch;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_chunks * per; i += gridDim.x * blockDim.x) {
        const int c = i / per, k = i % per / pitch, u = i % pitch, b = c * kN + k;
        float* const x = xd + size_t(c) * (per + kN);
        x[kN + k * pitch + u] = (u < users && b < M) ? __fmul_rn(a[size_t(u) * a_stride + b], wG) : 0.f;
        if (u == 0) x[k] = b < M ? dn[b] : 0.f;
    }
}

template <int NU>
__global__ void __launch_bounds__(kThreads, 1) gram_tmem_kernel(GramTmemArgs g)
{
    constexpr int MODE = kTF32x3;
    using T = OpTraits<MODE>;
    using X = ChunkData<NU>;
    extern __shared__ __align__(1024) uint8_t smem[];
    const int Kp = g.Kp, ks = min(kSliceK, Kp), n_slices = (Kp + kSliceK - 1) / kSliceK;
    const uint32_t half_bytes = uint32_t(kN) * ks * T::kElem; // hi or lo of a slice
    uint8_t* const sB = smem;                                 // [kStages][hi | lo]
    float* const sX = reinterpret_cast<float*>(sB + size_t(kStages) * 2 * half_bytes); // [kXStages][X::kFloats]
    float* const red = sX + kXStages * X::kFloats;            // [kTileM][NU]
    float* const sxn = red + kTileM * NU;                     // [kTileM]
    uint64_t* const bars = reinterpret_cast<uint64_t*>(sxn + kTileM);
    uint64_t* const full = bars;                  // [kStages]
    uint64_t* const empty = full + kStages;       // [kStages]
    uint64_t* const xfull = empty + kStages;      // [kXStages]
    uint64_t* const xempty = xfull + kXStages;    // [kXStages]
    uint64_t* const tfull = xempty + kXStages;    // [2]
    uint64_t* const tempty = tfull + 2;           // [2]
    uint64_t* const afull = tempty + 2;           // [1]
    uint64_t* const done = afull + 1;             // [1]
    uint32_t* const tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
    volatile int* const abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int tile = blockIdx.x, split = blockIdx.y;
    const int c0 = split * g.chunks_per_split;
    const int nch = max(0, min(g.n_chunks, c0 + g.chunks_per_split) - c0);

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int s = 0; s < kXStages; ++s) {
            mbar_init(&xfull[s], 1);
            mbar_init(&xempty[s], kEpiWarps);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&tfull[s], 1);
            mbar_init(&tempty[s], kEpiWarps);
        }
        mbar_init(afull, kEpiWarps);
        mbar_init(done, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kEpiWarps + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == kEpiWarps) {
        // ---------------- producer: per chunk its K slices, then its norms and coefficients ----------------
        if (lane == 0) {
            const size_t chunk_bytes = size_t(kN) * 2 * Kp * T::kElem;
            int issued = 0, xissued = 0;
            bool ok = true;
            for (int i = 0; i < nch && ok; ++i) {
                const uint8_t* const b = g.b_ops + size_t(c0 + i) * chunk_bytes;
                for (int f = 0; f < n_slices; ++f) {
                    const int s = issued % kStages;
                    if (issued >= kStages && !mbar_wait(&empty[s], ((issued / kStages) - 1) & 1, abort_flag, g.wait_ns)) {
                        ok = false;
                        break;
                    }
                    const int k0 = f * kSliceK;
                    const uint32_t bytes = uint32_t(kN) * min(kSliceK, Kp - k0) * T::kElem;
                    uint8_t* const d = sB + size_t(s) * 2 * half_bytes;
                    mbar_expect_tx(&full[s], 2 * bytes);
                    bulk_g2s(d, b + size_t(k0) * kN * T::kElem, bytes, &full[s]);
                    bulk_g2s(d + half_bytes, b + size_t(Kp + k0) * kN * T::kElem, bytes, &full[s]);
                    ++issued;
                }
                if (!ok) break;
                const int s = i % kXStages;
                if (i >= kXStages && !mbar_wait(&xempty[s], ((i / kXStages) - 1) & 1, abort_flag, g.wait_ns)) break;
                mbar_expect_tx(&xfull[s], X::kFloats * 4);
                bulk_g2s(sX + size_t(s) * X::kFloats, g.xd + size_t(c0 + i) * X::kFloats, X::kFloats * 4, &xfull[s]);
                ++xissued;
            }
            // no bulk copy may still be writing shared memory when the CTA exits
            for (int i = max(0, issued - kStages); i < issued; ++i) mbar_drain(&full[i % kStages], (i / kStages) & 1);
            for (int i = max(0, xissued - kXStages); i < xissued; ++i)
                mbar_drain(&xfull[i % kXStages], (i / kXStages) & 1);
        }
    } else if (warp == kEpiWarps + 1) {
        // ---------------- MMA issuer ----------------
        if (lane == 0 && mbar_wait(afull, 0, abort_flag, g.wait_ns)) {
            tc_fence_after();
            const uint32_t idesc = instr_desc<MODE>(kTileM, kN);
            constexpr uint32_t lbo = kN * 16;
            // One thread issues everything: descriptors are built once, a K step, the lo half or a stage is an
            // addition to their address field (units of 16 bytes).  Building them for every product took 100
            // cycles each, about what a product takes.
            constexpr uint64_t kStep = 2 * lbo / 16;
            const uint64_t db = smem_desc(sB, lbo, 128), lo_half = half_bytes / 16;
            int n = 0;
            bool ok = true;
            for (int i = 0; i < nch && ok; ++i) {
                const int buf = i & 1;
                if (i >= 2 && !mbar_wait(&tempty[buf], ((i >> 1) - 1) & 1, abort_flag, g.wait_ns)) break;
                const uint32_t d = tmem + uint32_t(buf * kN);
                for (int f = 0; f < n_slices; ++f, ++n) {
                    const int s = n % kStages;
                    if (!mbar_wait(&full[s], (n / kStages) & 1, abort_flag, g.wait_ns)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint64_t bh = db + uint64_t(s) * (2 * lo_half), bl = bh + lo_half;
                    const uint32_t ah = tmem + kAcol + uint32_t(f * kSliceK), al = ah + uint32_t(Kp);
                    const int steps = min(kSliceK, Kp - f * kSliceK) / T::kStepK;
#pragma unroll
                    for (int kk = 0; kk < kSliceK / T::kStepK; ++kk) {
                        if (kk >= steps) break;
                        // data hi / lo of a K step: T::kStepK tensor-memory columns each
                        umma_ts<MODE>(d, ah + kk * T::kStepK, bh + kk * kStep, idesc, (f > 0 || kk > 0) ? 1u : 0u);
                        umma_ts<MODE>(d, ah + kk * T::kStepK, bl + kk * kStep, idesc, 1u);
                        umma_ts<MODE>(d, al + kk * T::kStepK, bh + kk * kStep, idesc, 1u);
                    }
                    umma_commit(&empty[s]);
                }
                if (ok) umma_commit(&tfull[buf]);
            }
        }
        if (lane == 0) {
            // every MMA of this CTA has completed before tensor memory is released
            umma_commit(done);
            mbar_drain(done, 0);
        }
    } else {
        // ---------------- epilogue ----------------
        const int q = warp & 3, h = warp >> 2;
        const uint32_t tlane = tmem + (uint32_t(q * 32) << 16);
        {
            // this warp's 32 rows into its tensor-memory lanes: the hi half (h = 0, with the norms) or the lo half
            const int r = q * 32 + lane, row = tile * kTileM + r;
            const float* const x = g.rows + size_t(row) * g.Dp;
            float xn = 0.f;
            for (int k = 0; k < Kp; k += 8) {
                float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                if (row < g.n_samples) {
#pragma unroll
                    for (int j = 0; j < 8; j += 4)
                        if (k + j < g.Dp) {
                            const float4 t = __ldg(reinterpret_cast<const float4*>(x + k + j));
                            v[j] = t.x;
                            v[j + 1] = t.y;
                            v[j + 2] = t.z;
                            v[j + 3] = t.w;
                        }
                }
                uint32_t w[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    float hi, lo;
                    split_operand<MODE>(v[j], &hi, &lo);
                    w[j] = __float_as_uint(h ? lo : hi);
                    xn = fmaf(v[j], v[j], xn);
                }
                tmem_st8(tlane + kAcol + uint32_t(h * Kp + k), w);
            }
            if (h == 0) sxn[r] = xn;
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(afull);
            asm volatile("bar.sync 1, %0;" ::"r"(kEpiWarps * 32) : "memory");
        }
        const int r0 = q * 32 + (lane >> 2), cp = 2 * (lane & 3); // rows r0 + 8 m, columns cp, cp + 1 of each eight
        f32x2 xn[4];
#pragma unroll
        for (int m = 0; m < 4; ++m) xn[m] = pack2(sxn[r0 + 8 * m], sxn[r0 + 8 * m]);
        constexpr int NP = NU / 2 + (NU == 1); // packed users
        f32x2 acc[4][NP];
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
            for (int u = 0; u < NP; ++u) acc[m][u] = 0ull;
        const f32x2 minus2 = pack2(-2.f, -2.f);
        for (int i = 0; i < nch; ++i) {
            const int s = i % kXStages, buf = i & 1;
            const bool ready = mbar_wait(&xfull[s], (i / kXStages) & 1, abort_flag, g.wait_ns) &&
                               mbar_wait(&tfull[buf], (i >> 1) & 1, abort_flag, g.wait_ns);
            if (!__all_sync(0xffffffffu, ready)) break; // (the loads below are warp-wide)
            tc_fence_after();
            const float* const dn = sX + size_t(s) * X::kFloats + cp;
            const float* const aw = sX + size_t(s) * X::kFloats + kN + cp * X::kPitch;
#pragma unroll 1
            for (int cb = 0; cb < kN / 2; cb += 32) {
                const int col = h * (kN / 2) + cb;
                uint32_t v[2][16];
                tmem_ld_16x32(tlane + uint32_t(buf * kN + col), v[0]);
                tmem_ld_16x32(tlane + (16u << 16) + uint32_t(buf * kN + col), v[1]);
                tmem_ld_wait(v[0], v[1]);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int c8 = col + 8 * e;
                    const f32x2 dn2 = *reinterpret_cast<const f32x2*>(dn + c8);
                    float2 kv[4]; // (column cp, column cp + 1) of rows r0 + 8 m
#pragma unroll
                    for (int m = 0; m < 4; ++m) {
                        const uint32_t* const p = v[m >> 1] + 4 * e + 2 * (m & 1);
                        const float2 d2 = unpack2(fma2(minus2, pack2(__uint_as_float(p[0]), __uint_as_float(p[1])),
                                                       add2(xn[m], dn2)));
                        kv[m].x = ex2(g.ewl2 * fmaxf(d2.x, 0.f));
                        kv[m].y = ex2(g.ewl2 * fmaxf(d2.y, 0.f));
                    }
                    const float* const a = aw + c8 * X::kPitch;
                    if constexpr (NU == 1) {
                        const f32x2 a2 = *reinterpret_cast<const f32x2*>(a);
#pragma unroll
                        for (int m = 0; m < 4; ++m) acc[m][0] = fma2(a2, pack2(kv[m].x, kv[m].y), acc[m][0]);
                    } else {
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            f32x2 k2[4];
#pragma unroll
                            for (int m = 0; m < 4; ++m) {
                                const float t = j ? kv[m].y : kv[m].x;
                                k2[m] = pack2(t, t);
                            }
                            if constexpr (NU == 2) {
                                const f32x2 a2 = *reinterpret_cast<const f32x2*>(a + j * X::kPitch);
#pragma unroll
                                for (int m = 0; m < 4; ++m) acc[m][0] = fma2(a2, k2[m], acc[m][0]);
                            } else {
#pragma unroll
                                for (int u = 0; u < NP; u += 2) {
                                    const ulonglong2 a4 =
                                        *reinterpret_cast<const ulonglong2*>(a + j * X::kPitch + 2 * u);
#pragma unroll
                                    for (int m = 0; m < 4; ++m) acc[m][u] = fma2(a4.x, k2[m], acc[m][u]);
#pragma unroll
                                    for (int m = 0; m < 4; ++m) acc[m][u + 1] = fma2(a4.y, k2[m], acc[m][u + 1]);
                                }
                            }
                        }
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&tempty[buf]);
                mbar_arrive(&xempty[s]);
            }
        }
        // a row's sums: four lanes (columns modulo 8), two warps (column halves)
        float sum[4][NU];
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
            for (int u = 0; u < NP; ++u) {
                const float2 t = unpack2(acc[m][u]);
                if constexpr (NU == 1) {
                    sum[m][0] = t.x + t.y;
                } else {
                    sum[m][2 * u] = t.x;
                    sum[m][2 * u + 1] = t.y;
                }
            }
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
            for (int u = 0; u < NU; ++u) {
                sum[m][u] += __shfl_xor_sync(0xffffffffu, sum[m][u], 1);
                sum[m][u] += __shfl_xor_sync(0xffffffffu, sum[m][u], 2);
            }
        if (h == 1) {
#pragma unroll
            for (int m = 0; m < 4; ++m)
#pragma unroll
                for (int u = 0; u < NU; ++u)
                    if ((u & 3) == (lane & 3)) red[(r0 + 8 * m) * NU + u] = sum[m][u];
        }
        asm volatile("bar.sync 1, %0;" ::"r"(kEpiWarps * 32) : "memory");
        if (h == 0) {
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const int row = tile * kTileM + r0 + 8 * m;
#pragma unroll
                for (int u = 0; u < NU; ++u)
                    if ((u & 3) == (lane & 3) && u < g.users && row < g.n_samples)
                        g.part[(size_t(split) * g.users + u) * g.n_samples + row] = sum[m][u] + red[(r0 + 8 * m) * NU + u];
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == kEpiWarps + 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols));
    }
    if (threadIdx.x == 0 && *abort_flag) atomicExch(g.err, 1);
}

template <int NU> cudaError_t launch(const GramTmemArgs& g, int n_tiles, int splits, cudaStream_t s)
{
    const size_t need = size_t(kStages) * 2 * kN * std::min(kSliceK, g.Kp) * 4 +
                        sizeof(float) * (kXStages * ChunkData<NU>::kFloats + kTileM * (NU + 1)) +
                        sizeof(uint64_t) * (2 * kStages + 2 * kXStages + 6) + 16;
    // more than half of an SM's shared memory: one CTA per SM holds all its tensor memory
    const size_t smem = std::max<size_t>(need, 120 * 1024);
    const cudaError_t e = allow_smem(gram_tmem_kernel<NU>);
    if (e != cudaSuccess) return e;
    gram_tmem_kernel<NU><<<dim3(n_tiles, splits), kThreads, smem, s>>>(g);
    return cudaGetLastError();
}

} // namespace

size_t gram_tmem_data_floats(int users) { return size_t(kN) * (1 + coef_pitch(user_class(users))); }

cudaError_t launch_gram_tmem(const GramTmemArgs& g, const float* dn, const float* a, size_t a_stride, int M, float wG,
                             float* xd, int n_tiles, int splits, cudaStream_t s)
{
    const int nu = user_class(g.users), pitch = coef_pitch(nu);
    chunk_data_kernel<<<std::min(1184, (g.n_chunks * kN * pitch + 255) / 256), 256, 0, s>>>(dn, a, a_stride, g.users, M,
                                                                                          g.n_chunks, pitch, wG, xd);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    switch (nu) {
    case 1: return launch<1>(g, n_tiles, splits, s);
    case 2: return launch<2>(g, n_tiles, splits, s);
    case 4: return launch<4>(g, n_tiles, splits, s);
    case 8: return launch<8>(g, n_tiles, splits, s);
    default: return launch<16>(g, n_tiles, splits, s);
    }
}

} // namespace apsm
