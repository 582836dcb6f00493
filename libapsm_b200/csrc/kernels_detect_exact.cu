// Exact FP32 APSM detection (the "plain" form): the model
//   f(x_s) = wL <w, x_s> + sum_b (a_b wG) exp(ew ||d_b - x_s||^2)
// evaluated in the reference BALANCED kernel's order
// (cpp/lib/apsm/apsm_detect.cu:526-538 linear part, :690-808 Gaussian part,
// :810-876 reduction): lane l of the warp that owns sample s accumulates
// first the linear terms idx = l, l+32, ... and then the Gaussian terms of
// dictionary rows b = l, l+32, ... in ascending order; squared distances are
// sequential fma chains over the features; the 32 partials are combined with
// the shuffle-down tree.  Given the same coefficients the soft outputs are
// bit-identical to the reference's.
//
// Bound: FP32 arithmetic, one subtraction and one fma per feature and pair
// (sample, row), a product and a sum per user.  131072 samples x 16384 rows of
// 128 features, 16 users: 17.5 ms at the 126 lanes per clock measured for
// either instruction.  Taken: 20.4 ms (30.0 ms with two rows x four samples
// per lane and scalar arithmetic, which asked shared memory for 6 floats per
// 8 pairs and feature and filled every issue slot).
//
// Layout: each lane works on four rows (lane + 32 r of a tile of 128) for the
// eight samples of its warp, the samples packed by twos (the packed
// instructions round each half like the scalar ones).  Per feature a lane
// takes 4 + 8 floats from shared memory for 32 pairs; the samples are stored
// negated, so the difference is a packed sum.  More rows and fewer samples a
// lane (8 x 4, 12 warps) took 1.82 against 1.55 ms (37888 samples x 4096 rows
// of 128 features); 16 users' sums of eight samples take 128 registers, so one
// block of eight warps fills an SM.  Dictionary tiles arrive by asynchronous copies in chunks of FC
// features, two or three in flight.  The Gaussian value of a pair is computed
// once for all users of the cell (up to 16 per pass).
#include "apsm_kernels.cuh"
#include "packed_f32.cuh"

namespace apsm {

namespace {

// 16 or 4 bytes to shared memory; zeros where `live` is false (the source is not read then)
__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src, bool live)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst))),
                 "l"(gmem_src), "r"(live ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async4(void* smem_dst, const void* gmem_src, bool live)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst))),
                 "l"(gmem_src), "r"(live ? 4 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

constexpr int kRows = 128; // dictionary rows per tile: four per lane
constexpr int kRowsPerLane = kRows / 32;
constexpr int kSpw = 8;    // samples per warp
constexpr int kH = kSpw / 2;

// FC features per chunk, W warps per block, KU users per pass.
template <int FC, int W, int KU> struct Shape {
    static constexpr int kStages = FC > 32 ? 2 : 3; // chunks in flight
    static constexpr int kPitch = FC + 4; // floats per tile row: the float4s of eight neighbouring rows cover the banks
    static constexpr int kSamples = W * kSpw;
    static constexpr size_t smem(int Dp)
    {
        return sizeof(float) * (size_t(kStages) * kRows * kPitch + size_t(kStages) * KU * kRows + size_t(kSamples) * Dp);
    }
};

// One level of the warp's reduction of n values per lane: lanes with bit `off` keep the upper half of the
// values, the others the lower half, each adding its partner's.
template <int N> __device__ __forceinline__ void reduce_values(float (&v)[N], int lane)
{
    int n = N;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        if (n > 1) {
            const bool up = lane & off;
#pragma unroll
            for (int j = 0; j < N / 2; ++j)
                if (j < n / 2) {
                    const float keep = up ? v[j + n / 2] : v[j], give = up ? v[j] : v[j + n / 2];
                    v[j] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, give, off));
                }
            n >>= 1;
        } else {
            v[0] = __fadd_rn(v[0], __shfl_xor_sync(0xffffffffu, v[0], off));
        }
    }
}

template <int FC, int W, int KU>
__global__ void __launch_bounds__(W * 32, 8 / W) detect_exact_kernel(DetectArgs args)
{
    using S = Shape<FC, W, KU>;
    constexpr int P = S::kPitch, kStages = S::kStages, SPW = kSpw, H = kH;
    const int D = args.D, Dp = args.Dp, M = args.M;
    const ModelParams mp = args.mp;

    extern __shared__ __align__(16) float sm[];
    float* const tiles = sm;                              // [kStages][kRows][P]
    float* const coef = tiles + kStages * kRows * P;      // [kStages][KU][kRows]
    float* const xs = coef + kStages * KU * kRows;        // [kSamples / 2][Dp] pairs (-x_2i, -x_2i+1)

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int sb = blockIdx.x * S::kSamples;

    // the block's samples, negated and interleaved by twos; samples past the end are zero
    for (int idx = tid; idx < (S::kSamples / 2) * (Dp / 4); idx += W * 32) {
        const int i = idx / (Dp / 4), c = 4 * (idx - i * (Dp / 4));
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
        const int s = sb + 2 * i;
        const float4 u = s < args.n_samples ? __ldg(reinterpret_cast<const float4*>(args.Xs + size_t(s) * Dp + c)) : z;
        const float4 v =
            s + 1 < args.n_samples ? __ldg(reinterpret_cast<const float4*>(args.Xs + size_t(s + 1) * Dp + c)) : z;
        float4* dst = reinterpret_cast<float4*>(xs + 2 * (size_t(i) * Dp + c));
        dst[0] = make_float4(-u.x, -v.x, -u.y, -v.y);
        dst[1] = make_float4(-u.z, -v.z, -u.w, -v.w);
    }

    const int n_tiles = (M + kRows - 1) / kRows;
    const int nf = (Dp + FC - 1) / FC; // chunks of a tile
    const int n_chunks = n_tiles * nf;
    const float* const xw = xs + size_t(warp) * SPW * Dp;
    for (int uc = 0; uc < args.users; uc += KU) {
        const int nu = min(KU, args.users - uc);
        // chunk g = (tile, features) into stage g % kStages; with a tile's first chunk come its coefficients
        int st_t = 0, st_f = 0, st_slot = 0, co_slot = 0;
        auto stage = [&] {
            if (st_t < n_tiles) {
                const int b0 = st_t * kRows;
                float* const tb = tiles + st_slot * kRows * P;
#pragma unroll
                for (int idx = tid; idx < kRows * (FC / 4); idx += W * 32) {
                    const int r = idx / (FC / 4), c = 4 * (idx % (FC / 4));
                    const bool live = b0 + r < M && st_f * FC + c < Dp;
                    cp_async16(tb + r * P + c, args.dict + (live ? size_t(b0 + r) * Dp + st_f * FC + c : 0), live);
                }
                if (st_f == 0) {
                    float* const cb = coef + co_slot * KU * kRows;
                    for (int idx = tid; idx < KU * kRows; idx += W * 32) {
                        const int u = idx / kRows, b = b0 + idx % kRows;
                        const bool live = u < nu && b < M;
                        cp_async4(cb + idx, args.a + (live ? size_t(uc + u) * args.a_stride + b : 0), live);
                    }
                    co_slot = co_slot + 1 == kStages ? 0 : co_slot + 1;
                }
            }
            cp_async_commit(); // (an empty group past the end keeps the count)
            if (++st_f == nf) {
                st_f = 0;
                ++st_t;
            }
            st_slot = st_slot + 1 == kStages ? 0 : st_slot + 1;
        };
        __syncthreads(); // samples in place; an earlier pass has read its last chunk
#pragma unroll
        for (int g = 0; g + 1 < kStages; ++g) stage();

        // linear part first (kernel_apsm_detection_linear_shmem)
        f32x2 p[H][KU];
#pragma unroll
        for (int h = 0; h < H; ++h)
#pragma unroll
            for (int u = 0; u < KU; ++u) p[h][u] = 0ull;
        for (int idx = lane; idx < D; idx += 32) {
#pragma unroll
            for (int u = 0; u < KU; ++u)
                if (u < nu) {
                    const float wv = __ldg(args.w + size_t(uc + u) * D + idx);
                    const f32x2 w2 = pack2(wv, wv);
#pragma unroll
                    for (int h = 0; h < H; ++h) {
                        const float2 x = *reinterpret_cast<const float2*>(xw + 2 * (h * Dp + idx));
                        p[h][u] = add2(p[h][u], mul2(w2, pack2(__fmul_rn(mp.wL, -x.x), __fmul_rn(mp.wL, -x.y))));
                    }
                }
        }

        int slot = 0, cslot = 0;
        for (int t = 0; t < n_tiles; ++t) {
            f32x2 acc[kRowsPerLane][H];
#pragma unroll
            for (int r = 0; r < kRowsPerLane; ++r)
#pragma unroll
                for (int h = 0; h < H; ++h) acc[r][h] = 0ull;
            for (int f = 0; f < nf; ++f) {
                cp_async_wait<kStages - 2>();
                __syncthreads(); // this chunk is complete, the previous one's stage is free
                stage();
                const float* const d = tiles + (slot * kRows + lane) * P;
                const float* const x = xw + 2 * f * FC;
                const int fc = min(FC, Dp - f * FC);
                // four features: per feature all 16 packed differences, then the 16 independent sums
                auto four = [&](int c) {
                    ulonglong2 xv[2][H];
#pragma unroll
                    for (int k = 0; k < 2; ++k)
#pragma unroll
                        for (int h = 0; h < H; ++h)
                            xv[k][h] = *reinterpret_cast<const ulonglong2*>(x + 2 * (h * Dp + c + 2 * k));
                    float4 v[kRowsPerLane];
#pragma unroll
                    for (int r = 0; r < kRowsPerLane; ++r) v[r] = *reinterpret_cast<const float4*>(d + r * 32 * P + c);
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        f32x2 e[kRowsPerLane][H];
#pragma unroll
                        for (int r = 0; r < kRowsPerLane; ++r) {
                            const float q = k == 0 ? v[r].x : k == 1 ? v[r].y : k == 2 ? v[r].z : v[r].w;
                            const f32x2 q2 = pack2(q, q);
#pragma unroll
                            for (int h = 0; h < H; ++h)
                                e[r][h] = add2(q2, (k & 1) ? xv[k / 2][h].y : xv[k / 2][h].x);
                        }
#pragma unroll
                        for (int r = 0; r < kRowsPerLane; ++r)
#pragma unroll
                            for (int h = 0; h < H; ++h) acc[r][h] = fma2(e[r][h], e[r][h], acc[r][h]);
                    }
                };
                if (fc == FC) {
#pragma unroll 8
                    for (int c = 0; c < FC; c += 4) four(c);
                } else {
#pragma unroll 1
                    for (int c = 0; c < fc; c += 4) four(c);
                }
                slot = slot + 1 == kStages ? 0 : slot + 1;
            }
            // the lane's rows b = lane + 32 r of the tile in ascending order; users past the last have zero
            // coefficients (a test per user costs more than the work it saves: 1.89 with it, 1.58 ms without, 16 users,
            // 37888 samples x 4096 rows of 128 features)
            const float* const cb = coef + cslot * KU * kRows + lane;
            auto users_row = [&](int r) {
                f32x2 kv[H];
#pragma unroll
                for (int h = 0; h < H; ++h) {
                    const float2 q = unpack2(acc[r][h]);
                    kv[h] = pack2(expf(__fmul_rn(mp.ew, q.x)), expf(__fmul_rn(mp.ew, q.y)));
                }
#pragma unroll
                for (int u = 0; u < KU; ++u) {
                    const float a = __fmul_rn(cb[u * kRows + 32 * r], mp.wG); // apsm_detect.cu:802
                    const f32x2 a2 = pack2(a, a);
#pragma unroll
                    for (int h = 0; h < H; ++h) p[h][u] = add2(p[h][u], mul2(a2, kv[h]));
                }
            };
            const int rows = M - t * kRows;
            if (rows >= kRows) {
#pragma unroll
                for (int r = 0; r < kRowsPerLane; ++r) users_row(r);
            } else {
#pragma unroll
                for (int r = 0; r < kRowsPerLane; ++r)
                    if (lane + 32 * r < rows) users_row(r);
            }
            cslot = cslot + 1 == kStages ? 0 : cslot + 1;
        }
        // The warp's tree (apsm_detect.cu:830-833): the levels add the same two partials as a shuffle-down tree,
        // but every level also halves the values a lane still carries, so 32 values take 31 shuffles, not 160.
        constexpr int V = SPW * KU, B = V < 32 ? V : 32; // values of a warp, values per reduction
#pragma unroll
        for (int v0 = 0; v0 < V; v0 += B) {
            float v[B];
#pragma unroll
            for (int j = 0; j < B; j += 2) { // value v0 + j: user (v0 + j) / SPW, sample (v0 + j) % SPW
                const float2 q = unpack2(p[((v0 + j) % SPW) / 2][(v0 + j) / SPW]);
                v[j] = q.x;
                v[j + 1] = q.y;
            }
            reduce_values(v, lane);
            // the lane's value: its top log2(B) bits, from the first level down
            const int j = v0 + lane / (32 / B);
            const int u = j / SPW, si = sb + warp * SPW + j % SPW;
            if (lane % (32 / B) == 0 && u < nu && si < args.n_samples)
                args.out[size_t(uc + u) * args.out_stride + si] = v[0];
        }
    }
}

template <int FC, int W, int KU> cudaError_t launch_shape(const DetectArgs& args, cudaStream_t stream)
{
    using S = Shape<FC, W, KU>;
    const size_t smem = S::smem(args.Dp);
    if (const cudaError_t e = allow_smem(detect_exact_kernel<FC, W, KU>); e != cudaSuccess)
        return e; // the error stays for the caller's cudaGetLastError
    const int grid = (args.n_samples + S::kSamples - 1) / S::kSamples;
    detect_exact_kernel<FC, W, KU><<<grid, W * 32, smem, stream>>>(args);
    return cudaSuccess;
}

template <int FC, int W> void launch_users(const DetectArgs& args, cudaStream_t stream)
{
    if (args.users == 1) launch_shape<FC, W, 1>(args, stream);
    else if (args.users <= 4) launch_shape<FC, W, 4>(args, stream);
    else if (args.users <= 8) launch_shape<FC, W, 8>(args, stream);
    else launch_shape<FC, W, 16>(args, stream);
}

// Blocks of eight warps share a dictionary tile among 64 samples; where they would leave half of the SMs
// without one, blocks of four warps spread the samples over twice as many SMs.  Measured (kernel alone):
// 3600 samples x 1200 rows of 16 features, 57 or 113 blocks: 19 against 17 us; 7680 samples x 1370 rows of
// 32 features, 120 or 240 blocks: 47 against 50 us.
template <int FC> void launch_features(const DetectArgs& args, cudaStream_t stream)
{
    constexpr int kHalfOfSms = 148 / 2;
    if ((args.n_samples + 8 * kSpw - 1) / (8 * kSpw) > kHalfOfSms) launch_users<FC, 8>(args, stream);
    else launch_users<FC, 4>(args, stream);
}

} // namespace

void launch_detect_exact(const DetectArgs& args, cudaStream_t stream)
{
    if (args.n_samples <= 0) return;
    if (args.D <= 8) launch_features<8>(args, stream);
    else if (args.D <= 16) launch_features<16>(args, stream);
    else if (args.D <= 32) launch_features<32>(args, stream);
    else launch_features<64>(args, stream);
}

} // namespace apsm
