// Batched FP32 detection in pair form, all detection jobs of a class of
// antenna counts in one launch.
//
// For data sample s (rows 2s, 2s+1) the reference evaluates
// (cpp/lib/apsm/apsm_detect.cu:526-538 linear, :690-808 Gaussian)
//   f_{2s}   = wL <w, x_2s>   + sum_b a_{2b} K(2b, 2s)   + a_{2b+1} K(2b+1, 2s)
//   f_{2s+1} = wL <w, x_2s+1> + sum_b a_{2b} K(2b, 2s+1) + a_{2b+1} K(2b+1, 2s+1)
// Here each (sample, dictionary pair) costs one complex inner product
// y_b^H y_s (4N fma) and three exponentials instead of four distance loops
// and four exponentials.  Summation order differs from the reference; the
// FP32 bar is 1e-4 relative.
//
// Order of the Gaussian sum: the dictionary is cut into chunks of kChunk
// pairs; in a chunk lane l adds its pairs l, l + 32, ... from zero, the lanes
// are added by a tree, and the chunk sums are added in chunk order.  A launch
// may give one tile of samples to several blocks (grid.z "parts", for batches
// too small to fill the GPU, i.e. single requests): each block then stores its
// chunk sums ([chunk][sample], coalesced) and the tile's last block to arrive
// adds them in chunk order -- the same additions as one block doing every
// chunk, so the estimates do not depend on how a batch was split.
//
// Bound: FP32 arithmetic (4N + 8 fma per sample and pair) and the special
// function unit (3 exponentials).  16 jobs of 8064 samples x 1100 pairs: 95 and
// 94 us at 4 antennas, 539 and 94 us at 32.  Taken, before (one sample per thread against broadcast
// dictionary entries, scalar arithmetic) and in this form: 254 -> 207, 388 -> 287,
// 638 -> 450, 1119 -> 799 us at 4, 8, 16, 32 antennas.  Keeping kernel values below
// 2^-126 where they matter (low_estimates) moves these by +2, +10, +1, -3 us
// (choosing the exponential for every warp and chunk cost +9, +13, +13, +17).
//
// Layout: a lane works on four pairs (lane + 32 r of a tile of 128) for the
// eight samples of its warp, packed by twos, so 8 + 16 floats of shared memory
// per antenna serve 32 complex products.  The packed fma with three distinct
// operand pairs is short of register ports: the order of the main loop keeps
// the samples' operand for eight instructions (with the operands changing
// every instruction 32 antennas took 850 us; scalar arithmetic 960 us).  Three
// blocks of four warps per SM drift apart, so that one's exponentials run
// beside another's products (one block of eight: 916 us).
#include "apsm_batch.cuh"
#include "packed_f32.cuh"

namespace apsm {

namespace {

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src, bool live)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(smem_dst))),
                 "l"(gmem_src), "r"(live ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Base-2 exponential on the special function unit; results below 2^-126 are zero, or (SMALL) kept as FP32
// holds them, which takes three more instructions.
template <bool SMALL> __device__ __forceinline__ float ex2(float x)
{
    float y;
    if constexpr (SMALL) asm("ex2.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    else asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

constexpr float kLog2e = 1.4426950408889634f;
constexpr int kWarps = 4;
constexpr int kThreads = kWarps * 32;
constexpr int kSpw = 8;               // samples per warp
constexpr int kH = kSpw / 2;          // packed by twos
constexpr int kTile = kWarps * kSpw;  // samples per block
constexpr int kChunk = 128;           // dictionary pairs per chunk (= one shared-memory tile)
constexpr int kR = kChunk / 32;       // pairs per lane
constexpr int kStages = 2;

// KC antennas of a tile per copy
template <int KC> struct Shape {
    static constexpr int kPitch = 2 * KC + 4; // floats per tile row: the float4s of eight neighbouring rows cover the banks
    static constexpr size_t smem(int N)
    {
        return sizeof(float) * (size_t(kStages) * kChunk * kPitch + size_t(2) * kTile * ((N + 1) & ~1) + kTile);
    }
};

// The main loop drops kernel values below 2^-126: less than half a rounding of an estimate of kLow or more (n pairs
// with |a| wG up to 2^36 / n).  A smaller estimate is formed again with every value FP32 holds; models without a linear
// part have such estimates far from their dictionary, others hardly but for samples of zero.
constexpr float kLow = 0x1p-64f;

// Component (lane / 2) % 2 of <w, y_s> for the warp's sample lane / 4 (xw: its samples; sample i, antenna k at
// 4 ((i / 2) Np + k) + i % 2 and two further)
__device__ __forceinline__ float linear_part(const BatchDetectJob& jb, const float* xw, int Np, int lane)
{
    const float* const x = xw + 4 * (lane >> 3) * Np + (lane >> 2 & 1);
    const int N = jb.N;
    float l = 0.f;
    if (lane & 2)
        for (int k = 0; k < N; ++k) l = fmaf(__ldg(jb.w + k), x[4 * k + 2], fmaf(-__ldg(jb.w + N + k), x[4 * k], l));
    else
        for (int k = 0; k < N; ++k) l = fmaf(__ldg(jb.w + k), x[4 * k], fmaf(__ldg(jb.w + N + k), x[4 * k + 2], l));
    return l;
}

// The estimates of the warp's samples with a lane in the mask; sums in the order of the main loop.  Out of line, so
// that it takes no registers from there.
__device__ __noinline__ void low_estimates(const BatchDetectJob& jb, const float* xs, const float* nrm, float wL,
                                           float wG, int s0, uint32_t mask)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, N = jb.N, Np = jb.Np, Mp = jb.Mp;
    const float ew2 = jb.ew * kLog2e;
    const float* const xw = xs + 2 * size_t(warp) * kSpw * Np;
    float g = 0.f; // lanes 4 i + 2 c: component c of sample i
    for (int c0 = 0; c0 < Mp; c0 += kChunk) {
        float f[kSpw][2];
#pragma unroll
        for (int i = 0; i < kSpw; ++i) f[i][0] = f[i][1] = 0.f;
#pragma unroll 1
        for (int b = c0 + lane; b < min(Mp, c0 + kChunk); b += 32) {
            const float2* const y = jb.Yd + size_t(b) * Np;
            float re[kSpw], im[kSpw];
#pragma unroll
            for (int i = 0; i < kSpw; ++i) re[i] = im[i] = 0.f;
#pragma unroll 1
            for (int k = 0; k < N; ++k) {
                const float2 d = __ldg(y + k);
#pragma unroll
                for (int i = 0; i < kSpw; ++i) {
                    const float* const x = xw + 4 * ((i >> 1) * Np + k) + (i & 1);
                    re[i] = fmaf(d.x, x[0], fmaf(d.y, x[2], re[i]));
                    im[i] = fmaf(-d.y, x[0], fmaf(d.x, x[2], im[i]));
                }
            }
            const float a0 = __ldg(jb.a + 2 * b) * wG, a1 = __ldg(jb.a + 2 * b + 1) * wG, nb = __ldg(jb.nrm_d + b);
#pragma unroll
            for (int i = 0; i < kSpw; ++i) {
                const float q = fmaf(ew2, nb, ew2 * nrm[warp * kSpw + i]);
                const float kA = ex2<true>(fminf(fmaf(-2.f * ew2, re[i], q), 0.f));
                const float kP = ex2<true>(fminf(fmaf(-2.f * ew2, im[i], q), 0.f));
                const float kM = ex2<true>(fminf(fmaf(2.f * ew2, im[i], q), 0.f));
                f[i][0] = fmaf(a0, kA, fmaf(a1, kM, f[i][0]));
                f[i][1] = fmaf(a0, kP, fmaf(a1, kA, f[i][1]));
            }
        }
#pragma unroll
        for (int i = 0; i < kSpw; ++i)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                float v = f[i][c];
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
                if (lane == 4 * i + 2 * c) g += v;
            }
    }
    const int s = s0 + warp * kSpw + lane / 4;
    if (!(lane & 1) && (mask >> (lane & ~3) & 15u))
        reinterpret_cast<float*>(jb.out + s)[(lane >> 1) & 1] = fmaf(wL, linear_part(jb, xw, Np, lane), g);
}

template <int KC>
__global__ void __launch_bounds__(kThreads, 3) batch_detect_kernel(const BatchDetectJob* __restrict__ jobs, int nmax,
                                                                float wL, float wG)
{
    constexpr int P = Shape<KC>::kPitch;
    const BatchDetectJob& jb = jobs[blockIdx.y];
    const int s0 = blockIdx.x * kTile;
    const int S = jb.S;
    if (s0 >= S || jb.N > nmax) return;
    const int N = jb.N, Np = jb.Np, Mp = jb.Mp;
    const int n_chunks = (Mp + kChunk - 1) / kChunk;
    // this block's chunks: runs of cpb chunks, parts_j runs for this job
    const int cpb = n_chunks > 0 ? (n_chunks + int(gridDim.z) - 1) / int(gridDim.z) : 1;
    const int parts_j = n_chunks > 0 ? (n_chunks + cpb - 1) / cpb : 1;
    const int part = blockIdx.z;
    if (part >= parts_j) return;
    const bool split = parts_j > 1;
    const int c_begin = part * cpb, c_end = min(n_chunks, c_begin + cpb);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float ew2 = jb.ew * kLog2e;

    extern __shared__ __align__(16) float sm[];
    float* const tiles = sm;                           // [kStages][kChunk][P]
    float* const xs = tiles + kStages * kChunk * P;    // [kTile / 2][Np] of (re_2i, re_2i+1, im_2i, im_2i+1)
    float* const nrm = xs + 2 * kTile * Np;            // [kTile]
    __shared__ int s_last;

    const int nf = (Np + KC - 1) / KC; // copies of a tile
    int st_c = c_begin, st_f = 0, st_slot = 0;
    auto stage = [&] {
        if (st_c < c_end) {
            const int b0 = st_c * kChunk;
            float* const tb = tiles + st_slot * kChunk * P;
#pragma unroll
            for (int idx = tid; idx < kChunk * (KC / 2); idx += kThreads) {
                const int r = idx / (KC / 2), k = 2 * (idx % (KC / 2));
                const bool live = b0 + r < Mp && st_f * KC + k < Np;
                cp_async16(tb + r * P + 2 * k, jb.Yd + (live ? size_t(b0 + r) * Np + st_f * KC + k : 0), live);
            }
        }
        cp_async_commit(); // (an empty group past the end keeps the count)
        if (++st_f == nf) {
            st_f = 0;
            ++st_c;
        }
        st_slot = st_slot + 1 == kStages ? 0 : st_slot + 1;
    };
#pragma unroll
    for (int g = 0; g + 1 < kStages; ++g) stage();

    // the tile's samples straight from the antenna-major input (coalesced per antenna), packed by twos
    for (int idx = tid; idx < kTile * Np; idx += kThreads) {
        const int k = idx / kTile, i = idx % kTile;
        const float2 v = (k < N && s0 + i < S) ? __ldg(jb.rx + size_t(k) * S + s0 + i) : make_float2(0.f, 0.f);
        float* const dst = xs + 4 * (size_t(i >> 1) * Np + k) + (i & 1);
        dst[0] = v.x;
        dst[2] = v.y;
    }
    __syncthreads();
    if (tid < kTile) { // squared norms, real parts first (the order of the training rows' norms)
        const float* const v = xs + 4 * size_t(tid >> 1) * Np + (tid & 1);
        float ns = 0.f;
        for (int k = 0; k < N; ++k) ns = fmaf(v[4 * k], v[4 * k], ns);
        for (int k = 0; k < N; ++k) ns = fmaf(v[4 * k + 2], v[4 * k + 2], ns);
        nrm[tid] = ns;
    }
    __syncthreads();
    f32x2 ens[kH]; // ew2 ||y_s||^2
#pragma unroll
    for (int h = 0; h < kH; ++h)
        ens[h] = mul2(pack2(ew2, ew2), *reinterpret_cast<const f32x2*>(nrm + warp * kSpw + 2 * h));

    const float* const xw = xs + size_t(warp) * 2 * kSpw * Np;
    const f32x2 ew2_2 = pack2(ew2, ew2), pos = pack2(2.f * ew2, 2.f * ew2), neg = pack2(-2.f * ew2, -2.f * ew2);
    int slot = 0;
    float t = 0.f; // running sum of the chunk sums of the lane's (sample, component) (unsplit launches)
    for (int c = c_begin; c < c_end; ++c) {
        f32x2 re[kR][kH], im[kR][kH];
#pragma unroll
        for (int r = 0; r < kR; ++r)
#pragma unroll
            for (int h = 0; h < kH; ++h) re[r][h] = im[r][h] = 0ull;
        float2 ab[kR];
        float nb[kR];
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            const int b = c * kChunk + 32 * r + lane;
            ab[r] = b < Mp ? __ldg(reinterpret_cast<const float2*>(jb.a) + b) : make_float2(0.f, 0.f);
            nb[r] = b < Mp ? __ldg(jb.nrm_d + b) : 0.f;
        }
        for (int f = 0; f < nf; ++f) {
            cp_async_wait<kStages - 2>();
            __syncthreads(); // this copy is complete, the previous one's stage is free
            stage();
            const float* const d = tiles + (slot * kChunk + lane) * P;
            const float* const x = xw + 4 * f * KC;
            auto two = [&](int k) { // two antennas
                float4 v[kR];
#pragma unroll
                for (int r = 0; r < kR; ++r) v[r] = *reinterpret_cast<const float4*>(d + r * 32 * P + 2 * k);
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    ulonglong2 xv[kH]; // (real parts, imaginary parts) of two samples
#pragma unroll
                    for (int h = 0; h < kH; ++h) xv[h] = *reinterpret_cast<const ulonglong2*>(x + 4 * (h * Np + k + q));
                    f32x2 bx[kR], by[kR], bm[kR];
#pragma unroll
                    for (int r = 0; r < kR; ++r) {
                        const float vx = q ? v[r].z : v[r].x, vy = q ? v[r].w : v[r].y;
                        bx[r] = pack2(vx, vx);
                        by[r] = pack2(vy, vy);
                        bm[r] = pack2(-vy, -vy);
                    }
#pragma unroll
                    for (int h = 0; h < kH; ++h) {
#pragma unroll
                        for (int r = 0; r < kR; ++r) {
                            re[r][h] = fma2(by[r], xv[h].y, re[r][h]);
                            im[r][h] = fma2(bx[r], xv[h].y, im[r][h]);
                        }
#pragma unroll
                        for (int r = 0; r < kR; ++r) {
                            re[r][h] = fma2(bx[r], xv[h].x, re[r][h]);
                            im[r][h] = fma2(bm[r], xv[h].x, im[r][h]);
                        }
                    }
                }
            };
            const int nk = min(KC, Np - f * KC);
            if (nk == KC) {
#pragma unroll
                for (int k = 0; k < KC; k += 2) two(k);
            } else {
#pragma unroll 1
                for (int k = 0; k < nk; k += 2) two(k);
            }
            slot = slot + 1 == kStages ? 0 : slot + 1;
        }
        f32x2 f0[kH], f1[kH];
#pragma unroll
        for (int h = 0; h < kH; ++h) f0[h] = f1[h] = 0ull;
#pragma unroll
        for (int r = 0; r < kR; ++r) {
            // rows past the dictionary: copied as zeros, with zero coefficients and an exponent <= 0
            const f32x2 n2 = pack2(nb[r], nb[r]);
            const f32x2 a0 = pack2(ab[r].x * wG, ab[r].x * wG), a1 = pack2(ab[r].y * wG, ab[r].y * wG);
#pragma unroll
            for (int h = 0; h < kH; ++h) {
                const f32x2 sum = fma2(ew2_2, n2, ens[h]);
                const float2 qa = unpack2(fma2(neg, re[r][h], sum));
                const float2 qp = unpack2(fma2(neg, im[r][h], sum)); // K(2b, 2s+1)
                const float2 qm = unpack2(fma2(pos, im[r][h], sum)); // K(2b+1, 2s)
                const f32x2 kA = pack2(ex2<false>(fminf(qa.x, 0.f)), ex2<false>(fminf(qa.y, 0.f)));
                const f32x2 kP = pack2(ex2<false>(fminf(qp.x, 0.f)), ex2<false>(fminf(qp.y, 0.f)));
                const f32x2 kM = pack2(ex2<false>(fminf(qm.x, 0.f)), ex2<false>(fminf(qm.y, 0.f)));
                f0[h] = fma2(a0, kA, fma2(a1, kM, f0[h]));
                f1[h] = fma2(a0, kP, fma2(a1, kA, f1[h]));
            }
        }
        // the lanes' tree; every level halves the values a lane carries: value j = (sample j / 2, component j % 2)
        // ends in lanes 2j, 2j + 1
        float v[2 * kSpw];
#pragma unroll
        for (int h = 0; h < kH; ++h) {
            const float2 p0 = unpack2(f0[h]), p1 = unpack2(f1[h]);
            v[4 * h] = p0.x;
            v[4 * h + 1] = p1.x;
            v[4 * h + 2] = p0.y;
            v[4 * h + 3] = p1.y;
        }
        int n = 2 * kSpw;
#pragma unroll
        for (int off = 16; off > 1; off >>= 1) {
            const bool up = lane & off;
#pragma unroll
            for (int j = 0; j < kSpw; ++j)
                if (j < n / 2) {
                    const float keep = up ? v[j + n / 2] : v[j], give = up ? v[j] : v[j + n / 2];
                    v[j] = keep + __shfl_xor_sync(0xffffffffu, give, off);
                }
            n >>= 1;
        }
        const float sum = v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
        if (split) {
            const int s = s0 + warp * kSpw + lane / 4;
            if (!(lane & 1) && s < S)
                reinterpret_cast<float*>(jb.part + size_t(c) * S + s)[(lane >> 1) & 1] = sum;
        } else {
            t += sum;
        }
    }
    if (split) {
        // the tile's last block adds the chunk sums of all parts in chunk order
        __threadfence();
        __syncthreads();
        if (tid == 0) s_last = atomicAdd(jb.cnt + blockIdx.x, 1) == parts_j - 1;
        __syncthreads();
        if (!s_last) return;
        __threadfence();
    }
    // every warp finishes its own samples: the lane's value, with the linear part
    const int s = s0 + warp * kSpw + lane / 4, c = (lane >> 1) & 1;
    bool low = false;
    if (s < S) {
        if (split) {
            t = 0.f;
#pragma unroll 8
            for (int k = 0; k < n_chunks; ++k)
                t += __ldcg(reinterpret_cast<const float*>(jb.part + size_t(k) * S + s) + c);
        }
        const float est = fmaf(wL, linear_part(jb, xw, Np, lane), t);
        if (!(lane & 1)) reinterpret_cast<float*>(jb.out + s)[c] = est;
        low = fabsf(est) < kLow;
    }
    const uint32_t mask = __ballot_sync(0xffffffffu, low);
    if (mask) low_estimates(jb, xs, nrm, wL, wG, s0, mask);
}

template <int KC>
cudaError_t launch(const BatchDetectJob* d_jobs, dim3 grid, int nmax, float wL, float wG, cudaStream_t s)
{
    const size_t smem = Shape<KC>::smem(nmax);
    const cudaError_t e = allow_smem(batch_detect_kernel<KC>, 1024);
    if (e != cudaSuccess) return e;
    batch_detect_kernel<KC><<<grid, kThreads, smem, s>>>(d_jobs, nmax, wL, wG);
    return cudaGetLastError();
}

} // namespace

cudaError_t launch_batch_detect(const BatchDetectJob* d_jobs, int n_jobs, int max_tiles, int parts, int nmax, float wL,
                                float wG, cudaStream_t s)
{
    if (n_jobs <= 0 || max_tiles <= 0) return cudaSuccess;
    dim3 grid(max_tiles, n_jobs, parts > 1 ? parts : 1);
    switch (nmax) {
    case 4: return launch<4>(d_jobs, grid, nmax, wL, wG, s);
    case 8: return launch<8>(d_jobs, grid, nmax, wL, wG, s);
    case 16:
    case 32:
    case 64: return launch<16>(d_jobs, grid, nmax, wL, wG, s);
    default: return cudaErrorInvalidValue;
    }
}

int batch_detect_tile() { return kTile; }
int batch_detect_chunk() { return kChunk; }

} // namespace apsm
