// APSM training sweep with the projection window's kernel matrix in registers:
// one CTA per chain (one detector's, or one user's, sequence of training
// steps), the chains taken from a counter by one persistent launch.
//
// Step semantics are the reference's (cpp/lib/apsm/apsm_train.cu:100-166 host
// step loop, :271-432 kernel; prediction apsm_detect.cu:170-226): at every step
// each active window row j gets
//     f_j = wL <x_j, w> + sum_{b visible} a_b K(b, j),
//     c_j = hyperslab(y_j - f_j) / W / (wL |x_j|^2 + wG),
// then a_j += c_j and w += sum_j c_j x_j, all from the pre-step values.
//
// Evaluation.  With Kt = K + wL <x, x'> a step changes the predictions of the
// window by Kt c, so every window row keeps its prediction h_j and adds
// sum_i c_i Kt(i, j) after each step.  A pair of rows that leaves the window has
// final coefficients: it joins v += a_b x_b, and pairs entering later see it as
// a Gaussian term.  A pair n entering at step t + 1 starts from
//     wL <v, x_n> + sum_{b < F} a_b K(b, n) + sum_{F <= b < n} a_b Kt(b, n),
// F = max(n_first, n - 1 - qP): the first sum (the "frozen" part, over the
// whole dictionary) is formed one step ahead, off the chain's critical path;
// the second one runs over the window while the window's own update runs.  The
// kernel columns therefore hold plain Gaussian values below F and combined
// values from there on (BatchCommon::split).  w = v + sum_{window} a_b x_b.
//
// What bounds a step is its latency: two block barriers, the window's update
// (4 fma per pair of pairs: 27.6k fma at window 80, 215 cycles on one SM) and
// the correction chain between them.  The window matrix in shared memory (the
// form of kernels_batch_sweep.cu) costs 84 KB of shared-memory reads per step,
// 650 cycles at best; in registers it costs none.  12 warps hold the 84 x 96
// slots of a window of 80 (21 pair slots per lane, three floats each), so that
// one chain has the SM to itself; 4 more warps, one per scheduler, run the
// corrections between the updates and prepare entering pairs beside them (16
// warps: 128 registers a thread and 128 bytes spilled; 15 + 5 warps at 96
// registers took 4500 cycles a step).  Kernel columns arrive by bulk copies,
// groups of up to four columns several steps ahead, in a ring.
//
// Measured, before (kernels_sweep.cu for one detector, kernels_batch_sweep.cu for
// many) and now: 1000 pilots, 8 users, window 80: 3.65 ms, now 1.03; 600 pilots,
// window 20: 1.8 ms, now 0.59; 512 detectors (563k steps, window 80): 7.09 ms, now
// 4.1; 64 pilots appended to 16 dictionaries of 2000: 289 us, now 98.
#include "apsm_batch.cuh"
#include "packed_f32.cuh"
#include "apsm_tc.cuh"

#include <algorithm>

namespace apsm {

namespace {

using namespace tc;

constexpr int kHelpWarps = 4;           // warps 0, 1, 3: one thread per pair slot of the window; warp 2: copies and
constexpr int kPrepWarp = 2;            // the part of an entering pair's start that needs no new coefficients
constexpr int kRowThreads = 96;
constexpr int kGroups = 8;              // column copies in flight, in groups of up to kBatch columns
constexpr int kBatch = 4;
constexpr int kEvictAhead = 4;          // steps that an evicted pair's data is fetched ahead
constexpr int kSampleBatch = 8;         // entering pairs per copy group of samples, two groups in flight

// RG compute warps: lane l holds pair slots l, l + 32, .. (C of them) against the TR row slots of
// its warp, three registers each (A, Bp, Bm).  A warp reads its rows' corrections once for all its columns (a broadcast read costs the
// shared-memory pipe as much as any other).  BLOCKS: CTAs per SM that the register bound leaves
// room for.
template <int C_, int RG_, int TR_, int BLOCKS_> struct Shape {
    static constexpr int C = C_, RG = RG_, TR = TR_, kBlocks = BLOCKS_;
    static constexpr int kThreads = 32 * (kHelpWarps + RG);
    static constexpr int kCols = 32 * C;                       // pair slots (columns)
    static constexpr int kSlots = kCols > RG * TR ? kCols : RG * TR;
    static constexpr int kMatrix = C == 1 ? 1024 : (C == 2 ? 4096 : 8192); // RG TR x kCols entries, a power of two
    static constexpr int kRed = RG * 2 * kCols > kHelpWarps * kMaxFeatures ? RG * 2 * kCols : kHelpWarps * kMaxFeatures;
};

struct Layout {
    int stream; // column entries in flight (a power of two)
    int ring;   // coefficients of the frozen pairs (a power of two)
    int pitch;  // floats per sample
};

// Shared memory: the parts of fixed size first (their addresses are constants), then stream, ring
// and samples.
template <class S> struct alignas(128) Shared {
    float4 nbuf[S::kSlots];                      // entering pair's column by slot
    float4 evk[kEvictAhead * kRowThreads];       // evicted pair's entries by row thread
    float4 rec[64];                              // entering pairs: y0, y1, projection scale, by te
    float2 eva[kEvictAhead * kRowThreads];       // evicted pair's coefficients
    float2 cs[S::kSlots];                        // corrections by slot
    float2 aw[2 * S::kSlots];                    // window coefficients by step parity
    float2 prs[64];                              // old-pair sums of the entering pairs, by te
    float2 lp[4 * 32];                           // warp kPrepWarp's share of the starts, by te
    float red[S::kRed];                          // [RG][2 kCols] update partials
    float hw[2 * S::kSlots];                     // first predictions
    float4 low[32];                              // low parts of v (warp kPrepWarp)
    float vs[kMaxFeatures];
    uint64_t cfull[kGroups], xfull[2];           // column and sample groups have arrived
    BatchTrainJob js;
    int abort_flag, stop[2], job;                // stop: the abort flag as every thread of a step sees it
    uint32_t base[2];                            // column and sample groups of the jobs before (phases run on)
};

template <class S> __host__ __device__ inline size_t smem_bytes(const Layout& l)
{
    return sizeof(Shared<S>) + 16 * size_t(l.stream) + 8 * size_t(l.ring) + 4 * size_t(4) * kSampleBatch * l.pitch + 128;
}

// apsm_train.cu:380-401, without branches (a divergent branch costs the chain some 50 cycles)
__device__ __forceinline__ float hyperslab(float e, float eB)
{
    const float hi = __fsub_rn(e, eB), lo = __fadd_rn(e, eB);
    const float c = e < -eB ? lo : 0.f;
    return e > eB ? hi : c;
}

// a_{2b} K(2b, .) + a_{2b+1} K(2b+1, .) for the two rows of the column's pair
__device__ __forceinline__ void acc_pair(float2 ab, float4 kv, float& g0, float& g1)
{
    g0 = fmaf(ab.x, kv.x, fmaf(ab.y, kv.z, g0));
    g1 = fmaf(ab.x, kv.y, fmaf(ab.y, kv.x, g1));
}

__device__ __forceinline__ void warp_sum2(float& a, float& b)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, o);
        b += __shfl_xor_sync(0xffffffffu, b, o);
    }
}

// The sum of a over the warp in lanes 0-15, of b in lanes 16-31.
__device__ __forceinline__ float warp_sum_halves(float a, float b, int lane)
{
    const float other = __shfl_xor_sync(0xffffffffu, lane < 16 ? b : a, 16);
    float v = (lane < 16 ? a : b) + other;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Bounded wait for a copy (limit_ns; 0: no wait at all), kept short: the roles' step loops have to stay in the
// instruction cache.
__device__ __forceinline__ bool copy_wait(uint64_t* bar, uint32_t parity, volatile int* abort, unsigned long long limit_ns)
{
    if (mbar_test_wait(bar, parity)) return true;
    const unsigned long long t0 = global_ns();
#pragma unroll 1
    while (limit_ns == 0 || !mbar_try_wait(bar, parity)) {
        if (*abort) return false;
        if (limit_ns == 0 || global_ns() - t0 > limit_ns) {
            *abort = 1;
            return false;
        }
    }
    return true;
}

// Barriers of a step, arrived at from each role's own loop.
template <int ID, int THREADS> __device__ __forceinline__ void step_sync()
{
    __syncwarp();
    asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(THREADS) : "memory");
}
template <int ID, int THREADS> __device__ __forceinline__ void step_arrive()
{
    __syncwarp();
    asm volatile("bar.arrive %0, %1;" ::"n"(ID), "n"(THREADS) : "memory");
}

// Register updates of the tile in place (selects on the register arrays made the compiler copy the whole tile
// several times a step).
__device__ __forceinline__ void set(float& a, float& p, float& m, float na, float np, float nm)
{
    asm volatile("mov.b32 %0, %3;\n\tmov.b32 %1, %4;\n\tmov.b32 %2, %5;"
                 : "+f"(a), "+f"(p), "+f"(m)
                 : "f"(na), "f"(np), "f"(nm));
}
__device__ __forceinline__ void load_if(float& a, float& p, float& m, uint32_t addr, int pred)
{
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.s32 q, %4, 0;\n\t@q ld.shared.v2.f32 {%0, %1}, [%3];\n\t"
                 "@q ld.shared.f32 %2, [%3 + 8];\n\t}"
                 : "+f"(a), "+f"(p), "+f"(m)
                 : "r"(addr), "r"(pred)
                 : "memory");
}

// asynchronous global -> shared copies of a thread (complete at cp_wait)
__device__ __forceinline__ void cp_async8(void* dst, const void* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A job as one role of the kernel sees it, read afresh from shared memory where it is needed: values held
// across the step loops would take registers from the window tile.
struct JobView {
    int hi0, T0, hiL, n_first, capP, nP, qP, RP;
    uint32_t magic;
    bool pro;
    const float4* Kc; // column n's entry 0 less its place among the columns from 0
    const BatchTrainJob& j;

    // The schedule (window_schedule below): step t of the first pass sees pairs up to hi0 + t, the last
    // min(qP, ..) of them its window; later passes repeat the last window with 1, 2, .. active pairs (ramp)
    // or all of them.  Pair hi0 + te - 1 enters at step te of the first pass.
    __device__ __forceinline__ JobView(const BatchTrainJob& job, const BatchCommon& cm)
        : hi0(job.hi0), T0(job.t_pass), hiL(job.hi0 + job.t_pass - 1), n_first(job.n_first), capP(job.capP), nP(job.nP),
          qP(cm.qP), RP(cm.XSP), pro(job.pro != nullptr), Kc(job.Kc - job.kc_base), j(job)
    {
        // n mod RP by a product with ceil(2^32 / RP) (pair indices are far below 2^32 / RP), one fixup
        magic = uint32_t((0x100000000ull + uint32_t(RP) - 1) / uint32_t(RP));
    }
    __device__ __forceinline__ int hi_of(int t) const { return hi0 + min(t, T0 - 1); }
    __device__ __forceinline__ int start_of(int hi) const { return max(0, hi - qP); }
    __device__ __forceinline__ int slot_of(int n) const
    {
        const int r = n - int(__umulhi(uint32_t(n), magic)) * RP;
        return r < 0 ? r + RP : (r >= RP ? r - RP : r);
    }
    __device__ __forceinline__ int pair_of_slot(int q, int s, int los) const { return s + (q >= los ? q - los : q - los + RP); }
    __device__ __forceinline__ const float4* col_ptr(int n) const
    {
        return Kc + column_prefix(n, 1, nP, capP) - col_begin(n, capP);
    }
    __device__ __forceinline__ float2 y_at(int n, int k) const
    {
        const float* p = j.Yf + size_t(n) * j.y_pitch + size_t(k) * j.y_m;
        return make_float2(p[0], p[j.y_off]);
    }
    // frozen range [frozen_lo, frozen_hi) of the pair n entering the window
    __device__ __forceinline__ int frozen_hi(int n) const { return band_begin(n, n_first, qP); }
    __device__ __forceinline__ int frozen_lo(int n) const { return max(col_begin(n, capP), j.flo); }
    // sums of the old pairs [.., n_first) of column n that the kernel-column launch formed, one per pass
    __device__ __forceinline__ int pro_passes(int n) const
    {
        if (j.pro_passes > 0) return j.pro_passes;
        const int g0 = n_first + (n - n_first) / kKcolGroup * kKcolGroup;
        const int gl = min(g0 + kKcolGroup, nP) - 1;
        return (col_end(gl, 1, nP) - col_begin(g0, capP) + kKcolRows - 1) / kKcolRows;
    }
};

template <class S>
__global__ void __launch_bounds__(S::kThreads, S::kBlocks)
    window_sweep_kernel(const BatchTrainJob* __restrict__ jobs, int n_jobs, BatchCommon cm, Layout lay, int* counter,
                        int* err, unsigned long long wait_ns)
{
    constexpr int C = S::C, RG = S::RG, TR = S::TR, kCols = S::kCols, kSlots = S::kSlots;
    constexpr int kAll = S::kThreads, kSampleGroups = 2;
    extern __shared__ __align__(128) uint8_t smem_raw[];
    Shared<S>& m = *reinterpret_cast<Shared<S>*>(smem_raw);
    float4* const stream = reinterpret_cast<float4*>(smem_raw + sizeof(Shared<S>)); // columns of the entering pairs
    float2* const ring = reinterpret_cast<float2*>(stream + lay.stream); // coefficients, pair b at b mod ring
    // [2 kSampleBatch][2][lay.pitch] samples of the entering pairs and of those that join v with them, by te
    float* const xs = reinterpret_cast<float*>(ring + lay.ring);
    float4 *const nbuf = m.nbuf, *const evk = m.evk, *const rec = m.rec;
    float2 *const eva = m.eva, *const cs = m.cs, *const aw = m.aw, *const prs = m.prs, *const lp = m.lp;
    float *const red = m.red, *const hw = m.hw, *const vs = m.vs;
    uint64_t *const cfull = m.cfull, *const xfull = m.xfull;
    volatile int *const abort_flag = &m.abort_flag, *const stop = m.stop, *const job_s = &m.job;
    volatile uint32_t* const base_s = m.base;
    BatchTrainJob& js = m.js;
    const uint32_t smask = uint32_t(lay.stream) - 1, rmask = uint32_t(lay.ring) - 1;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cw = warp - kHelpWarps; // compute warp (< 0: helper)
    const float wL = cm.wL, wG = cm.wG, eB = cm.eB;

    if (tid == 0) {
        for (int i = 0; i < kGroups; ++i) mbar_init(&cfull[i], 1);
        for (int i = 0; i < kSampleGroups; ++i) mbar_init(&xfull[i], 1);
        abort_flag[0] = 0;
        stop[0] = stop[1] = 0;
        base_s[0] = base_s[1] = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }

    // (A, Bp, Bm) of row slots cw TR + k against pair slots lane + 32 j, at j TR + k
    float tA[TR * C], tP[TR * C], tM[TR * C];

    for (;;) {
        __syncthreads();
        if (tid == 0) {
            *job_s = atomicAdd(counter, 1);
            if (*job_s < n_jobs) {
                js = jobs[*job_s];
                js.flo = js.pro ? js.n_first : 0;
            }
        }
        for (int i = tid; i < S::kRed; i += S::kThreads) red[i] = 0.f;
        for (int i = tid; i < kSlots; i += S::kThreads) cs[i] = aw[i] = aw[kSlots + i] = make_float2(0.f, 0.f);
        for (int i = tid; i < 2 * kSlots; i += S::kThreads) hw[i] = 0.f;
        for (int i = tid; i < kSlots; i += S::kThreads) nbuf[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncthreads();
        if (*job_s >= n_jobs) break;
        if (js.n_steps <= 0) continue; // w unchanged
        {
        const JobView v(js, cm);
        const int N = js.N, n_first = v.n_first, used0 = js.used_beforeP, hi0 = v.hi0;
        const float* ag = js.a;
        const int s0 = v.start_of(hi0), lo0 = max(0, hi0 - v.capP);
        const bool pro = v.pro;
        const bool warm = used0 > 0;  // the dictionary holds trained pairs

        // ---------------- v, the coefficients, the window ----------------
        // v: residual weights with every pair before the window (js.r covers all but the last qP pairs
        // of the dictionary); or, from the weights alone, w less the window's old pairs
        const int v_from = js.w_init ? used0 : max(0, used0 - v.qP);
        for (int d = tid; d < 2 * N; d += S::kThreads) {
            float vd = js.fresh && !js.w_init ? 0.f : (js.w_init ? js.w[d] : js.r[d]);
            const int k = d < N ? d : d - N;
            for (int b = min(v_from, n_first); b < max(v_from, n_first); ++b) {
                float2 ab = *reinterpret_cast<const float2*>(ag + 2 * b);
                if (v_from > n_first) ab = make_float2(-ab.x, -ab.y);
                const float2 y = v.y_at(b, k);
                vd = d < N ? fmaf(ab.x, y.x, fmaf(ab.y, y.y, vd)) : fmaf(ab.x, y.y, fmaf(-ab.y, y.x, vd));
            }
            vs[d] = vd;
        }
        if (warm)
            for (int b = (pro ? n_first : lo0) + tid; b < n_first; b += S::kThreads)
                ring[b & rmask] = *reinterpret_cast<const float2*>(ag + 2 * b);
        __syncthreads();
        const int los0 = v.slot_of(s0);
        // the window's predictions: linear part and the pairs before the window (a row group's partial of
        // the tile below adds the window's own pairs)
        if (warm || js.w_init)
            for (int j = s0 + warp; j < hi0; j += S::kThreads / 32) {
                float g0 = 0.f, g1 = 0.f;
                if (pro) {
                    const float2* pr = js.pro + size_t(j - n_first) * js.pro_stride;
                    for (int ps = lane; ps < v.pro_passes(j); ps += 32) {
                        g0 += pr[ps].x;
                        g1 += pr[ps].y;
                    }
                } else if (warm) {
                    const float4* col = v.col_ptr(j);
#pragma unroll 8
                    for (int b = lo0 + lane; b < n_first; b += 32) acc_pair(ring[b & rmask], __ldg(col + b), g0, g1);
                }
                for (int k = lane; k < N; k += 32) {
                    const float2 y = v.y_at(j, k);
                    const float v0 = wL * vs[k], v1 = wL * vs[N + k];
                    g0 = fmaf(v0, y.x, fmaf(v1, y.y, g0));
                    g1 = fmaf(v0, y.y, fmaf(-v1, y.x, g1));
                }
                warp_sum2(g0, g1);
                if (lane == 0) *reinterpret_cast<float2*>(hw + 2 * v.slot_of(j)) = make_float2(g0, g1);
            }
        // the window's kernel matrix, by slots in the stream buffer (rows of kCols), then into the tile
        for (int i = tid; i < RG * TR * kCols; i += S::kThreads) stream[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncthreads();
        for (int j = s0 + warp; j < hi0; j += S::kThreads / 32) {
            const float4* col = v.col_ptr(j);
            const int sj = v.slot_of(j);
            for (int b = s0 + lane; b <= j; b += 32) {
                const float4 kv = __ldg(col + b);
                const int sb = v.slot_of(b);
                stream[sb * kCols + sj] = kv;
                stream[sj * kCols + sb] = make_float4(kv.x, kv.z, kv.y, kv.w); // transposed: Bp, Bm swapped
            }
        }
        __syncthreads();
        }
        if (cw >= 0) {
#pragma unroll
            for (int i = 0; i < TR * C; ++i) {
                const float4 kv = stream[(cw * TR + i % TR) * kCols + 32 * (i / TR) + lane];
                tA[i] = kv.x;
                tP[i] = kv.y;
                tM[i] = kv.z;
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // these accesses before the columns' copies
        __syncthreads();

        // ---------------- the steps, each warp in its role ----------------
        // Two barriers a step: phase 1 (corrections; the pair that enters joins the tile), phase 2 (the window's
        // update; beside it the next pairs' starts).  Roles meet at the barriers alone; warp kPrepWarp works a
        // step ahead and does not wait at the first one.  A step costs what its longest chain of dependent
        // instructions costs, so roles keep to straight code and read shared memory early.
        uint32_t issued_c = 0, issued_x = 0; // column and sample groups issued (warp kPrepWarp)
        if (cw >= 0) {
            const int T0 = js.t_pass, n_steps = js.n_steps, RP = cm.XSP;
            // the window's update: red[cw] = sum of this warp's rows' corrections times the tile
            const float2* cu = cs + cw * TR;
            float2* my_red = reinterpret_cast<float2*>(red + cw * 2 * kCols) + lane;
            auto window_update = [&](float g0, float g1, int jn) {
                // (this warp's share of the entering pair's start is summed beside the products: its shuffles wait on
                // nothing here)
                const float g = warp_sum_halves(g0, g1, lane);
                const float s0 = __shfl_sync(0xffffffffu, g, 0), s1 = __shfl_sync(0xffffffffu, g, 16);
                float x0[C], x1[C], y0[C], y1[C];
#pragma unroll
                for (int j = 0; j < C; ++j) x0[j] = x1[j] = y0[j] = y1[j] = 0.f;
#pragma unroll
                for (int k = 0; k < TR; ++k) {
                    const float2 c = cu[k];
#pragma unroll
                    for (int j = 0; j < C; ++j) {
                        x0[j] = fmaf(c.x, tA[j * TR + k], x0[j]);
                        x1[j] = fmaf(c.x, tP[j * TR + k], x1[j]);
                        y0[j] = fmaf(c.y, tM[j * TR + k], y0[j]);
                        y1[j] = fmaf(c.y, tA[j * TR + k], y1[j]);
                    }
                }
#pragma unroll
                for (int j = 0; j < C; ++j)
                    my_red[32 * j] = make_float2(x0[j] + y0[j] + (j == jn ? s0 : 0.f), x1[j] + y1[j] + (j == jn ? s1 : 0.f));
            };
            step_sync<1, kAll>(); // the window's coefficients are in cs
            if (js.used_beforeP > 0) window_update(0.f, 0.f, -1);
            // the pair n entering next: its slot, the place of its column
            int qn, n = js.hi0;
            const volatile BatchTrainJob& jv = js; // (read in every step: registers are the tile's)
            uint32_t pos = 0;
            {
                const JobView v(js, cm);
                qn = v.slot_of(n);
            }
            step_sync<2, kAll>();
#pragma unroll 1
            for (int t = 0; t < n_steps; ++t) {
                const int halt = stop[(t + 1) & 1]; // (written in the step before: the same for every thread)
                float g0 = 0.f, g1 = 0.f;
                const int jn = t + 1 < T0 && lane == (qn & 31) ? qn >> 5 : -1; // the entering pair is in this lane's column jn
                if (t + 1 < T0) {
                    // The pair that enters at the next step joins the tile (its corrections are zero until then);
                    // its prediction starts, in this warp's share, from the frozen sum and the window's terms with the
                    // coefficients before this step; the update below adds this step's
                    const int n_first = jv.n_first;
                    const int lo = max(n + 1 - jv.capP, jv.flo), cnt = max(n_first, n - 1 - cm.qP) - lo;
                    const int fi = tid - 32 * kHelpWarps;
                    const bool in = fi < cnt;
                    float4 k1 = stream[(pos + (in ? fi : 0)) & smask];
                    float2 a1 = ring[(lo + fi) & rmask];
                    const float4 k0 = nbuf[lane < TR ? cw * TR + lane : 0];
                    float2 a0 = aw[((t + 1) & 1) * kSlots + (lane < TR ? cw * TR + lane : 0)];
                    a0 = make_float2(lane < TR ? a0.x : 0.f, lane < TR ? a0.y : 0.f);
                    a1 = make_float2(in ? a1.x : 0.f, in ? a1.y : 0.f);
                    if (!in) k1 = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (cw == 0) {
                        const float2 l = lp[((t + 1) & 3) * 32 + lane];
                        g0 = l.x;
                        g1 = l.y;
                    }
                    acc_pair(a0, k0, g0, g1);
                    acc_pair(a1, k1, g0, g1);
#pragma unroll 1
                    for (int i = fi + 32 * RG; i < cnt; i += 32 * RG)
                        acc_pair(ring[(lo + i) & rmask], stream[(pos + i) & smask], g0, g1);
                    const int kn = qn - cw * TR;
                    if (kn >= 0 && kn < TR) { // its row: K(n, j) from column n
                        float4 kv[C];
#pragma unroll
                        for (int j = 0; j < C; ++j) kv[j] = nbuf[32 * j + lane];
#pragma unroll
                        for (int k = 0; k < TR; ++k)
                            if (kn == k) {
#pragma unroll
                                for (int j = 0; j < C; ++j) set(tA[j * TR + k], tP[j * TR + k], tM[j * TR + k], kv[j].x, kv[j].z, kv[j].y);
                            }
                    }
                    // its column
                    const uint32_t tr = smem_u32(nbuf + cw * TR);
                    const int mine = lane == (qn & 31), jc = qn >> 5;
                    if (jc == 0) {
#pragma unroll
                        for (int i = 0; i < TR; ++i) load_if(tA[i], tP[i], tM[i], tr + 16 * i, mine);
                    } else if (C == 2 || (C > 2 && jc == 1)) {
                        constexpr int o = C > 1 ? TR : 0;
#pragma unroll
                        for (int i = 0; i < TR; ++i) load_if(tA[o + i], tP[o + i], tM[o + i], tr + 16 * i, mine);
                    } else if (C > 2) {
                        constexpr int o = C > 2 ? 2 * TR : 0;
#pragma unroll
                        for (int i = 0; i < TR; ++i) load_if(tA[o + i], tP[o + i], tM[o + i], tr + 16 * i, mine);
                    }
                    pos += uint32_t(n + 1 - lo);
                    ++n;
                    qn = qn + 1 == RP ? 0 : qn + 1;
                }
                if (halt) break;
                if (tid == 32 * kHelpWarps) stop[t & 1] = *abort_flag;
                step_sync<1, kAll>();
                window_update(g0, g1, jn);
                step_sync<2, kAll>();
            }
        } else if (warp != kPrepWarp) {
            // window rows: predictions, coefficients, targets and projection scale of this thread's pair slot
            const JobView v(js, cm);
            const int T0 = v.T0, n_steps = js.n_steps, RP = v.RP, capP = v.capP, qP = v.qP, hi0 = v.hi0, n_first = v.n_first;
            const int s0 = v.start_of(hi0), los0 = v.slot_of(s0);
            const int q = 32 * (warp < 2 ? warp : 2) + lane;
            float* const ag = js.a;
            const bool row = q < RP;
            int d = q - los0; // place in the window
            if (d < 0) d += RP;
            float2 h = make_float2(0.f, 0.f), a = h, y = h, ev = h;
            float rd = 0.f;
            if (row && d < hi0 - s0) {
                const int j = s0 + d;
                h = *reinterpret_cast<const float2*>(hw + 2 * q);
                a = *reinterpret_cast<const float2*>(ag + 2 * j);
                y = make_float2(js.y[2 * j], js.y[2 * j + 1]);
                rd = __frcp_rn(fmaf(wL, js.nrm[size_t(j) * js.nrm_stride], wG));
                cs[q] = a; // the window's own pairs enter the predictions by one product
                aw[kSlots + q] = a;
            }
            // the pair evicted before step t + 1 (the window pairs of step t + 1 that are in the window already
            // lose its term): its entry in the column of this thread's slot and its coefficients
            auto evict_fetch = [&](int t) {
                const int hi = v.hi_of(t), b = hi - capP;
                if (b >= 0 && t + 1 < T0 && row) {
                    const int s_next = v.start_of(hi + 1);
                    const int j = v.pair_of_slot(q, s_next, v.slot_of(s_next));
                    float4* dst = evk + (t % kEvictAhead) * kRowThreads + q;
                    if (j < hi) cp_async16(dst, v.col_ptr(j) + b);
                    else *dst = make_float4(0.f, 0.f, 0.f, 0.f);
                    cp_async8(eva + (t % kEvictAhead) * kRowThreads + q, ag + 2 * b);
                }
                cp_commit();
            };
            const bool evicts = v.hiL > capP, ramps = js.ramp != 0;
            const int flo = js.flo;
            int hi = hi0, s = s0, w = hi0 - s0;
            uint32_t pos = 0; // place of the column of the pair n = hi
            // that column's entries by slot: the window's pairs, the pair that left last, the pair itself
            auto spread = [&]() {
                const int lo = max(hi + 1 - capP, flo);
                const bool last = d == RP - 1 && s > n_first;
                float4 k = stream[(pos + uint32_t(last ? s - 1 - lo : s + d - lo)) & smask];
                if (!(d <= w || last)) k = make_float4(0.f, 0.f, 0.f, 0.f);
                if (row) nbuf[q] = k;
                pos += uint32_t(hi + 1 - lo);
            };
            step_sync<1, kAll>();
            if (1 < T0) spread();
            if (evicts)
#pragma unroll 1
                for (int t = 0; t < kEvictAhead - 1; ++t) evict_fetch(t);
            step_sync<2, kAll>();
            float* const snap = js.snap_a;
            const size_t snap_stride = size_t(js.snap_stride);
            int ramp = 0;
            float inv_w = __frcp_rn(float(2 * w));
            const f32x2* const rp = reinterpret_cast<const f32x2*>(red) + q;
            bool grows = 1 < T0, slides = grows && w == qP; // a pair enters at the next step; the first one leaves
            bool entered = false;
            int na = w;
#pragma unroll 1
            for (int t = 0; t < n_steps; ++t) {
                const int halt = stop[(t + 1) & 1];
                if (row) {
                    f32x2 r[RG];
#pragma unroll
                    for (int g = 0; g < RG; ++g) r[g] = rp[g * kCols];
                    const float4 re = rec[t & 63];
                    if (entered) {
                        h = ev = a = make_float2(0.f, 0.f); // (its whole prediction is in red)
                        y = make_float2(re.x, re.y);
                        rd = re.z;
                    }
                    h.x -= ev.x;
                    h.y -= ev.y;
#pragma unroll
                    for (int o = 1; o < RG; o *= 2)
#pragma unroll
                        for (int g = 0; g + o < RG; g += 2 * o) r[g] = add2(r[g], r[g + o]);
                    const float2 rs = unpack2(r[0]);
                    h.x += rs.x;
                    h.y += rs.y;
                    const float sc = d < na ? inv_w * rd : 0.f;
                    const float2 c = make_float2(d < na ? hyperslab(__fsub_rn(y.x, h.x), eB) * sc : 0.f,
                                                 d < na ? hyperslab(__fsub_rn(y.y, h.y), eB) * sc : 0.f);
                    cs[q] = c;
                    a.x += c.x;
                    a.y += c.y;
                    aw[(t & 1) * kSlots + q] = d < w ? a : make_float2(0.f, 0.f);
                    if (d == 0 && slides) {
                        ring[s & rmask] = a;
                        *reinterpret_cast<float2*>(ag + 2 * s) = a;
                    }
                    if (snap && d < na) *reinterpret_cast<float2*>(snap + size_t(t) * snap_stride + 2 * d) = a;
                }
                if (halt) break;
                step_sync<1, kAll>();
                if (evicts) {
                    ev = make_float2(0.f, 0.f);
                    if (grows && hi >= capP) {
                        cp_wait<kEvictAhead - 2>();
                        if (row)
                            acc_pair(eva[(t % kEvictAhead) * kRowThreads + q], evk[(t % kEvictAhead) * kRowThreads + q],
                                     ev.x, ev.y);
                    }
                    evict_fetch(t + kEvictAhead - 1);
                }
                // the next step
                if (grows) {
                    ++hi;
                    if (slides) {
                        ++s;
                        d = d == 0 ? RP - 1 : d - 1;
                    } else {
                        ++w;
                        inv_w = __frcp_rn(float(2 * w));
                    }
                }
                entered = grows && d == w - 1;
                na = w;
                grows = t + 2 < T0;
                slides = grows && w == qP;
                if (t + 1 >= T0 && ramps) {
                    ramp = ramp >= T0 ? 1 : ramp + 1;
                    na = min(w, ramp);
                }
                if (grows) spread();
                step_sync<2, kAll>();
            }
            if (row && d < w) *reinterpret_cast<float2*>(ag + 2 * (s + d)) = a;
            cp_wait<0>();
        } else {
            // v in registers (features lane and lane + 32)
            const JobView v(js, cm);
            const int T0 = v.T0, n_steps = js.n_steps, hi0 = v.hi0, hiL = v.hiL, n_first = v.n_first, N = js.N;
            const int pitch = lay.pitch, y_m = js.y_m, y_off = js.y_off;
            const uint32_t base_c = base_s[0], base_x = base_s[1];
            int vF = n_first;
            const int k1 = lane + 32;
            const bool has0 = lane < N, has1 = k1 < N;
            float2 v0 = make_float2(0.f, 0.f), v1 = v0;
            if (has0) v0 = make_float2(vs[lane], vs[N + lane]);
            if (has1) v1 = make_float2(vs[k1], vs[N + k1]);
            const float* const x_lane = xs + lane * y_m;
            auto sample = [&](int at, bool has) { // of the row at `at`, this lane's feature (+ 32 y_m: the second one)
                return has ? make_float2(x_lane[at], x_lane[at + y_off]) : make_float2(0.f, 0.f);
            };
            const float2 zero = make_float2(0.f, 0.f);
            // A pair joins v with Kahan's summation (a plain sum over thousands of pairs was the largest error of w:
            // 0.3-1.4e-6 against 0.1-0.2e-6).
            // (the low parts wait in shared memory: registers are short here)
            m.low[lane] = make_float4(0.f, 0.f, 0.f, 0.f);
            auto join = [](float& v, float& l, float p) {
                const float y = __fadd_rn(p, l), t = __fadd_rn(v, y);
                l = __fsub_rn(y, __fsub_rn(t, v));
                v = t;
            };
            auto join_v = [&](float2 ab, float2 u0, float2 u1) {
                float4 l = m.low[lane];
                join(v0.x, l.x, fmaf(ab.x, u0.x, ab.y * u0.y));
                join(v0.y, l.y, fmaf(ab.x, u0.y, -ab.y * u0.x));
                if (N > 32) {
                    join(v1.x, l.z, fmaf(ab.x, u1.x, ab.y * u1.y));
                    join(v1.y, l.w, fmaf(ab.x, u1.y, -ab.y * u1.x));
                }
                m.low[lane] = l;
            };
            // Columns, from their first frozen entry to the pair itself, one after the other around the stream
            // buffer; lane l plans those of the entering steps te = l mod 32 (and their pairs' targets, scales and
            // old-pair sums) when the block of 32 begins.  They are copied in groups of `batch`, so far ahead that
            // `lead` columns fit (a column is read up to the step before te).
            const int n_last = hiL - 1;
            const int longest = T0 > 1 ? n_last + 1 - v.frozen_lo(n_last) : 1; // (columns never get shorter)
            const int lead = min(kBatch * (kGroups - 1), int(uint32_t(lay.stream) / uint32_t(longest)));
            const int batch = lead >= 2 * kBatch ? kBatch : 1;
            const float4* c_src = nullptr;
            int c_len = 0;
            uint32_t c_pos = 0, c_next = 0; // place of this lane's column, of the next block's first
            auto plan = [&](int first) {
                const int te = first + lane;
                c_len = 0;
                if (te >= 1 && te < T0) {
                    const int n = hi0 + te - 1, lo = v.frozen_lo(n);
                    c_len = n + 1 - lo;
                    c_src = v.col_ptr(n) + lo;
                    rec[te & 63] = make_float4(js.y[2 * n], js.y[2 * n + 1],
                                               __frcp_rn(fmaf(wL, js.nrm[size_t(n) * js.nrm_stride], wG)), 0.f);
                    float2 g = zero;
                    if (v.pro) {
                        const float2* pr = js.pro + size_t(n - n_first) * js.pro_stride;
                        for (int ps = 0; ps < v.pro_passes(n); ++ps) {
                            g.x += pr[ps].x;
                            g.y += pr[ps].y;
                        }
                    }
                    prs[te & 63] = g;
                }
                int sum = c_len;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int u = __shfl_up_sync(0xffffffffu, sum, o);
                    if (lane >= o) sum += u;
                }
                c_pos = c_next + uint32_t(sum - c_len);
                c_next += uint32_t(__shfl_sync(0xffffffffu, sum, 31));
            };
            int c_te = 0; // columns of steps before c_te are issued (a multiple of batch)
            auto issue = [&](int te_end) { // groups that end by te_end (exclusive)
#pragma unroll 1
                while (c_te + batch <= te_end && c_te < T0) {
                    if ((c_te & 31) == 0) plan(c_te);
                    const uint32_t e = base_c + issued_c;
                    uint64_t* bar = &cfull[e % kGroups];
                    const int i = lane - (c_te & 31);
                    const bool on = i >= 0 && i < batch && c_len > 0;
                    const int total = __reduce_add_sync(0xffffffffu, on ? c_len : 0);
                    if (lane == 0) mbar_expect_tx(bar, uint32_t(16 * total)); // (an empty group completes at once)
                    if (on) {
                        const uint32_t p = c_pos & smask;
                        const int c1 = min(c_len, int(uint32_t(lay.stream) - p));
                        bulk_g2s(stream + p, c_src, uint32_t(16 * c1), bar);
                        if (c_len > c1) bulk_g2s(stream, c_src + c1, uint32_t(16 * (c_len - c1)), bar);
                    }
                    ++issued_c;
                    c_te += batch;
                }
            };
            uint32_t seen_c = 0; // groups that have arrived
            auto arrived = [&](int te) {
                if (te >= T0 || int(seen_c) * batch > te) return;
                copy_wait(&cfull[(base_c + seen_c) % kGroups], ((base_c + seen_c) / kGroups) & 1u, abort_flag, wait_ns);
                ++seen_c;
            };
            // samples, in groups of kSampleBatch entering pairs, one lane each
            auto sample_issue = [&](int te) { // te = 1, 1 + kSampleBatch, ..: the group's first step
                const uint32_t e = base_x + issued_x;
                uint64_t* bar = &xfull[e % kSampleGroups];
                const int ti = te + lane, n = hi0 + ti - 1, nb = v.frozen_hi(n) - 1; // (the pair that joins with n)
                const bool on = lane < kSampleBatch && ti < T0, joins = on && nb >= n_first;
                const uint32_t bytes = uint32_t(4 * js.y_row);
                const int cnt = __popc(__ballot_sync(0xffffffffu, on)) + __popc(__ballot_sync(0xffffffffu, joins));
                if (lane == 0) mbar_expect_tx(bar, uint32_t(cnt) * bytes);
                float* dst = xs + ((ti - 1) & (2 * kSampleBatch - 1)) * 2 * pitch;
                if (on) bulk_g2s(dst, js.Yf + size_t(n) * js.y_pitch, bytes, bar);
                if (joins) bulk_g2s(dst + pitch, js.Yf + size_t(nb) * js.y_pitch, bytes, bar);
                ++issued_x;
            };
            uint32_t seen_x = 0;
            auto samples_arrived = [&]() {
                copy_wait(&xfull[(base_x + seen_x) % kSampleGroups], ((base_x + seen_x) / kSampleGroups) & 1u, abort_flag,
                          wait_ns);
                ++seen_x;
            };
            // old-pair sums and linear part of the pair entering at step te (called for te = 1, 2, ..)
            auto prepare = [&](int te) {
                if (te >= T0) return;
                const int n = hi0 + te - 1;
                if ((te - 1) % kSampleBatch == 0) {
                    if (te + kSampleBatch < T0) sample_issue(te + kSampleBatch);
                    if (te > 1) samples_arrived();
                }
                const int at = ((te - 1) & (2 * kSampleBatch - 1)) * 2 * pitch;
                const float2 x0 = sample(at, has0), x1 = sample(at + 32 * y_m, has1);
                const float2 b0 = sample(at + pitch, has0), b1 = sample(at + pitch + 32 * y_m, has1);
                const float2 ab = ring[vF & rmask];
                const float2 ps = prs[te & 63];
                if (v.frozen_hi(n) > vF) { // the pair vF joins v
                    join_v(ab, b0, b1);
                    ++vF;
                }
                float g0 = fmaf(v0.x, x0.x, v0.y * x0.y), g1 = fmaf(v0.x, x0.y, -v0.y * x0.x);
                if (N > 32) {
                    g0 = fmaf(v1.x, x1.x, fmaf(v1.y, x1.y, g0));
                    g1 = fmaf(v1.x, x1.y, fmaf(-v1.y, x1.x, g1));
                }
                lp[(te & 3) * 32 + lane] = make_float2(fmaf(wL, g0, lane == 0 ? ps.x : 0.f), fmaf(wL, g1, lane == 0 ? ps.y : 0.f));
            };
            issue(min(lead, T0 + batch)); // (steps before lead)
            if (1 < T0) {
                sample_issue(1);
                samples_arrived(); // (right behind its issue: a limit of 0 expires here in every job)
            }
            arrived(0);
            arrived(1);
            step_sync<1, kAll>();
            prepare(1);
            step_sync<2, kAll>();
            bool ok = true;
#pragma unroll 1
            for (int t = 0; t < n_steps; ++t) {
                const int halt = stop[(t + 1) & 1];
                arrived(t + 2);
                if (halt) {
                    ok = false;
                    break;
                }
                step_arrive<1, kAll>();
                issue(t + 1 + lead);
                prepare(t + 2);
                step_sync<2, kAll>();
            }
            if (ok) {
                for (const int sL = v.start_of(hiL); vF < sL; ++vF) // pairs that left after the last entry
                    join_v(ring[vF & rmask], has0 ? v.y_at(vF, lane) : zero, has1 ? v.y_at(vF, k1) : zero);
                if (has0) {
                    vs[lane] = v0.x;
                    vs[N + lane] = v0.y;
                }
                if (has1) {
                    vs[k1] = v1.x;
                    vs[N + k1] = v1.y;
                }
            }
        }
        __syncthreads();
        if (*abort_flag) { // (the same for every thread: nothing sets it after the barrier)
            if (warp == kPrepWarp && lane == 0) { // this CTA's copies land before it leaves
                for (uint32_t i = issued_c > kGroups ? issued_c - kGroups : 0u; i < issued_c; ++i)
                    mbar_drain(&cfull[(base_s[0] + i) % kGroups], ((base_s[0] + i) / kGroups) & 1u);
                for (uint32_t i = issued_x > kSampleGroups ? issued_x - kSampleGroups : 0u; i < issued_x; ++i)
                    mbar_drain(&xfull[(base_s[1] + i) % kSampleGroups], ((base_s[1] + i) / kSampleGroups) & 1u);
                atomicExch(err, 1);
            }
            break;
        }
        // ---------------- w = v + the window's pairs; v stays with the detector ----------------
        const JobView v(js, cm);
        const int N = js.N, hiL = v.hiL, sL = v.start_of(hiL);
        const float* ag = js.a;
        float* part = red; // [kHelpWarps][kMaxFeatures]
        if (warp < kHelpWarps)
            for (int k = lane; k < N; k += 32) {
                float w0 = 0.f, w1 = 0.f;
#pragma unroll 4
                for (int b = sL + warp; b < hiL; b += kHelpWarps) {
                    const float2 ab = *reinterpret_cast<const float2*>(ag + 2 * b);
                    const float2 y = v.y_at(b, k);
                    w0 = fmaf(ab.x, y.x, fmaf(ab.y, y.y, w0));
                    w1 = fmaf(ab.x, y.y, fmaf(-ab.y, y.x, w1));
                }
                part[warp * kMaxFeatures + k] = w0;
                part[warp * kMaxFeatures + N + k] = w1;
            }
        __syncthreads();
        for (int d = tid; d < 2 * N; d += S::kThreads) {
            float acc = 0.f;
#pragma unroll
            for (int i = 0; i < kHelpWarps; ++i) acc += part[i * kMaxFeatures + d];
            js.w[d] = vs[d] + acc;
            if (js.r) js.r[d] = vs[d];
        }
        // barrier phases of the next job run on from this one's copies
        if (tid == 32 * kPrepWarp) { // (read by the next job's roles, after its barriers)
            base_s[0] += issued_c;
            base_s[1] += issued_x;
        }
    }
}

using Shape32 = Shape<1, 8, 4, 2>;  // up to 32 pair slots
using Shape64 = Shape<2, 8, 8, 1>;  // up to 64
using Shape84 = Shape<3, 12, 7, 1>; // up to 84

// Buffer sizes: at least three columns of `range` + 1 entries in flight (one read by the step, one
// by the step ahead, one on its way), up to 8192 entries; a CTA's share of an SM's shared memory
// where several run on one.
template <class S> bool layout_for(int range, int pitch, Layout* l)
{
    l->pitch = pitch;
    for (l->ring = 256; l->ring < range + 16; l->ring *= 2) {}
    for (int blocks = S::kBlocks; blocks >= 1; --blocks)
        for (l->stream = 8192; l->stream >= S::kMatrix && l->stream >= 3 * (range + 1); l->stream /= 2)
            if (smem_bytes<S>(*l) <= kMaxSmem / blocks - 2048) return true;
    return false;
}

template <class F> bool with_shape(int slots, F&& f)
{
    if (slots <= 32) return f(Shape32());
    if (slots <= 64) return f(Shape64());
    if (slots <= 84) return f(Shape84());
    return false;
}

} // namespace

bool window_schedule(const std::vector<TrainStep>& steps, int qP, int capP, bool full_start, int* hi0, int* t_pass)
{
    if (steps.empty()) return false;
    *hi0 = steps[0].hi / 2;
    int T0 = 1;
    while (T0 < int(steps.size()) && steps[T0].hi > steps[T0 - 1].hi) ++T0;
    *t_pass = T0;
    for (int t = 0; t < int(steps.size()); ++t) {
        const int hi = *hi0 + std::min(t, T0 - 1), w = std::min(qP, hi);
        const int na = t < T0 || full_start ? w : std::min(w, (t - T0) % T0 + 1);
        const TrainStep& s = steps[t];
        if (s.hi != 2 * hi || s.wk != 2 * w || s.n_active != 2 * na || w > capP) return false;
    }
    return true;
}

bool window_sweep_supports(int qP, int sp, int capP, int range, int np)
{
    // one pair per step; evicted pairs lie before every window pair's combined entries, their
    // coefficients final when they are fetched kEvictAhead steps early
    if (sp != 1 || capP < 2 * qP + 2 * kEvictAhead || range < 1) return false;
    return with_shape(qP + 3, [&](auto s) {
        Layout l;
        return layout_for<decltype(s)>(range, int(round_up(2 * uint32_t(np), 4)), &l);
    });
}

cudaError_t window_sweep_occupancy(const BatchCommon& cm, int range, int* ctas_per_sm)
{
    *ctas_per_sm = 0;
    cudaError_t e = cudaErrorInvalidValue;
    with_shape(cm.XSP, [&](auto s) {
        using S = decltype(s);
        Layout l;
        if (!layout_for<S>(range, int(round_up(2 * uint32_t(cm.Np), 4)), &l)) return false;
        const size_t smem = smem_bytes<S>(l);
        e = allow_smem(window_sweep_kernel<S>);
        if (e == cudaSuccess)
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas_per_sm, window_sweep_kernel<S>, S::kThreads, smem);
        return true;
    });
    return e;
}

cudaError_t launch_window_sweep(const BatchTrainJob* d_jobs, int n_jobs, BatchCommon cm, int range, int grid,
                                int* d_counter, int* d_err, cudaStream_t s)
{
    if (n_jobs <= 0) return cudaSuccess;
    cudaError_t e = cudaErrorInvalidValue;
    with_shape(cm.XSP, [&](auto shape) {
        using S = decltype(shape);
        Layout l;
        if (!layout_for<S>(range, int(round_up(2 * uint32_t(cm.Np), 4)), &l)) return false;
        const size_t smem = smem_bytes<S>(l);
        e = allow_smem(window_sweep_kernel<S>);
        if (e != cudaSuccess) return true;
        window_sweep_kernel<S><<<grid, S::kThreads, smem, s>>>(d_jobs, n_jobs, cm, l, d_counter, d_err, wait_limit_ns());
        e = cudaGetLastError();
        return true;
    });
    return e;
}

} // namespace apsm
