// egg_simple.cu -- brute-force GPU SynC, the second drop-in.
//
// Replaces GPU_DynamicalClustering (src/algorithms/simple_GPU_SynC.cu:29-238,
// reached from GPU_DynamicalClustering_wrapper, src/maps/map.cpp:27-29): every
// iteration updates each point from all points within eps (itself included),
//   x_p += (1/N) sum_q sin(x_q - x_p),
// and the loop stops once the mean local order parameter
// r_local = mean_p (1/N) sum_q exp(-|x_p - x_q|) reaches lam, or after max_iter
// iterations (the reference's cap is 100).  Labels: a point whose eps-ball
// holds more than one point gets the rank of the smallest index in that ball
// among all such smallest indices (simple_GPU_SynC.cu:70-100), else -1.
//
// The neighbour test is the reference's `sqrt(sum of diff^2) <= eps` with the
// square sum accumulated by fused multiply-adds, i.e. d2 <= the largest float
// whose sqrtf is <= eps.  Each point's sums are formed in the reference's
// order (neighbours by index).  r_local is summed in FP64 in a fixed order
// (the reference adds per-point floats with atomics, in no fixed order).
//
// Bound by instruction issue: n^2 distance tests, and sines and an
// exponential for the few percent of pairs within eps.  A warp takes
// kTargets points: the lanes test a staged tile of source points, a run of
// eight each, the neighbours queue up in index order, and 32 at a time a lane evaluates its neighbour's terms, which lane
// k then adds for component k in queue order.  One point per thread ran the
// sines and the exponential for any lane of 32 with a neighbour (80% of the
// steps at 5% neighbours) and left all but 157 of the chip's 592 schedulers
// with one warp at 20,000 points: 4.4 -> 0.8 ms per iteration at 20k x 2D (1.6
// with a push per 32 tests instead of one scan per tile).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "eggsync.h"
#include "egg_common.cuh"
#include "egg_host_common.h"

namespace egg {

namespace {

constexpr int kSimpleBlock = 128;  // four warps
constexpr int kTargets = 2;        // points per warp
constexpr int kSimplePerBlock = kSimpleBlock / 32 * kTargets;

// source points per staged tile (at most 16 KB)
__host__ __device__ constexpr int simple_tile(int D) { return D >= 1 && D <= 8 ? 256 : (D == 16 ? 128 : 64); }
constexpr int kSimpleTerms = 32;  // components of the contributions held at a time
__host__ __device__ constexpr int simple_queue(int D) { return simple_tile(D) + 32; }  // one target's queue

// Lane L tests the TS / 32 sources from L * TS / 32 on: source j of the tile
// lies at (j mod run) * 32 + j / run, so that the lanes' k-th ones are a row.
template <int TS>
__device__ __forceinline__ int simple_slot(int j) {
    constexpr int run = TS / 32;
    return (j % run) * 32 + j / run;
}

// sources [t0, t0 + m) into tile[l][TS], by the whole block
template <int TS>
__device__ __forceinline__ void simple_stage(const float* __restrict__ cur, int t0, int m, int d, float* tile) {
    __syncthreads();
    for (int k = threadIdx.x; k < m * d; k += kSimpleBlock) {
        const int j = k / d, l = k - j * d;
        tile[l * TS + simple_slot<TS>(j)] = __ldg(cur + (size_t)t0 * d + k);
    }
    __syncthreads();
}

// one iteration; rp[p] = the point's mean of exp(-distance)
template <int D>
__global__ void __launch_bounds__(kSimpleBlock) k_simple_iter(const float* __restrict__ cur, float* __restrict__ next,
                                                              int n, int dd, float t_eps, double* __restrict__ rp) {
    constexpr int DM = D > 0 ? D : kMaxDims;
    constexpr int TS = simple_tile(D);
    constexpr int SLOTS = (DM + 1 + 31) / 32;  // components per lane: d sums, then r
    constexpr int QS = simple_queue(D), RUN = TS / 32;
    const int d = D > 0 ? D : dd;
    extern __shared__ float sh[];  // tile [d][TS], then per warp: terms [32][33], queues [kTargets][QS]
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float* const tile = sh;
    float* const terms = sh + (size_t)TS * d + wid * (kSimpleTerms * 33 + QS * kTargets);
    int* const queues = reinterpret_cast<int*>(terms + kSimpleTerms * 33);
    const int p0 = (blockIdx.x * (kSimpleBlock / 32) + wid) * kTargets;
    float x[kTargets][DM], acc[kTargets][SLOTS];
    int cnt[kTargets], qn[kTargets];
#pragma unroll
    for (int t = 0; t < kTargets; t++) {
        for (int l = 0; l < d; l++) x[t][l] = cur[(size_t)min(p0 + t, n - 1) * d + l];
#pragma unroll
        for (int j = 0; j < SLOTS; j++) acc[t][j] = 0.f;
        cnt[t] = qn[t] = 0;
    }
    // m <= 32 queued neighbours of target t from `head` on, a lane each
    auto flush = [&](int t, int head, int m) {
        const int* q = queues + QS * t + head;
        const int j = lane < m ? q[lane] : 0;
        float d2 = 0.f;
        if (D > 0 && D + 1 <= kSimpleTerms) {
            if (lane < m) {
                for (int l = 0; l < d; l++) {
                    const float v = __ldg(cur + (size_t)j * d + l);
                    d2 = dist_step(x[t][l], v, d2);
                    terms[l * 33 + lane] = sinf(__fsub_rn(v, x[t][l]));
                }
                terms[d * 33 + lane] = expf(-sqrtf(d2));
            }
            __syncwarp();
            if (lane <= d) {
                float a = acc[t][0];
#pragma unroll 4
                for (int b = 0; b < m; b++) a += terms[lane * 33 + b];
                acc[t][0] = a;
            }
            __syncwarp();
        } else {
            if (lane < m)
                for (int l = 0; l < d; l++) d2 = dist_step(x[t][l], __ldg(cur + (size_t)j * d + l), d2);
            for (int c0 = 0; c0 <= d; c0 += kSimpleTerms) {
                const int ce = min(c0 + kSimpleTerms, d + 1);
                if (lane < m)
                    for (int c = c0; c < ce; c++)
                        terms[(c - c0) * 33 + lane] =
                            c < d ? sinf(__fsub_rn(__ldg(cur + (size_t)j * d + c), x[t][c])) : expf(-sqrtf(d2));
                __syncwarp();
                if (c0 + lane < ce) {
                    float a = 0.f;
#pragma unroll
                    for (int s = 0; s < SLOTS; s++)
                        if (s == c0 / 32) a = acc[t][s];
                    for (int b = 0; b < m; b++) a += terms[lane * 33 + b];
#pragma unroll
                    for (int s = 0; s < SLOTS; s++)
                        if (s == c0 / 32) acc[t][s] = a;
                }
                __syncwarp();
            }
        }
    };
    for (int t0 = 0; t0 < n; t0 += TS) {
        const int m = min(TS, n - t0);
        simple_stage<TS>(cur, t0, m, d, tile);
        // a lane's neighbours among its run of sources, as bits (past m: an
        // older tile's points, not counted)
        unsigned hits[kTargets];
#pragma unroll
        for (int t = 0; t < kTargets; t++) hits[t] = 0;
#pragma unroll
        for (int k = 0; k < RUN; k++) {
            float d2[kTargets];
#pragma unroll
            for (int t = 0; t < kTargets; t++) d2[t] = 0.f;
            for (int l = 0; l < d; l++) {
                const float v = tile[l * TS + k * 32 + lane];
#pragma unroll
                for (int t = 0; t < kTargets; t++) d2[t] = dist_step(x[t][l], v, d2[t]);
            }
            const bool in = lane * RUN + k < m;
#pragma unroll
            for (int t = 0; t < kTargets; t++) hits[t] |= (in && d2[t] <= t_eps) ? 1u << k : 0u;
        }
        // their places in the queues: one scan for all targets (counts up to
        // TS <= 256 in nine bits each)
        static_assert(kTargets * 10 <= 32, "counts of all targets in one word");
        unsigned mine = 0;
#pragma unroll
        for (int t = 0; t < kTargets; t++) mine |= (unsigned)__popc(hits[t]) << (10 * t);
        if (__any_sync(0xffffffffu, mine != 0)) {
            unsigned upto = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned v = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= o) upto += v;
            }
            const unsigned all = __shfl_sync(0xffffffffu, upto, 31);
            upto -= mine;
#pragma unroll
            for (int t = 0; t < kTargets; t++) {
                int* q = queues + QS * t;
                int pos = qn[t] + (int)((upto >> (10 * t)) & 1023u);
                for (unsigned h = hits[t]; h; h &= h - 1) q[pos++] = t0 + lane * RUN + __ffs(h) - 1;
                const int got = (int)((all >> (10 * t)) & 1023u);
                qn[t] += got;
                cnt[t] += got;
            }
            __syncwarp();
#pragma unroll
            for (int t = 0; t < kTargets; t++) {
                int* q = queues + QS * t;
                int head = 0;
                for (; qn[t] - head >= 32; head += 32) flush(t, head, 32);
                if (head) {
                    const int rest = lane < qn[t] - head ? q[head + lane] : 0;
                    __syncwarp();
                    if (lane < qn[t] - head) q[lane] = rest;
                    qn[t] -= head;
                    __syncwarp();
                }
            }
        }
    }
#pragma unroll
    for (int t = 0; t < kTargets; t++) {
        if (qn[t] > 0) flush(t, 0, qn[t]);
        const int p = p0 + t;
        if (p >= n) break;
#pragma unroll
        for (int s = 0; s < SLOTS; s++) {
            const int c = lane + 32 * s;
            if (c < d) next[(size_t)p * d + c] = __ldg(cur + (size_t)p * d + c) + acc[t][s] / (float)cnt[t];
            if (c == d) rp[p] = (double)(acc[t][s] / (float)cnt[t]);
        }
    }
}

// mean of rp over the points: a fixed tree over fixed strides
__global__ void __launch_bounds__(1024) k_simple_rsum(const double* __restrict__ rp, int n, double* r) {
    __shared__ double s_r[1024];
    double s = 0.0;
    for (int p = threadIdx.x; p < n; p += 1024) s += rp[p];
    s_r[threadIdx.x] = s;
    __syncthreads();
    for (int o = 512; o > 0; o >>= 1) {
        if (threadIdx.x < o) s_r[threadIdx.x] += s_r[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) *r = s_r[0] / n;
}

// smallest index within eps (count > 1): rep[p], and mark that index.  The
// sources come in index order, so a warp is done with its second neighbour
// (the first is the smallest); the block ends when all its warps are.
template <int D>
__global__ void __launch_bounds__(kSimpleBlock) k_simple_reps(const float* __restrict__ X, int n, int dd, float t_eps,
                                                              int* rep, int* incl) {
    constexpr int DM = D > 0 ? D : kMaxDims;
    constexpr int TS = simple_tile(D), RUN = TS / 32;
    const int d = D > 0 ? D : dd;
    extern __shared__ float sh[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int p0 = (blockIdx.x * (kSimpleBlock / 32) + wid) * kTargets;
    float x[kTargets][DM];
    int first[kTargets], cnt[kTargets];
#pragma unroll
    for (int t = 0; t < kTargets; t++) {
        for (int l = 0; l < d; l++) x[t][l] = X[(size_t)min(p0 + t, n - 1) * d + l];
        first[t] = -1;
        cnt[t] = 0;
    }
    for (int t0 = 0; t0 < n; t0 += TS) {
        bool done = true;
#pragma unroll
        for (int t = 0; t < kTargets; t++) done = done && (p0 + t >= n || cnt[t] > 1);
        if (__syncthreads_and(done)) break;
        const int m = min(TS, n - t0);
        simple_stage<TS>(X, t0, m, d, sh);
        unsigned hits[kTargets];
#pragma unroll
        for (int t = 0; t < kTargets; t++) hits[t] = 0;
#pragma unroll
        for (int k = 0; k < RUN; k++) {
            float d2[kTargets];
#pragma unroll
            for (int t = 0; t < kTargets; t++) d2[t] = 0.f;
            for (int l = 0; l < d; l++) {
                const float v = sh[l * TS + k * 32 + lane];
#pragma unroll
                for (int t = 0; t < kTargets; t++) d2[t] = dist_step(x[t][l], v, d2[t]);
            }
            const bool in = lane * RUN + k < m;
#pragma unroll
            for (int t = 0; t < kTargets; t++) hits[t] |= (in && d2[t] <= t_eps) ? 1u << k : 0u;
        }
#pragma unroll
        for (int t = 0; t < kTargets; t++) {
            const int low = hits[t] ? t0 + lane * RUN + __ffs(hits[t]) - 1 : 0x7fffffff;
            const int mn = __reduce_min_sync(0xffffffffu, low);
            if (first[t] < 0 && mn != 0x7fffffff) first[t] = mn;
            cnt[t] += __reduce_add_sync(0xffffffffu, __popc(hits[t]));
        }
    }
    if (lane == 0)
        for (int t = 0; t < kTargets && p0 + t < n; t++) {
            rep[p0 + t] = cnt[t] > 1 ? first[t] : -1;
            if (cnt[t] > 1) incl[first[t]] = 1;
        }
}

// ranks of the marked indices: exclusive prefix counts, one block of 1024
// threads walking the array in chunks; *total = how many are marked
__global__ void __launch_bounds__(1024) k_simple_rank(const int* __restrict__ incl, int n, int* rank, int* total) {
    __shared__ int ws[32];
    __shared__ int carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int base = 0; base < n; base += 1024) {
        const int i = base + threadIdx.x;
        const int v = i < n ? incl[i] : 0;
        int x = v;
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) ws[wid] = x;
        __syncthreads();
        if (wid == 0) {
            int s = ws[lane], t = s;
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, t, o);
                if (lane >= o) t += y;
            }
            ws[lane] = t - s;
        }
        __syncthreads();
        if (i < n) rank[i] = carry + ws[wid] + x - v;
        __syncthreads();
        if (threadIdx.x == 1023) carry += ws[wid] + x;
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
}

__global__ void k_simple_finite(const float* __restrict__ x, size_t cnt, int* bad) {
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < cnt; t += (size_t)gridDim.x * blockDim.x)
        if (!isfinite(x[t])) *bad = 1;
}

__global__ void k_simple_labels(const int* __restrict__ rep, const int* __restrict__ rank, int n, int* out) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x)
        out[p] = rep[p] >= 0 ? rank[rep[p]] : -1;
}

#define EGG_SIMPLE_D(d, KERNEL, ...)                  \
    switch (d) {                                      \
        case 1: KERNEL<1> __VA_ARGS__; break;         \
        case 2: KERNEL<2> __VA_ARGS__; break;         \
        case 3: KERNEL<3> __VA_ARGS__; break;         \
        case 4: KERNEL<4> __VA_ARGS__; break;         \
        case 5: KERNEL<5> __VA_ARGS__; break;         \
        case 8: KERNEL<8> __VA_ARGS__; break;         \
        case 16: KERNEL<16> __VA_ARGS__; break;       \
        default: KERNEL<0> __VA_ARGS__; break;        \
    }

float sq_threshold_f(float e) {
    float t = e * e;
    while (t > 0.0f && sqrtf(t) > e) t = nextafterf(t, 0.0f);
    for (;;) {
        const float u = nextafterf(t, INFINITY);
        if (sqrtf(u) <= e) t = u; else break;
    }
    return t;
}

}  // namespace

int simple_run(const float* x, int64_t n64, int32_t d, float eps, float lam, int32_t max_iter, int32_t* labels,
               float* positions_out, egg_stats* stats, void* stream) {
    if (!x || !labels) throw ArgError{EGG_ERR_ARG, "x and labels must not be NULL"};
    if (n64 < 1 || n64 > (1 << 26)) throw ArgError{EGG_ERR_ARG, "n out of range"};
    if (d < 1 || d > kMaxDims) throw ArgError{EGG_ERR_ARG, "d must be in [1, 64]"};
    if (!(eps > 0.f) || !std::isfinite(eps)) throw ArgError{EGG_ERR_ARG, "eps must be positive and finite"};
    if (max_iter < 0) throw ArgError{EGG_ERR_ARG, "max_iter must be >= 0"};
    const int n = (int)n64;
    const int cap = max_iter > 0 ? max_iter : 100;
    const float t_eps = sq_threshold_f(eps);
    cudaStream_t st = (cudaStream_t)stream;
    const int blocks = (n + kSimplePerBlock - 1) / kSimplePerBlock;
    const int ts = d <= 5 || d == 8 ? 256 : (d == 16 ? 128 : 64);  // simple_tile of the dispatched kernel
    const size_t smem_reps = sizeof(float) * (size_t)ts * d;
    const size_t smem = smem_reps + sizeof(float) * (kSimpleBlock / 32) * (kSimpleTerms * 33 + (ts + 32) * kTargets);
    std::vector<void*> tmp;
    auto alloc = [&](size_t bytes) {
        void* p = nullptr;
        EGG_CHECK(dev_alloc((void**)&p, std::max<size_t>(bytes, 4)));
        tmp.push_back(p);
        return p;
    };
    cudaEvent_t ev[6] = {};
    int iters = 0;
    double r_local = 0.0;
    std::vector<float> itr;
    try {
        for (auto& e : ev) EGG_CHECK(cudaEventCreate(&e));
        EGG_CHECK(cudaEventRecord(ev[0], st));
        float* cur = (float*)alloc(4 * (size_t)n * d);
        float* nxt = (float*)alloc(4 * (size_t)n * d);
        double* rp = (double*)alloc(8 * (size_t)n);
        double* rd = (double*)alloc(16);
        int* flags = (int*)(rd + 1);  // non-finite input, marked indices
        EGG_CHECK(cudaMemcpyAsync(cur, x, 4 * (size_t)n * d, cudaMemcpyDefault, st));
        EGG_CHECK(cudaMemsetAsync(flags, 0, 8, st));
        k_simple_finite<<<(int)std::min<size_t>(((size_t)n * d + 255) / 256, 148 * 8), 256, 0, st>>>(
            cur, (size_t)n * d, flags);
        int hf[2] = {0, 0};
        EGG_CHECK(cudaMemcpyAsync(hf, flags, 8, cudaMemcpyDeviceToHost, st));
        EGG_CHECK(cudaStreamSynchronize(st));
        if (hf[0]) throw ArgError{EGG_ERR_INPUT, "input holds NaN or Inf"};
        EGG_CHECK(cudaEventRecord(ev[1], st));
        while (r_local < (double)lam && iters < cap) {
            EGG_CHECK(cudaEventRecord(ev[4], st));
            EGG_SIMPLE_D(d, k_simple_iter, <<<blocks, kSimpleBlock, smem, st>>>(cur, nxt, n, d, t_eps, rp));
            k_simple_rsum<<<1, 1024, 0, st>>>(rp, n, rd);
            EGG_CHECK(cudaMemcpyAsync(&r_local, rd, 8, cudaMemcpyDeviceToHost, st));
            EGG_CHECK(cudaEventRecord(ev[5], st));
            EGG_CHECK(cudaStreamSynchronize(st));
            float ms = 0.f;
            EGG_CHECK(cudaEventElapsedTime(&ms, ev[4], ev[5]));
            itr.push_back(ms);
            std::swap(cur, nxt);
            iters++;
        }
        EGG_CHECK(cudaEventRecord(ev[2], st));
        int* rep = (int*)alloc(4 * (size_t)n);
        int* incl = (int*)alloc(4 * (size_t)n);
        int* rank = (int*)alloc(4 * (size_t)n);
        const bool dev_out = is_device_ptr(labels);
        int* lab = dev_out ? labels : (int*)alloc(4 * (size_t)n);
        EGG_CHECK(cudaMemsetAsync(incl, 0, 4 * (size_t)n, st));
        EGG_SIMPLE_D(d, k_simple_reps, <<<blocks, kSimpleBlock, smem_reps, st>>>(cur, n, d, t_eps, rep, incl));
        k_simple_rank<<<1, 1024, 0, st>>>(incl, n, rank, flags + 1);
        k_simple_labels<<<std::min((n + kSimpleBlock - 1) / kSimpleBlock, 148 * 16), kSimpleBlock, 0, st>>>(rep, rank, n, lab);
        EGG_CHECK(cudaMemcpyAsync(hf, flags, 8, cudaMemcpyDeviceToHost, st));
        EGG_CHECK(cudaEventRecord(ev[3], st));
        if (!dev_out) EGG_CHECK(cudaMemcpyAsync(labels, lab, 4 * (size_t)n, cudaMemcpyDeviceToHost, st));
        if (positions_out)
            EGG_CHECK(cudaMemcpyAsync(positions_out, cur, 4 * (size_t)n * d, cudaMemcpyDefault, st));
        EGG_CHECK(cudaStreamSynchronize(st));
        EGG_CHECK(cudaGetLastError());
        if (stats) {
            float t01, t12, t23, t03;
            EGG_CHECK(cudaEventElapsedTime(&t01, ev[0], ev[1]));
            EGG_CHECK(cudaEventElapsedTime(&t12, ev[1], ev[2]));
            EGG_CHECK(cudaEventElapsedTime(&t23, ev[2], ev[3]));
            EGG_CHECK(cudaEventElapsedTime(&t03, ev[0], ev[3]));
            stats->iterations = iters;
            stats->converged = r_local >= (double)lam;
            stats->n_clusters = hf[1];
            stats->order_param = r_local;
            stats->order_param_lo = stats->order_param_hi = r_local;
            stats->workspace_bytes = (int64_t)(4 * (size_t)n * d * 2 + 24 * (size_t)n);
            stats->stage_ms[0] = t01;
            stats->stage_ms[2] = t12;
            stats->stage_ms[4] = t23;
            stats->total_ms = t03;
            stats->launches = 2 * iters + 4;
            if (stats->itr_ms)
                for (int i = 0; i < std::min(iters, stats->itr_cap); i++) stats->itr_ms[i] = itr[i];
        }
    } catch (...) {
        for (void* p : tmp) cudaFree(p);
        for (auto e : ev)
            if (e) cudaEventDestroy(e);
        throw;
    }
    for (void* p : tmp) cudaFree(p);
    for (auto e : ev) cudaEventDestroy(e);
    return r_local >= (double)lam ? EGG_OK : EGG_MAX_ITER;
}

}  // namespace egg

extern "C" __attribute__((visibility("default"))) int egg_simple_sync_run(const float* x, int64_t n, int32_t d,
                                                                          float eps, float lam, int32_t max_iter,
                                                                          int32_t* labels, float* positions_out,
                                                                          egg_stats* stats, void* stream) {
    return egg::guarded(
        [&] { return egg::simple_run(x, n, d, eps, lam, max_iter, labels, positions_out, stats, stream); });
}
