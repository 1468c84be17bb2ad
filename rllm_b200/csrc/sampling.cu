// On-device token sampling: one cluster of CTAs per logits row, the row never leaves the GPU.
//   temperature <= 0 : argmax, lowest index on ties, NaNs never win (no candidate: id 0);
//   otherwise        : x = logit / T; candidates x >= threshold, where the threshold is found by
//                      40 bisection steps on the value (top_k: largest t with count(x >= t) >= k;
//                      top_p: largest t whose candidates hold >= top_p of the mass of the top_k
//                      set); the token is argmax(x + g), g = -ln(-ln(u)) Gumbel noise with
//                      u = hash(seed, counter, token) in (0,1): an exact draw from softmax(x)
//                      that is reproducible whatever else is in the batch.
// Semantics and hash constants: crates/rllm-core/src/sample.rs:19-109 of AxiomOperator/rllm;
// its device counterpart is sample_rows (crates/rllm-cuda/kernels/kernels.cu:885-954).
#include "common.cuh"
#include <math.h>

#include <cooperative_groups.h>
namespace cg = cooperative_groups;

#define SAMPLE_THREADS 1024
#define SAMPLE_CTAS 8              // CTAs of a row's cluster
#define SAMPLE_SLICE_BYTES (200 * 1024)   // largest slice that is kept in shared memory
#define BISECT_STEPS 40
#define BISECT_AT_ONCE 3           // bisection steps per pass over the row: 2^3 - 1 thresholds
#define BISECT_POINTS 7

__device__ __forceinline__ float hash_uniform(unsigned long long seed, unsigned long long counter,
                                              unsigned int token) {
    unsigned long long z = seed ^ (counter * 0x9E3779B97F4A7C15ull) ^
                           ((unsigned long long)token * 0xD1B54A32D192ED03ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return ((float)(z >> 40) + 0.5f) * (1.0f / 16777216.0f);
}

struct KeyIdx { float key; int idx; };
__device__ __forceinline__ KeyIdx better(KeyIdx a, KeyIdx b) {
    // larger key wins; equal keys: lower index; idx < 0 means "no candidate"
    if (b.idx < 0) return a;
    if (a.idx < 0) return b;
    if (b.key > a.key || (b.key == a.key && b.idx < a.idx)) return b;
    return a;
}
__device__ KeyIdx block_best(KeyIdx v, KeyIdx* sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        KeyIdx other;
        other.key = __shfl_xor_sync(0xffffffffu, v.key, o);
        other.idx = __shfl_xor_sync(0xffffffffu, v.idx, o);
        v = better(v, other);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    __syncthreads();
    if (lane == 0) sh[warp] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        KeyIdx t = sh[0];
        for (int i = 1; i < nw; ++i) t = better(t, sh[i]);
        sh[32] = t;
    }
    __syncthreads();
    return sh[32];
}

struct SampleShared {
    float warp_part[BISECT_POINTS][32];
    float part[2][BISECT_POINTS];          // what the other CTAs read, in turn
    float sum[BISECT_POINTS];
    KeyIdx best[33];
    KeyIdx best_part;
};

// Sums (or maxima) of N values over the row's whole cluster, in a fixed order: butterfly, warps, CTAs.  Every thread
// gets them.  `turn` alternates between the two buffers: who writes one again has passed a cluster barrier that every
// reader of its old contents reached afterwards.
template <int N, bool MAX>
__device__ void cluster_reduce(float (&v)[N], SampleShared& sm, int& turn) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        v[i] = MAX ? warp_max(v[i]) : warp_sum(v[i]);
        if (lane == 0) sm.warp_part[i][warp] = v[i];
    }
    __syncthreads();
    if (threadIdx.x < N) {
        float t = sm.warp_part[threadIdx.x][0];
        for (int w = 1; w < SAMPLE_THREADS / 32; ++w) {
            const float o = sm.warp_part[threadIdx.x][w];
            t = MAX ? fmaxf(t, o) : t + o;
        }
        sm.part[turn][threadIdx.x] = t;
    }
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    if (threadIdx.x < N) {
        float p[SAMPLE_CTAS];
#pragma unroll
        for (int c = 0; c < SAMPLE_CTAS; ++c) p[c] = *cluster.map_shared_rank(&sm.part[turn][threadIdx.x], c);
        float t = p[0];
#pragma unroll
        for (int c = 1; c < SAMPLE_CTAS; ++c) t = MAX ? fmaxf(t, p[c]) : t + p[c];
        sm.sum[threadIdx.x] = t;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = sm.sum[i];
    turn ^= 1;
}

// The best candidate of the cluster, valid in CTA 0; nobody leaves before it has been read.
__device__ KeyIdx cluster_best(KeyIdx b, SampleShared& sm) {
    b = block_best(b, sm.best);
    if (threadIdx.x == 0) sm.best_part = b;
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    if (cluster.block_rank() == 0 && threadIdx.x == 0)
        for (int c = 1; c < SAMPLE_CTAS; ++c) b = better(b, *cluster.map_shared_rank(&sm.best_part, c));
    cluster.sync();
    return b;
}

// 40 bisection steps of [a, b] on "mass(t) >= wanted", mass(t) being the sum of weight(x) over the row's x >= t: three steps a
// pass, which evaluates the seven points that those three steps can come to.
template <typename Weight>
__device__ float bisect(const float* xs, int n, float inv_t, float a, float b, float wanted, Weight weight, SampleShared& sm, int& turn) {
    for (int s = 0; s < BISECT_STEPS; s += BISECT_AT_ONCE) {
        float t[BISECT_POINTS], mass[BISECT_POINTS];
        t[3] = 0.5f * (a + b);
        t[1] = 0.5f * (a + t[3]); t[5] = 0.5f * (t[3] + b);
        t[0] = 0.5f * (a + t[1]); t[2] = 0.5f * (t[1] + t[3]); t[4] = 0.5f * (t[3] + t[5]); t[6] = 0.5f * (t[5] + b);
#pragma unroll
        for (int i = 0; i < BISECT_POINTS; ++i) mass[i] = 0.f;
#pragma unroll 4
        for (int i = threadIdx.x; i < n; i += SAMPLE_THREADS) {
            const float v = xs[i] * inv_t;
            if (v >= t[0]) {
                const float e = weight(v);
#pragma unroll
                for (int j = 0; j < BISECT_POINTS; ++j) mass[j] += v >= t[j] ? e : 0.f;
            }
        }
        cluster_reduce<BISECT_POINTS, false>(mass, sm, turn);
        int at = 3;
#pragma unroll
        for (int d = 2; d >= 0; --d) {             // the point under test lies d levels above the leaves
            if (s + 2 - d >= BISECT_STEPS) break;
            float m = 0.f, x = 0.f;
#pragma unroll
            for (int j = 0; j < BISECT_POINTS; ++j)
                if (j == at) { m = mass[j]; x = t[j]; }
            const int half = d == 2 ? 2 : 1;
            if (m >= wanted) { a = x; at += half; } else { b = x; at -= half; }
        }
    }
    return a;
}

// One cluster of 8 CTAs per row, an eighth of the row in each one's shared memory, read from memory once.  Bound by the
// passes of the two bisections (every element compared with a threshold, and its exponential for top_p): 14 passes on
// 8 SMs where it was 40 on one.  Two rows of 151,936 with top_p: 573 -> 86 us a launch.
__global__ void __launch_bounds__(SAMPLE_THREADS)
sample_rows_kernel(const float* logits, long long row_stride, int vocab, int slice, int resident,
                   const float* __restrict__ temperature, const int* __restrict__ top_k,
                   const float* __restrict__ top_p, const unsigned long long* __restrict__ seed,
                   const unsigned long long* __restrict__ counter, int* __restrict__ out) {
    extern __shared__ float kept[];
    __shared__ SampleShared sm;
    pdl_wait();
    pdl_launch_dependents();
    const int r = blockIdx.x / SAMPLE_CTAS, tid = threadIdx.x;
    const int i0 = (blockIdx.x % SAMPLE_CTAS) * slice, n = max(0, min(slice, vocab - i0));
    const float* x = logits + (size_t)r * row_stride + i0;
    const float T = temperature ? temperature[r] : 0.f;
    int turn = 0;

    if (!(T > 0.f)) {
        KeyIdx b; b.key = -INFINITY; b.idx = -1;
#pragma unroll 4
        for (int i = tid; i < n; i += SAMPLE_THREADS) {
            const float v = x[i];
            if (v > b.key) { b.key = v; b.idx = i0 + i; }     // NaN compares false
        }
        b = cluster_best(b, sm);
        if (tid == 0 && i0 == 0) out[r] = b.idx < 0 ? 0 : b.idx;
        return;
    }
    const float inv_t = 1.0f / T;
    float ends[2] = {-INFINITY, -INFINITY};                   // largest value, largest of the values turned round
    for (int i = tid; i < n; i += SAMPLE_THREADS) {
        const float u = x[i], v = u * inv_t;
        if (resident) kept[i] = u;                            // read again by this thread only
        ends[0] = fmaxf(ends[0], v);
        ends[1] = fmaxf(ends[1], -v);
    }
    cluster_reduce<2, true>(ends, sm, turn);
    const float* xs = resident ? kept : x;
    const float vmax = ends[0], hi = ends[0];
    float lo = -ends[1], thr = -INFINITY;
    const int k = top_k ? top_k[r] : 0;
    const float p = top_p ? top_p[r] : 1.0f;
    if (k > 0 && k < vocab) {                                 // counts < 2^24 are exact in float
        thr = bisect(xs, n, inv_t, lo, hi, (float)k, [](float) { return 1.f; }, sm, turn);
        lo = thr;
    }
    if (p < 1.0f) {
        float total[1] = {0.f};
        for (int i = tid; i < n; i += SAMPLE_THREADS) {
            const float v = xs[i] * inv_t;
            if (v >= thr) total[0] += expf(v - vmax);
        }
        cluster_reduce<1, false>(total, sm, turn);
        thr = bisect(xs, n, inv_t, lo, hi, p * total[0], [vmax](float v) { return expf(v - vmax); }, sm, turn);
    }
    const unsigned long long sd = seed ? seed[r] : 0ull, ct = counter ? counter[r] : 0ull;
    KeyIdx b; b.key = -INFINITY; b.idx = -1;
    for (int i = tid; i < n; i += SAMPLE_THREADS) {
        const float v = xs[i] * inv_t;
        if (v >= thr) {
            const float u = hash_uniform(sd, ct, (unsigned)(i0 + i));
            const float key = v + (-logf(-logf(u)));
            if (key > b.key) { b.key = key; b.idx = i0 + i; }
        }
    }
    b = cluster_best(b, sm);
    if (tid == 0 && i0 == 0) out[r] = b.idx < 0 ? 0 : b.idx;
}

// logits[index[i]] += delta[i] (logit bias, frequency and presence penalties): index is the flat
// position row * row_stride + token; the caller has summed the deltas of equal positions, so no
// two threads touch one value (crates/rllm-cuda/kernels/kernels.cu:875-880).
__global__ void logit_adjust_kernel(float* __restrict__ logits, const long long* __restrict__ index,
                                    const float* __restrict__ delta, int n) {
    pdl_wait();
    pdl_launch_dependents();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) logits[index[i]] += delta[i];
}

RLLM_API int rllm_logit_adjust(float* logits, const long long* index, const float* delta, int n, cudaStream_t stream) {
    if (n <= 0) return 0;
    return rllm_launch(logit_adjust_kernel, dim3((n + 255) / 256), dim3(256), 0, stream, logits, index, delta, n);
}

RLLM_API int rllm_sample_rows(const float* logits, long long row_stride, int rows, int vocab,
                              const float* temperature, const int* top_k, const float* top_p,
                              const unsigned long long* seed, const unsigned long long* counter,
                              int* out, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (vocab <= 0 || vocab >= (1 << 24)) return (int)cudaErrorInvalidValue;
    const int slice = (vocab + SAMPLE_CTAS - 1) / SAMPLE_CTAS;
    const size_t bytes = (size_t)slice * sizeof(float);
    const int resident = temperature != nullptr && bytes <= SAMPLE_SLICE_BYTES;      // the greedy form reads the row once
    if (resident) {
        const int e = (int)cudaFuncSetAttribute(sample_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SAMPLE_SLICE_BYTES);
        if (e) return e;
    }
    return rllm_launch_clusters(sample_rows_kernel, dim3(rows * SAMPLE_CTAS), dim3(SAMPLE_THREADS), resident ? bytes : 0, stream,
                                dim3(SAMPLE_CTAS), logits, row_stride, vocab, slice, resident, temperature, top_k, top_p, seed,
                                counter, out);
}

// the packed-argument forms (common.cuh) for the host runtime's replay of recorded launches
RLLM_PACKED(rllm_logit_adjust)
RLLM_PACKED(rllm_sample_rows)
