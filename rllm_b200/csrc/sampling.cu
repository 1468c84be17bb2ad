// On-device token sampling: one block or one cluster of blocks per logits row, the row never leaves the GPU.
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
#define BISECT_STEPS 40
#define SAMPLE_CTAS 8              // CTAs of a row's cluster
#define SAMPLE_CLASSES (SAMPLE_THREADS / SAMPLE_CTAS)     // columns modulo SAMPLE_THREADS that one of them holds
#define SAMPLE_KEPT_BYTES (200 * 1024)    // shared memory for them
#define BISECT_AT_ONCE 3           // bisection steps per pass of a cluster: 2^3 - 1 thresholds
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

// One block per row, many rows or a small vocabulary: a row is read again (from L2) for each of up to 80 bisection steps.
// A sum over the row: thread i adds up the columns i, i + 1,024, ..., then warp_sum, then the warps in order.  (Products are
// written out so that this kernel and the next one round alike.)
__global__ void __launch_bounds__(SAMPLE_THREADS)
sample_rows_kernel(const float* logits, long long row_stride, int vocab,
                   const float* __restrict__ temperature, const int* __restrict__ top_k,
                   const float* __restrict__ top_p, const unsigned long long* __restrict__ seed,
                   const unsigned long long* __restrict__ counter, int* __restrict__ out) {
    __shared__ float red[33];
    __shared__ KeyIdx best_sh[33];
    pdl_wait();
    pdl_launch_dependents();
    const int r = blockIdx.x, tid = threadIdx.x;
    const float* x = logits + (size_t)r * row_stride;
    const float T = temperature ? temperature[r] : 0.f;

    if (!(T > 0.f)) {
        KeyIdx b; b.key = -INFINITY; b.idx = -1;
        for (int i = tid; i < vocab; i += SAMPLE_THREADS) {
            const float v = x[i];
            if (v > b.key) { b.key = v; b.idx = i; }     // NaN compares false
        }
        b = block_best(b, best_sh);
        if (tid == 0) out[r] = b.idx < 0 ? 0 : b.idx;
        return;
    }
    const float inv_t = 1.0f / T;
    float lo = INFINITY, hi = -INFINITY;
    for (int i = tid; i < vocab; i += SAMPLE_THREADS) {
        const float v = __fmul_rn(x[i], inv_t);
        lo = fminf(lo, v); hi = fmaxf(hi, v);
    }
    hi = block_max(hi, red);
    lo = -block_max(-lo, red);
    const float vmax = hi;
    float thr = -INFINITY;
    const int k = top_k ? top_k[r] : 0;
    const float p = top_p ? top_p[r] : 1.0f;
    if (k > 0 && k < vocab) {
        float a = lo, b = hi;
        for (int s = 0; s < BISECT_STEPS; ++s) {
            const float mid = 0.5f * (a + b);
            float c = 0.f;
            for (int i = tid; i < vocab; i += SAMPLE_THREADS) c += (__fmul_rn(x[i], inv_t) >= mid) ? 1.f : 0.f;
            c = block_sum(c, red);                       // counts < 2^24 are exact in float
            if (c >= (float)k) a = mid; else b = mid;
        }
        thr = a; lo = a;
    }
    if (p < 1.0f) {
        float total = 0.f;
        for (int i = tid; i < vocab; i += SAMPLE_THREADS) {
            const float v = __fmul_rn(x[i], inv_t);
            if (v >= thr) total += expf(v - vmax);
        }
        total = block_sum(total, red);
        float a = lo, b = hi;
        for (int s = 0; s < BISECT_STEPS; ++s) {
            const float mid = 0.5f * (a + b);
            float ms = 0.f;
            for (int i = tid; i < vocab; i += SAMPLE_THREADS) {
                const float v = __fmul_rn(x[i], inv_t);
                if (v >= mid) ms += expf(v - vmax);
            }
            ms = block_sum(ms, red);
            if (ms >= p * total) a = mid; else b = mid;
        }
        thr = a;
    }
    const unsigned long long sd = seed ? seed[r] : 0ull, ct = counter ? counter[r] : 0ull;
    KeyIdx b; b.key = -INFINITY; b.idx = -1;
    for (int i = tid; i < vocab; i += SAMPLE_THREADS) {
        const float v = __fmul_rn(x[i], inv_t);
        if (v >= thr) {
            const float u = hash_uniform(sd, ct, (unsigned)i);
            const float key = v + (-logf(-logf(u)));
            if (key > b.key) { b.key = key; b.idx = i; }
        }
    }
    b = block_best(b, best_sh);
    if (tid == 0) out[r] = b.idx < 0 ? 0 : b.idx;
}

// One cluster of eight CTAs per row, few rows of a large vocabulary: a CTA holds the columns of 128 threads of the kernel above
// (columns c with c mod 1,024 in [128 rank, 128 rank + 128)) in shared memory, scaled, with their exponentials where both
// fit, and a pass over them takes three bisection steps: the sums for the seven thresholds that those steps can come to,
// each the same sum in the same order as above, so a draw does not
// depend on how many rows there are.  Bound by the issue slots of four warps in the passes and by the cluster's barriers.
struct ClusterShared {
    float part[2][BISECT_POINTS][SAMPLE_CLASSES / 32];     // what the other CTAs read, in turn
    float ends[2];
    float all[BISECT_POINTS];
    float red[33];
    KeyIdx best[33];
    KeyIdx best_part;
};

__global__ void __launch_bounds__(SAMPLE_THREADS)
sample_rows_cluster_kernel(const float* logits, long long row_stride, int vocab, int kept_e,
                           const float* __restrict__ temperature, const int* __restrict__ top_k,
                           const float* __restrict__ top_p, const unsigned long long* __restrict__ seed,
                           const unsigned long long* __restrict__ counter, int* __restrict__ out) {
    extern __shared__ float kept[];                        // [steps][128] values, then their exponentials
    __shared__ ClusterShared sm;
    pdl_wait();
    pdl_launch_dependents();
    cg::cluster_group cluster = cg::this_cluster();
    const int r = blockIdx.x / SAMPLE_CTAS, tid = threadIdx.x, lane = tid & 31, rank = blockIdx.x % SAMPLE_CTAS;
    const int steps = (vocab + SAMPLE_THREADS - 1) / SAMPLE_THREADS, n = steps * SAMPLE_CLASSES;
    const float* x = logits + (size_t)r * row_stride;
    const float T = temperature ? temperature[r] : 0.f;
    // column of the block's e-th value
    auto column = [&](int e) { return e / SAMPLE_CLASSES * SAMPLE_THREADS + rank * SAMPLE_CLASSES + e % SAMPLE_CLASSES; };
    auto finish = [&](KeyIdx b) {
        b = block_best(b, sm.best);
        if (tid == 0) sm.best_part = b;
        cluster.sync();
        if (rank == 0 && tid == 0) {
            for (int c = 1; c < SAMPLE_CTAS; ++c) b = better(b, *cluster.map_shared_rank(&sm.best_part, c));
            out[r] = b.idx < 0 ? 0 : b.idx;
        }
        cluster.sync();                                    // nobody leaves before it has been read
    };

    if (!(T > 0.f)) {
        KeyIdx b; b.key = -INFINITY; b.idx = -1;
        const int end = min(vocab, (rank + 1) * n);        // an eighth of the row in one piece
#pragma unroll 4
        for (int i = rank * n + tid; i < end; i += SAMPLE_THREADS) {
            const float v = x[i];
            if (v > b.key) { b.key = v; b.idx = i; }       // NaN compares false
        }
        finish(b);
        return;
    }
    const float inv_t = 1.0f / T, nan = __int_as_float(0x7fffffff);
    float hi = -INFINITY, neg_lo = -INFINITY;
#pragma unroll 4
    for (int e = tid; e < n; e += SAMPLE_THREADS) {
        const int i = column(e);
        const float v = i < vocab ? __fmul_rn(x[i], inv_t) : nan;          // not a number: at or above no threshold
        kept[e] = v;
        hi = fmaxf(hi, v);
        neg_lo = fmaxf(neg_lo, -v);
    }
    hi = block_max(hi, sm.red);
    neg_lo = block_max(neg_lo, sm.red);
    if (tid == 0) { sm.ends[0] = hi; sm.ends[1] = neg_lo; }
    cluster.sync();
#pragma unroll
    for (int c = 0; c < SAMPLE_CTAS; ++c) {
        const float* o = cluster.map_shared_rank(sm.ends, c);
        hi = fmaxf(hi, o[0]);
        neg_lo = fmaxf(neg_lo, o[1]);
    }
    const float vmax = hi;
    float lo = -neg_lo, thr = -INFINITY;
    const int k = top_k ? top_k[r] : 0;
    const float p = top_p ? top_p[r] : 1.0f;
    float* exps = kept + n;
    if (kept_e && p < 1.0f)
        for (int e = tid; e < n; e += SAMPLE_THREADS) exps[e] = expf(kept[e] - vmax);     // seen by others behind the next barrier
    // Sums over the columns at or above each of the thresholds, counted or with their exponentials, in sm.all.  A thread of the
    // first 128 adds up one column class for all seven: seven chains side by side for one read of a value.
    int turn = 0;
    auto sums = [&](const float (&t)[BISECT_POINTS], bool mass) {
        __syncthreads();
        if (tid < SAMPLE_CLASSES) {
            float s[BISECT_POINTS];
#pragma unroll
            for (int j = 0; j < BISECT_POINTS; ++j) s[j] = 0.f;
            auto add = [&](float v, float w) {
#pragma unroll
                for (int j = 0; j < BISECT_POINTS; ++j)
                    if (v >= t[j]) s[j] += w;
            };
            if (!mass) {
#pragma unroll 8
                for (int e = tid; e < n; e += SAMPLE_CLASSES) add(kept[e], 1.f);
            } else if (kept_e) {
#pragma unroll 8
                for (int e = tid; e < n; e += SAMPLE_CLASSES) add(kept[e], exps[e]);
            } else {
#pragma unroll 4
                for (int e = tid; e < n; e += SAMPLE_CLASSES) {
                    const float v = kept[e];
                    add(v, expf(v - vmax));
                }
            }
#pragma unroll
            for (int j = 0; j < BISECT_POINTS; ++j) {
                s[j] = warp_sum(s[j]);
                if (lane == 0) sm.part[turn][j][tid / 32] = s[j];
            }
        }
        cluster.sync();
        if (tid < BISECT_POINTS) {
            float w[SAMPLE_CTAS][SAMPLE_CLASSES / 32], s = 0.f;
#pragma unroll
            for (int c = 0; c < SAMPLE_CTAS; ++c)
#pragma unroll
                for (int i = 0; i < SAMPLE_CLASSES / 32; ++i) w[c][i] = cluster.map_shared_rank(sm.part[turn][tid], c)[i];
#pragma unroll
            for (int c = 0; c < SAMPLE_CTAS; ++c)
#pragma unroll
                for (int i = 0; i < SAMPLE_CLASSES / 32; ++i) s += w[c][i];
            sm.all[tid] = s;
        }
        turn ^= 1;                     // who writes a buffer again has passed a barrier that its readers reached afterwards
        __syncthreads();
    };
    auto bisect = [&](float a, float b, float wanted, bool mass) {
        for (int s = 0; s < BISECT_STEPS; s += BISECT_AT_ONCE) {
            float t[BISECT_POINTS];
            t[3] = 0.5f * (a + b);
            t[1] = 0.5f * (a + t[3]); t[5] = 0.5f * (t[3] + b);
            t[0] = 0.5f * (a + t[1]); t[2] = 0.5f * (t[1] + t[3]); t[4] = 0.5f * (t[3] + t[5]); t[6] = 0.5f * (t[5] + b);
            sums(t, mass);
            int at = 3;
#pragma unroll
            for (int d = 2; d >= 0; --d) {             // the point under test lies d levels above the leaves
                if (s + 2 - d >= BISECT_STEPS) break;
                float mid = 0.f;
#pragma unroll
                for (int j = 0; j < BISECT_POINTS; ++j)
                    if (j == at) mid = t[j];
                const int half = d == 2 ? 2 : 1;
                if (sm.all[at] >= wanted) { a = mid; at += half; } else { b = mid; at -= half; }
            }
        }
        return a;
    };
    if (k > 0 && k < vocab) {                              // counts < 2^24 are exact in float
        thr = bisect(lo, hi, (float)k, false);
        lo = thr;
    }
    if (p < 1.0f) {
        const float same[BISECT_POINTS] = {thr, thr, thr, thr, thr, thr, thr};
        sums(same, true);
        thr = bisect(lo, hi, p * sm.all[0], true);
    }
    const unsigned long long sd = seed ? seed[r] : 0ull, ct = counter ? counter[r] : 0ull;
    KeyIdx b; b.key = -INFINITY; b.idx = -1;
    for (int e = tid; e < n; e += SAMPLE_THREADS) {
        const float v = kept[e];
        if (v >= thr) {
            const int i = column(e);
            const float u = hash_uniform(sd, ct, (unsigned)i);
            const float key = v + (-logf(-logf(u)));
            if (key > b.key) { b.key = key; b.idx = i; }
        }
    }
    finish(b);
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
    // A cluster takes a fraction of a block's time, but 15 of them run at once (16 rows take twice the time of 15) where 148
    // blocks do: clusters while their waves cost less, which the vocabulary and the kinds of limit say.  us a launch, block /
    // clusters: 151,936 x 1 row with top_p 478 / 68, x 64 531 / 331; with top_k 292 / 56 and 293 / 277; with neither 74 / 19, and
    // 74 / 93 for 64 rows.  32,768 x 8 with top_p 125 / 39, x 64 126 / 190.  1,000 x 64 with top_p 36 / 144.  A row that the
    // cluster cannot keep is left to a block.  Greedy rows are read once: 151,936 x 1 8.7 / 8.1, x 64 9.4 / 30.
    const bool greedy = temperature == nullptr;
    const size_t bytes = (size_t)((vocab + SAMPLE_THREADS - 1) / SAMPLE_THREADS) * SAMPLE_CLASSES * sizeof(float);
    const int waves = (int)(((long long)rows * SAMPLE_CTAS + 119) / 120);
    int paid = 1;
    if (top_p) paid = vocab / 16000 > 7 ? 7 : vocab / 16000;
    else if (top_k) paid = vocab / 30000 > 6 ? 6 : vocab / 30000;
    else paid = vocab / 38000 > 4 ? 4 : vocab / 38000;
    if (greedy ? vocab >= 100000 && waves == 1
               : vocab >= 4096 && (waves == 1 || waves <= paid) && bytes <= SAMPLE_KEPT_BYTES) {
        const int kept_e = !greedy && top_p && 2 * bytes <= SAMPLE_KEPT_BYTES;
        if (!greedy) {
            const int e = (int)cudaFuncSetAttribute(sample_rows_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                    SAMPLE_KEPT_BYTES);
            if (e) return e;
        }
        return rllm_launch_clusters(sample_rows_cluster_kernel, dim3(rows * SAMPLE_CTAS), dim3(SAMPLE_THREADS),
                                    greedy ? 0 : bytes * (1 + kept_e), stream, dim3(SAMPLE_CTAS), logits, row_stride, vocab,
                                    kept_e, temperature, top_k, top_p, seed, counter, out);
    }
    return rllm_launch(sample_rows_kernel, dim3(rows), dim3(SAMPLE_THREADS), 0, stream, logits, row_stride, vocab,
                       temperature, top_k, top_p, seed, counter, out);
}

// the packed-argument forms (common.cuh) for the host runtime's replay of recorded launches
RLLM_PACKED(rllm_logit_adjust)
RLLM_PACKED(rllm_sample_rows)
