// Row-wise helpers that several kinds of layers share; float32 arithmetic whatever the storage
// type, accurate expf / tanhf / log1pf (no fast-math):
//
//   rows_act        out[t, c] = factor * f1(row_scale[t] * in[t, c] + bias[c]) * f2(mul[t, c / mul_group])   (row_scale, bias, mul optional;
//                   mul_group > 1: one factor for each run of that many columns, a gate per head)
//   axpby           out = a * x + b * y                                      (float32)
//   cat2_cast       out[t] = [x[t] + s * delta[t] | y[t]] in the activation type (delta optional)
//   qkv_rownorm_store  biased q/k/v projection row -> RMSNorm over the WHOLE q row and the whole k
//                   row (one weight per column), then optionally the rotation of the first `rot` entries
//                   of every query and key head by the step's angles; queries out, keys and values into
//                   the paged cache; the value heads may have another size than the key heads, or the
//                   values are the key columns as projected (v_off = the keys' first column)
//
// f1, f2: the activations of activations.cuh.
#include "common.cuh"
#include "activations.cuh"

__device__ __forceinline__ float ld_any(const void* p, int dt, size_t i) {
    return dt == RLLM_F32 ? ((const float*)p)[i] : __bfloat162float(((const bf16*)p)[i]);
}
__device__ __forceinline__ void st_any(void* p, int dt, size_t i, float v) {
    if (dt == RLLM_F32) ((float*)p)[i] = v;
    else ((bf16*)p)[i] = __float2bfloat16_rn(v);
}

// four neighbouring entries (16 or 8 bytes, aligned)
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 ld4(const bf16* p) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void st4(bf16* p, float4 v) {
    uint2 u;
    *reinterpret_cast<__nv_bfloat162*>(&u.x) = __floats2bfloat162_rn(v.x, v.y);
    *reinterpret_cast<__nv_bfloat162*>(&u.y) = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(p) = u;
}
__device__ __forceinline__ float4 ld4_any(const void* p, int dt, size_t i) {
    return dt == RLLM_F32 ? ld4((const float*)p + i) : ld4((const bf16*)p + i);
}
static inline bool al16(const void* p) { return ((uintptr_t)p & 15) == 0; }

// Threads of a block laid over rows of `cols` columns, four a thread: a power of two of them per row, up to the whole block,
// so that a thread finds its place with shifts and a block of narrow rows takes many of them.
#define ROWS4_THREADS 256
struct Rows4 {
    int n, cols, shift;                                // 1 << shift threads a row
    __device__ __forceinline__ size_t row() const { return (size_t)blockIdx.x * (ROWS4_THREADS >> shift) + (threadIdx.x >> shift); }
    __device__ __forceinline__ int column() const { return ((int)(blockIdx.y << shift) + (int)(threadIdx.x & ((1 << shift) - 1))) * 4; }
};
static inline dim3 rows4_grid(int n, int cols, Rows4& at) {
    at = {n, cols, 0};
    while (at.shift < 8 && (4 << at.shift) < cols) ++at.shift;
    const int rows = ROWS4_THREADS >> at.shift, wide = 4 << at.shift;
    return dim3((n + rows - 1) / rows, (cols + wide - 1) / wide);
}
// the activation of four values side by side (one after the other they are a chain of four calls)
__device__ __forceinline__ void act4(float (&x)[4], int act) {
#define ACT4(A) case A: _Pragma("unroll") for (int i = 0; i < 4; ++i) x[i] = act_apply(x[i], A); break;
    switch (act) { ACT4(ACT_SILU) ACT4(ACT_RELU2) ACT4(ACT_SIGMOID) ACT4(ACT_TANH) ACT4(ACT_SOFTPLUS) default: break; }
#undef ACT4
}

// rows_act on rows that can be read four entries at a time (every stride a multiple of 4, bases on 16 bytes): bound by its
// bytes.  No thread divides by the row's length (a 64-bit division per element cost more than the memory).
// relu^2, float32 to bfloat16, inputs not in the cache: 2,048 x 12,288 103 us one element a thread, 36 one row a block and one
// activation after the other, now 29 (5.3 TB/s); 2,048 x 64 2.0 / 2.7 / 1.3; 8 x 64 1.4 / 1.6 / 1.2.
__global__ void __launch_bounds__(ROWS4_THREADS)
rows_act4_kernel(const void* in, int in_dt, long long in_stride, const float* __restrict__ bias, int act1, const void* mul,
                 int mul_dt, long long mul_stride, int act2, void* out, int out_dt, long long out_stride, const Rows4 at, int mul_group,
                 float factor, const float* row_scale) {
    pdl_wait();
    pdl_launch_dependents();
    const size_t t = at.row();
    const int c = at.column();
    if (t >= at.n || c >= at.cols) return;
    float4 v = ld4_any(in, in_dt, t * in_stride + c);
    float x[4] = {v.x, v.y, v.z, v.w}, m[4];
    if (mul) {
        if (mul_group == 1) {
            const float4 f = ld4_any(mul, mul_dt, t * mul_stride + c);
            m[0] = f.x; m[1] = f.y; m[2] = f.z; m[3] = f.w;
        } else m[0] = m[1] = m[2] = m[3] = ld_any(mul, mul_dt, t * mul_stride + c / mul_group);
    }
    const float s = row_scale ? row_scale[t] : 1.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (row_scale) x[i] *= s;
        if (bias) x[i] += bias[c + i];
    }
    act4(x, act1);
    if (mul) act4(m, act2);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        x[i] *= factor;
        if (mul) x[i] *= m[i];
    }
    v = make_float4(x[0], x[1], x[2], x[3]);
    if (out_dt == RLLM_F32) st4((float*)out + t * out_stride + c, v);
    else st4((bf16*)out + t * out_stride + c, v);
}

__global__ void rows_act_kernel(const void* in, int in_dt, long long in_stride, const float* __restrict__ bias,
                                int act1, const void* mul, int mul_dt, long long mul_stride, int act2, void* out,
                                int out_dt, long long out_stride, int cols, size_t total, int mul_group, float factor,
                                const float* row_scale) {
    pdl_wait();
    pdl_launch_dependents();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const size_t t = i / cols;
    const int c = (int)(i - t * cols);
    float v = ld_any(in, in_dt, t * in_stride + c);
    if (row_scale) v *= row_scale[t];
    if (bias) v += bias[c];
    v = act_apply(v, act1) * factor;
    if (mul) v *= act_apply(ld_any(mul, mul_dt, t * mul_stride + c / mul_group), act2);
    st_any(out, out_dt, t * out_stride + c, v);
}

// The gate of an attention's heads on bfloat16 rows: out[t, c] = in[t, c] * f2(mul[t, c / group]) with eight
// columns (16 bytes) a thread; `group` a multiple of 8, so the eight share a factor.
__global__ void rows_gate_bf16_kernel(const bf16* in, long long in_stride, const float* mul, long long mul_stride, int act2,
                                      bf16* out, long long out_stride, int cols8, int group8, size_t total, float factor) {
    pdl_wait();
    pdl_launch_dependents();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const size_t t = i / cols8;
    const int c8 = (int)(i - t * cols8);
    const float f = factor * act_apply(mul[t * mul_stride + c8 / group8], act2);
    uint4 u = *reinterpret_cast<const uint4*>(in + t * in_stride + 8 * (size_t)c8);
    __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float2 v = __bfloat1622float2(p[q]);
        p[q] = __floats2bfloat162_rn(v.x * f, v.y * f);
    }
    *reinterpret_cast<uint4*>(out + t * out_stride + 8 * (size_t)c8) = u;
}

RLLM_API int rllm_rows_act(const void* in, int in_dt, long long in_stride, const float* bias, int act1,
                           const void* mul, int mul_dt, long long mul_stride, int act2, void* out, int out_dt,
                           long long out_stride, int n, int cols, int mul_group, float factor, const float* row_scale,
                           cudaStream_t stream) {
    const size_t total = (size_t)n * cols;
    if (total == 0) return 0;
    if (mul_group <= 0) return (int)cudaErrorInvalidValue;
    if (in_dt == RLLM_BF16 && out_dt == RLLM_BF16 && mul && mul_dt == RLLM_F32 && !bias && !row_scale && act1 == ACT_NONE &&
        mul_group % 8 == 0 && cols % 8 == 0 && in_stride % 8 == 0 && out_stride % 8 == 0 && al16(in) && al16(out)) {
        const size_t t8 = total / 8;
        return rllm_launch(rows_gate_bf16_kernel, dim3((unsigned)((t8 + 255) / 256)), dim3(256), 0, stream, (const bf16*)in,
                           in_stride, (const float*)mul, mul_stride, act2, (bf16*)out, out_stride, cols / 8, mul_group / 8, t8, factor);
    }
    if (cols % 4 == 0 && in_stride % 4 == 0 && out_stride % 4 == 0 && al16(in) && al16(out) &&
        (!mul || mul_group % 4 == 0 || (mul_group == 1 && mul_stride % 4 == 0 && al16(mul))) &&
        cols <= 4 * ROWS4_THREADS * 65535) {
        Rows4 at;
        const dim3 grid = rows4_grid(n, cols, at);
        return rllm_launch(rows_act4_kernel, grid, dim3(ROWS4_THREADS), 0, stream, in, in_dt, in_stride, bias, act1, mul, mul_dt,
                           mul_stride, act2, out, out_dt, out_stride, at, mul_group, factor, row_scale);
    }
    return rllm_launch(rows_act_kernel, dim3((unsigned)((total + 255) / 256)), dim3(256), 0, stream, in, in_dt,
                       in_stride, bias, act1, mul, mul_dt, mul_stride, act2, out, out_dt, out_stride, cols, total,
                       mul_group, factor, row_scale);
}

__global__ void axpby_kernel(float a, const float* x, float b, const float* y, float* out, size_t total) {
    pdl_wait();
    pdl_launch_dependents();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < total) out[i] = a * x[i] + b * y[i];
}
// four elements a thread: 2,048 x 4,096, not in the cache, 35 -> 16 us (6.3 TB/s)
__global__ void axpby4_kernel(float a, const float* x, float b, const float* y, float* out, size_t quads) {
    pdl_wait();
    pdl_launch_dependents();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= quads) return;
    const float4 u = ld4(x + 4 * i), v = ld4(y + 4 * i);
    st4(out + 4 * i, make_float4(a * u.x + b * v.x, a * u.y + b * v.y, a * u.z + b * v.z, a * u.w + b * v.w));
}
RLLM_API int rllm_axpby(float a, const float* x, float b, const float* y, float* out, long long total,
                        cudaStream_t stream) {
    if (total <= 0) return 0;
    if (total % 4 == 0 && al16(x) && al16(y) && al16(out)) {
        const size_t quads = (size_t)total / 4;
        return rllm_launch(axpby4_kernel, dim3((unsigned)((quads + 255) / 256)), dim3(256), 0, stream, a, x, b, y, out, quads);
    }
    return rllm_launch(axpby_kernel, dim3((unsigned)((total + 255) / 256)), dim3(256), 0, stream, a, x, b, y, out,
                       (size_t)total);
}

// out[t, 0:d] = x[t] (+ s * delta[t]),  out[t, d:2d] = y[t]; x and y float32 [n, d].
__global__ void cat2_cast_kernel(const float* x, const void* delta, int delta_dt, float s, const float* y, void* out,
                                 int out_dt, int d, size_t total) {
    pdl_wait();
    pdl_launch_dependents();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= total) return;
    const size_t t = i / d;
    const int c = (int)(i - t * d);
    float v = x[i];
    if (delta) v += s * ld_any(delta, delta_dt, i);
    st_any(out, out_dt, t * 2 * d + c, v);
    st_any(out, out_dt, t * 2 * d + d + c, y[i]);
}
// four columns a thread, no division: 2,048 x 4,096 to bfloat16, not in the cache, 43 -> 16.5 us
__global__ void __launch_bounds__(ROWS4_THREADS)
cat2_cast4_kernel(const float* x, const void* delta, int delta_dt, float s, const float* y, void* out, int out_dt, const Rows4 at) {
    pdl_wait();
    pdl_launch_dependents();
    const size_t t = at.row();
    const int c = at.column(), d = at.cols;
    if (t >= at.n || c >= d) return;
    float4 v = ld4(x + t * d + c);
    const float4 w = ld4(y + t * d + c);
    if (delta) {
        const float4 e = ld4_any(delta, delta_dt, t * d + c);
        v = make_float4(v.x + s * e.x, v.y + s * e.y, v.z + s * e.z, v.w + s * e.w);
    }
    if (out_dt == RLLM_F32) {
        st4((float*)out + t * 2 * d + c, v);
        st4((float*)out + t * 2 * d + d + c, w);
    } else {
        st4((bf16*)out + t * 2 * d + c, v);
        st4((bf16*)out + t * 2 * d + d + c, w);
    }
}
RLLM_API int rllm_cat2_cast(const float* x, const void* delta, int delta_dt, float s, const float* y, void* out,
                            int out_dt, int n, int d, cudaStream_t stream) {
    const size_t total = (size_t)n * d;
    if (total == 0) return 0;
    if (d % 4 == 0 && al16(x) && al16(y) && al16(out) && (!delta || al16(delta)) && d <= 4 * ROWS4_THREADS * 65535) {
        Rows4 at;
        const dim3 grid = rows4_grid(n, d, at);
        return rllm_launch(cat2_cast4_kernel, grid, dim3(ROWS4_THREADS), 0, stream, x, delta, delta_dt, s, y, out, out_dt, at);
    }
    return rllm_launch(cat2_cast_kernel, dim3((unsigned)((total + 255) / 256)), dim3(256), 0, stream, x, delta,
                       delta_dt, s, y, out, out_dt, d, total);
}

// One block per token.  qkv[t] = [q (wq) | k (wk) | v (wv) | ...] with rows `ld` apart (the projection
// may hold more columns behind v, an output gate for instance) (+ bias); q and k rows are divided by
// their root mean square over the whole row (eps inside the root) and multiplied by a weight per
// column when the weight is given; q -> q_out[t]; k, v -> the paged cache at slots[t]
// (layouts [page][kv_head][bs][dk] and [page][kv_head][bs][dv]); slot < 0 writes nothing, a slot
// beyond the pool sets the error word.
// STAGED: the q and k columns (with their bias) are read from global memory once, into shared memory
// ((wq + wk) floats), and the norm, the rotation and its partner reads work from there.
template <typename TI, typename TO, bool STAGED>
__global__ void __launch_bounds__(1024)
qkv_rownorm_store_kernel(const TI* qkv, const float* __restrict__ bias, const float* __restrict__ q_norm_w,
                         const float* __restrict__ k_norm_w, const int* __restrict__ slots, TO* q_out, TO* k_cache,
                         TO* v_cache, long long ld, int wq, int wk, int wv, int G, int dk, int dv, int bs, float eps,
                         int write_kv, int n_slots, int* err, const float2* cs_table, int rot, int pairs, int v_off) {
    __shared__ float red[33];
    extern __shared__ float staged_row[];
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x, tid = threadIdx.x;
    const TI* row = qkv + (size_t)t * ld;
    float sq = 0.f, sk = 0.f;
    for (int c = tid; c < wq; c += blockDim.x) {
        const float v = to_f<TI>(row[c]) + (bias ? bias[c] : 0.f);
        if (STAGED) staged_row[c] = v;
        sq += v * v;
    }
    for (int c = tid; c < wk; c += blockDim.x) {
        const float v = to_f<TI>(row[wq + c]) + (bias ? bias[wq + c] : 0.f);
        if (STAGED) staged_row[wq + c] = v;
        sk += v * v;
    }
    sq = block_sum(sq, red);
    sk = block_sum(sk, red);
    const float rq = q_norm_w ? 1.0f / sqrtf(sq / (float)wq + eps) : 1.f;
    const float rk = k_norm_w ? 1.0f / sqrtf(sk / (float)wk + eps) : 1.f;
    // The rotation: entry e of a head's first `rot` turns with its partner (e +- rot/2, or its neighbour
    // in the pair layout) by the token's angle of that pair; a thread reads both normed values.
    const int half = rot >> 1;
    const float2* cs = rot ? cs_table + (size_t)t * half : nullptr;
    auto normed = [&](int base, int c, const float* w, float r) {
        float v = STAGED ? staged_row[base + c] : to_f<TI>(row[base + c]) + (bias ? bias[base + c] : 0.f);
        if (w) v = v * r * w[c];
        return v;
    };
    auto turned = [&](int base, int c, const float* w, float r) {
        const float v = normed(base, c, w, r);
        const int e = c % dk;
        if (e >= rot) return v;
        int pair, other;
        bool first;
        if (pairs) { pair = e >> 1; first = !(e & 1); other = first ? c + 1 : c - 1; }
        else { first = e < half; pair = first ? e : e - half; other = first ? c + half : c - half; }
        const float o = normed(base, other, w, r);
        const float2 a = cs[pair];
        return first ? v * a.x - o * a.y : v * a.x + o * a.y;
    };
    for (int c = tid; c < wq; c += blockDim.x) q_out[(size_t)t * wq + c] = from_f<TO>(turned(0, c, q_norm_w, rq));
    if (!write_kv) return;
    int slot = slots[t];
    if (slot >= n_slots) {
        if (tid == 0 && err) atomicExch(err, RLLM_ERR_SLOT);
        slot = -1;
    }
    if (slot < 0) return;
    const size_t page = slot / bs, off = slot % bs;
    for (int c = tid; c < wk; c += blockDim.x)
        k_cache[((page * G + c / dk) * bs + off) * dk + c % dk] = from_f<TO>(turned(wq, c, k_norm_w, rk));
    for (int c = tid; c < wv; c += blockDim.x) {
        const float v = to_f<TI>(row[v_off + c]) + (bias ? bias[v_off + c] : 0.f);
        v_cache[((page * G + c / dv) * bs + off) * dv + c % dv] = from_f<TO>(v);
    }
}

// The same without a rotation, on float32 rows that can be read four entries at a time: the q and k columns stay in
// registers (NV float4 a thread) between the sums and the stores, both sums are taken in one exchange.  Bound by its bytes;
// 2,048 rows of 4,096 + 1,024 + 1,024: 51 us through shared memory an entry at a time, now 32 us; 8 rows 9.9 -> 5.9 us, with
// the weights and values on their way early (EARLY) 4.1 -> 2.7 us between kernels of its own kind.
// AL: biases and norm weights can be read four columns at a time (elsewhere one at a time: 8 rows of 4,096 + 1,024 + 1,024 2.6 us,
// 2,048 rows 18.4 against 16.9; by the kernel above, which adds in another order, 5.3 and 39).
template <typename TO, int NV, bool EARLY, bool AL>
__global__ void __launch_bounds__(1024)
qkv_rownorm_store4_kernel(const float* qkv, const float* __restrict__ bias, const float* __restrict__ q_norm_w,
                          const float* __restrict__ k_norm_w, const int* __restrict__ slots, TO* q_out, TO* k_cache, TO* v_cache,
                          long long ld, int wq, int wk, int wv, int G, int dk, int dv, int bs, float eps, int write_kv,
                          int n_slots, int* err, int v_off) {
    __shared__ float red[2][32];
    pdl_launch_dependents();
    const int t = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    // EARLY: few tokens wait for memory, not for bandwidth: biases and norm weights, which do not depend on the kernels before,
    // are here when the rows are, and the first value columns when they are stored.  With many tokens the registers that
    // takes cost more (2,048 rows of 1,024 + 256 + 256: 8.7 -> 9.8 us).
    float4 wgt[EARLY ? NV : 1], off4[EARLY ? NV : 1];
    auto four = [](const float* p) { return AL ? ld4(p) : make_float4(p[0], p[1], p[2], p[3]); };
    auto norm_weight = [&](int c) {
        const float* w = c < wq ? q_norm_w : k_norm_w;
        return w ? four(w + (c < wq ? c : c - wq)) : make_float4(1.f, 1.f, 1.f, 1.f);
    };
    if (EARLY) {
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const int c = 4 * (tid + i * blockDim.x);
            wgt[EARLY ? i : 0] = c < wq + wk ? norm_weight(c) : make_float4(1.f, 1.f, 1.f, 1.f);
            off4[EARLY ? i : 0] = bias && c < wq + wk ? four(bias + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    pdl_wait();
    const float* row = qkv + (size_t)t * ld;
    auto biased = [&](int c) {
        float4 v = ld4(row + c);
        if (bias) { v.x += bias[c]; v.y += bias[c + 1]; v.z += bias[c + 2]; v.w += bias[c + 3]; }
        return v;
    };
    int slot = write_kv ? slots[t] : -1;
    float4 val[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int c = 4 * (tid + i * blockDim.x);
        if (c < wq + wk) val[i] = ld4(row + c);
    }
    float4 first_v = make_float4(0.f, 0.f, 0.f, 0.f);           // a thread's first four value columns, on their way meanwhile
    if (EARLY && 4 * tid < wv) first_v = biased(v_off + 4 * tid);
    float sq = 0.f, sk = 0.f;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int c = 4 * (tid + i * blockDim.x);
        if (c >= wq + wk) continue;
        if (bias) {
            const float4 b = EARLY ? off4[EARLY ? i : 0] : four(bias + c);
            val[i].x += b.x; val[i].y += b.y; val[i].z += b.z; val[i].w += b.w;
        }
        const float s = val[i].x * val[i].x + val[i].y * val[i].y + val[i].z * val[i].z + val[i].w * val[i].w;
        if (c < wq) sq += s; else sk += s;
    }
    sq = warp_sum(sq);
    sk = warp_sum(sk);
    if (lane == 0) { red[0][tid >> 5] = sq; red[1][tid >> 5] = sk; }
    __syncthreads();
    const bool in = lane < (int)(blockDim.x >> 5);
    sq = warp_sum(in ? red[0][lane] : 0.f);
    sk = warp_sum(in ? red[1][lane] : 0.f);
    const float rq = 1.0f / sqrtf(sq / (float)wq + eps), rk = 1.0f / sqrtf(sk / (float)wk + eps);
    if (slot >= n_slots) {
        if (tid == 0 && err) atomicExch(err, RLLM_ERR_SLOT);
        slot = -1;
    }
    const size_t page = slot < 0 ? 0 : slot / bs, off = slot < 0 ? 0 : slot % bs;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        int c = 4 * (tid + i * blockDim.x);
        if (c >= wq + wk) continue;
        const bool is_q = c < wq;
        float4 v = val[i];
        if (is_q ? q_norm_w != nullptr : k_norm_w != nullptr) {
            const float r = is_q ? rq : rk;
            const float4 w = EARLY ? wgt[EARLY ? i : 0] : norm_weight(c);
            v = make_float4(v.x * r * w.x, v.y * r * w.y, v.z * r * w.z, v.w * r * w.w);
        }
        if (!is_q) c -= wq;
        if (is_q) st4(q_out + (size_t)t * wq + c, v);
        else if (slot >= 0) st4(k_cache + ((page * G + c / dk) * bs + off) * dk + c % dk, v);
    }
    if (slot < 0) return;
    for (int c = 4 * tid; c < wv; c += 4 * blockDim.x)
        st4(v_cache + ((page * G + c / dv) * bs + off) * dv + c % dv, EARLY && c == 4 * tid ? first_v : biased(v_off + c));
}

RLLM_API int rllm_qkv_rownorm_store(const void* qkv, int in_dt, long long ld, const float* bias, const float* q_norm_w,
                                    const float* k_norm_w, const int* slots, void* q_out, void* k_cache,
                                    void* v_cache, int out_dt, int n, int H, int G, int dk, int dv, int bs,
                                    float eps, int write_kv, long long n_slots, int* err, const void* cs_table,
                                    int rot, int pairs, int v_off, cudaStream_t stream) {
    if (n <= 0) return 0;
    if (H <= 0 || G <= 0 || dk <= 0 || dv <= 0 || bs <= 0 || v_off < 0 || ld < (long long)v_off + (long long)G * dv ||
        ld < (long long)(H + G) * dk ||
        rot < 0 || rot > dk || (rot & 1) || (rot && !cs_table))
        return (int)cudaErrorInvalidValue;
    const int ns = (int)(n_slots > 0x7fffffffLL ? 0x7fffffffLL : n_slots);
    // a block per token: few tokens (a decode step) get more threads each, since the row's sums keep it in one block
    const int threads = n < 128 ? 1024 : 256;
    const int qk = (H + G) * dk, nv = (qk / 4 + threads - 1) / threads;
    if (in_dt == RLLM_F32 && !rot && nv <= 8 && ld % 4 == 0 && dk % 4 == 0 && dv % 4 == 0 && v_off % 4 == 0 && al16(qkv) &&
        al16(q_out) && al16(k_cache) && al16(v_cache)) {
        const bool al = al16(bias) && al16(q_norm_w) && al16(k_norm_w);
#define LAUNCH4(TO, NV, EARLY)                                                                                                 \
    return rllm_launch(al ? qkv_rownorm_store4_kernel<TO, NV, EARLY, true> : qkv_rownorm_store4_kernel<TO, NV, EARLY, false>,  \
                       dim3(n), dim3(threads), 0, stream, (const float*)qkv, bias, q_norm_w, k_norm_w, slots, (TO*)q_out,      \
                       (TO*)k_cache, (TO*)v_cache, ld, H * dk, G * dk, G * dv, G, dk, dv, bs, eps, write_kv, ns, err, v_off)
        if (out_dt == RLLM_F32) {
            if (nv <= 2 && n < 128) { LAUNCH4(float, 2, true); }
            if (nv <= 2) { LAUNCH4(float, 2, false); }
            LAUNCH4(float, 8, false);
        }
        if (nv <= 2 && n < 128) { LAUNCH4(bf16, 2, true); }
        if (nv <= 2) { LAUNCH4(bf16, 2, false); }
        LAUNCH4(bf16, 8, false);
#undef LAUNCH4
    }
    const size_t smem = (size_t)(H + G) * dk * sizeof(float);
#define LAUNCH(TI, TO)                                                                                         \
    if (smem <= 40 * 1024)                                                                                     \
        return rllm_launch(qkv_rownorm_store_kernel<TI, TO, true>, dim3(n), dim3(threads), smem, stream, (const TI*)qkv, \
                           bias, q_norm_w, k_norm_w, slots, (TO*)q_out, (TO*)k_cache, (TO*)v_cache, ld, H * dk, G * dk, \
                           G * dv, G, dk, dv, bs, eps, write_kv, ns, err, (const float2*)cs_table, rot, pairs, v_off);    \
    return rllm_launch(qkv_rownorm_store_kernel<TI, TO, false>, dim3(n), dim3(threads), 0, stream, (const TI*)qkv, bias, \
                       q_norm_w, k_norm_w, slots, (TO*)q_out, (TO*)k_cache, (TO*)v_cache, ld, H * dk, G * dk, G * dv, \
                       G, dk, dv, bs, eps, write_kv, ns, err, (const float2*)cs_table, rot, pairs, v_off)
    if (in_dt == RLLM_F32 && out_dt == RLLM_F32) { LAUNCH(float, float); }
    if (in_dt == RLLM_F32 && out_dt == RLLM_BF16) { LAUNCH(float, bf16); }
    if (in_dt == RLLM_BF16 && out_dt == RLLM_BF16) { LAUNCH(bf16, bf16); }
    return (int)cudaErrorInvalidValue;
#undef LAUNCH
}

RLLM_PACKED(rllm_rows_act)
RLLM_PACKED(rllm_axpby)
RLLM_PACKED(rllm_cat2_cast)
RLLM_PACKED(rllm_qkv_rownorm_store)
