// Paged causal attention of the float32 path for key and value heads of 64 or 128: the function that
// attention_generic.cu computes (masks, caps, slopes and sinks as its head describes them), with float32 arithmetic
// throughout, for the shapes in which a block per (token, head) that reads its keys from memory by itself is slow.
//
// attn_f32_rows_kernel, requests of few tokens: bound by the latency of the key and value reads.  A block per (token,
// key/value head and up to 4 of its query heads); 16 warps take chunks of 32 keys in turn (chunk c belongs to warp
// c mod 16), eight lanes read one key's row in whole lines, one softmax per warp, merged in the order of the warps.
//
// attn_f32_tile_kernel, prompt portions: 32 rows (tokens x query heads of one key/value head) against tiles of 32 keys,
// which cp.async brings in one tile ahead; a score is a chain over the head's entries, rows of 132 floats keep the
// reads of eight keys in different banks.  Keys are read once per 32 rows where they were read once per row.
//
// In both kernels chunks and tiles start at multiples of 32 of the key's position, so a token's result depends only on
// its own keys and on whether its request has few tokens in the step, never on the requests around it.  A key that a row
// does not see adds nothing to it, not even where its value is infinite: tiles with masked pairs test the weight.
//
// Measured (head size 128, 16 query heads on 8): requests of 300 keys, two decoding 108 -> 12 us a layer,
// portions of 300 and 161 tokens 540 -> 64 us.
#include "common.cuh"
#include <math.h>

#define A32_KEYS 32
#define A32_WARPS 16
#define A32_HEADS 4
#define A32_ROWS 32

struct F32Mask {
    float scale, softcap;
    int window, keep_first, chunk;
};

// first key that a token at `pos` sees (the kept first ones aside)
__device__ __forceinline__ int first_key(const F32Mask& k, int pos) {
    int first = (k.window > 0 && pos + 1 - k.window > 0) ? pos + 1 - k.window : 0;
    if (k.chunk > 0) first = max(first, pos - pos % k.chunk);
    return first;
}
__device__ __forceinline__ int page_of(const int* table, int p, int bs, int n_pages, int* err) {
    int page = table[p / bs];
    if (page < 0 || page >= n_pages) {            // refused: read page 0, report
        if (err) atomicExch(err, RLLM_ERR_PAGE);
        page = 0;
    }
    return page;
}
__device__ __forceinline__ float shape_score(const F32Mask& k, float dot, const float* slopes, int head, int distance) {
    float s = dot * k.scale;
    if (k.softcap > 0.f) s = k.softcap * tanhf(s / k.softcap);
    if (slopes) s -= slopes[head] * (float)distance;
    return s;
}
__device__ __forceinline__ float dot4(float4 a, float4 b, float c) {
    return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, c))));
}

// four entries of the row that starts at `off`; zeros (and no access) for a key that is not seen
__device__ __forceinline__ float4 load_or_zero(const float* cache, long long off, int at) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (off >= 0) v = *reinterpret_cast<const float4*>(cache + off + at);
    return v;
}

// ---------------------------------------------------------------- few tokens

template <int HD, int G>
__global__ void __launch_bounds__(A32_WARPS * 32)
attn_f32_rows_kernel(const float* q, const float* k_cache, const float* v_cache, float* out, const int* __restrict__ positions,
                     const int* __restrict__ seq_ids, const int* __restrict__ tokens, const int* __restrict__ block_table,
                     int table_stride, int H, int K, int head_chunks, int bs, F32Mask mask, int n_pages, int* err,
                     const float* __restrict__ sink, const float* __restrict__ slopes) {
    constexpr int X = HD / 32;                     // float4 of a key row per lane, eight lanes a key
    constexpr int LPK = HD / 4, KPP = 32 / LPK;    // lanes per value row, value rows at a time
    constexpr int PB = G >= 2 ? 2 : 4, VB = G >= 4 ? 4 : 8;
    __shared__ float sc[A32_WARPS][G][A32_KEYS];
    __shared__ float ml[2][A32_WARPS][G];
    __shared__ __align__(16) float os[A32_WARPS][G][HD];
    pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = tokens[blockIdx.x];
    const int kvh = blockIdx.y / head_chunks, g = H / K, g0 = (blockIdx.y % head_chunks) * G;
    const int pos = positions[t], first = first_key(mask, pos);
    const int* table = block_table + (size_t)seq_ids[t] * table_stride;
    const int kept = min(mask.keep_first, first);

    float4 qv[G][X];
#pragma unroll
    for (int j = 0; j < G; ++j) {
        const int h = kvh * g + min(g0 + j, g - 1);
        const float4* row = reinterpret_cast<const float4*>(q + ((size_t)t * H + h) * HD);
#pragma unroll
        for (int x = 0; x < X; ++x) qv[j][x] = row[(lane & 7) + 8 * x];
    }
    float m_run[G], l_run[G];
    float4 acc[G];
#pragma unroll
    for (int j = 0; j < G; ++j) {
        m_run[j] = -INFINITY;
        l_run[j] = 0.f;
        acc[j] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (int run = 0; run < 2; ++run) {            // the kept first keys outside the window, then the window
        const int lo = run == 0 ? 0 : first, hi = run == 0 ? kept : pos + 1;
        for (int c = lo / A32_KEYS + (warp - lo / A32_KEYS % A32_WARPS + A32_WARPS) % A32_WARPS; c * A32_KEYS < hi; c += A32_WARPS) {
            const int p = c * A32_KEYS + lane;
            const bool seen = p >= lo && p < hi;
            long long off = -1;                    // where the key's row starts, -1: not seen
            if (seen) off = (((long long)page_of(table, p, bs, n_pages, err) * K + kvh) * bs + p % bs) * HD;
            // the loads of PB passes are in flight together (a pass: four keys)
#pragma unroll
            for (int i0 = 0; i0 < 8; i0 += PB) {
                float4 kv[PB][X];
#pragma unroll
                for (int b = 0; b < PB; ++b) {
                    const long long o = __shfl_sync(0xffffffffu, off, 4 * (i0 + b) + (lane >> 3));
#pragma unroll
                    for (int x = 0; x < X; ++x) kv[b][x] = load_or_zero(k_cache, o, 4 * ((lane & 7) + 8 * x));
                }
#pragma unroll
                for (int b = 0; b < PB; ++b)
#pragma unroll
                    for (int j = 0; j < G; ++j) {
                        float d = 0.f;
#pragma unroll
                        for (int x = 0; x < X; ++x) d = dot4(qv[j][x], kv[b][x], d);
                        d += __shfl_xor_sync(0xffffffffu, d, 1);
                        d += __shfl_xor_sync(0xffffffffu, d, 2);
                        d += __shfl_xor_sync(0xffffffffu, d, 4);
                        if ((lane & 7) == j) sc[warp][j][4 * (i0 + b) + (lane >> 3)] = d;
                    }
            }
            __syncwarp();
#pragma unroll
            for (int j = 0; j < G; ++j) {
                const float s = seen ? shape_score(mask, sc[warp][j][lane], slopes, kvh * g + min(g0 + j, g - 1), pos - p) : -INFINITY;
                const float m_new = fmaxf(m_run[j], warp_max(s));
                const float e = seen ? expf(s - m_new) : 0.f;
                const float alpha = m_run[j] == -INFINITY ? 0.f : expf(m_run[j] - m_new);
                l_run[j] = l_run[j] * alpha + warp_sum(e);
                m_run[j] = m_new;
                acc[j].x *= alpha; acc[j].y *= alpha; acc[j].z *= alpha; acc[j].w *= alpha;
                __syncwarp();
                sc[warp][j][lane] = e;
            }
            __syncwarp();
#pragma unroll
            for (int i0 = 0; i0 < A32_KEYS; i0 += VB * KPP) {
                float4 v[VB];
#pragma unroll
                for (int b = 0; b < VB; ++b)
                    v[b] = load_or_zero(v_cache, __shfl_sync(0xffffffffu, off, i0 + b * KPP + lane / LPK), 4 * (lane % LPK));
#pragma unroll
                for (int b = 0; b < VB; ++b)
#pragma unroll
                    for (int j = 0; j < G; ++j) {
                        const float e = sc[warp][j][i0 + b * KPP + lane / LPK];
                        acc[j].x = fmaf(e, v[b].x, acc[j].x); acc[j].y = fmaf(e, v[b].y, acc[j].y);
                        acc[j].z = fmaf(e, v[b].z, acc[j].z); acc[j].w = fmaf(e, v[b].w, acc[j].w);
                    }
            }
            __syncwarp();
        }
    }
#pragma unroll
    for (int j = 0; j < G; ++j) {
#pragma unroll
        for (int o = LPK; o < 32; o <<= 1) {
            acc[j].x += __shfl_xor_sync(0xffffffffu, acc[j].x, o); acc[j].y += __shfl_xor_sync(0xffffffffu, acc[j].y, o);
            acc[j].z += __shfl_xor_sync(0xffffffffu, acc[j].z, o); acc[j].w += __shfl_xor_sync(0xffffffffu, acc[j].w, o);
        }
        if (lane < LPK) *reinterpret_cast<float4*>(&os[warp][j][4 * lane]) = acc[j];
        if (lane == 0) {
            ml[0][warp][j] = m_run[j];
            ml[1][warp][j] = l_run[j];
        }
    }
    __syncthreads();
    for (int x = threadIdx.x; x < G * HD; x += A32_WARPS * 32) {
        const int j = x / HD, d = x % HD, h = kvh * g + g0 + j;
        if (g0 + j >= g) continue;
        float m = sink ? sink[h] : -INFINITY;
        for (int w = 0; w < A32_WARPS; ++w) m = fmaxf(m, ml[0][w][j]);
        float l = sink ? expf(sink[h] - m) : 0.f, o = 0.f;
        for (int w = 0; w < A32_WARPS; ++w) {
            const float lw = ml[1][w][j];
            if (lw == 0.f) continue;               // no keys: a warp that saw one has a sum that is not zero
            const float f = expf(ml[0][w][j] - m);
            l = fmaf(lw, f, l);
            o = fmaf(os[w][j][d], f, o);
        }
        out[((size_t)t * H + h) * HD + d] = o * (1.0f / l);
    }
}

// ---------------------------------------------------------------- prompt portions

__device__ __forceinline__ void copy_row16(float* dst, const float* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes)
                 : "memory");
}

template <int HD>
struct TileShared {
    float q[A32_ROWS][HD + 4];
    float k[2][A32_KEYS][HD + 4];
    float v[2][A32_KEYS][HD + 4];
    float p[A32_ROWS][A32_KEYS + 4];
    float alpha[A32_ROWS];
    float l[A32_ROWS];
};

template <int HD>
__global__ void __launch_bounds__(128)
attn_f32_tile_kernel(const float* q, const float* k_cache, const float* v_cache, float* out, const int* __restrict__ positions,
                     const int* __restrict__ cu_q, const int* __restrict__ tile_req, const int* __restrict__ tile_tok0,
                     const int* __restrict__ block_table, int table_stride, int H, int K, int TT, int GH, int head_chunks, int bs,
                     F32Mask mask, int n_pages, int* err, const float* __restrict__ sink, const float* __restrict__ slopes) {
    extern __shared__ __align__(16) unsigned char raw[];
    TileShared<HD>& sm = *reinterpret_cast<TileShared<HD>*>(raw);
    constexpr int F4 = HD / 4, C4 = HD / 64;
    pdl_wait();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int req = tile_req[blockIdx.x], tok0 = tile_tok0[blockIdx.x];
    const int n_tok = min(TT, cu_q[req + 1] - tok0);
    const int kvh = blockIdx.y / head_chunks, g = H / K, g0 = (blockIdx.y % head_chunks) * GH;
    const int* table = block_table + (size_t)req * table_stride;
    const int pos0 = positions[tok0], pos1 = pos0 + n_tok - 1;
    const int first0 = first_key(mask, pos0), kept1 = min(mask.keep_first, first_key(mask, pos1));

    // row r: token tok0 + r / GH, head g0 + r % GH of the group; rows without one read token tok0's and are not written
    for (int x = tid; x < A32_ROWS * F4; x += 128) {
        const int r = x / F4, f = x % F4, tt = r / GH, hh = g0 + r % GH;
        const bool in = tt < n_tok && hh < g;
        const float4 v = *reinterpret_cast<const float4*>(q + ((size_t)(tok0 + (in ? tt : 0)) * H + kvh * g + (in ? hh : 0)) * HD + 4 * f);
        *reinterpret_cast<float4*>(&sm.q[r][4 * f]) = v;
    }
    // scores: rows rs + 16 * i, keys ks + 8 * j; output: rows ro + 8 * i, columns 4 * (co + 16 * j)
    const int ks = lane & 7, rs = warp * 4 + (lane >> 3), co = lane & 15, ro = warp * 2 + (lane >> 4);
    float m_run[2], l_run[2];
    int rpos[2], rfirst[2], rkept[2], rhead[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int r = rs + 16 * i, tt = r / GH;
        rhead[i] = kvh * g + min(g0 + r % GH, g - 1);
        rpos[i] = pos0 + min(tt, n_tok - 1);
        rfirst[i] = first_key(mask, rpos[i]);
        rkept[i] = min(mask.keep_first, rfirst[i]);
        m_run[i] = sink ? sink[rhead[i]] : -INFINITY;
        l_run[i] = sink ? 1.f : 0.f;
    }
    float4 acc[4][C4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < C4; ++j) acc[i][j] = make_float4(0.f, 0.f, 0.f, 0.f);

    // key tiles: those of the kept first keys, then those from the first row's first key on
    const int kept_tiles = (kept1 + A32_KEYS - 1) / A32_KEYS, t_first = first0 / A32_KEYS;
    const int n_tiles = kept_tiles + pos1 / A32_KEYS + 1 - t_first;
    auto tile_start = [&](int t) { return (t < kept_tiles ? t : t_first + t - kept_tiles) * A32_KEYS; };
    auto fetch = [&](int t) {
        const int c0 = tile_start(t), lo = t < kept_tiles ? 0 : first0, hi = t < kept_tiles ? kept1 : pos1 + 1;
        // a warp's eight keys: their pages in eight lanes, their rows by all
        const int mine = c0 + warp * 8 + (lane & 7);
        long long off = -1;
        if (mine >= lo && mine < hi) off = (((long long)page_of(table, mine, bs, n_pages, err) * K + kvh) * bs + mine % bs) * HD;
#pragma unroll
        for (int i = 0; i < 8 * F4 / 32; ++i) {
            const int x = i * 32 + lane, key = x / F4, f = x % F4;
            const long long o = __shfl_sync(0xffffffffu, off, key);
            const int bytes = o >= 0 ? 16 : 0;
            const long long at = o >= 0 ? o + 4 * f : 0;
            copy_row16(&sm.k[t & 1][warp * 8 + key][4 * f], k_cache + at, bytes);
            copy_row16(&sm.v[t & 1][warp * 8 + key][4 * f], v_cache + at, bytes);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(0);
    for (int t = 0; t < n_tiles; ++t) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                  // tile t is here (and q); nobody reads tile t - 1 any more
        if (t + 1 < n_tiles) fetch(t + 1);
        const int c0 = tile_start(t);
        const bool kept_run = t < kept_tiles;
        float s[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 8
        for (int f = 0; f < HD; f += 4) {
            float4 a[2], b[4];
#pragma unroll
            for (int i = 0; i < 2; ++i) a[i] = *reinterpret_cast<const float4*>(&sm.q[rs + 16 * i][f]);
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(&sm.k[t & 1][ks + 8 * j][f]);
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) s[i][j] = dot4(a[i], b[j], s[i][j]);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int lo = kept_run ? 0 : rfirst[i], hi = kept_run ? rkept[i] : rpos[i] + 1;
            float top = -INFINITY;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int p = c0 + ks + 8 * j;
                s[i][j] = p >= lo && p < hi ? shape_score(mask, s[i][j], slopes, rhead[i], rpos[i] - p) : -INFINITY;
                top = fmaxf(top, s[i][j]);
            }
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 1));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 2));
            top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, 4));
            const float m_new = fmaxf(m_run[i], top);
            const float alpha = m_run[i] == -INFINITY ? 0.f : expf(m_run[i] - m_new);
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int p = c0 + ks + 8 * j;
                const float e = p >= lo && p < hi ? expf(s[i][j] - m_new) : 0.f;
                sm.p[rs + 16 * i][ks + 8 * j] = e;
                sum += e;
            }
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            sum += __shfl_xor_sync(0xffffffffu, sum, 4);
            l_run[i] = l_run[i] * alpha + sum;
            m_run[i] = m_new;
            if (ks == 0) sm.alpha[rs + 16 * i] = alpha;
        }
        __syncthreads();                                  // weights and factors are there
        // every pair of the tile is seen where the last key is at or before the first row and the first key is in all rows' windows
        const bool whole = !kept_run && c0 + A32_KEYS - 1 <= pos0 && c0 >= first_key(mask, pos1);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float f = sm.alpha[ro + 8 * i];
#pragma unroll
            for (int j = 0; j < C4; ++j) { acc[i][j].x *= f; acc[i][j].y *= f; acc[i][j].z *= f; acc[i][j].w *= f; }
        }
#pragma unroll 2
        for (int key = 0; key < A32_KEYS; key += 4) {
            float4 w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) w[i] = *reinterpret_cast<const float4*>(&sm.p[ro + 8 * i][key]);
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int j = 0; j < C4; ++j) {
                    const float4 v = *reinterpret_cast<const float4*>(&sm.v[t & 1][key + x][4 * (co + 16 * j)]);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const float e = x == 0 ? w[i].x : x == 1 ? w[i].y : x == 2 ? w[i].z : w[i].w;
                        if (whole || e != 0.f) {
                            acc[i][j].x = fmaf(e, v.x, acc[i][j].x); acc[i][j].y = fmaf(e, v.y, acc[i][j].y);
                            acc[i][j].z = fmaf(e, v.z, acc[i][j].z); acc[i][j].w = fmaf(e, v.w, acc[i][j].w);
                        }
                    }
                }
        }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
        if (ks == 0) sm.l[rs + 16 * i] = l_run[i];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = ro + 8 * i, tt = r / GH, hh = g0 + r % GH;
        if (tt >= n_tok || hh >= g) continue;
        const float inv = 1.0f / sm.l[r];
        float* row = out + ((size_t)(tok0 + tt) * H + kvh * g + hh) * HD;
#pragma unroll
        for (int j = 0; j < C4; ++j) {
            const float4 o = acc[i][j];
            *reinterpret_cast<float4*>(row + 4 * (co + 16 * j)) = make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv);
        }
    }
}

// ---------------------------------------------------------------- launch

static bool f32_shape_ok(int H, int K, int hd, int bs, int keep_first, int chunk) {
    return (hd == 64 || hd == 128) && K > 0 && H % K == 0 && bs > 0 && keep_first >= 0 && chunk >= 0;
}

// Tokens tokens[0..n_tokens): one block per token and up to 4 query heads of one key/value head.
RLLM_API int rllm_attn_f32_rows(const float* q, const float* k_cache, const float* v_cache, float* out, const int* positions,
                                const int* seq_ids, const int* tokens, int n_tokens, const int* block_table, int table_stride, int H,
                                int K, int hd, int bs, float scale, int window, int keep_first, int chunk, float softcap,
                                int n_pages, int* err, const float* sink, const float* slopes, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (!f32_shape_ok(H, K, hd, bs, keep_first, chunk)) return (int)cudaErrorInvalidValue;
    const F32Mask mask = {scale, softcap, window, keep_first, chunk};
    const int g = H / K, G = g >= 3 ? 4 : g, chunks = (g + G - 1) / G;
#define ROWS(HD, GG)                                                                                                            \
    if (hd == HD && G == GG)                                                                                                    \
        return rllm_launch_after(attn_f32_rows_kernel<HD, GG>, dim3(n_tokens, K * chunks), dim3(A32_WARPS * 32), 0, stream, q, k_cache, \
                           v_cache, out, positions, seq_ids, tokens, block_table, table_stride, H, K, chunks, bs, mask, n_pages, \
                           err, sink, slopes);
    ROWS(64, 1) ROWS(64, 2) ROWS(64, 4) ROWS(128, 1) ROWS(128, 2) ROWS(128, 4)
#undef ROWS
    return (int)cudaErrorInvalidValue;
}

// Tiles of TT tokens of one request x GH query heads of one key/value head, TT * GH <= 32.
RLLM_API int rllm_attn_f32_tiles(const float* q, const float* k_cache, const float* v_cache, float* out, const int* positions,
                                 const int* cu_q, const int* tile_req, const int* tile_tok0, int n_tiles, int TT, int GH,
                                 int head_chunks, const int* block_table, int table_stride, int H, int K, int hd, int bs, float scale,
                                 int window, int keep_first, int chunk, float softcap, int n_pages, int* err, const float* sink,
                                 const float* slopes, cudaStream_t stream) {
    if (n_tiles <= 0) return 0;
    if (!f32_shape_ok(H, K, hd, bs, keep_first, chunk) || TT < 1 || GH < 1 || TT * GH > A32_ROWS || GH * head_chunks < H / K)
        return (int)cudaErrorInvalidValue;
    const F32Mask mask = {scale, softcap, window, keep_first, chunk};
#define TILES(HD)                                                                                                              \
    if (hd == HD) {                                                                                                            \
        const int e = (int)cudaFuncSetAttribute(attn_f32_tile_kernel<HD>, cudaFuncAttributeMaxDynamicSharedMemorySize,          \
                                                (int)sizeof(TileShared<HD>));                                                  \
        if (e) return e;                                                                                                       \
        return rllm_launch_after(attn_f32_tile_kernel<HD>, dim3(n_tiles, K * head_chunks), dim3(128), sizeof(TileShared<HD>), stream, \
                           q, k_cache, v_cache, out, positions, cu_q, tile_req, tile_tok0, block_table, table_stride, H, K, TT, \
                           GH, head_chunks, bs, mask, n_pages, err, sink, slopes);                                              \
    }
    TILES(64) TILES(128)
#undef TILES
    return (int)cudaErrorInvalidValue;
}

// the packed-argument forms (common.cuh) for the host runtime's replay of recorded launches
RLLM_PACKED(rllm_attn_f32_rows)
RLLM_PACKED(rllm_attn_f32_tiles)
