// Paged causal attention of the float32 path for key and value heads of 64 or 128: the function that
// attention_generic.cu computes (masks, caps, slopes and sinks as its head describes them), with float32 arithmetic
// throughout, for the shapes in which a block per (token, head) that reads its keys from memory by itself is slow.
//
// Both kernels give a token the same bits, so its result depends on its own keys alone: not on the requests around it, not on
// how its prompt was cut into portions, not on which of the two ran.  The order that they share: keys in chunks of 32 that
// start at multiples of 32 of the position (those of the kept first keys, then those of the window), and per chunk
//   a score  eight sums, lane q of eight over the entries 4 (q + 8 x) .. + 3 in ascending order, added as a tree of pairs;
//   M        the largest score so far, this chunk's included;
//   the sum  of the weights exp(s - M): four keys 8 apart one after the other, then a tree of pairs over the eight;
//   o        the weighted values: one chain over the keys for heads of 128, one each over even and odd keys for heads of 64;
//   l = l * exp(M before - M) + sum,  acc = acc * exp(M before - M) + o   (one fused multiply-add each).
// A key that a row does not see adds nothing to it, not even where its value is infinite.  Scores of -inf weigh nothing beside
// finite ones wherever those are.
//
// attn_f32_rows_kernel: bound by the latency of the key and value reads.  A block per (token, key/value head and up to 4 of its
// query heads); its warps take one chunk each, eight lanes read one key's row in whole lines, and a round of chunks is
// merged in order by all threads.  M is known before the weights are worked out (a maximum has no order), so only the
// merge is a chain.
//
// attn_f32_tile_kernel: 32 rows (tokens x query heads of one key/value head) against tiles of 32 keys, which cp.async brings
// in one tile ahead; rows of 132 floats keep the reads of eight keys in different banks.  Keys are read once per 32 rows,
// but a tile's keys are one chain on one SM, 4.8 us each.
//
// Measured (head size 128, 16 query heads on 8) against the plain kernel, us a launch: two decoding requests of 300 keys
// 38 -> 7.0, of 4,096 471 -> 46, 32 of 300 102 -> 17; one portion of 461 tokens 964 -> 89, two of 300 793 -> 61.
#include "common.cuh"
#include <math.h>

#define A32_KEYS 32
#define A32_MAX_WARPS 16
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
// (written out, so that both kernels round alike)
__device__ __forceinline__ float shape_score(const F32Mask& k, float dot, const float* slopes, int head, int distance) {
    float s = __fmul_rn(dot, k.scale);
    if (k.softcap > 0.f) s = __fmul_rn(k.softcap, tanhf(s / k.softcap));
    if (slopes) s = fmaf(-slopes[head], (float)distance, s);
    return s;
}
// the factor of what was summed up to a largest score of `before` when it has become `now`
__device__ __forceinline__ float rescale(float before, float now) { return before == -INFINITY ? 0.f : expf(before - now); }
// the weight of score s (-inf only: nothing seen yet, every weight zero)
__device__ __forceinline__ float weight(float s, float top) { return expf(s - (top == -INFINITY ? 0.f : top)); }
__device__ __forceinline__ float dot4(float4 a, float4 b, float c) {
    return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, c))));
}

// four entries of the row that starts at `off`; zeros (and no access) for a key that is not seen
__device__ __forceinline__ float4 load_or_zero(const float* cache, long long off, int at) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (off >= 0) v = *reinterpret_cast<const float4*>(cache + off + at);
    return v;
}

// ---------------------------------------------------------------- token by token

// dynamic shared memory, in floats: q [G][HD], scores and weights [warps][G][32], o [warps][G][HD], the warps' largest score,
// factor and sum [3][warps][G]
static size_t rows_smem(int hd, int G, int warps) { return (size_t)(G * hd + warps * G * (A32_KEYS + hd + 3)) * sizeof(float); }

template <int HD, int G>
__global__ void __launch_bounds__(A32_MAX_WARPS * 32)
attn_f32_rows_kernel(const float* q, const float* k_cache, const float* v_cache, float* out, const int* __restrict__ positions,
                     const int* __restrict__ seq_ids, const int* __restrict__ tokens, const int* __restrict__ block_table,
                     int table_stride, int H, int K, int head_chunks, int bs, F32Mask mask, int n_pages, int* err,
                     const float* __restrict__ sink, const float* __restrict__ slopes) {
    constexpr int X = HD / 32;                     // float4 of a key row per lane, eight lanes a key
    constexpr int LPK = HD / 4, KPP = 32 / LPK;    // lanes per value row, value rows at a time
    constexpr int PB = 16 / X;                     // passes (of four keys) whose loads are in flight together
    constexpr int VB = 16;                         // value rows in flight
    constexpr int PER = (G * HD + 127) / 128;      // outputs a thread merges, at most (blocks have 128 threads or more)
    extern __shared__ __align__(16) float shared[];
    const int threads = blockDim.x, warps = threads >> 5, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    float* sq = shared;
    float* sc = sq + G * HD + warp * (G * A32_KEYS);
    float* os = sq + G * HD + warps * (G * A32_KEYS);
    float* s_top = os + warps * (G * HD);
    float* s_factor = s_top + warps * G;
    float* s_sum = s_factor + warps * G;
    pdl_wait();
    const int t = tokens[blockIdx.x];
    const int kvh = blockIdx.y / head_chunks, g = H / K, g0 = (blockIdx.y % head_chunks) * G;
    const int pos = positions[t], first = first_key(mask, pos);
    const int* table = block_table + (size_t)seq_ids[t] * table_stride;
    const int kept = min(mask.keep_first, first);
    for (int x = tid; x < G * LPK; x += threads) {
        const int h = kvh * g + min(g0 + x / LPK, g - 1);
        reinterpret_cast<float4*>(sq)[x] = reinterpret_cast<const float4*>(q + ((size_t)t * H + h) * HD)[x % LPK];
    }
    float m_run[G], acc[PER], l[PER];
#pragma unroll
    for (int j = 0; j < G; ++j) m_run[j] = sink ? sink[kvh * g + min(g0 + j, g - 1)] : -INFINITY;
#pragma unroll
    for (int r = 0; r < PER; ++r) {
        acc[r] = 0.f;
        l[r] = sink ? 1.f : 0.f;
    }
    __syncthreads();

    const int n_kept = (kept + A32_KEYS - 1) / A32_KEYS, c_first = first / A32_KEYS;
    const int n_chunks = n_kept + pos / A32_KEYS + 1 - c_first;
    // where the row of this lane's key of chunk c starts, -1: the key is not seen
    auto row_of = [&](int c, int& p) -> long long {
        const bool in_kept = c < n_kept;
        const int lo = in_kept ? 0 : first, hi = in_kept ? kept : pos + 1;
        p = (in_kept ? c : c_first + c - n_kept) * A32_KEYS + lane;
        if (c >= n_chunks || p < lo || p >= hi) return -1;
        return (((long long)page_of(table, p, bs, n_pages, err) * K + kvh) * bs + p % bs) * HD;
    };
    int p, p_next;
    long long off_next = row_of(warp, p_next);
    for (int base = 0; base < n_chunks; base += warps) {
        const int n_live = min(warps, n_chunks - base);
        const bool live = warp < n_live;
        const long long off = off_next;
        p = p_next;
        const bool seen = off >= 0;
        const uint32_t any = __ballot_sync(0xffffffffu, seen);       // runs of keys of which none is seen are passed over
        float s[G];
        float4 v[VB];
        auto load_values = [&](int i0) {
#pragma unroll
            for (int b = 0; b < VB; ++b)
                v[b] = load_or_zero(v_cache, __shfl_sync(0xffffffffu, off, i0 + b * KPP + lane / LPK), 4 * (lane % LPK));
        };
        if (live) {
#pragma unroll
            for (int i0 = 0; i0 < 8; i0 += PB) {
                if (!(any >> (4 * i0) & (uint32_t)((1ull << (4 * PB)) - 1))) continue;
                float4 kv[PB][X];
#pragma unroll
                for (int b = 0; b < PB; ++b) {
                    const long long o = __shfl_sync(0xffffffffu, off, 4 * (i0 + b) + (lane >> 3));
#pragma unroll
                    for (int x = 0; x < X; ++x) kv[b][x] = load_or_zero(k_cache, o, 4 * ((lane & 7) + 8 * x));
                }
#pragma unroll
                for (int j = 0; j < G; ++j) {
                    float d[PB];
#pragma unroll
                    for (int b = 0; b < PB; ++b) d[b] = 0.f;
#pragma unroll
                    for (int x = 0; x < X; ++x) {
                        const float4 qv = reinterpret_cast<const float4*>(sq)[j * LPK + (lane & 7) + 8 * x];
#pragma unroll
                        for (int b = 0; b < PB; ++b) d[b] = dot4(qv, kv[b][x], d[b]);
                    }
#pragma unroll
                    for (int b = 0; b < PB; ++b) {
                        d[b] += __shfl_xor_sync(0xffffffffu, d[b], 1);
                        d[b] += __shfl_xor_sync(0xffffffffu, d[b], 2);
                        d[b] += __shfl_xor_sync(0xffffffffu, d[b], 4);
                        if ((lane & 7) == j) sc[j * A32_KEYS + 4 * (i0 + b) + (lane >> 3)] = d[b];
                    }
                }
            }
            __syncwarp();
#pragma unroll
            for (int j = 0; j < G; ++j) {
                s[j] = seen ? shape_score(mask, sc[j * A32_KEYS + lane], slopes, kvh * g + min(g0 + j, g - 1), pos - p) : -INFINITY;
                const float top = warp_max(s[j]);
                if (lane == 0) s_top[warp * G + j] = top;
            }
            load_values(0);                        // on their way while the block meets
        }
        off_next = row_of(base + warps + warp, p_next);
        __syncthreads();                           // the round's maxima are there
#pragma unroll
        for (int j = 0; j < G; ++j) {
            const float v = lane < n_live ? s_top[lane * G + j] : -INFINITY;
            const float before = fmaxf(m_run[j], warp_max(lane < warp ? v : -INFINITY));
            m_run[j] = fmaxf(m_run[j], warp_max(v));
            if (live) {
                const float now = fmaxf(before, s_top[warp * G + j]);
                sc[j * A32_KEYS + lane] = seen ? weight(s[j], now) : 0.f;
                if (lane == 0) s_factor[warp * G + j] = rescale(before, now);
            }
        }
        __syncwarp();
        if (live) {
            float4 o[G];
#pragma unroll
            for (int j = 0; j < G; ++j) {
                const float* e = sc + j * A32_KEYS + (lane & 7);
                float sum = e[0] + e[8] + e[16] + e[24];
                sum += __shfl_xor_sync(0xffffffffu, sum, 1);
                sum += __shfl_xor_sync(0xffffffffu, sum, 2);
                sum += __shfl_xor_sync(0xffffffffu, sum, 4);
                if (lane == 0) s_sum[warp * G + j] = sum;
                o[j] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int i0 = 0; i0 < A32_KEYS; i0 += VB * KPP) {
                if (i0 > 0) {
                    if (!(any >> i0)) continue;
                    load_values(i0);
                }
#pragma unroll
                for (int b = 0; b < VB; ++b)
#pragma unroll
                    for (int j = 0; j < G; ++j) {
                        const float e = sc[j * A32_KEYS + i0 + b * KPP + lane / LPK];
                        o[j].x = fmaf(e, v[b].x, o[j].x); o[j].y = fmaf(e, v[b].y, o[j].y);
                        o[j].z = fmaf(e, v[b].z, o[j].z); o[j].w = fmaf(e, v[b].w, o[j].w);
                    }
            }
#pragma unroll
            for (int j = 0; j < G; ++j) {
                if (KPP == 2) {
                    o[j].x += __shfl_xor_sync(0xffffffffu, o[j].x, 16); o[j].y += __shfl_xor_sync(0xffffffffu, o[j].y, 16);
                    o[j].z += __shfl_xor_sync(0xffffffffu, o[j].z, 16); o[j].w += __shfl_xor_sync(0xffffffffu, o[j].w, 16);
                }
                if (lane < LPK) *reinterpret_cast<float4*>(os + (warp * G + j) * HD + 4 * lane) = o[j];
            }
        }
        __syncthreads();                           // the round's parts are there; they are written again behind the next barrier but one
#pragma unroll
        for (int r = 0; r < PER; ++r) {
            const int x = tid + r * threads, j = x / HD;
            if (x >= G * HD) break;
            for (int w = 0; w < n_live; ++w) {
                const float f = s_factor[w * G + j];
                acc[r] = fmaf(acc[r], f, os[w * (G * HD) + x]);
                l[r] = fmaf(l[r], f, s_sum[w * G + j]);
            }
        }
    }
    pdl_launch_dependents();
#pragma unroll
    for (int r = 0; r < PER; ++r) {
        const int x = tid + r * threads, j = x / HD;
        if (x >= G * HD) break;
        if (g0 + j < g) out[((size_t)t * H + kvh * g + g0 + j) * HD + x % HD] = acc[r] * (1.0f / l[r]);
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
    float p[A32_ROWS][A32_KEYS + 4];               // weights; -1 where the row does not see the key
    float alpha[A32_ROWS];
    float l[A32_ROWS];
};

template <int HD>
__global__ void __launch_bounds__(128, HD == 64 ? 4 : 2)      // as many as shared memory allows
attn_f32_tile_kernel(const float* q, const float* k_cache, const float* v_cache, float* out, const int* __restrict__ positions,
                     const int* __restrict__ cu_q, const int* __restrict__ tile_req, const int* __restrict__ tile_tok0,
                     const int* __restrict__ block_table, int table_stride, int H, int K, int TT, int GH, int head_chunks, int bs,
                     F32Mask mask, int n_pages, int* err, const float* __restrict__ sink, const float* __restrict__ slopes) {
    extern __shared__ __align__(16) unsigned char raw[];
    TileShared<HD>& sm = *reinterpret_cast<TileShared<HD>*>(raw);
    constexpr int F4 = HD / 4, C4 = HD / 64, KPP = 128 / HD;
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
        // the eight sums of a score, as a tree of pairs
        float s[2][4];
        auto part = [&](int q, float (&d)[2][4]) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) d[i][j] = 0.f;
#pragma unroll
            for (int f = 4 * q; f < HD; f += 32) {
                float4 a[2], b[4];
#pragma unroll
                for (int i = 0; i < 2; ++i) a[i] = *reinterpret_cast<const float4*>(&sm.q[rs + 16 * i][f]);
#pragma unroll
                for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(&sm.k[t & 1][ks + 8 * j][f]);
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) d[i][j] = dot4(a[i], b[j], d[i][j]);
            }
        };
        auto add = [](float (&to)[2][4], const float (&d)[2][4]) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) to[i][j] += d[i][j];
        };
#pragma unroll
        for (int q = 0; q < 8; q += 4) {
            float d0[2][4], d1[2][4], d2[2][4];
            part(q, d0); part(q + 1, d1);
            add(d0, d1);
            part(q + 2, d1); part(q + 3, d2);
            add(d1, d2);
            add(d0, d1);
            if (q == 0) {
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) s[i][j] = d0[i][j];
            } else add(s, d0);
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
            const float alpha = rescale(m_run[i], m_new);
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int p = c0 + ks + 8 * j;
                const bool seen = p >= lo && p < hi;
                const float e = seen ? weight(s[i][j], m_new) : 0.f;
                sm.p[rs + 16 * i][ks + 8 * j] = seen ? e : -1.f;
                sum += e;
            }
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            sum += __shfl_xor_sync(0xffffffffu, sum, 4);
            l_run[i] = fmaf(l_run[i], alpha, sum);
            m_run[i] = m_new;
            if (ks == 0) sm.alpha[rs + 16 * i] = alpha;
        }
        __syncthreads();                                  // weights and factors are there
        // every pair of the tile is seen where the last key is at or before the first row and the first key is in all rows' windows
        const bool whole = !kept_run && c0 + A32_KEYS - 1 <= pos0 && c0 >= first_key(mask, pos1);
        float4 o[KPP][4][C4];                             // heads of 64: even and odd keys apart
#pragma unroll
        for (int e = 0; e < KPP; ++e)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < C4; ++j) o[e][i][j] = make_float4(0.f, 0.f, 0.f, 0.f);
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
                        float4& to = o[x % KPP][i][j];
                        if (whole || !(e < 0.f)) {
                            to.x = fmaf(e, v.x, to.x); to.y = fmaf(e, v.y, to.y);
                            to.z = fmaf(e, v.z, to.z); to.w = fmaf(e, v.w, to.w);
                        }
                    }
                }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float f = sm.alpha[ro + 8 * i];
#pragma unroll
            for (int j = 0; j < C4; ++j) {
                float4 v = o[0][i][j];
                if (KPP == 2) { v.x += o[KPP - 1][i][j].x; v.y += o[KPP - 1][i][j].y; v.z += o[KPP - 1][i][j].z; v.w += o[KPP - 1][i][j].w; }
                acc[i][j].x = fmaf(acc[i][j].x, f, v.x); acc[i][j].y = fmaf(acc[i][j].y, f, v.y);
                acc[i][j].z = fmaf(acc[i][j].z, f, v.z); acc[i][j].w = fmaf(acc[i][j].w, f, v.w);
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
    // keys that a token can see, from the table's width; a warp per chunk of them up to 16 (the order does not depend on it)
    long long span = (long long)table_stride * bs;
    if (chunk > 0 && (long long)chunk + keep_first < span) span = (long long)chunk + keep_first;
    if (window > 0 && (long long)window + keep_first < span) span = (long long)window + keep_first;
    const int warps = span <= 4 * A32_KEYS ? 4 : span <= 8 * A32_KEYS ? 8 : A32_MAX_WARPS;
    // Query heads per block: as few as still run all at once (16 warps of 128 registers fill an SM), so that a block's chain is
    // short; up to four share the reads of their keys otherwise.  (One token of 32 heads on 8: with four heads a block 9.3 us
    // for one key and 88 for 4,096, with one 4.1 and 46.)
    const int g = H / K;
    const long long slots = (long long)rllm_sm_count() * (A32_MAX_WARPS / warps);
    int G = 1;
    while (G < 4 && G < g && (long long)n_tokens * K * ((g + G - 1) / G) > slots) G *= 2;
    const int chunks = (g + G - 1) / G;
#define ROWS(HD, GG)                                                                                                            \
    if (hd == HD && G == GG)                                                                                                    \
        return rllm_launch_after(attn_f32_rows_kernel<HD, GG>, dim3(n_tokens, K * chunks), dim3(warps * 32),                     \
                                 rows_smem(HD, GG, warps), stream, q, k_cache, v_cache, out, positions, seq_ids, tokens,         \
                                 block_table, table_stride, H, K, chunks, bs, mask, n_pages, err, sink, slopes);
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
