// The float32 product C[m,n] (+)= A[m,k] . W[n,k]^T with float32 multiply-add: the path that every float32
// model takes.  Two kernels, ONE order of summation, so that a row's bits depend neither on m nor on the kernel:
//
//   the k axis is dealt out in runs of 8 to 32 classes (class of element e: (e / 8) mod 32); a class's sum is one
//   chain of fused multiply-adds over its elements in ascending order, and the 32 class sums are added one after
//   the other, class 0 first.  (A chain of k/32 terms and a chain of 32 instead of one of k: a smaller error.)
//
// gemv_f32_kernel, up to GEMV_ROWS rows: bound by the bytes of W.  A warp takes NR rows of W, a lane is a class, so
// a warp reads whole lines of W and no W element passes through shared memory; NR * U = 4 row segments of 1 KB are
// in flight per warp.  NR grows with the rows of A because each 32 bytes of A that come out of L1 then serve NR
// rows of W (22 bytes per clock and SM of W leave L1 room for about four times as many bytes of A).
//
// gemm_f32_kernel, more rows: bound by the FMA pipe (74 TFLOP/s).  cp.async tiles of 16 k values (two runs, of one class
// or of two neighbours) in rows of 20 floats: eight rows' float4 then lie in eight different 16-byte bank groups, so no
// transposition is needed and every shared-memory read of a warp is one wavefront.  Per 4 k values a thread reads
// TM + TN float4 for TM * TN * 4 multiply-adds.  128 x 64 tiles (8 x 8 a thread) where they fill the SMs, 64 x 64 (4 x 8) where
// they do and there are no more rows than that, else 64 x 32 (4 x 4): a launch of fewer blocks than SMs is as slow as its
// one block.
//
// Measured in place of one kernel for every shape (64 x 64 tiles, one chain over k, 16 shared-memory reads of 4 bytes per
// 16 multiply-adds, a block per 64 columns also for a single row): float32 requests of 300 and 161 tokens at the 0.6B
// sizes with 8 decode steps 258 -> 65.5 ms; the head of 151,936 x 1,024 for one row 94 us (6.6 TB/s), 4,096 columns of
// 1,024 for 1,024 rows 30 TFLOP/s.
//
// Both are launched behind the kernel before, not early beside its end: they fill the SMs, and blocks that wait there keep
// the rest of the kernel before from its place (the same requests 39.3 ms launched early, 36.9 ms so).
#include "common.cuh"

#define F32_CLASSES 32
#define F32_RUN 8
#define F32_STEP (F32_CLASSES * F32_RUN)
#define GEMV_WARPS 8

// ---------------------------------------------------------------- few rows

// 8 elements of a row from element e on; what lies behind k reads as zero.
template <bool VEC>
__device__ __forceinline__ void load_run(float (&r)[F32_RUN], const float* row, int e, int k) {
    if (VEC) {                                      // k is a multiple of 4 and the row starts on 16 bytes
        float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
        if (e < k) a = *reinterpret_cast<const float4*>(row + e);
        if (e + 4 < k) b = *reinterpret_cast<const float4*>(row + e + 4);
        r[0] = a.x; r[1] = a.y; r[2] = a.z; r[3] = a.w;
        r[4] = b.x; r[5] = b.y; r[6] = b.z; r[7] = b.w;
    } else {
#pragma unroll
        for (int i = 0; i < F32_RUN; ++i) r[i] = e + i < k ? row[e + i] : 0.f;
    }
}

template <int M, int NR, int U, bool VEC>
__global__ void __launch_bounds__(GEMV_WARPS * 32, M >= 4 ? 2 : 3)
gemv_f32_kernel(const float* A, const float* W, float* C, int m, int n, int k, int lda, int ldw, int ldc, int accumulate,
                long long sa, long long sw, long long sc) {
    __shared__ float part[GEMV_WARPS][M * NR][F32_CLASSES + 1];
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int m0 = blockIdx.y * M;
    A += (size_t)blockIdx.z * sa + (size_t)m0 * lda;
    W += (size_t)blockIdx.z * sw;
    C += (size_t)blockIdx.z * sc + (size_t)m0 * ldc;
    const int rows = min(M, m - m0);
    const int groups = (n + NR - 1) / NR;
    const float* arow[M];
#pragma unroll
    for (int i = 0; i < M; ++i) arow[i] = A + (size_t)min(i, rows - 1) * lda;
    for (int g = blockIdx.x * GEMV_WARPS + warp; g < groups; g += gridDim.x * GEMV_WARPS) {
        const float* wrow[NR];
#pragma unroll
        for (int j = 0; j < NR; ++j) wrow[j] = W + (size_t)min(g * NR + j, n - 1) * ldw;
        // the lane that writes an output also fetches the value it adds to, ahead of the loop
        const int oi = lane / NR, oj = g * NR + lane % NR;
        const bool writes = lane < M * NR && oi < rows && oj < n;
        float old = 0.f;
        if (writes && accumulate) old = C[(size_t)oi * ldc + oj];
        float acc[M][NR];
#pragma unroll
        for (int i = 0; i < M; ++i)
#pragma unroll
            for (int j = 0; j < NR; ++j) acc[i][j] = 0.f;
        for (int e0 = lane * F32_RUN; e0 < k; e0 += U * F32_STEP) {
            float w[U][NR][F32_RUN];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int j = 0; j < NR; ++j) load_run<VEC>(w[u][j], wrow[j], e0 + u * F32_STEP, k);
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int i = 0; i < M; ++i) {
                    float a[F32_RUN];
                    load_run<VEC>(a, arow[i], e0 + u * F32_STEP, k);
#pragma unroll
                    for (int x = 0; x < F32_RUN; ++x)
#pragma unroll
                        for (int j = 0; j < NR; ++j) acc[i][j] = fmaf(a[x], w[u][j][x], acc[i][j]);
                }
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < M; ++i)
#pragma unroll
            for (int j = 0; j < NR; ++j) part[warp][i * NR + j][lane] = acc[i][j];
        __syncwarp();
        if (writes) {
            float t = 0.f;
#pragma unroll
            for (int c = 0; c < F32_CLASSES; ++c) t += part[warp][lane][c];
            C[(size_t)oi * ldc + oj] = t + old;
        }
    }
}

// ---------------------------------------------------------------- many rows

#define GEMM_BK 16
#define GEMM_LD 20
#define GEMM_STAGES 3

__device__ __forceinline__ void copy_async16(uint32_t dst, const float* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void copy_async4(uint32_t dst, const float* src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// TY x TX threads of TM x TN outputs; a thread's rows are ty + TY * i, its columns tx + TX * j.
template <int TY, int TX, int TM, int TN, bool VEC>
__global__ void __launch_bounds__(TY * TX)
gemm_f32_kernel(const float* A, const float* W, float* C, int m, int n, int k, int lda, int ldw, int ldc, int accumulate,
                long long sa, long long sw, long long sc) {
    constexpr int BM = TY * TM, BN = TX * TN, THREADS = TY * TX, ROWS = BM + BN;
    __shared__ __align__(16) float tile[GEMM_STAGES][ROWS * GEMM_LD];
    pdl_wait();
    const int tid = threadIdx.x;
    // a warp covers 4 rows x 8 columns of threads: its stores fill 32-byte sectors
    const int lane = tid & 31, warp = tid >> 5;
    constexpr int WX = TX / 8;
    const int tx = (warp % WX) * 8 + (lane & 7), ty = (warp / WX) * 4 + (lane >> 3);
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    A += (size_t)blockIdx.z * sa;
    W += (size_t)blockIdx.z * sw;
    C += (size_t)blockIdx.z * sc;

    const int per_class = (k + F32_STEP - 1) / F32_STEP;                      // runs of one class
    const int runs = per_class * min(F32_CLASSES, (k + F32_RUN - 1) / F32_RUN);
    const int tiles = (runs + 1) / 2;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(&tile[0][0]);

    constexpr int PARTS = VEC ? GEMM_BK / 4 : GEMM_BK;                        // copies per row of a tile
    const int f = tid % PARTS * (GEMM_BK / PARTS);                            // a thread's place in its rows
    auto fetch = [&](int t) {
        // the tile's runs: number 2 t and the next one, of the same class or of the class behind it
        const int q0 = 2 * t / per_class, p0 = 2 * t - q0 * per_class;
        const bool turns = p0 + 1 == per_class;
        const int e0 = p0 * F32_STEP + q0 * F32_RUN, e1 = 2 * t + 1 == runs ? k : turns ? (q0 + 1) * F32_RUN : e0 + F32_STEP;
        const uint32_t to = base + (t % GEMM_STAGES) * (ROWS * GEMM_LD * 4);
        const int e = (f < F32_RUN ? e0 : e1) + f % F32_RUN;
#pragma unroll
        for (int r = tid / PARTS; r < ROWS; r += THREADS / PARTS) {
            const bool is_a = r < BM;
            const int row = is_a ? m0 + r : n0 + r - BM;
            const bool in = row < (is_a ? m : n) && e < k;
            const float* src = is_a ? A : W;
            if (in) src += (size_t)row * (is_a ? lda : ldw) + e;
            const uint32_t dst = to + (r * GEMM_LD + f) * 4;
            if (VEC) copy_async16(dst, src, in ? 16 : 0);
            else copy_async4(dst, src, in ? 4 : 0);
        }
    };

    float acc[TM][TN], total[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = total[i][j] = 0.f;

#pragma unroll
    for (int s = 0; s < GEMM_STAGES - 1; ++s) {
        if (s < tiles) fetch(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    int left = per_class;
    for (int t = 0; t < tiles; ++t) {
        asm volatile("cp.async.wait_group %0;" ::"n"(GEMM_STAGES - 2) : "memory");
        __syncthreads();                                   // tile t has arrived; nobody reads tile t - 1 any more
        if (t + GEMM_STAGES - 1 < tiles) fetch(t + GEMM_STAGES - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* as = tile[t % GEMM_STAGES] + ty * GEMM_LD;
        const float* ws = tile[t % GEMM_STAGES] + (BM + tx) * GEMM_LD;
#pragma unroll
        for (int f = 0; f < GEMM_BK; f += 4) {
            float4 a[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(as + i * TY * GEMM_LD + f);
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const float4 w = *reinterpret_cast<const float4*>(ws + j * TX * GEMM_LD + f);
#pragma unroll
                for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].x, w.x, acc[i][j]);
#pragma unroll
                for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].y, w.y, acc[i][j]);
#pragma unroll
                for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].z, w.z, acc[i][j]);
#pragma unroll
                for (int i = 0; i < TM; ++i) acc[i][j] = fmaf(a[i].w, w.w, acc[i][j]);
            }
            if (f % F32_RUN != 0 && --left == 0) {         // a run ends, and the class with it
                left = per_class;
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) {
                        total[i][j] += acc[i][j];
                        acc[i][j] = 0.f;
                    }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int row = m0 + ty + TY * i;
        if (row >= m) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int col = n0 + tx + TX * j;
            if (col >= n) continue;
            float* c = C + (size_t)row * ldc + col;
            *c = total[i][j] + (accumulate ? *c : 0.f);
        }
    }
}

// ---------------------------------------------------------------- launch

// Rows up to which W is streamed by warps (in groups of 8 rows of A, each of which reads W again, from L2 where it fits):
// 16 rows of 6,144 x 1,024 take 17 us this way, 24 rows take 53 us in tiles, which are mostly empty then.
#define GEMV_ROWS 16
// With less k most lanes of the streaming kernel have nothing to do: 16 rows of 8,192 x 16 take 5.7 us streamed, 2.5 in tiles.
#define GEMV_MIN_K 32
// Products of so little k are over before their blocks could be in the way: launched early, 16 rows of 8,192 x 16 2.85 -> 2.5 us.
#define EARLY_MAX_K 64

RLLM_API int rllm_gemm_f32_batched(const float* A, const float* W, float* C, int m, int n, int k, int lda, int ldw, int ldc,
                                   int accumulate, int batch, long long sa, long long sw, long long sc, cudaStream_t stream) {
    if (m <= 0 || n <= 0 || batch <= 0) return 0;
    if (k <= 0 || batch > 65535) return (int)cudaErrorInvalidValue;
    const bool vec = ((uintptr_t)A | (uintptr_t)W) % 16 == 0 && (k | lda | ldw) % 4 == 0 && (batch == 1 || (sa | sw) % 4 == 0);
    const int n_sm = rllm_sm_count();
#define GEMV(M, NR, U)                                                                                                   \
    {                                                                                                                    \
        const int need = ((n + NR - 1) / NR + GEMV_WARPS - 1) / GEMV_WARPS, most = n_sm * (M >= 4 ? 2 : 3);               \
        dim3 grid(need < most ? need : most, (m + M - 1) / M, batch);                                                     \
        return vec ? rllm_launch_after(gemv_f32_kernel<M, NR, U, true>, grid, dim3(GEMV_WARPS * 32), 0, stream, A, W, C, m, n,  \
                                 k, lda, ldw, ldc, accumulate, sa, sw, sc)                                                \
                   : rllm_launch_after(gemv_f32_kernel<M, NR, U, false>, grid, dim3(GEMV_WARPS * 32), 0, stream, A, W, C, m, n, \
                                 k, lda, ldw, ldc, accumulate, sa, sw, sc);                                               \
    }
    if (m <= GEMV_ROWS && k > GEMV_MIN_K) {
        if (m == 1) GEMV(1, 1, 4)
        if (m == 2) GEMV(2, 1, 4)
        if (m <= 4) GEMV(4, 2, 2)
        GEMV(8, 4, 1)
    }
#undef GEMV
#define GEMM(TY, TX, TM, TN)                                                                                             \
    {                                                                                                                    \
        dim3 grid((n + TX * TN - 1) / (TX * TN), (m + TY * TM - 1) / (TY * TM), batch);                                   \
        auto kern = vec ? gemm_f32_kernel<TY, TX, TM, TN, true> : gemm_f32_kernel<TY, TX, TM, TN, false>;                 \
        if (k <= EARLY_MAX_K)                                                                                            \
            return rllm_launch(kern, grid, dim3(TY * TX), 0, stream, A, W, C, m, n, k, lda, ldw, ldc, accumulate, sa, sw, sc); \
        return rllm_launch_after(kern, grid, dim3(TY * TX), 0, stream, A, W, C, m, n, k, lda, ldw, ldc, accumulate, sa, sw, sc); \
    }
    const long long large = (long long)((n + 63) / 64) * ((m + 127) / 128) * batch;
    if (large >= n_sm) {
        if (m > 64) GEMM(16, 8, 8, 8)
        GEMM(16, 8, 4, 8)
    }
    GEMM(16, 8, 4, 4)
#undef GEMM
}
