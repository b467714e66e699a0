// True fp32 matrix product for the 32-bit path: C[M,N] = A[M,K] . W[N,K]^T.
//
// Plain FFMA on CUDA cores, no tensor-core mode of any kind. Each output
// element is one chain of fused multiply-adds over k = 0..K-1 in ascending
// order, so its bits depend only on its row of A and its row of W: not on M,
// not on the tile it falls in, not on what else is in the batch. That makes
// the 32-bit path bit-stable under every way of cutting the work, which is
// what lets it expose faults of the cache or the batch. All three kernels
// below walk the same chain, so which of them a size takes does not show.
//
// Weights are [out, in] row-major and y = W.x as in the reference
// (mynah-slm src/arch_qwen3.c:51-52).
#include "common.cuh"

namespace {

__device__ __forceinline__ void copy16(uint32_t dst, const float* src, bool valid) {
    const int n = valid ? 16 : 0;                                    // 0 source bytes: the 16 bytes are zero-filled
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(n));
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// A 16-byte read of shared memory that stays where it is written: ahead of the multiply-adds it is to hide behind, behind the barrier
// that says that the slab is there (the clobber: nothing that touches memory moves across it).
__device__ __forceinline__ float4 read16(uint32_t at) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at) : "memory");
    return v;
}

// ---- rows that are not 16-byte aligned, or no multiple of four long: scalar loads, any size

constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;   // 256 threads, 4x4 outputs each

__global__ void __launch_bounds__(256)
gemm_f32_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C,
                int M, int N, int K, int lda, int ldw, int ldc) {
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tx = tid % 16, ty = tid / 16;            // tx -> columns (n), ty -> rows (m)
    float acc[TM][TN] = {};

    // each thread stages 4 elements of A and 4 of W per k-slab
    const int lr = tid / 4;            // 0..63: row inside the tile
    const int lk = (tid % 4) * 4;      // 0,4,8,12: first k inside the slab

    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int k = k0 + lk + j;
            const int am = m0 + lr, wn = n0 + lr;
            As[lk + j][lr] = (am < M && k < K) ? A[(size_t)am * lda + k] : 0.f;
            Ws[lk + j][lr] = (wn < N && k < K) ? W[(size_t)wn * ldw + k] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; k++) {
            float a[TM], w[TN];
#pragma unroll
            for (int i = 0; i < TM; i++) a[i] = As[k][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; j++) w[j] = Ws[k][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; i++)
#pragma unroll
                for (int j = 0; j < TN; j++) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; i++) {
        const int m = m0 + ty * TM + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; j++) {
            const int n = n0 + tx * TN + j;
            if (n < N) C[(size_t)m * ldc + n] = acc[i][j];
        }
    }
}

// ---- many rows: tiles of BM x BN outputs, a thread TM x TN of them, slabs of 32 or 64 k brought by 16-byte asynchronous
// copies into three stages. Both operands stay as they lie in memory ([row][k], rows padded by 4 words, so that eight
// rows' 16-byte reads meet no bank twice); a thread reads four k of its TM + TN rows at a time, a step ahead of their use, and
// walks them in order. Bound by the reads of shared memory (four cycles of an SM for a warp's 16-byte read of sixteen rows, two for
// two) and by how few warps a product of few rows makes. us for 161 rows, 4,096 x 1,024 / 1,024 x 2,048 / 6,144 x 1,024 /
// 1,024 x 3,072 outputs x k: 73 / 64 / 74 / 90 with reads where they are used -> 55 / 46 / 72 / 66.

constexpr int GRID_ROWS = 65535;                                     // tiles of rows that a launch's grid can name
constexpr int TILE_STAGES = 3;

template <int BM, int BN, int TM, int TN, int SLAB>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C,
                     int M, int N, int K, int lda, int ldw, int ldc) {
    constexpr int PITCH = SLAB + 4, TX = BN / TN, THREADS = TX * (BM / TM), CHUNKS = (BM + BN) * (SLAB / 4);
    static_assert(CHUNKS % THREADS == 0, "whole rounds of copies");
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int slabs = (K + SLAB - 1) / SLAB;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(smem);

    auto fetch = [&](int s) {
        if (s < slabs) {
            const uint32_t stage = base + (uint32_t)(s % TILE_STAGES) * ((BM + BN) * PITCH * 4);
#pragma unroll
            for (int c = 0; c < CHUNKS / THREADS; c++) {
                const int i = tid + c * THREADS, row = i / (SLAB / 4), kc = (i % (SLAB / 4)) * 4, k = s * SLAB + kc;
                const bool is_a = row < BM;
                const int r = is_a ? m0 + row : n0 + row - BM;
                const bool ok = k < K && r < (is_a ? M : N);
                const float* src = is_a ? A + (ok ? (size_t)r * lda + k : 0) : W + (ok ? (size_t)r * ldw + k : 0);
                copy16(stage + (row * PITCH + kc) * 4, src, ok);
            }
        }
        copy_commit();                                               // (an empty group beyond the end keeps the count in step)
    };

    griddep_wait();
    float acc[TM][TN] = {};
#pragma unroll
    for (int s = 0; s < TILE_STAGES - 1; s++) fetch(s);
    for (int s = 0; s < slabs; s++) {
        copy_wait<TILE_STAGES - 2>();
        __syncthreads();                                             // slab s is there; slab s - 1 has been read by all
        fetch(s + TILE_STAGES - 1);
        // four k of the thread's rows a step; the next step's are on their way while these are multiplied
        const uint32_t a_at = base + (uint32_t)((s % TILE_STAGES) * ((BM + BN) * PITCH) + ty * PITCH) * 4;
        const uint32_t w_at = base + (uint32_t)((s % TILE_STAGES) * ((BM + BN) * PITCH) + (BM + tx) * PITCH) * 4;
        struct Piece { float4 a[TM], w[TN]; } piece[2];
        auto load = [&](Piece& p, int k) {
#pragma unroll
            for (int j = 0; j < TN; j++) p.w[j] = read16(w_at + (j * TX * PITCH + k) * 4);
#pragma unroll
            for (int i = 0; i < TM; i++) p.a[i] = read16(a_at + (i * (BM / TM) * PITCH + k) * 4);
        };
        load(piece[0], 0);
#pragma unroll
        for (int k = 0; k < SLAB; k += 4) {
            if (k + 4 < SLAB) load(piece[(k / 4 + 1) & 1], k + 4);
            const Piece& p = piece[(k / 4) & 1];
#pragma unroll
            for (int i = 0; i < TM; i++)
#pragma unroll
                for (int j = 0; j < TN; j++) acc[i][j] = fmaf(p.a[i].x, p.w[j].x, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TM; i++)
#pragma unroll
                for (int j = 0; j < TN; j++) acc[i][j] = fmaf(p.a[i].y, p.w[j].y, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TM; i++)
#pragma unroll
                for (int j = 0; j < TN; j++) acc[i][j] = fmaf(p.a[i].z, p.w[j].z, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TM; i++)
#pragma unroll
                for (int j = 0; j < TN; j++) acc[i][j] = fmaf(p.a[i].w, p.w[j].w, acc[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < TM; i++) {
        const int m = m0 + ty + i * (BM / TM);
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; j++) {
            const int n = n0 + tx + j * TX;
            if (n < N) C[(size_t)m * ldc + n] = acc[i][j];
        }
    }
}

template <int BM, int BN, int TM, int TN, int SLAB>
int launch_tile(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, cudaStream_t stream) {
    auto kern = gemm_f32_tile_kernel<BM, BN, TM, TN, SLAB>;
    constexpr int smem = TILE_STAGES * (BM + BN) * (SLAB + 4) * 4;
    if (smem > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e != cudaSuccess) return mynah_fail("gemm_f32: %s", cudaGetErrorString(e));
    }
    mynah_launch(kern, dim3(ceil_div(N, BN), ceil_div(M, BM)), dim3((BM / TM) * (BN / TN)), smem, stream, A, W, C, M, N, K, lda, ldw, ldc);
    return mynah_check_launch("gemm_f32");
}

// ---- a step's few rows (at most 16): bound by the weights' one pass over memory, and by the chain of K dependent
// multiply-adds (four cycles each: 2 us for K = 1,024), which no split may shorten. All threads of a CTA copy slabs of
// 128 k of its BN weight rows (and of the input rows) into a ring; one thread an output row and MR input rows
// multiplies. The weights' first slabs are asked for before the kernel in front has ended. Two rows of the 0.6B shape:
// 13 to 17 us a product of a layer and 107 us for the head (622 MB, 5.8 TB/s); with the scalar kernel 163 us a product.

constexpr int ROW_THREADS = 128, ROW_MAX_M = 16;

template <int BN, int MR, int STAGES, int ROW_SLAB>
__global__ void __launch_bounds__(ROW_THREADS)
gemm_f32_rows_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C,
                     int M, int N, int K, int lda, int ldw, int ldc) {
    constexpr int ROW_PITCH = ROW_SLAB + 4;
    extern __shared__ __align__(16) float smem[];
    const int tid = threadIdx.x, n0 = blockIdx.x * BN;
    const int groups = (M + MR - 1) / MR, rows_a = groups * MR;      // input rows, rounded up; those beyond M are zeros
    const int stage_words = (BN + rows_a) * ROW_PITCH;
    const int slabs = (K + ROW_SLAB - 1) / ROW_SLAB;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(smem);

    auto fetch_w = [&](int s) {
        const uint32_t stage = base + (uint32_t)(s % STAGES) * (stage_words * 4);
#pragma unroll
        for (int c = 0; c < BN * (ROW_SLAB / 4) / ROW_THREADS; c++) {
            const int i = tid + c * ROW_THREADS, row = i / (ROW_SLAB / 4), kc = (i % (ROW_SLAB / 4)) * 4, k = s * ROW_SLAB + kc;
            const bool ok = k < K && n0 + row < N;
            copy16(stage + (row * ROW_PITCH + kc) * 4, W + (ok ? (size_t)(n0 + row) * ldw + k : 0), ok);
        }
    };
    auto fetch_a = [&](int s) {
        const uint32_t stage = base + (uint32_t)(s % STAGES) * (stage_words * 4) + BN * ROW_PITCH * 4;
        for (int i = tid; i < rows_a * (ROW_SLAB / 4); i += ROW_THREADS) {
            const int row = i / (ROW_SLAB / 4), kc = (i % (ROW_SLAB / 4)) * 4, k = s * ROW_SLAB + kc;
            const bool ok = k < K && row < M;
            copy16(stage + (row * ROW_PITCH + kc) * 4, A + (ok ? (size_t)row * lda + k : 0), ok);
        }
    };
#pragma unroll
    for (int s = 0; s < STAGES - 1; s++)
        if (s < slabs) fetch_w(s);
    griddep_wait();
#pragma unroll
    for (int s = 0; s < STAGES - 1; s++) {
        if (s < slabs) fetch_a(s);
        copy_commit();                                               // (the first group holds all the weights' slabs too)
    }
    constexpr int AHEAD = MR == 4 ? 8 : 16;
    struct Piece {
        float4 w[AHEAD / 4], a[MR][AHEAD / 4];
        __device__ __forceinline__ void load(uint32_t wp, uint32_t ap, int k) {
#pragma unroll
            for (int i = 0; i < AHEAD / 4; i++) {
                w[i] = read16(wp + (k + 4 * i) * 4);
#pragma unroll
                for (int r = 0; r < MR; r++) a[r][i] = read16(ap + (r * ROW_PITCH + k + 4 * i) * 4);
            }
        }
        __device__ __forceinline__ void multiply(float (&acc)[MR]) const {
#pragma unroll
            for (int i = 0; i < AHEAD / 4; i++)
#pragma unroll
                for (int r = 0; r < MR; r++) {
                    acc[r] = fmaf(a[r][i].x, w[i].x, acc[r]);
                    acc[r] = fmaf(a[r][i].y, w[i].y, acc[r]);
                    acc[r] = fmaf(a[r][i].z, w[i].z, acc[r]);
                    acc[r] = fmaf(a[r][i].w, w[i].w, acc[r]);
                }
        }
    };
    const int n = tid % BN, mg = tid / BN;
    const bool works = mg < groups;
    float acc[MR] = {};
    for (int s = 0; s < slabs; s++) {
        copy_wait<STAGES - 2>();
        __syncthreads();
        if (s + STAGES - 1 < slabs) {
            fetch_w(s + STAGES - 1);
            fetch_a(s + STAGES - 1);
        } else if (s + STAGES - 1 == slabs) {
            griddep_launch_late();
        }
        copy_commit();
        if (works) {
            const uint32_t w = base + (uint32_t)((s % STAGES) * stage_words + n * ROW_PITCH) * 4;
            const uint32_t a = base + (uint32_t)((s % STAGES) * stage_words + (BN + mg * MR) * ROW_PITCH) * 4;
            if constexpr (BN == 16 && MR == 4) {
                // two CTAs an SM and more cover one another's reads; the registers of reading ahead only cost (16 rows, 6,144 x 1,024: 20.7 us
                // against 19.6; 9,728 x 2,560: 79.0 / 74.8; 12 rows of 16,384 x 1,024: 46.8 / 43.7; two rows of 6,144 x 1,024 the other way: 10.9 / 11.2)
                const float* wf = smem + (size_t)(s % STAGES) * stage_words + n * ROW_PITCH;
                const float* af = smem + (size_t)(s % STAGES) * stage_words + (BN + mg * MR) * ROW_PITCH;
#pragma unroll 8
                for (int k = 0; k < ROW_SLAB; k += 4) {
                    const float4 wv = *reinterpret_cast<const float4*>(wf + k);
#pragma unroll
                    for (int r = 0; r < MR; r++) {
                        const float4 av = *reinterpret_cast<const float4*>(af + r * ROW_PITCH + k);
                        acc[r] = fmaf(av.x, wv.x, acc[r]);
                        acc[r] = fmaf(av.y, wv.y, acc[r]);
                        acc[r] = fmaf(av.z, wv.z, acc[r]);
                        acc[r] = fmaf(av.w, wv.w, acc[r]);
                    }
                }
            } else {
                // the next AHEAD k are on their way from shared memory while these are multiplied
                Piece p0, p1;
                p0.load(w, a, 0);
#pragma unroll 1
                for (int k = 0; k < ROW_SLAB; k += 2 * AHEAD) {
                    p1.load(w, a, k + AHEAD);
                    p0.multiply(acc);
                    p0.load(w, a, min(k + 2 * AHEAD, ROW_SLAB - AHEAD));
                    p1.multiply(acc);
                }
            }
        }
    }
    if (works && n0 + n < N) {
#pragma unroll
        for (int r = 0; r < MR; r++)
            if (mg * MR + r < M) C[(size_t)(mg * MR + r) * ldc + n0 + n] = acc[r];
    }
}

template <int BN, int MR, int STAGES, int ROW_SLAB>
int launch_rows(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, cudaStream_t stream) {
    constexpr int ROW_PITCH = ROW_SLAB + 4;
    auto kern = gemm_f32_rows_kernel<BN, MR, STAGES, ROW_SLAB>;
    const int smem = STAGES * (BN + ceil_div(M, MR) * MR) * ROW_PITCH * 4;
    constexpr int most = STAGES * (BN + (MR == 4 ? ROW_MAX_M : MR)) * ROW_PITCH * 4;
    if (most > 48 * 1024) {
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
        if (e != cudaSuccess) return mynah_fail("gemm_f32: %s", cudaGetErrorString(e));
    }
    mynah_launch(kern, dim3(ceil_div(N, BN)), dim3(ROW_THREADS), smem, stream, A, W, C, M, N, K, lda, ldw, ldc);
    return mynah_check_launch("gemm_f32");
}

template <int BN, int STAGES, int SLAB>
int launch_rows_m(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, cudaStream_t stream) {
    if (M == 1) return launch_rows<BN, 1, STAGES, SLAB>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    if (M == 2) return launch_rows<BN, 2, STAGES, SLAB>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    return launch_rows<BN, 4, STAGES, SLAB>(A, W, C, M, N, K, lda, ldw, ldc, stream);
}

}  // namespace

MYNAH_API int mynah_gemm_f32(const float* A, const float* W, float* C, int M, int N, int K,
                             int lda, int ldw, int ldc, cudaStream_t stream) {
    if (M == 0 || N == 0) return 0;
    MYNAH_REQUIRE(M > 0 && N > 0 && K > 0, "gemm_f32: bad sizes M=%d N=%d K=%d", M, N, K);
    MYNAH_REQUIRE(lda >= K && ldw >= K && ldc >= N, "gemm_f32: a leading dimension is smaller than its row");
    MYNAH_REQUIRE(ceil_div(M, BM) <= GRID_ROWS, "gemm_f32: %d rows exceed one launch (%d)", M, GRID_ROWS * BM);
    const bool vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && ((uintptr_t)A | (uintptr_t)W) % 16 == 0;
    // A single slab of 32 k or less: a step's rows would be multiplied with four times as many zeros. us a product of K = 32, general
    // kernel / few rows: 16 x 16,384 4.8 / 8.1, 12 x 3,072 3.6 / 4.0, 8 x 3,072 3.6 / 3.9, 5 x 16,384 4.7 / 5.4, 4 x 16,384 4.7 / 5.0;
    // 5 x 6,144 3.6 / 3.4, 4 x 6,144 3.6 / 3.3, 2 x 16,384 4.6 / 4.0. (Leaving the zeros out in that kernel costs one row of
    // K = 1,024 to 3,072 10%.)
    const bool thin = K <= 32 && M <= ROW_MAX_M && (M >= 8 ? N >= 3072 : (long long)M * N > 32768);
    if (!vec || thin) {
        const dim3 grid(ceil_div(N, BN), ceil_div(M, BM));
        gemm_f32_kernel<<<grid, 256, 0, stream>>>(A, W, C, M, N, K, lda, ldw, ldc);
        return mynah_check_launch("gemm_f32");
    }
    if (M <= ROW_MAX_M) {
        // enough CTAs that every SM streams (two an SM and more), else as many weight rows a CTA as keep its threads busy
        const int sms = mynah_sm_count();
        if (N >= 32 * 4 * sms) return launch_rows_m<32, 3, 128>(A, W, C, M, N, K, lda, ldw, ldc, stream);
        if (N >= 16 * 2 * sms) return launch_rows_m<16, 4, 128>(A, W, C, M, N, K, lda, ldw, ldc, stream);
        // long slabs where a CTA an SM is all there is (half as many barriers; 1,024 outputs, K = 3,072: 1 row 21 -> 17 us, 2 rows 25 -> 20,
        // 16 rows 36 -> 30); with more CTAs their shared memory would keep some waiting (8 rows of 4,096: 21 -> 25)
        if (ceil_div(N, 8) <= sms && K >= 512) return launch_rows_m<8, 4, 256>(A, W, C, M, N, K, lda, ldw, ldc, stream);
        return launch_rows_m<8, 6, 128>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    }
    // Tiles of 32 x 32 with 64 threads unless they leave SMs idle (then twice the threads a tile: 40 rows of 1,024 x 3,072 46 us against
    // 58) or there are many and a tile of 64 is more than half full (tiles of 64 x 64 read half as much from L2: 800 rows of 6,144 x 1,024 260
    // against 264, 64 rows of 151,936 x 1,024 477 / 496; 32 rows 466 / 259; 161 rows of 4,096 x 1,024, fewer than five a SM, 69 / 55).
    // The larger the product the better they stand against the tile of 128 x 128 without reads ahead that they took the place of: rows of
    // 6,144 x 1,024, us: 500 246 -> 170, 1,024 369 -> 312, 2,048 735 -> 591, 4,000 1,342 -> 1,146.
    const int sms = mynah_sm_count();
    const long long small = ceil_div_ll(M, 32) * ceil_div_ll(N, 32), large = ceil_div_ll(M, 64) * ceil_div_ll(N, 64);
    if ((large >= 5 * sms && M > 32) || ceil_div(M, 32) > GRID_ROWS) return launch_tile<64, 64, 8, 4, 32>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    if (small <= sms) return launch_tile<32, 32, 4, 2, 64>(A, W, C, M, N, K, lda, ldw, ldc, stream);
    return launch_tile<32, 32, 4, 4, 32>(A, W, C, M, N, K, lda, ldw, ldc, stream);
}
