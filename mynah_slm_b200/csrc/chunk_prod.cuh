// What two linear recurrences share whose prompts go chunk by chunk (retention, the gated delta rule): fp32 products of a chunk's
// rows from shared memory, in pairs of multiply-adds (fma.rn.f32x2: the same roundings at half the instructions), and the
// outputs of a chunk from its queries, keys, values and the state before it.
#pragma once
#include "common.cuh"

namespace {

constexpr int RC_THREADS = 256;

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float lo, float hi) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ void fma2(f32x2& c, f32x2 a, f32x2 b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b)); }
__device__ __forceinline__ void mul2(f32x2& c, f32x2 a) { asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(c) : "l"(a)); }

struct alignas(16) Pairs { f32x2 lo, hi; };                 // four floats as two pairs, one 16-byte load
__device__ __forceinline__ Pairs pairs_at(const float* p) { return *reinterpret_cast<const Pairs*>(p); }

// A chunk's rows of one head into shared memory, rows from nt on as zeros (C rows, d values, d + 4 apart).
template <int C>
__device__ __forceinline__ void stage_rows(float* dst, const float* __restrict__ src, size_t row, int d, int nt) {
#pragma unroll 4
    for (int idx = threadIdx.x; idx < C * (d / 4); idx += RC_THREADS) {
        const int tt = idx / (d / 4), i4 = (idx % (d / 4)) * 4;
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (tt < nt) x = *reinterpret_cast<const float4*>(src + (size_t)tt * row + i4);
        *reinterpret_cast<float4*>(dst + tt * (d + 4) + i4) = x;
    }
}

// A chunk's values of one head, columns [j0, j0 + JT), times `weight(token)`; what does not exist is zero.
template <typename T, int C, int JT, typename F>
__device__ __forceinline__ void stage_values(float* vs, const T* __restrict__ v, int ldv, int j0, int vd, int nt, F weight) {
#pragma unroll 4
    for (int idx = threadIdx.x; idx < C * JT; idx += RC_THREADS) {
        const int tt = idx / JT, c = idx % JT;
        vs[idx] = (tt < nt && j0 + c < vd) ? weight(tt) * to_f32(v[(size_t)tt * ldv + j0 + c]) : 0.f;
    }
}

// Outputs of one chunk of C tokens (nt of them exist) and one head, for the columns [j0, j0 + JT) of vd, by RC_THREADS threads:
//
//   o_t = sum_{s <= t} w(t, s) (q_t . k_s) v_s  +  before(t) S^T q_t
//
// q, k: the chunk's first rows (d values, ld_qk apart; d a multiple of 32); v: the head's values, ldv apart; S: [d][cols] from
// column j0 on; out: the head's output columns, ldo apart. `weigh.fill(W)` runs while nothing else uses W [C][C + 4] (it may
// leave weights there), `weigh.score(t, s, W)` is w(t, s) for s <= t, read by the thread that then writes the product there.
// Thread (ty, tx) owns tokens ty * RT + u and columns tx * 4 + {0..3} (of either half, when the tile has 128). The keys' place in
// shared memory is used again by the old state, 32 rows at a time, and then by the values. `sm`: chunk_outputs_floats(...).
template <int C, int JT>
__host__ __device__ constexpr size_t chunk_outputs_floats(int d) {
    const size_t rows = (size_t)C * (d + 4), pieces = (size_t)64 * JT;
    return rows + (size_t)C * (C + 4) + (rows > pieces ? rows : pieces);
}
template <typename T, int C, int JT, class WEIGH>
__device__ __forceinline__ void chunk_outputs(float* sm, const float* __restrict__ q, const float* __restrict__ k, size_t ld_qk, int d,
                                              const T* __restrict__ v, int ldv, int j0, int vd, const float* __restrict__ S_before,
                                              int cols, float* __restrict__ out, size_t ldo, int nt, const WEIGH& weigh) {
    constexpr int RT = C / 16, G = JT / 64, LDW = C + 4, SR = 32;
    const int ldr = d + 4;
    float* qs = sm;                        // [C][ldr]
    float* Ws = qs + C * ldr;              // [C][LDW]
    float* xs = Ws + C * LDW;              // [C][ldr] keys; [2][SR][JT] state rows; [C][JT] values
    weigh.fill(Ws);
    stage_rows<C>(qs, q, ld_qk, d, nt);
    stage_rows<C>(xs, k, ld_qk, d, nt);
    __syncthreads();
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
    {   // scores: tokens ty + 16 u, keys tx + 16 w; even and odd values of a head are summed apart, then added
        f32x2 acc[RT][RT];
#pragma unroll
        for (int u = 0; u < RT; u++)
#pragma unroll
            for (int w = 0; w < RT; w++) acc[u][w] = 0ull;
#pragma unroll 2
        for (int i = 0; i < d; i += 4) {
            Pairs qv[RT], kv[RT];
#pragma unroll
            for (int u = 0; u < RT; u++) qv[u] = pairs_at(qs + (ty + 16 * u) * ldr + i);
#pragma unroll
            for (int w = 0; w < RT; w++) kv[w] = pairs_at(xs + (tx + 16 * w) * ldr + i);
#pragma unroll
            for (int u = 0; u < RT; u++)
#pragma unroll
                for (int w = 0; w <= u; w++) {              // (keys behind every token of the group: not needed)
                    fma2(acc[u][w], qv[u].lo, kv[w].lo);
                    fma2(acc[u][w], qv[u].hi, kv[w].hi);
                }
        }
#pragma unroll
        for (int u = 0; u < RT; u++)
#pragma unroll
            for (int w = 0; w < RT; w++) {
                const int t = ty + 16 * u, s = tx + 16 * w;
                const float2 x = unpack2(acc[u][w]);
                Ws[t * LDW + s] = s <= t ? weigh.score(t, s, Ws) * (x.x + x.y) : 0.f;
            }
    }
    __syncthreads();                                        // the scores are there, the keys are done with
    f32x2 acc[RT][G][2];
#pragma unroll
    for (int u = 0; u < RT; u++)
#pragma unroll
        for (int w = 0; w < G; w++) acc[u][w][0] = acc[u][w][1] = 0ull;
    // one product's four steps of k: rows [ty * RT, + RT) of `lhs` from column i, rows [i, i + 4) of `rhs`
    auto steps = [&](const float* lhs, int ld, const float* rhs) {
        float4 x[RT];
#pragma unroll
        for (int u = 0; u < RT; u++) x[u] = *reinterpret_cast<const float4*>(lhs + (ty * RT + u) * ld);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            Pairs y[G];
#pragma unroll
            for (int w = 0; w < G; w++) y[w] = pairs_at(rhs + k * JT + w * 64 + tx * 4);
#pragma unroll
            for (int u = 0; u < RT; u++) {
                const float xk = k == 0 ? x[u].x : k == 1 ? x[u].y : k == 2 ? x[u].z : x[u].w;
                const f32x2 x2 = pack2(xk, xk);
#pragma unroll
                for (int w = 0; w < G; w++) {
                    fma2(acc[u][w][0], x2, y[w].lo);
                    fma2(acc[u][w][1], x2, y[w].hi);
                }
            }
        }
    };
    // ---- the old state, in pieces of SR rows; a piece is on its way while the one before is multiplied
    auto fetch = [&](int piece) {
        if (piece * SR < d) {
            float* dst = xs + (piece & 1) * SR * JT;
#pragma unroll
            for (int idx = threadIdx.x; idx < SR * JT / 4; idx += RC_THREADS) {
                const int i = idx / (JT / 4), c = (idx % (JT / 4)) * 4;
                const uint32_t s = (uint32_t)__cvta_generic_to_shared(dst + i * JT + c);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(s), "l"(S_before + (size_t)(piece * SR + i) * cols + c) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(0);
    for (int p = 0; p * SR < d; p++) {
        fetch(p + 1);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const float* S = xs + (p & 1) * SR * JT;
#pragma unroll 2
        for (int i = 0; i < SR; i += 4) steps(qs + p * SR + i, ldr, S + i * JT);
        __syncthreads();                                    // the piece's place may be filled again
    }
#pragma unroll
    for (int u = 0; u < RT; u++) {
        const float gt = weigh.before(ty * RT + u);
#pragma unroll
        for (int w = 0; w < G; w++) {
            mul2(acc[u][w][0], pack2(gt, gt));
            mul2(acc[u][w][1], pack2(gt, gt));
        }
    }
    // ---- scores times values
    stage_values<T, C, JT>(xs, v, ldv, j0, vd, nt, [](int) { return 1.f; });
    __syncthreads();
    const int s_end = ((ty | 1) + 1) * RT;                  // keys behind the last token of the warp's rows weigh nothing
    for (int s = 0; s < s_end; s += 4) steps(Ws + s, LDW, xs + s * JT);
#pragma unroll
    for (int u = 0; u < RT; u++) {
        const int t = ty * RT + u;
        if (t >= nt) break;
        float* row = out + (size_t)t * ldo;
#pragma unroll
        for (int w = 0; w < G; w++) {
            const int j = j0 + w * 64 + tx * 4;
            const float2 x = unpack2(acc[u][w][0]), y = unpack2(acc[u][w][1]);
            if (j + 3 < vd && (vd & 3) == 0) {
                *reinterpret_cast<float4*>(row + j) = make_float4(x.x, x.y, y.x, y.y);
            } else {
                if (j < vd) row[j] = x.x;
                if (j + 1 < vd) row[j + 1] = x.y;
                if (j + 2 < vd) row[j + 2] = y.x;
                if (j + 3 < vd) row[j + 3] = y.y;
            }
        }
    }
}

}  // namespace
