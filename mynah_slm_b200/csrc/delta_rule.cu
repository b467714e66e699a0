// Gated delta rule: a linear-attention recurrence whose per-head state S [dim x vd] is decayed, corrected
// towards the new value along the new key, and read with the query, token after token:
//
//   S <- g_t S;   u = beta_t (v_t - S^T k_t);   S <- S + k_t u^T;   o_t = S^T q_t
//
// (the read-out sees the token's own write). Three kernels:
//
//   delta_prep    q, k -> unit vectors per head, x / sqrt(sum(x^2) + 1e-6), q also times dim^(-1/2);
//                 beta = sigmoid(b_raw);  g = exp(-exp(A_log_h) * softplus(a_raw + dt_bias_h))       (fp32 out)
//   delta_rule    the recurrence. The columns of S are independent given k, q, g and beta, so a CTA takes a
//                 tile of columns of one head of one sequence; a column's dim values are spread over L adjacent
//                 lanes (about 16 values a lane, in registers) that add their parts of the two dot products
//                 by shuffles in a fixed order. Half of the CTA's threads compute; the other half stage the next
//                 sixteen tokens' keys, queries, values, decays and betas in shared memory (two buffers) and
//                 write the last sixteen outputs, so that the chain from token to token waits on no load from
//                 global memory. S is fp32 [n_slots + 1][H][dim][vd], carried per slot.
//   gated_rmsnorm out = o / rms(o over the head's vd) * w[d] * act(gate),  act = silu or sigmoid
//
// The decay is one number a head, or one a head and key channel (g then has H * dim values a row and multiplies
// the rows of S: S <- diag(g_t) S); the recurrence kernel stages such a decay like a key.
//
// All arithmetic is fp32. A sequence's rows are walked in order, so a prompt run whole, in pieces or token by token performs the
// same operations in the same order, except that long bfloat16 pieces go chunk by chunk (see below).
#include "chunk_prod.cuh"
#include "layout.cuh"

namespace {

__device__ __forceinline__ float softplus_f(float v) { return v > 20.f ? v : log1pf(expf(v)); }

struct DeltaPrepArgs {
    int H, G, dim, ldc, ldab;
    float q_scale;
};

// grid (rows, parts): a warp a head of q or k, four of them a part; the last part also forms the gates. (One CTA a row, each warp
// with every fourth head, took 9.2 us for two rows of 8 heads each, one round trip to memory after the other; now 4.5.)
template <typename T>
__global__ void __launch_bounds__(128)
delta_prep_kernel(const T* __restrict__ qk, const T* __restrict__ a_raw, const T* __restrict__ b_raw,
                  VecRef A_log, VecRef dt_bias, float* __restrict__ qn, float* __restrict__ kn,
                  float* __restrict__ g_out, float* __restrict__ beta_out, DeltaPrepArgs a,
                  const float* __restrict__ a_ch, int lda) {
    griddep_launch_small();
    griddep_wait();
    const int row = blockIdx.x;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const T* src = qk + (size_t)row * a.ldc;
    for (int hh = warp + 4 * blockIdx.y; hh < 2 * a.G; hh += 4 * gridDim.y) {
        const T* v = src + (size_t)hh * a.dim;                  // q heads, then k heads
        float ss = 0.f;
        for (int d = lane; d < a.dim; d += 32) {
            const float f = to_f32(v[d]);
            ss = fmaf(f, f, ss);
        }
        const float r = (1.0f / sqrtf(warp_sum(ss) + 1e-6f)) * (hh < a.G ? a.q_scale : 1.0f);
        float* dst = hh < a.G ? qn + ((size_t)row * a.G + hh) * a.dim : kn + ((size_t)row * a.G + (hh - a.G)) * a.dim;
        for (int d = lane; d < a.dim; d += 32) dst[d] = to_f32(v[d]) * r;
    }
    if (blockIdx.y + 1 < gridDim.y) return;
    for (int h = threadIdx.x; h < a.H; h += blockDim.x) {
        const float bv = to_f32(b_raw[(size_t)row * a.ldab + h]);
        if (a_ch == nullptr) {
            const float av = to_f32(a_raw[(size_t)row * a.ldab + h]);
            g_out[(size_t)row * a.H + h] = expf(-expf(A_log.at(h)) * softplus_f(av + dt_bias.at(h)));
        }
        beta_out[(size_t)row * a.H + h] = 1.0f / (1.0f + expf(-bv));
    }
    if (a_ch != nullptr) {                                      // one decay a head and key channel
        const int n = a.H * a.dim;
        for (int i = threadIdx.x; i < n; i += blockDim.x)
            g_out[(size_t)row * n + i] = expf(-expf(A_log.at(i / a.dim)) * softplus_f(a_ch[(size_t)row * lda + i] + dt_bias.at(i)));
    }
}

constexpr int DELTA_THREADS = 128;
constexpr int DELTA_TB = 16;                // tokens staged in shared memory at a time (8 where 16 do not fit)

struct DeltaArgs {
    int B, H, G, dim, vd, n_slots, ldv;
    int L;                                   // lanes a column (a power of two)
    int per;                                 // key values a lane: ceil(dim / L) rounded up to a multiple of 4
    int vec;                                 // 1: keys and queries can be fetched four values at a time
};

// Keys and queries of a staged token lie in shared memory lane chunk by lane chunk: `per` values, then zeros up to
// RMAX (what a lane reads), then 4 unused floats, so that the L lanes of a column read their chunks (as 16-byte
// vectors) from different banks.
__device__ __forceinline__ int kq_slot(int i, int per, int stride) { return (i / per) * stride + i % per; }

template <typename T, int RMAX, bool CH, int TB>
__global__ void __launch_bounds__(2 * DELTA_THREADS)
delta_rule_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const T* __restrict__ v,
                  const float* __restrict__ g, const float* __restrict__ beta, float* __restrict__ state,
                  float* __restrict__ o, const int* __restrict__ cu_q, const int* __restrict__ slots, DeltaArgs a) {
    extern __shared__ float sm[];
    griddep_wait();
    const int b = blockIdx.z, h = blockIdx.y;
    const int slot = slots[b];
    const int q0 = cu_q[b], q1 = cu_q[b + 1];
    if (slot < 0 || slot >= a.n_slots || q1 <= q0) return;
    const int L = a.L, per = a.per;
    const int JT = DELTA_THREADS / L;                            // columns of this CTA
    const bool stager = threadIdx.x >= DELTA_THREADS;            // the second half of the CTA stages, the first computes
    const int tid = threadIdx.x % DELTA_THREADS;
    const int l = tid % L, jl = tid / L;
    const int j = blockIdx.x * JT + jl;
    const bool on = j < a.vd;
    const int jj = on ? j : a.vd - 1;
    const int kvh = h / (a.H / a.G);
    constexpr int CS = RMAX + 4;                                 // floats of a lane's chunk
    const int row = CS * L;                                      // floats of a staged key (or query)
    const int nk = TB * row, nv = TB * JT;
    float* ks = sm;                                              // [2][TB][row]
    float* qs = ks + 2 * nk;                                     // [2][TB][row]
    float* vs = qs + 2 * nk;                                     // [2][TB][JT]
    float* os = vs + 2 * nv;                                     // [2][TB][JT]
    float* gs = os + 2 * nv;                                     // [2][2][TB]: decay, beta
    float* gv = gs + 4 * TB;                               // [2][TB][row]: a decay per key channel (CH)
    for (int i = threadIdx.x; i < 4 * nk; i += 2 * DELTA_THREADS) ks[i] = 0.f;      // the unused slots stay zero
    if (CH)
        for (int i = threadIdx.x; i < 2 * nk; i += 2 * DELTA_THREADS) gv[i] = 0.f;
    __syncthreads();

    auto stage = [&](int k) {                                    // block k of the sequence's rows -> buffer k & 1
        const int t0 = q0 + k * TB, nt = min(TB, q1 - t0), buf = k & 1;
        if (a.vec) {
            // four consecutive values a load, four loads of k and of q a thread issued before the first is used
            const int d4 = a.dim / 4, total = nt * d4;
            for (int base = tid; base < total; base += 4 * DELTA_THREADS) {
                float4 kk[4], qq[4], gg[4];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int idx = base + e * DELTA_THREADS;
                    if (idx < total) {
                        const size_t src = ((size_t)(t0 + idx / d4) * a.G + kvh) * a.dim + (size_t)(idx % d4) * 4;
                        kk[e] = *reinterpret_cast<const float4*>(kn + src);
                        qq[e] = *reinterpret_cast<const float4*>(qn + src);
                        if (CH) gg[e] = *reinterpret_cast<const float4*>(g + ((size_t)(t0 + idx / d4) * a.H + h) * a.dim + (size_t)(idx % d4) * 4);
                    }
                }
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    const int idx = base + e * DELTA_THREADS;
                    if (idx < total) {
                        const int at = buf * nk + (idx / d4) * row + kq_slot((idx % d4) * 4, per, CS);
                        *reinterpret_cast<float4*>(ks + at) = kk[e];
                        *reinterpret_cast<float4*>(qs + at) = qq[e];
                        if (CH) *reinterpret_cast<float4*>(gv + at) = gg[e];
                    }
                }
            }
        }
#pragma unroll 4
        for (int idx = tid; idx < (a.vec ? 0 : nt * a.dim); idx += DELTA_THREADS) {
            const int tt = idx / a.dim, i = idx % a.dim;
            const size_t src = ((size_t)(t0 + tt) * a.G + kvh) * a.dim + i;
            const int at = buf * nk + tt * row + kq_slot(i, per, CS);
            ks[at] = kn[src];
            qs[at] = qn[src];
            if (CH) gv[at] = g[((size_t)(t0 + tt) * a.H + h) * a.dim + i];
        }
        for (int idx = tid; idx < nt * JT; idx += DELTA_THREADS) {
            const int tt = idx / JT, col = blockIdx.x * JT + idx % JT;
            vs[buf * nv + idx] = col < a.vd ? to_f32(v[(size_t)(t0 + tt) * a.ldv + (size_t)h * a.vd + col]) : 0.f;
        }
        if (tid < nt) {
            gs[buf * 2 * TB + tid] = CH ? 1.0f : g[(size_t)(t0 + tid) * a.H + h];
            gs[buf * 2 * TB + TB + tid] = beta[(size_t)(t0 + tid) * a.H + h];
        }
    };
    auto write_out = [&](int k) {
        const int t0 = q0 + k * TB, nt = min(TB, q1 - t0), buf = k & 1;
        for (int idx = tid; idx < nt * JT; idx += DELTA_THREADS) {
            const int tt = idx / JT, col = blockIdx.x * JT + idx % JT;
            if (col < a.vd) o[(size_t)(t0 + tt) * a.H * a.vd + (size_t)h * a.vd + col] = os[buf * nv + idx];
        }
    };

    float S[RMAX];
    float* st = state + (((size_t)slot * a.H + h) * a.dim) * a.vd + jj;
    const int i0 = l * per;
    if (!stager) {
#pragma unroll
        for (int r = 0; r < RMAX; r++) S[r] = (r < per && i0 + r < a.dim) ? st[(size_t)(i0 + r) * a.vd] : 0.f;
    } else {
        stage(0);
    }
    __syncthreads();
    const int n_blocks = (q1 - q0 + TB - 1) / TB;
    for (int k = 0; k < n_blocks; k++) {
        if (stager) {
            if (k + 1 < n_blocks) stage(k + 1);
            if (k > 0) write_out(k - 1);
        } else {
            const int nt = min(TB, q1 - q0 - k * TB), buf = k & 1;
            for (int tt = 0; tt < nt; tt++) {
                const float gt = gs[buf * 2 * TB + tt], bt = gs[buf * 2 * TB + TB + tt];
                const float4* k4 = reinterpret_cast<const float4*>(ks + buf * nk + tt * row + l * CS);
                const float4* q4 = reinterpret_cast<const float4*>(qs + buf * nk + tt * row + l * CS);
                float kr[RMAX];
                float d4[4] = {0.f, 0.f, 0.f, 0.f};             // four partial sums: four short chains instead of a long one
#pragma unroll
                for (int r = 0; r < RMAX; r += 4) {
                    const float4 kk = k4[r >> 2];
                    kr[r] = kk.x; kr[r + 1] = kk.y; kr[r + 2] = kk.z; kr[r + 3] = kk.w;
                }
                if (CH) {
                    const float4* g4 = reinterpret_cast<const float4*>(gv + buf * nk + tt * row + l * CS);
#pragma unroll
                    for (int r = 0; r < RMAX; r += 4) {
                        const float4 gg = g4[r >> 2];
                        S[r] *= gg.x; S[r + 1] *= gg.y; S[r + 2] *= gg.z; S[r + 3] *= gg.w;
                    }
                }
#pragma unroll
                for (int r = 0; r < RMAX; r++) {
                    if (!CH) S[r] *= gt;
                    d4[r & 3] = fmaf(S[r], kr[r], d4[r & 3]);
                }
                float dot = (d4[0] + d4[1]) + (d4[2] + d4[3]);
                for (int s = L >> 1; s > 0; s >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, s);
                const float u = bt * (vs[buf * nv + tt * JT + jl] - dot);
                float o4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int r = 0; r < RMAX; r += 4) {
                    const float4 qq = q4[r >> 2];
                    S[r] = fmaf(kr[r], u, S[r]);
                    S[r + 1] = fmaf(kr[r + 1], u, S[r + 1]);
                    S[r + 2] = fmaf(kr[r + 2], u, S[r + 2]);
                    S[r + 3] = fmaf(kr[r + 3], u, S[r + 3]);
                    o4[0] = fmaf(S[r], qq.x, o4[0]);
                    o4[1] = fmaf(S[r + 1], qq.y, o4[1]);
                    o4[2] = fmaf(S[r + 2], qq.z, o4[2]);
                    o4[3] = fmaf(S[r + 3], qq.w, o4[3]);
                }
                float out = (o4[0] + o4[1]) + (o4[2] + o4[3]);
                for (int s = L >> 1; s > 0; s >>= 1) out += __shfl_xor_sync(0xffffffffu, out, s);
                if (l == 0) os[buf * nv + tt * JT + jl] = out;
            }
        }
        __syncthreads();
    }
    if (stager) {
        write_out(n_blocks - 1);
    } else if (on) {
#pragma unroll
        for (int r = 0; r < RMAX; r++)
            if (r < per && i0 + r < a.dim) st[(size_t)(i0 + r) * a.vd] = S[r];
    }
}

// a warp a (row, head)
template <typename T>
__global__ void __launch_bounds__(128)
gated_rmsnorm_kernel(const float* __restrict__ o, const T* __restrict__ gate, int ldg, VecRef w, T* __restrict__ out,
                     int n_heads_total, int H, int vd, float eps, int gate_sigmoid) {
    griddep_launch_small();
    griddep_wait();
    const int idx = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (idx >= n_heads_total) return;
    const int lane = threadIdx.x & 31;
    const int row = idx / H, h = idx % H;
    const float* src = o + ((size_t)row * H + h) * vd;
    float ss = 0.f;
    for (int d = lane; d < vd; d += 32) ss = fmaf(src[d], src[d], ss);
    const float r = 1.0f / sqrtf(warp_sum(ss) / (float)vd + eps);
    const T* gt = gate + (size_t)row * ldg + (size_t)h * vd;
    T* dst = out + ((size_t)row * H + h) * vd;
    for (int d = lane; d < vd; d += 32) {
        const float z = to_f32(gt[d]);
        const float sg = 1.0f / (1.0f + expf(-z));
        dst[d] = from_f32<T>(src[d] * r * w.at(d) * (gate_sigmoid ? sg : z * sg));
    }
}

// ---- the recurrence chunk by chunk, for bfloat16 prompts whose decay is one number a head (the 32-bit path keeps its one order) ----
// With a chunk of C tokens, S the state before it, p(t, s) = g_(s+1) ... g_t and G_t = g_0 ... g_t (products taken one by one, as the
// recurrence takes them):
//
//   u_t = beta_t (v_t - G_t S^T k_t - sum_{s < t} p(t, s) (k_t . k_s) u_s)
//   o_t = G_t S^T q_t + sum_{s <= t} p(t, s) (q_t . k_s) u_s
//   S_new = G_last S + sum_s p(last, s) k_s u_s^T
//
// The first line is a lower triangular system with two right-hand sides that do not depend on S: u = U - W S with U and W its
// solutions for beta_t v_t and beta_t G_t k_t. Three kernels, all sums fp32:
//
//   delta_solve   U and W of every chunk and head: a thread a column, by substitution, eight rows at a time in registers
//   delta_chain   the chain: a CTA takes 32 columns of a head's state through its sequence's chunks: u = U - W S (written over U),
//                 S_new; the state before every chunk goes to scratch. The next chunk's rows arrive under the products.
//   delta_out     the outputs of a chunk, which need nothing else (chunk_prod.cuh)
//
// The chain bounds it: two products of 64 x 128 x 32 a chunk, whose reads of shared memory take about 4 us, and three barriers.
// A step's chunks go in passes, so that scratch is bounded. Sums run in another order than token by token: the two forms
// agree to rounding. Measured (3,248 tokens of two sequences, 16 heads of 128 on 8 of
// keys), us a layer: 104 + 185 + 123; token by token 802. Outputs lie 1.1e-7 to 3.3e-7 from 64 bits, token by token 0.8e-7 to 2.8e-7
// (a token's sums over 128 channels are one chain here, four there). From 128 tokens on: shorter prompts leave too few chunks a chain.
constexpr int DC = 64, DC_COLS = 32, DC_TILE = 128;         // tokens a chunk, columns a CTA of the chain, columns solved at a time

struct DeltaChunkArgs {
    int B, H, G, dim, vd, n_slots, ldv, cols;              // cols: columns of a state and of U in scratch (vd padded to whole tiles)
    int first;                                              // the pass's first chunk
    float *W, *U, *states, *decays;                         // scratch: [chunk][H][DC][dim], [..][DC][cols], [..][dim][cols], [..][DC][2]
};

__global__ void __launch_bounds__(RC_THREADS, 2)
delta_solve_kernel(const float* __restrict__ kn, const bf16* __restrict__ v, const float* __restrict__ g, const float* __restrict__ beta,
                   const int* __restrict__ cu_q, DeltaChunkArgs a) {
    constexpr int LDA = DC + 4;
    extern __shared__ __align__(16) float sm[];
    __shared__ float gs[DC], bs[DC], Gs[DC];
    griddep_wait();
    int b, tile;
    if (!find_query_tile(cu_q, a.B, DC, a.first + (int)blockIdx.x, b, tile)) return;
    const int h = blockIdx.y, d = a.dim, ldk = d + 4, tid = threadIdx.x;
    const int t0 = cu_q[b] + tile * DC, nt = min(DC, cu_q[b + 1] - t0);
    float* ks = sm;                        // [DC][ldk]: keys; W's columns go over them
    float* At = ks + DC * ldk;             // [DC][LDA]: the matrix transposed
    float* us = At + DC * LDA;             // [DC][DC_TILE]: U's columns
    if (tid < DC) {
        gs[tid] = tid < nt ? g[(size_t)(t0 + tid) * a.H + h] : 1.f;
        bs[tid] = tid < nt ? beta[(size_t)(t0 + tid) * a.H + h] : 0.f;
    }
    const size_t n = (size_t)a.G * d;
    stage_rows<DC>(ks, kn + (size_t)t0 * n + (size_t)(h / (a.H / a.G)) * d, n, d, nt);
    stage_values<bf16, DC, DC_TILE>(us, v + (size_t)t0 * a.ldv + (size_t)h * a.vd, a.ldv, 0, a.vd, nt, [](int) { return 1.f; });
    __syncthreads();
    const size_t unit = (size_t)blockIdx.x * a.H + h;
    if (tid < DC) {                                         // column s of the decays between two tokens
        float p = 1.f;
        for (int t = 0; t < DC; t++) {
            if (t > tid) p *= gs[t];
            At[tid * LDA + t] = t >= tid ? p : 0.f;
        }
        a.decays[(unit * DC + tid) * 2] = At[tid * LDA + nt - 1];
    } else if (tid == DC) {
        float p = 1.f;
        for (int t = 0; t < DC; t++) Gs[t] = p *= gs[t];
    }
    __syncthreads();
    if (tid < DC) a.decays[(unit * DC + tid) * 2 + 1] = Gs[tid];
    {   // the matrix below its diagonal: tokens ty + 16 u, keys tx + 16 w
        const int ty = tid >> 4, tx = tid & 15;
        f32x2 acc[4][4];
#pragma unroll
        for (int u = 0; u < 4; u++)
#pragma unroll
            for (int w = 0; w < 4; w++) acc[u][w] = 0ull;
#pragma unroll 2
        for (int i = 0; i < d; i += 4) {
            Pairs x[4], y[4];
#pragma unroll
            for (int u = 0; u < 4; u++) x[u] = pairs_at(ks + (ty + 16 * u) * ldk + i);
#pragma unroll
            for (int w = 0; w < 4; w++) y[w] = pairs_at(ks + (tx + 16 * w) * ldk + i);
#pragma unroll
            for (int u = 0; u < 4; u++)
#pragma unroll
                for (int w = 0; w <= u; w++) {
                    fma2(acc[u][w], x[u].lo, y[w].lo);
                    fma2(acc[u][w], x[u].hi, y[w].hi);
                }
        }
#pragma unroll
        for (int u = 0; u < 4; u++)
#pragma unroll
            for (int w = 0; w < 4; w++) {
                const int t = ty + 16 * u, s = tx + 16 * w;
                const float2 x = unpack2(acc[u][w]);
                At[s * LDA + t] = s < t ? bs[t] * (At[s * LDA + t] * (x.x + x.y)) : 0.f;
            }
    }
    __syncthreads();
    // the first half of the threads solves for W (d <= DC_TILE columns), the second for U, DC_TILE columns a round
    const bool is_w = tid < DC_TILE;
    for (int j = tid % DC_TILE; j < (is_w ? d : a.cols); j += is_w ? d : DC_TILE) {
        const bf16* vc = v + (size_t)t0 * a.ldv + (size_t)h * a.vd + j;
        float* dst = is_w ? a.W + unit * DC * d + j : a.U + unit * DC * a.cols + j;
        float* own = is_w ? ks + j : us + j % DC_TILE;      // this thread's column: nobody else's
        const int ldd = is_w ? d : a.cols, ldo = is_w ? ldk : DC_TILE;
        if (!is_w && j >= DC_TILE) {                        // (the first round's values are there)
#pragma unroll 16
            for (int t = 0; t < DC; t++) own[t * DC_TILE] = t < nt && j < a.vd ? to_f32(vc[(size_t)t * a.ldv]) : 0.f;
        }
        for (int r0 = 0; r0 < DC; r0 += 8) {
            float x[8], y[4][8] = {};                       // four sums a row: short chains
#pragma unroll
            for (int e = 0; e < 8; e++) x[e] = bs[r0 + e] * ((is_w ? Gs[r0 + e] : 1.f) * own[(r0 + e) * ldo]);
            for (int s = 0; s < r0; s += 4) {
                float xs[4];
                float4 m0[4], m1[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    xs[q] = own[(s + q) * ldo];
                    m0[q] = *reinterpret_cast<const float4*>(At + (s + q) * LDA + r0);
                    m1[q] = *reinterpret_cast<const float4*>(At + (s + q) * LDA + r0 + 4);
                }
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const float m[8] = {m0[q].x, m0[q].y, m0[q].z, m0[q].w, m1[q].x, m1[q].y, m1[q].z, m1[q].w};
#pragma unroll
                    for (int e = 0; e < 8; e++) y[q][e] = fmaf(m[e], xs[q], y[q][e]);
                }
            }
#pragma unroll
            for (int e = 0; e < 8; e++) x[e] -= (y[0][e] + y[1][e]) + (y[2][e] + y[3][e]);
#pragma unroll
            for (int s = 0; s < 8; s++)
#pragma unroll
                for (int e = s + 1; e < 8; e++) x[e] = fmaf(-At[(r0 + s) * LDA + r0 + e], x[s], x[e]);
#pragma unroll
            for (int e = 0; e < 8; e++) {
                own[(r0 + e) * ldo] = x[e];
                dst[(size_t)(r0 + e) * ldd] = x[e];         // (rows from nt on are zeros)
            }
        }
    }
}

// grid (cols / DC_COLS, H, B)
__global__ void __launch_bounds__(RC_THREADS)
delta_chain_kernel(const float* __restrict__ kn, float* __restrict__ state, const int* __restrict__ cu_q, const int* __restrict__ slots,
                   DeltaChunkArgs a, int n_pass) {
    constexpr int LDU = DC_COLS + 4;
    extern __shared__ __align__(16) float sm[];
    __shared__ int parts[RC_THREADS / 32];
    griddep_wait();
    const int b = blockIdx.z, h = blockIdx.y, j0 = blockIdx.x * DC_COLS, d = a.dim, ldk = d + 4, tid = threadIdx.x;
    const int q0 = cu_q[b], q1 = cu_q[b + 1], slot = slots[b];
    int before = 0;                                         // chunks of the sequences before this one
    for (int i = tid; i < b; i += RC_THREADS) before += (cu_q[i + 1] - cu_q[i] + DC - 1) / DC;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    if ((tid & 31) == 0) parts[tid >> 5] = before;
    __syncthreads();
    before = 0;
#pragma unroll
    for (int w = 0; w < RC_THREADS / 32; w++) before += parts[w];
    const int tiles = (q1 - q0 + DC - 1) / DC;
    // chunk t of the sequence is number before + tiles - 1 - t; this pass holds the numbers [first, first + n_pass)
    const int last_no = before + tiles - 1;
    const int t_lo = max(0, last_no - (a.first + n_pass - 1)), t_hi = min(tiles, last_no - a.first + 1);
    if (t_lo >= t_hi || slot < 0 || slot >= a.n_slots) return;
    const int stage_words = 2 * DC * ldk + DC * DC_COLS + 2 * DC;
    float* Ss = sm + 2 * stage_words;      // [d][DC_COLS]
    float* us = Ss + d * DC_COLS;          // [DC][LDU]: u, times its decay to the chunk's end
    const size_t n = (size_t)a.G * d;
    const float* keys = kn + (size_t)(h / (a.H / a.G)) * d;
    auto copy = [](float* dst, const float* src, bool valid) {
        const int bytes = valid ? 16 : 0;                   // 0: the 16 bytes are zero-filled
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
    };
    auto fetch = [&](int t) {                               // W [DC][ldk], k [DC][ldk], U [DC][DC_COLS], decays [DC][2]
        if (t < t_hi) {
            float* ws = sm + (t & 1) * stage_words;
            float* ks = ws + DC * ldk;
            float* u0 = ks + DC * ldk;
            const size_t unit = (size_t)(last_no - t - a.first) * a.H + h;
            const int row0 = q0 + t * DC, nt = min(DC, q1 - row0);
            for (int idx = tid; idx < DC * (d / 4); idx += RC_THREADS) {
                const int r = idx / (d / 4), c = (idx % (d / 4)) * 4;
                copy(ws + r * ldk + c, a.W + (unit * DC + r) * d + c, true);
                copy(ks + r * ldk + c, keys + (size_t)(row0 + (r < nt ? r : 0)) * n + c, r < nt);
            }
            for (int idx = tid; idx < DC * (DC_COLS / 4); idx += RC_THREADS) {
                const int r = idx / (DC_COLS / 4), c = (idx % (DC_COLS / 4)) * 4;
                copy(u0 + r * DC_COLS + c, a.U + (unit * DC + r) * a.cols + j0 + c, true);
            }
            if (tid < DC / 2) copy(u0 + DC * DC_COLS + tid * 4, a.decays + unit * DC * 2 + tid * 4, true);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(t_lo);
    // a thread's part of the state: rows i0 + r, columns c0 + {0..3}
    const int i0 = (tid >> 3) * 4, c0 = (tid & 7) * 4;
    const bool owns = i0 < d;
    f32x2 S[4][2];
    float* sp = state + (((size_t)slot * a.H + h) * d + i0) * a.vd + j0 + c0;
#pragma unroll
    for (int r = 0; r < 4; r++) {
        float x[4];
#pragma unroll
        for (int e = 0; e < 4; e++) x[e] = owns && j0 + c0 + e < a.vd ? sp[(size_t)r * a.vd + e] : 0.f;
        S[r][0] = pack2(x[0], x[1]);
        S[r][1] = pack2(x[2], x[3]);
    }
    // a thread's part of u: tokens ty * 4 + r, columns tx * 2 + {0, 1}
    const int ty = tid >> 4, tx = tid & 15;
    for (int t = t_lo; t < t_hi; t++) {
        fetch(t + 1);
        const float* ws = sm + (t & 1) * stage_words;
        const float* ks = ws + DC * ldk;
        const float* u0 = ks + DC * ldk;
        const float* dec = u0 + DC * DC_COLS;
        const size_t unit = (size_t)(last_no - t - a.first) * a.H + h;
        const int nt = min(DC, q1 - q0 - t * DC);
        if (owns) {
            float* to = a.states + (unit * d + i0) * a.cols + j0 + c0;
#pragma unroll
            for (int r = 0; r < 4; r++) {
                *reinterpret_cast<Pairs*>(Ss + (i0 + r) * DC_COLS + c0) = Pairs{S[r][0], S[r][1]};
                *reinterpret_cast<Pairs*>(to + (size_t)r * a.cols) = Pairs{S[r][0], S[r][1]};
            }
        }
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();                                    // this chunk's rows and the state are there
        {
            f32x2 acc[4] = {0ull, 0ull, 0ull, 0ull};
#pragma unroll 4
            for (int i = 0; i < d; i += 4) {
                float4 x[4];
#pragma unroll
                for (int r = 0; r < 4; r++) x[r] = *reinterpret_cast<const float4*>(ws + (ty * 4 + r) * ldk + i);
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const f32x2 y = *reinterpret_cast<const f32x2*>(Ss + (i + k) * DC_COLS + tx * 2);
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        const float xk = k == 0 ? x[r].x : k == 1 ? x[r].y : k == 2 ? x[r].z : x[r].w;
                        fma2(acc[r], pack2(xk, xk), y);
                    }
                }
            }
            float* to = a.U + (unit * DC + ty * 4) * a.cols + j0 + tx * 2;
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const float2 s = unpack2(acc[r]), w = *reinterpret_cast<const float2*>(u0 + (ty * 4 + r) * DC_COLS + tx * 2);
                const float2 u = make_float2(w.x - s.x, w.y - s.y);
                *reinterpret_cast<float2*>(to + (size_t)r * a.cols) = u;
                const float p = dec[(ty * 4 + r) * 2];
                *reinterpret_cast<float2*>(us + (ty * 4 + r) * LDU + tx * 2) = make_float2(p * u.x, p * u.y);
            }
        }
        __syncthreads();                                    // u is there
        if (owns) {
            const float ge = dec[(nt - 1) * 2 + 1];
#pragma unroll
            for (int r = 0; r < 4; r++) {
                mul2(S[r][0], pack2(ge, ge));
                mul2(S[r][1], pack2(ge, ge));
            }
#pragma unroll 4
            for (int s = 0; s < nt; s++) {
                const float4 k4 = *reinterpret_cast<const float4*>(ks + s * ldk + i0);
                const Pairs u2 = pairs_at(us + s * LDU + c0);
                const float kk[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
                for (int r = 0; r < 4; r++) {
                    const f32x2 k2 = pack2(kk[r], kk[r]);
                    fma2(S[r][0], k2, u2.lo);
                    fma2(S[r][1], k2, u2.hi);
                }
            }
        }
        __syncthreads();                                    // this chunk's place may be filled again
    }
    if (owns) {
#pragma unroll
        for (int r = 0; r < 4; r++) {
            const float2 x = unpack2(S[r][0]), y = unpack2(S[r][1]);
            const float z[4] = {x.x, x.y, y.x, y.y};
#pragma unroll
            for (int e = 0; e < 4; e++)
                if (j0 + c0 + e < a.vd) sp[(size_t)r * a.vd + e] = z[e];
        }
    }
}

struct DeltaWeights {
    const float* gs;                                        // the chunk's decays
    const float* Gs;                                        // their running product
    __device__ __forceinline__ void fill(float* W) const {
        const int s = threadIdx.x;
        if (s < DC) {
            float p = 1.f;
            for (int t = s; t < DC; t++) {
                if (t > s) p *= gs[t];
                W[t * (DC + 4) + s] = p;
            }
        }
    }
    __device__ __forceinline__ float score(int t, int s, const float* W) const { return W[t * (DC + 4) + s]; }
    __device__ __forceinline__ float before(int t) const { return Gs[t]; }
};

// grid (chunks of the pass, H, cols / JT)
template <int JT>
__global__ void __launch_bounds__(RC_THREADS, 2)
delta_out_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const float* __restrict__ g, float* __restrict__ o,
                 const int* __restrict__ cu_q, const int* __restrict__ slots, DeltaChunkArgs a) {
    extern __shared__ __align__(16) float sm[];
    __shared__ float gs[DC], Gs[DC];
    griddep_wait();
    int b, tile;
    if (!find_query_tile(cu_q, a.B, DC, a.first + (int)blockIdx.x, b, tile)) return;
    const int slot = slots[b];
    if (slot < 0 || slot >= a.n_slots) return;
    const int h = blockIdx.y, d = a.dim, j0 = blockIdx.z * JT;
    const int t0 = cu_q[b] + tile * DC, nt = min(DC, cu_q[b + 1] - t0);
    const size_t unit = (size_t)blockIdx.x * a.H + h;
    if (threadIdx.x < DC) {
        gs[threadIdx.x] = (int)threadIdx.x < nt ? g[(size_t)(t0 + threadIdx.x) * a.H + h] : 1.f;
        Gs[threadIdx.x] = a.decays[(unit * DC + threadIdx.x) * 2 + 1];
    }
    __syncthreads();
    const size_t n = (size_t)a.G * d, at = (size_t)t0 * n + (size_t)(h / (a.H / a.G)) * d;
    chunk_outputs<float, DC, JT>(sm, qn + at, kn + at, n, d, a.U + unit * DC * a.cols, a.cols, j0, a.vd,
                                 a.states + unit * d * a.cols + j0, a.cols, o + (size_t)t0 * a.H * a.vd + (size_t)h * a.vd,
                                 (size_t)a.H * a.vd, nt, DeltaWeights{gs, Gs});
}

// How a step's chunks go: columns a tile, padded columns, chunks at most, chunks a pass.
struct DeltaPlan {
    int JT, cols, total, n_pass;
    long long unit;                                         // floats of scratch a chunk
    DeltaPlan(int rows, int B, int H, int dim, int vd) {
        JT = vd > 64 ? 128 : 64;
        cols = ceil_div(vd, JT) * JT;
        total = rows / DC + B;
        unit = (long long)H * ((long long)DC * (dim + cols) + (long long)dim * cols + DC * 2);
        const long long fit = (256ll << 20) / 4 / unit;
        const int least = ceil_div(2 * mynah_sm_count(), H);
        const int most = (int)(fit < least ? least : fit > total ? total : fit);
        n_pass = ceil_div(total, ceil_div(total, most));
    }
};

int launch_chunks(const float* qn, const float* kn, const bf16* v, const float* g, const float* beta, float* state, float* o,
                  const int* cu_q, const int* slots, DeltaChunkArgs a, const DeltaPlan& plan, float* scratch, cudaStream_t stream) {
    const int d = a.dim;
    const size_t solve = ((size_t)DC * (d + 4) + (size_t)DC * (DC + 4) + (size_t)DC * DC_TILE) * sizeof(float);
    const size_t chain = (2 * ((size_t)2 * DC * (d + 4) + DC * DC_COLS + 2 * DC) + (size_t)d * DC_COLS + (size_t)DC * (DC_COLS + 4)) * sizeof(float);
    const size_t out = (plan.JT == 128 ? chunk_outputs_floats<DC, 128>(d) : chunk_outputs_floats<DC, 64>(d)) * sizeof(float);
    auto out_kernel = plan.JT == 128 ? delta_out_kernel<128> : delta_out_kernel<64>;
    if (cudaFuncSetAttribute(delta_solve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024) != cudaSuccess ||
        cudaFuncSetAttribute(delta_chain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) != cudaSuccess ||
        cudaFuncSetAttribute(out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 112 * 1024) != cudaSuccess)
        return mynah_fail("delta_rule: %zu bytes of shared memory are not to be had", chain);
    a.W = scratch;
    a.U = a.W + (size_t)plan.n_pass * a.H * DC * d;
    a.states = a.U + (size_t)plan.n_pass * a.H * DC * a.cols;
    a.decays = a.states + (size_t)plan.n_pass * a.H * d * a.cols;
    // a sequence's chunks are numbered from its last to its first, so the passes go from the last to the first too
    for (int p = (plan.total - 1) / plan.n_pass; p >= 0; p--) {
        a.first = p * plan.n_pass;
        mynah_launch(delta_solve_kernel, dim3(plan.n_pass, a.H), dim3(RC_THREADS), solve, stream, kn, v, g, beta, cu_q, a);
        mynah_launch(delta_chain_kernel, dim3(a.cols / DC_COLS, a.H, a.B), dim3(RC_THREADS), chain, stream, kn, state, cu_q, slots, a, plan.n_pass);
        mynah_launch(out_kernel, dim3(plan.n_pass, a.H, a.cols / plan.JT), dim3(RC_THREADS), out, stream, qn, kn, g, o, cu_q, slots, a);
        if (mynah_check_launch("delta_rule (chunks)") != 0) return -1;
    }
    return 0;
}

}  // namespace

// 0: every step walks token by token; otherwise prompts whose longest piece has at least this many tokens go chunk by chunk.
static int g_delta_chunk_min = 128;
MYNAH_API int mynah_delta_chunk_min(int n) {
    const int before = g_delta_chunk_min;
    g_delta_chunk_min = n;
    return before;
}

// Floats of scratch that mynah_delta_rule wants for a step of `rows` rows (0: it walks token by token), and its launches.
MYNAH_API long long mynah_delta_scratch_floats(int rows, int B, int H, int dim, int vd, int max_q_len, int channel_decay, int dtype, int* launches) {
    *launches = 1;
    if (g_delta_chunk_min <= 0 || max_q_len < g_delta_chunk_min || channel_decay || dtype != MYNAH_BF16 || dim % 32 != 0 || dim > 128 || rows <= 0) return 0;
    const DeltaPlan plan(rows, B, H, dim, vd);
    *launches = 3 * ceil_div(plan.total, plan.n_pass);
    return plan.n_pass * plan.unit;
}

// qk [T, ldc]: G*dim query then G*dim key values a row (after their convolution and activation); a_raw, b_raw
// [T, ldab] with H values a row; all in dtype. A_log, dt_bias [H] in w_dtype. Outputs fp32: qn, kn [T, G*dim],
// g, beta [T, H].
// a_ch, when given (fp32 [T, lda], H*dim values a row), makes the decay one a head and key channel: dt_bias then has
// H*dim values, g [T, H*dim], and a_raw is not read.
MYNAH_API int mynah_delta_prep(const void* qk, int ldc, const void* a_raw, const void* b_raw, int ldab, int dtype,
                               const void* A_log, const void* dt_bias, int w_dtype,
                               float* qn, float* kn, float* g, float* beta,
                               int T, int H, int G, int dim, const float* a_ch, int lda, cudaStream_t stream) {
    if (T == 0) return 0;
    MYNAH_REQUIRE(T > 0 && H > 0 && G > 0 && dim > 0 && H % G == 0, "delta_prep: bad sizes T=%d H=%d G=%d dim=%d", T, H, G, dim);
    const DeltaPrepArgs a{H, G, dim, ldc, ldab, 1.0f / sqrtf((float)dim)};
    const VecRef al{A_log, w_dtype}, db{dt_bias, w_dtype};
    const dim3 grid(T, ceil_div(2 * G, 4) + 1 <= 65535 && T <= 64 ? ceil_div(2 * G, 4) + 1 : 1);      // (a prompt's rows are CTAs enough)
    if (dtype == MYNAH_F32)
        mynah_launch(delta_prep_kernel<float>, grid, dim3(128), 0, stream, (const float*)qk, (const float*)a_raw,
                     (const float*)b_raw, al, db, qn, kn, g, beta, a, a_ch, lda);
    else if (dtype == MYNAH_BF16)
        mynah_launch(delta_prep_kernel<bf16>, grid, dim3(128), 0, stream, (const bf16*)qk, (const bf16*)a_raw,
                     (const bf16*)b_raw, al, db, qn, kn, g, beta, a, a_ch, lda);
    else
        return mynah_fail("delta_prep: unsupported dtype %d", dtype);
    return mynah_check_launch("delta_prep");
}

// v [T, ldv] in dtype with head h at h*vd; state fp32 [n_slots + 1, H, dim, vd]; o fp32 [T, H*vd]. g fp32 [T, H], or
// [T, H*dim] with channel_decay. rows: the step's rows; scratch: mynah_delta_scratch_floats(...) floats, or null (token by token).
MYNAH_API int mynah_delta_rule(const float* qn, const float* kn, const void* v, int ldv, int dtype,
                               const float* g, const float* beta, float* state, int n_slots, float* o,
                               const int* cu_q, const int* slots, int B, int H, int G, int dim, int vd,
                               int channel_decay, int rows, float* scratch, cudaStream_t stream) {
    if (B == 0) return 0;
    MYNAH_REQUIRE(B > 0 && H > 0 && G > 0 && dim > 0 && vd > 0 && H % G == 0, "delta_rule: bad sizes B=%d H=%d G=%d dim=%d vd=%d", B, H, G, dim, vd);
    MYNAH_REQUIRE(dim <= 1024, "delta_rule: a key of %d values exceeds 1024", dim);
    MYNAH_REQUIRE(B <= 65535 && H <= 65535, "delta_rule: B=%d or H=%d exceeds one launch", B, H);
    if (scratch != nullptr && dtype == MYNAH_BF16 && !channel_decay && dim % 32 == 0 && dim <= 128 &&
        (((uintptr_t)qn | (uintptr_t)kn | (uintptr_t)scratch) & 15) == 0) {
        const DeltaPlan plan(rows, B, H, dim, vd);
        MYNAH_REQUIRE(plan.cols / plan.JT <= 65535, "delta_rule: too many columns for one launch");
        const DeltaChunkArgs ca{B, H, G, dim, vd, n_slots, ldv, plan.cols, 0, nullptr, nullptr, nullptr, nullptr};
        return launch_chunks(qn, kn, (const bf16*)v, g, beta, state, o, cu_q, slots, ca, plan, scratch, stream);
    }
    int L = 1;
    while (L * 16 < dim && L < 32) L <<= 1;                     // about 16 key values a lane
    const int per = (ceil_div(dim, L) + 3) / 4 * 4;
    const int vec = dim % 4 == 0 && ((reinterpret_cast<uintptr_t>(qn) | reinterpret_cast<uintptr_t>(kn) |
                                      (channel_decay ? reinterpret_cast<uintptr_t>(g) : 0)) & 15) == 0;
    const DeltaArgs a{B, H, G, dim, vd, n_slots, ldv, L, per, vec};
    const int JT = DELTA_THREADS / L;
    const dim3 grid(ceil_div(vd, JT), H, B);
    const int rmax = per <= 16 ? 16 : 32;
    auto smem_for = [&](int tb) {
        return sizeof(float) * ((size_t)(channel_decay ? 6 : 4) * tb * (rmax + 4) * L + (size_t)4 * tb * JT + 4 * tb);
    };
    // a decay per channel is staged like a third key: with the longest keys only half as many tokens fit
    const int tb = smem_for(DELTA_TB) <= 200 * 1024 ? DELTA_TB : DELTA_TB / 2;
    const size_t smem = smem_for(tb);
#define DELTA_LAUNCH(T, RMAX, CH)                                                                                      \
    if (tb == DELTA_TB) { DELTA_LAUNCH_TB(T, RMAX, CH, DELTA_TB); }                                                    \
    else { DELTA_LAUNCH_TB(T, RMAX, CH, DELTA_TB / 2); }
#define DELTA_LAUNCH_TB(T, RMAX, CH, TB)                                                                                   \
    if (smem > 48 * 1024 &&                                                                                            \
        cudaFuncSetAttribute(delta_rule_kernel<T, RMAX, CH, TB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) \
        return mynah_fail("delta_rule: %zu bytes of shared memory are not to be had", smem);                          \
    mynah_launch(delta_rule_kernel<T, RMAX, CH, TB>, grid, dim3(2 * DELTA_THREADS), smem, stream, qn, kn, (const T*)v, g, beta, state, o, \
                 cu_q, slots, a)
#define DELTA_LAUNCH_R(T, CH)                  \
    if (rmax == 16) { DELTA_LAUNCH(T, 16, CH); } \
    else { DELTA_LAUNCH(T, 32, CH); }
    if (dtype != MYNAH_F32 && dtype != MYNAH_BF16) return mynah_fail("delta_rule: unsupported dtype %d", dtype);
    if (channel_decay) {
        if (dtype == MYNAH_F32) { DELTA_LAUNCH_R(float, true); }
        else { DELTA_LAUNCH_R(bf16, true); }
    } else {
        if (dtype == MYNAH_F32) { DELTA_LAUNCH_R(float, false); }
        else { DELTA_LAUNCH_R(bf16, false); }
    }
#undef DELTA_LAUNCH_R
#undef DELTA_LAUNCH_TB
#undef DELTA_LAUNCH
    return mynah_check_launch("delta_rule");
}

// out[t, h, :] = o[t, h, :] / rms(o[t, h, :]) * w * act(gate[t, h, :]), act = silu, or sigmoid with gate_sigmoid;
// o fp32 [T, H*vd], gate [T, ldg] and out [T, H*vd] in dtype, w [vd] in w_dtype.
MYNAH_API int mynah_gated_rmsnorm(const float* o, const void* gate, int ldg, int dtype, const void* w, int w_dtype,
                                  void* out, int T, int H, int vd, float eps, int gate_sigmoid, cudaStream_t stream) {
    if (T == 0) return 0;
    MYNAH_REQUIRE(T > 0 && H > 0 && vd > 0, "gated_rmsnorm: bad sizes T=%d H=%d vd=%d", T, H, vd);
    const long long total = (long long)T * H;
    MYNAH_REQUIRE(total <= 0x7fffffffLL, "gated_rmsnorm: too many heads");
    const VecRef wv{w, w_dtype};
    const dim3 grid((unsigned)ceil_div_ll(total, 4));
    if (dtype == MYNAH_F32)
        mynah_launch(gated_rmsnorm_kernel<float>, grid, dim3(128), 0, stream, o, (const float*)gate, ldg, wv, (float*)out,
                     (int)total, H, vd, eps, gate_sigmoid);
    else if (dtype == MYNAH_BF16)
        mynah_launch(gated_rmsnorm_kernel<bf16>, grid, dim3(128), 0, stream, o, (const bf16*)gate, ldg, wv, (bf16*)out,
                     (int)total, H, vd, eps, gate_sigmoid);
    else
        return mynah_fail("gated_rmsnorm: unsupported dtype %d", dtype);
    return mynah_check_launch("gated_rmsnorm");
}
