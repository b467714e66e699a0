// Retention: linear attention with a fixed decay per head, no softmax and no denominator. Per head, with
// S [dim x vd] the state (fp32, carried per slot):
//
//   S_t = decay_h S_(t-1) + k_t v_t^T,      o_t = S_t^T q_t
//
// Kernels (the per-head unit RMS and the gate that follow are `gated_rmsnorm`):
//
//   retention_prep   q, k rows -> fp32, the first `rot` dims of every head rotated by the position's table row
//                    (pairs (i, i + rot/2), or (2i, 2i+1)), k then multiplied by k_scale
//   retention_scan   the recurrence. The columns of S are independent, so a CTA takes a tile of columns of one
//                    head of one sequence; a column's dim values lie in the registers of L adjacent lanes (up to
//                    32 values a lane), which add their parts of o by shuffles in a fixed order. Keys, queries and
//                    values of 32 tokens at a time pass through shared memory.
//   retention_local, _states, _out   the same recurrence for pieces of 16 tokens and more, a chunk of tokens at a time (see below)
//   retention_step   all of a decode step's row behind its projection, the RMS and the gate with it (see below)
//
// All arithmetic is fp32. Which form a sequence's rows take depends on their number alone, so a step's rows have the same bits in any
// company. Token by token the rows are walked in order, whatever pieces they come in; chunk by chunk the sums run in another
// order (the forms agree to rounding), so a prompt run whole and the same prompt in pieces differ by roundings.
#include "layout.cuh"

namespace {

struct RetPrepArgs {
    int H, dim, ld, q_off, k_off;    // heads, head size, row stride, first columns of q and k
    int rot, interleaved, n_pos;
    float k_scale;
};

// one CTA a token
template <typename T>
__global__ void __launch_bounds__(128)
retention_prep_kernel(const T* __restrict__ qk, float* __restrict__ qn, float* __restrict__ kn,
                      const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                      const int* __restrict__ tok_seq, const int* __restrict__ tok_pos, RetPrepArgs a,
                      int* __restrict__ status) {
    griddep_launch_small();
    griddep_wait();
    const int t = blockIdx.x;
    if (tok_seq[t] < 0) return;
    const int pos = tok_pos[t];
    const bool rotate = a.rot > 0 && cos_t != nullptr;
    if (rotate && (pos < 0 || pos >= a.n_pos)) {
        if (threadIdx.x == 0) atomicOr(status, MYNAH_ST_POS_RANGE);
        return;
    }
    const int half = a.rot >> 1;
    const float* cr = rotate ? cos_t + (size_t)pos * half : nullptr;
    const float* sr = rotate ? sin_t + (size_t)pos * half : nullptr;
    const int n = a.H * a.dim;
    const T* row = qk + (size_t)t * a.ld;
    for (int idx = threadIdx.x; idx < 2 * n; idx += blockDim.x) {
        const bool is_k = idx >= n;
        const int e = is_k ? idx - n : idx;
        const int h = e / a.dim, d = e % a.dim;
        const T* src = row + (is_k ? a.k_off : a.q_off) + (size_t)h * a.dim;
        float v = to_f32(src[d]);
        if (rotate && d < a.rot) {
            int i, other;
            float sign;
            if (a.interleaved) {
                i = d >> 1; other = d ^ 1; sign = (d & 1) ? 1.f : -1.f;
            } else {
                i = d < half ? d : d - half; other = d < half ? d + half : d - half; sign = d < half ? -1.f : 1.f;
            }
            v = v * cr[i] + sign * to_f32(src[other]) * sr[i];
        }
        if (is_k) kn[(size_t)t * n + e] = v * a.k_scale;
        else qn[(size_t)t * n + e] = v;
    }
}

// The same where eight values lie on 16-byte boundaries and a rotated pair's two halves do too: a thread takes eight of a head
// (and fetches the eight they are paired with), so that every access is a vector and a step of any size has all its loads in
// flight at once. 16 heads of 128, us: 4 rows 13.8 -> 2.7, 3,837 rows 57 -> 28.
template <typename T>
__global__ void __launch_bounds__(128)
retention_prep_vec_kernel(const T* __restrict__ qk, float* __restrict__ qn, float* __restrict__ kn,
                          const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                          const int* __restrict__ tok_seq, const int* __restrict__ tok_pos, RetPrepArgs a, int n_tok,
                          int* __restrict__ status) {
    griddep_launch_small();
    griddep_wait();
    const int n = a.H * a.dim, per = n / 8;                 // pieces of eight, q's then k's
    const int piece = blockIdx.x * blockDim.x + threadIdx.x, t = blockIdx.y + blockIdx.z * gridDim.y;
    if (piece >= 2 * per || t >= n_tok || tok_seq[t] < 0) return;
    const int pos = tok_pos[t];
    const bool rotate = a.rot > 0 && cos_t != nullptr;
    if (rotate && (pos < 0 || pos >= a.n_pos)) {
        if (piece == 0) atomicOr(status, MYNAH_ST_POS_RANGE);
        return;
    }
    const bool is_k = piece >= per;
    const int e = (is_k ? piece - per : piece) * 8, h = e / a.dim, d = e % a.dim;
    const T* src = qk + (size_t)t * a.ld + (is_k ? a.k_off : a.q_off) + (size_t)h * a.dim;
    auto load = [](const T* p, float (&x)[8]) {
        uint4 w[sizeof(T) / 2];
#pragma unroll
        for (int i = 0; i < (int)sizeof(T) / 2; i++) w[i] = reinterpret_cast<const uint4*>(p)[i];
        const T* y = reinterpret_cast<const T*>(w);
#pragma unroll
        for (int i = 0; i < 8; i++) x[i] = to_f32(y[i]);
    };
    float x[8], r[8];
    load(src + d, x);
#pragma unroll
    for (int j = 0; j < 8; j++) r[j] = x[j];
    if (rotate && d < a.rot) {
        const int half = a.rot >> 1;
        const float* cr = cos_t + (size_t)pos * half;
        const float* sr = sin_t + (size_t)pos * half;
        if (a.interleaved) {
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const float sign = (j & 1) ? 1.f : -1.f;
                r[j] = x[j] * cr[(d + j) >> 1] + sign * x[j ^ 1] * sr[(d + j) >> 1];
            }
        } else {
            const int i = d < half ? d : d - half;
            const float sign = d < half ? -1.f : 1.f;
            float y[8];
            load(src + (d < half ? d + half : d - half), y);
#pragma unroll
            for (int j = 0; j < 8; j++) r[j] = x[j] * cr[i + j] + sign * y[j] * sr[i + j];
        }
    }
    const float scale = is_k ? a.k_scale : 1.f;
    float4* dst = reinterpret_cast<float4*>((is_k ? kn : qn) + (size_t)t * n + e);
    dst[0] = make_float4(r[0] * scale, r[1] * scale, r[2] * scale, r[3] * scale);
    dst[1] = make_float4(r[4] * scale, r[5] * scale, r[6] * scale, r[7] * scale);
}

constexpr int RET_THREADS = 128;
constexpr int RET_TB = 32;                 // tokens staged in shared memory at a time
constexpr int RET_RMAX = 32;               // state values a lane keeps

struct RetArgs {
    int B, H, dim, vd, n_slots, ldv, v_off;
    int L, per;                            // lanes a column (a power of two <= 32), values a lane (<= RET_RMAX)
};

// Rows [q0, q1) of one sequence and head, columns [j0, j0 + THREADS / L), by a CTA of THREADS threads that stages TB tokens at a time in
// `sm` (walk_floats). A column's arithmetic does not depend on THREADS or TB.
__host__ __device__ constexpr size_t walk_floats(int threads, int tb, int L, int per) {
    return (size_t)2 * tb * (per + 1) * L + (size_t)tb * (threads / L);
}
template <typename T, int THREADS, int TB>
__device__ __forceinline__ void walk_tokens(float* sm, const float* __restrict__ qn, const float* __restrict__ kn, const T* __restrict__ v,
                                            float g, float* __restrict__ state, float* __restrict__ o, int q0, int q1, int slot, int h, int j0,
                                            const RetArgs& a) {
    qn += (size_t)h * a.dim;
    kn += (size_t)h * a.dim;
    v += a.v_off + (size_t)h * a.vd;
    o += (size_t)h * a.vd;
    const int L = a.L, per = a.per;
    const int JT = THREADS / L;
    const int l = threadIdx.x % L, jl = threadIdx.x / L;
    const int j = j0 + jl;
    const bool on = j < a.vd;
    const int CS = per + 1;                                      // floats of a lane's chunk (padded against bank conflicts)
    const int rowf = CS * L;
    float* ks = sm;                                              // [TB][rowf]
    float* qs = ks + TB * rowf;                                  // [TB][rowf]
    float* vs = qs + TB * rowf;                                  // [TB][JT]
    for (int i = threadIdx.x; i < 2 * TB * rowf; i += THREADS) ks[i] = 0.f;    // slots beyond dim stay zero
    float S[RET_RMAX];
    float* sp = state + (((size_t)slot * a.H + h) * a.dim) * a.vd;
#pragma unroll
    for (int r = 0; r < RET_RMAX; r++) {
        const int i = l * per + r;
        S[r] = (on && r < per && i < a.dim) ? sp[(size_t)i * a.vd + j] : 0.f;
    }
    const int n = a.H * a.dim;
    for (int t0 = q0; t0 < q1; t0 += TB) {
        const int nt = min(TB, q1 - t0);
        __syncthreads();
        for (int idx = threadIdx.x; idx < nt * a.dim; idx += THREADS) {
            const int tt = idx / a.dim, i = idx % a.dim;
            const size_t src = (size_t)(t0 + tt) * n + i;
            const int dst = tt * rowf + (i / per) * CS + i % per;
            ks[dst] = kn[src];
            qs[dst] = qn[src];
        }
        for (int idx = threadIdx.x; idx < nt * JT; idx += THREADS) {
            const int tt = idx / JT, c = idx % JT;
            vs[idx] = j0 + c < a.vd ? to_f32(v[(size_t)(t0 + tt) * a.ldv + j0 + c]) : 0.f;
        }
        __syncthreads();
        for (int tt = 0; tt < nt; tt++) {
            const float* kk = ks + tt * rowf + l * CS;
            const float* qq = qs + tt * rowf + l * CS;
            const float vj = vs[tt * JT + jl];
            float acc = 0.f;
#pragma unroll
            for (int r = 0; r < RET_RMAX; r++) {
                if (r < per) {
                    S[r] = fmaf(kk[r], vj, g * S[r]);
                    acc = fmaf(S[r], qq[r], acc);
                }
            }
            for (int m = 1; m < L; m <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
            if (on && l == 0) o[(size_t)(t0 + tt) * a.H * a.vd + j] = acc;
        }
    }
    if (on) {
#pragma unroll
        for (int r = 0; r < RET_RMAX; r++) {
            const int i = l * per + r;
            if (r < per && i < a.dim) sp[(size_t)i * a.vd + j] = S[r];
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(RET_THREADS)
retention_scan_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const T* __restrict__ v,
                      const float* __restrict__ decay, float* __restrict__ state, float* __restrict__ o,
                      const int* __restrict__ cu_q, const int* __restrict__ slots, RetArgs a) {
    extern __shared__ float scan_sm[];
    griddep_wait();
    const int b = blockIdx.z, h = blockIdx.y;
    const int slot = slots[b];
    const int q0 = cu_q[b], q1 = cu_q[b + 1];
    if (slot < 0 || slot >= a.n_slots || q1 <= q0) return;
    walk_tokens<T, RET_THREADS, RET_TB>(scan_sm, qn, kn, v, decay[h], state, o, q0, q1, slot, h, blockIdx.x * (RET_THREADS / a.L), a);
}

// ---- a decode step: preparation, one token of the recurrence, the unit RMS and the gate ----
// A CTA a (row, head), L lanes a column as in retention_scan: the state's 64 KB (128 x 128) are asked for at once and everything
// else is worked out meanwhile, so the step is one trip to memory instead of three launches. The arithmetic and its order are those of
// retention_prep, retention_scan and gated_rmsnorm. Rows without a sequence give zeros. Measured (16 heads of
// 128, us against the three launches): 2 rows 8.4 / 8.7, 4 rows 8.6 / 9.5, 8 rows 9.2 / 12.8; where the CTAs no longer run side by side the
// scan's many small ones win (16 rows 18.9 / 19.3, 32 rows 36.6 / 29.8), and one row leaves most SMs idle (8.3 / 7.9).
struct RetStepArgs {
    int H, dim, vd, n_slots, L, per, ld, q_off, k_off, v_off, g_off, ldo;
    int rot, interleaved, n_pos;
    float k_scale, eps;
};

template <typename T>
__global__ void __launch_bounds__(512)
retention_step_kernel(const T* __restrict__ p, const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                      const float* __restrict__ decay, float* __restrict__ state, VecRef w, T* __restrict__ out,
                      const int* __restrict__ tok_seq, const int* __restrict__ tok_pos, const int* __restrict__ slots, RetStepArgs a,
                      int* __restrict__ status) {
    __shared__ float qs[128 + 32], ks[128 + 32], os[512], zs[512];    // q and k: a lane's chunk, one float apart from the next
    griddep_launch_small();
    griddep_wait();
    const int h = blockIdx.x, b = blockIdx.y, tid = threadIdx.x;
    const int slot = slots[b], pos = tok_pos[b];
    const T* row = p + (size_t)b * a.ld;
    T* dst = out + (size_t)b * a.ldo + (size_t)h * a.vd;
    const bool rotate = a.rot > 0 && cos_t != nullptr;
    const bool bad_pos = rotate && (pos < 0 || pos >= a.n_pos);
    if (tok_seq[b] < 0 || slot < 0 || slot >= a.n_slots || bad_pos) {
        if (tok_seq[b] >= 0 && bad_pos && tid == 0) atomicOr(status, MYNAH_ST_POS_RANGE);
        for (int j = tid; j < a.vd; j += blockDim.x) dst[j] = from_f32<T>(0.f);
        return;
    }
    const int L = a.L, per = a.per, l = tid % L, j = tid / L;
    const bool on = j < a.vd;
    float* sp = state + (((size_t)slot * a.H + h) * a.dim) * a.vd;
    float S[RET_RMAX];
#pragma unroll
    for (int r = 0; r < RET_RMAX; r++) {
        const int i = l * per + r;
        S[r] = (on && r < per && i < a.dim) ? sp[(size_t)i * a.vd + j] : 0.f;
    }
    for (int e = tid; e < 2 * a.dim; e += blockDim.x) {
        const bool is_k = e >= a.dim;
        const int d = is_k ? e - a.dim : e, half = a.rot >> 1;
        const T* src = row + (is_k ? a.k_off : a.q_off) + (size_t)h * a.dim;
        float v = to_f32(src[d]);
        if (rotate && d < a.rot) {
            int i, other;
            float sign;
            if (a.interleaved) {
                i = d >> 1; other = d ^ 1; sign = (d & 1) ? 1.f : -1.f;
            } else {
                i = d < half ? d : d - half; other = d < half ? d + half : d - half; sign = d < half ? -1.f : 1.f;
            }
            v = v * cos_t[(size_t)pos * half + i] + sign * to_f32(src[other]) * sin_t[(size_t)pos * half + i];
        }
        (is_k ? ks : qs)[d + d / per] = is_k ? v * a.k_scale : v;
    }
    for (int d = tid; d < a.vd; d += blockDim.x) zs[d] = to_f32(row[a.g_off + (size_t)h * a.vd + d]);
    const float vj = on ? to_f32(row[a.v_off + (size_t)h * a.vd + j]) : 0.f, g = decay[h];
    __syncthreads();
    float acc = 0.f;
#pragma unroll
    for (int r = 0; r < RET_RMAX; r++) {
        if (r < per && l * per + r < a.dim) {
            S[r] = fmaf(ks[l * (per + 1) + r], vj, g * S[r]);
            acc = fmaf(S[r], qs[l * (per + 1) + r], acc);
        }
    }
    for (int m = 1; m < L; m <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
    if (on && l == 0) os[j] = acc;
#pragma unroll
    for (int r = 0; r < RET_RMAX; r++) {
        const int i = l * per + r;
        if (on && r < per && i < a.dim) sp[(size_t)i * a.vd + j] = S[r];
    }
    __syncthreads();
    if (tid >= 32) return;
    float ss = 0.f;
    for (int d = tid; d < a.vd; d += 32) ss = fmaf(os[d], os[d], ss);
    const float r = 1.0f / sqrtf(warp_sum(ss) / (float)a.vd + a.eps);
    for (int d = tid; d < a.vd; d += 32) {
        const float z = zs[d], sg = 1.0f / (1.0f + expf(-z));
        dst[d] = from_f32<T>(os[d] * r * w.at(d) * (z * sg));
    }
}

// ---- the recurrence chunk by chunk, for prompts ----
// With a chunk of C tokens, S the state before it and g the head's decay:
//
//   o_t   = sum_{s <= t} g^(t-s) (q_t . k_s) v_s  +  g^(t+1) S^T q_t                      t, s inside the chunk
//   S_new = g^n S + U,   U = sum_s g^(n-1-s) k_s v_s^T                                   n tokens in the chunk
//
// U does not depend on S, and o depends on nothing but S and the chunk, so only the elementwise recurrence over the
// chunks' states is a chain. Three kernels, all sums fp32:
//
//   retention_local   U of every chunk and head, into scratch [chunk][H][dim][columns]
//   retention_states  the chain: a thread takes four values of a state through its sequence's chunks, puts the state before
//                     a chunk in U's place and the last one into the slot
//   retention_out     the decayed scores of a chunk (kept in shared memory), the read of its old state, scores times values
//
// What bounds them: the multiply-adds (49,000 a token and head of 128 x 128, 3.1e9 a layer for 4,000 tokens of 16 heads: 88 us at
// the FFMA rate) and the reads of shared memory that feed them; the products run in pairs (fma.rn.f32x2, the same roundings),
// which halves the instructions beside the loads. Scratch is bounded: a step's chunks go in passes of about 96 MB of states
// (what the cache holds), in the order of their sequences. Measured (3,837 tokens of 4 sequences,
// 16 heads of 128), us a layer: 85 + 46 + 137; a chain of CTAs that each walked a head's 32 columns through its chunks took 625.
//
// Sequences of fewer than 16 rows in such a step are walked token by token, by the CTAs of retention_out that have their rows: a
// decode row beside a prompt costs a row's work, and has the bits it has among its like.
//
// Where no sequence has more than one chunk nothing is a chain: retention_out reads the old state from its slot and leaves the
// new one there, one launch instead of three. us with the preparation and the gated norm, 16 heads of 128: one sequence of 20, 48,
// 64 rows 36.2, 40.3, 42.4 -> 23.4, 28.5, 31.1; 16 of 32 83 -> 41; 64 of 40 424 -> 175; a prompt of 70 beside 60 decode rows 322 -> 103.
//
// The powers of g come from a table made by repeated multiplication. Sums run in another order than token by token:
// the two forms agree to rounding.
constexpr int RC_THREADS = 256;
constexpr int WALK_TB = 16;                                 // tokens staged at a time where the chunks' CTAs walk a short sequence

struct RetChunkArgs {
    int H, dim, vd, n_slots, ldv, v_off, B, cols;          // cols: columns of a state in scratch (vd padded to whole tiles)
    int first;                                              // the pass's first chunk
    int least;                                              // rows from which a sequence goes chunk by chunk
    RetArgs walk;                                           // shorter ones are walked token by token
};

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

// gp[n] = g^n, n <= C
template <int C>
__device__ __forceinline__ void decay_powers(float* gp, float g) {
    if (threadIdx.x == 0) {
        float p = 1.f;
        for (int n = 0; n <= C; n++) {
            gp[n] = p;
            p *= g;
        }
    }
}

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

// A thread's part of U from a chunk's keys (rows ldk apart) and values in shared memory: eight state rows, four columns of either half
// of the tile. WEIGH: the values are yet to be multiplied by the powers of the decay.
template <int JT, bool WEIGH>
__device__ __forceinline__ void chunk_update(const float* kr, int ldk, const float* vr, int nt, const float* gp, f32x2 (&acc)[8][4]) {
#pragma unroll
    for (int u = 0; u < 8; u++)
#pragma unroll
        for (int w = 0; w < 4; w++) acc[u][w] = 0ull;
#pragma unroll 2
    for (int s = 0; s < nt; s++) {
        const float4 k0 = *reinterpret_cast<const float4*>(kr + s * ldk), k1 = *reinterpret_cast<const float4*>(kr + s * ldk + 4);
        Pairs v0 = pairs_at(vr + s * JT), v1 = pairs_at(vr + s * JT + JT / 2);
        if (WEIGH) {
            const f32x2 w = pack2(gp[nt - 1 - s], gp[nt - 1 - s]);
            mul2(v0.lo, w);
            mul2(v0.hi, w);
            mul2(v1.lo, w);
            mul2(v1.hi, w);
        }
        const float kk[8] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w};
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const f32x2 k2 = pack2(kk[u], kk[u]);
            fma2(acc[u][0], k2, v0.lo);
            fma2(acc[u][1], k2, v0.hi);
            fma2(acc[u][2], k2, v1.lo);
            fma2(acc[u][3], k2, v1.hi);
        }
    }
}

// grid (chunks of the pass, H, cols / JT): the step's chunks are numbered sequence by sequence (layout.cuh: find_query_tile).
// Thread (ti, tj) owns state rows ti * 8 + u and columns tj * 4 + {0..3} of either half of the tile.
template <typename T, int C, int JT>
__global__ void __launch_bounds__(RC_THREADS, 2)
retention_local_kernel(const float* __restrict__ kn, const T* __restrict__ v, const float* __restrict__ decay, float* __restrict__ states,
                       const int* __restrict__ cu_q, RetChunkArgs a) {
    extern __shared__ __align__(16) float sm[];
    __shared__ float gp[C + 1];
    griddep_wait();
    int b, tile;
    if (!find_query_tile(cu_q, a.B, C, a.first + (int)blockIdx.x, b, tile) || cu_q[b + 1] - cu_q[b] < a.least) return;
    const int h = blockIdx.y, d = a.dim, j0 = blockIdx.z * JT;
    const int t0 = cu_q[b] + tile * C, nt = min(C, cu_q[b + 1] - t0);
    float* ks = sm;                        // [C][d + 4]
    float* vs = ks + C * (d + 4);          // [C][JT]
    decay_powers<C>(gp, decay[h]);
    const size_t n = (size_t)a.H * d;
    stage_rows<C>(ks, kn + (size_t)t0 * n + (size_t)h * d, n, d, nt);
    __syncthreads();
    stage_values<T, C, JT>(vs, v + (size_t)t0 * a.ldv + a.v_off + (size_t)h * a.vd, a.ldv, j0, a.vd, nt,
                           [&](int tt) { return gp[nt - 1 - tt]; });
    __syncthreads();
    const int ti = threadIdx.x / (JT / 8), tj = threadIdx.x % (JT / 8);
    if (ti * 8 >= d) return;
    f32x2 acc[8][4];
    chunk_update<JT, false>(ks + ti * 8, d + 4, vs + tj * 4, nt, gp, acc);
    float* out = states + (((size_t)blockIdx.x * a.H + h) * d + ti * 8) * a.cols + j0 + tj * 4;
#pragma unroll
    for (int u = 0; u < 8; u++) {
        *reinterpret_cast<Pairs*>(out + (size_t)u * a.cols) = Pairs{acc[u][0], acc[u][1]};
        *reinterpret_cast<Pairs*>(out + (size_t)u * a.cols + JT / 2) = Pairs{acc[u][2], acc[u][3]};
    }
}

// grid (dim * cols / 4 / 256, H, B): four values of one state a thread, through the pass's chunks of sequence b.
__global__ void __launch_bounds__(RC_THREADS)
retention_states_kernel(const float* __restrict__ decay, float* __restrict__ states, float* __restrict__ state,
                        const int* __restrict__ cu_q, const int* __restrict__ slots, RetChunkArgs a, int C, int n_pass) {
    __shared__ int parts[RC_THREADS / 32];
    griddep_wait();
    const int b = blockIdx.z, h = blockIdx.y;
    const int q0 = cu_q[b], q1 = cu_q[b + 1], slot = slots[b];
    // the sequence's first chunk number: those of the sequences before it
    int before = 0;
    for (int i = threadIdx.x; i < b; i += RC_THREADS) before += (cu_q[i + 1] - cu_q[i] + C - 1) / C;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
    if ((threadIdx.x & 31) == 0) parts[threadIdx.x >> 5] = before;
    __syncthreads();
    before = 0;
#pragma unroll
    for (int w = 0; w < RC_THREADS / 32; w++) before += parts[w];
    const int tiles = (q1 - q0 + C - 1) / C;
    // tile t of the sequence is number before + tiles - 1 - t; this pass holds the numbers [first, first + n_pass)
    const int last_no = before + tiles - 1;
    const int t_lo = max(0, last_no - (a.first + n_pass - 1)), t_hi = min(tiles, last_no - a.first + 1);
    if (t_lo >= t_hi || slot < 0 || slot >= a.n_slots || q1 - q0 < a.least) return;
    const int e = blockIdx.x * RC_THREADS + threadIdx.x, per_row = a.cols / 4;
    const int i = e / per_row, c = (e % per_row) * 4;
    if (i >= a.dim || c >= a.vd) return;
    const float g = decay[h];
    float gc = 1.f, gl = 1.f;                               // the decay over a whole chunk, over the sequence's last
    for (int k = 0; k < C; k++) {
        if (k == q1 - q0 - (tiles - 1) * C) gl = gc;
        gc *= g;
    }
    if (q1 - q0 == tiles * C) gl = gc;
    float* sp = state + (((size_t)slot * a.H + h) * a.dim + i) * a.vd + c;
    const int have = min(4, a.vd - c);
    float S[4];
#pragma unroll
    for (int k = 0; k < 4; k++) S[k] = k < have ? sp[k] : 0.f;
    const size_t one = (size_t)a.H * a.dim * a.cols;        // floats of a chunk
    float* at = states + ((size_t)h * a.dim + i) * a.cols + c;
    constexpr int AHEAD = 8;
    for (int t = t_lo; t < t_hi; t += AHEAD) {
        float4 u[AHEAD];
#pragma unroll
        for (int k = 0; k < AHEAD; k++)
            if (t + k < t_hi) u[k] = *reinterpret_cast<const float4*>(at + (size_t)(last_no - (t + k) - a.first) * one);
#pragma unroll
        for (int k = 0; k < AHEAD; k++) {
            if (t + k < t_hi) {
                *reinterpret_cast<float4*>(at + (size_t)(last_no - (t + k) - a.first) * one) = make_float4(S[0], S[1], S[2], S[3]);
                const float gn = t + k == tiles - 1 ? gl : gc;
                S[0] = fmaf(gn, S[0], u[k].x);
                S[1] = fmaf(gn, S[1], u[k].y);
                S[2] = fmaf(gn, S[2], u[k].z);
                S[3] = fmaf(gn, S[3], u[k].w);
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (k < have) sp[k] = S[k];
}

// The same grid as retention_local. Thread (ty, tx) owns tokens ty * RT + u and columns tx * 4 + {0..3} (of either half, when the
// tile has 128). The keys' place in shared memory is used again by the old state, 32 rows at a time, and then by the values.
// ONE: grid (B, H, cols / JT), a sequence's only chunk: the old state comes from its slot (vd a multiple of 4), whose columns of this
// tile nobody else touches, and the new one goes there, in the operations of retention_local and retention_states.
template <typename T, int C, int JT, bool ONE>
__global__ void __launch_bounds__(RC_THREADS, 2)
retention_out_kernel(const float* __restrict__ qn, const float* __restrict__ kn, const T* __restrict__ v, const float* __restrict__ decay,
                     const float* __restrict__ states, float* state, float* __restrict__ o, const int* __restrict__ cu_q,
                     const int* __restrict__ slots, RetChunkArgs a) {
    constexpr int RT = C / 16, G = JT / 64, LDW = C + 4, SR = 32;
    extern __shared__ __align__(16) float sm[];
    __shared__ float gp[C + 1];
    griddep_wait();
    int b = blockIdx.x, tile = 0;
    if (!ONE && !find_query_tile(cu_q, a.B, C, a.first + (int)blockIdx.x, b, tile)) return;
    const int slot = slots[b];
    if (slot < 0 || slot >= a.n_slots || cu_q[b + 1] <= cu_q[b]) return;
    if (cu_q[b + 1] - cu_q[b] < a.least) {                  // (uniform)
        if (tile == 0) {
            const int wide = RC_THREADS / a.walk.L, j_end = min(a.vd, ((int)blockIdx.z + 1) * JT);
            for (int j = blockIdx.z * JT; j < j_end; j += wide) {
                walk_tokens<T, RC_THREADS, WALK_TB>(sm, qn, kn, v, decay[blockIdx.y], state, o, cu_q[b], cu_q[b + 1], slot, blockIdx.y, j, a.walk);
                __syncthreads();                            // shared memory is free again
            }
        }
        return;
    }
    const int h = blockIdx.y, d = a.dim, j0 = blockIdx.z * JT, ldr = d + 4;
    const int t0 = cu_q[b] + tile * C, nt = min(C, cu_q[b + 1] - t0);
    float* qs = sm;                        // [C][ldr]
    float* Ws = qs + C * ldr;              // [C][LDW]
    float* xs = Ws + C * LDW;              // [C][ldr] keys; [2][SR][JT] state rows; [C][JT] values
    decay_powers<C>(gp, decay[h]);
    const size_t n = (size_t)a.H * d;
    stage_rows<C>(qs, qn + (size_t)t0 * n + (size_t)h * d, n, d, nt);
    stage_rows<C>(xs, kn + (size_t)t0 * n + (size_t)h * d, n, d, nt);
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
            for (int u = 0; u < RT; u++) {
                if (16 * u >= nt) break;                    // uniform: no token of the group exists
#pragma unroll
                for (int w = 0; w <= u; w++) {              // (keys behind every token of the group: not needed)
                    fma2(acc[u][w], qv[u].lo, kv[w].lo);
                    fma2(acc[u][w], qv[u].hi, kv[w].hi);
                }
            }
        }
#pragma unroll
        for (int u = 0; u < RT; u++)
#pragma unroll
            for (int w = 0; w < RT; w++) {
                const int t = ty + 16 * u, s = tx + 16 * w;
                const float2 x = unpack2(acc[u][w]);
                Ws[t * LDW + s] = s <= t ? gp[t - s] * (x.x + x.y) : 0.f;
            }
    }
    __syncthreads();                                        // the scores are there, the keys are done with
    f32x2 acc[RT][G][2];
#pragma unroll
    for (int u = 0; u < RT; u++)
#pragma unroll
        for (int w = 0; w < G; w++) acc[u][w][0] = acc[u][w][1] = 0ull;
    // one product's four steps of k: rows [ty * RT, + RT) of `lhs` from column i, rows [i, i + 4) of `rhs`
    auto steps = [&](const float* lhs, int ld, const float* rhs, f32x2 (&acc)[RT][G][2]) {
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
    const int ldS = ONE ? a.vd : a.cols;
    float* own = ONE ? state + (((size_t)slot * a.H + h) * d) * a.vd + j0 : nullptr;
    const float* from = ONE ? own : states + ((size_t)blockIdx.x * a.H + h) * d * a.cols + j0;
    const bool busy = (ty & ~1) * RT < nt;                  // a token of the warp's rows exists
    auto fetch = [&](int piece) {
        if (piece * SR < d) {
            float* dst = xs + (piece & 1) * SR * JT;
#pragma unroll
            for (int idx = threadIdx.x; idx < SR * JT / 4; idx += RC_THREADS) {
                const int i = idx / (JT / 4), c = (idx % (JT / 4)) * 4;
                const uint32_t s = (uint32_t)__cvta_generic_to_shared(dst + i * JT + c);
                const bool in = !ONE || j0 + c < a.vd;      // (beyond the state's columns: zeros, nothing read)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(s), "l"(from + (in ? (size_t)(piece * SR + i) * ldS + c : 0)), "r"(in ? 16 : 0) : "memory");
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
        for (int i = 0; i < SR; i += 4)
            if (busy) steps(qs + p * SR + i, ldr, S + i * JT, acc);
        __syncthreads();                                    // the piece's place may be filled again
    }
    // ---- scores times values, summed apart from the state's part: the roundings of a sum are of its own size
    if (ONE) stage_rows<C>(qs, kn + (size_t)t0 * n + (size_t)h * d, n, d, nt);      // (the keys once more, where the queries were)
    stage_values<T, C, JT>(xs, v + (size_t)t0 * a.ldv + a.v_off + (size_t)h * a.vd, a.ldv, j0, a.vd, nt, [](int) { return 1.f; });
    __syncthreads();
    f32x2 within[RT][G][2];
#pragma unroll
    for (int u = 0; u < RT; u++)
#pragma unroll
        for (int w = 0; w < G; w++) within[u][w][0] = within[u][w][1] = 0ull;
    const int s_end = busy ? ((ty | 1) + 1) * RT : 0;       // keys behind the last token of the warp's rows weigh nothing
    for (int s = 0; s < s_end; s += 4) steps(Ws + s, LDW, xs + s * JT, within);
#pragma unroll
    for (int u = 0; u < RT; u++) {
        const int t = ty * RT + u;
        if (t >= nt) break;
        const f32x2 gt = pack2(gp[t + 1], gp[t + 1]);
        float* row = o + (size_t)(t0 + t) * a.H * a.vd + (size_t)h * a.vd;
#pragma unroll
        for (int w = 0; w < G; w++) {
            const int j = j0 + w * 64 + tx * 4;
            fma2(within[u][w][0], gt, acc[u][w][0]);
            fma2(within[u][w][1], gt, acc[u][w][1]);
            const float2 x = unpack2(within[u][w][0]), y = unpack2(within[u][w][1]);
            if (j + 3 < a.vd && (a.vd & 3) == 0) {
                *reinterpret_cast<float4*>(row + j) = make_float4(x.x, x.y, y.x, y.y);
            } else {
                if (j < a.vd) row[j] = x.x;
                if (j + 1 < a.vd) row[j + 1] = x.y;
                if (j + 2 < a.vd) row[j + 2] = y.x;
                if (j + 3 < a.vd) row[j + 3] = y.y;
            }
        }
    }
    if constexpr (ONE) {                                    // the state
        const int ti = threadIdx.x / (JT / 8), tj = threadIdx.x % (JT / 8);
        if (ti * 8 >= d) return;
        f32x2 U[8][4];
        chunk_update<JT, true>(qs + ti * 8, ldr, xs + tj * 4, nt, gp, U);
        const float gn = gp[nt];
#pragma unroll
        for (int half = 0; half < 2; half++) {
            const int c = tj * 4 + half * (JT / 2);
            if (j0 + c >= a.vd) continue;
#pragma unroll
            for (int u = 0; u < 8; u++) {
                float4* at = reinterpret_cast<float4*>(own + (size_t)(ti * 8 + u) * a.vd + c);
                const float4 S = *at;
                const float2 x = unpack2(U[u][2 * half]), y = unpack2(U[u][2 * half + 1]);
                *at = make_float4(fmaf(gn, S.x, x.x), fmaf(gn, S.y, x.y), fmaf(gn, S.z, y.x), fmaf(gn, S.w, y.y));
            }
        }
    }
}

// How a step's chunks go: tokens a chunk, columns a tile, padded columns of a state, chunks a pass.
struct RetPlan {
    int C, JT, cols, total, n_pass;
    bool one;                                               // no sequence has more than one chunk, and a launch does it all
    RetPlan(int rows, int B, int H, int dim, int vd, int max_q_len) {
        C = dim <= 128 ? 64 : 32;                           // (q and k of a chunk and a piece of the state: 86 KB a CTA, two an SM)
        one = max_q_len <= C && vd % 4 == 0;
        total = one ? B : rows / C + B;                     // at most
        // narrow tiles while even those leave no SM two CTAs (16 heads of 128: one sequence of 200 rows 43.9 -> 38.2 us, of 300 rows, with 160
        // narrow CTAs, 45.4 -> 48.5)
        JT = dim <= 128 && vd > 64 && (long long)total * H * ceil_div(vd, 64) > mynah_sm_count() ? 128 : 64;
        cols = ceil_div(vd, JT) * JT;
        const long long one = (long long)H * dim * cols;
        const long long fit = (96ll << 20) / 4 / one;
        const int least = ceil_div(2 * mynah_sm_count(), H);
        const int most = (int)(fit < least ? least : fit > total ? total : fit);
        const int passes = ceil_div(total, most);
        n_pass = ceil_div(total, passes);
    }
    long long floats(int H, int dim) const { return one ? 0 : (long long)n_pass * H * dim * cols; }
    int launches() const { return one ? 1 : 3 * ceil_div(total, n_pass); }
};

template <typename T, int C, int JT>
int launch_chunked(const float* qn, const float* kn, const void* v, const float* decay, float* states, float* state, float* o,
                   const int* cu_q, const int* slots, RetChunkArgs a, const RetPlan& plan, cudaStream_t stream) {
    const int d = a.dim;
    const size_t local = ((size_t)C * (d + 4) + (size_t)C * JT) * sizeof(float);
    const size_t shared_part = (size_t)C * (d + 4) > (size_t)64 * JT ? (size_t)C * (d + 4) : (size_t)64 * JT;
    const size_t out = ((size_t)C * (d + 4) + (size_t)C * (C + 4) + shared_part) * sizeof(float);
    if (walk_floats(RC_THREADS, WALK_TB, a.walk.L, a.walk.per) * sizeof(float) > out) return mynah_fail("retention_scan: a short sequence's walk does not fit");
    if (cudaFuncSetAttribute(retention_local_kernel<T, C, JT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 112 * 1024) != cudaSuccess ||
        cudaFuncSetAttribute(retention_out_kernel<T, C, JT, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 112 * 1024) != cudaSuccess ||
        cudaFuncSetAttribute(retention_out_kernel<T, C, JT, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 112 * 1024) != cudaSuccess)
        return mynah_fail("retention_scan: %zu bytes of shared memory are not to be had", out);
    if (plan.one) {
        mynah_launch(retention_out_kernel<T, C, JT, true>, dim3(a.B, a.H, plan.cols / JT), dim3(RC_THREADS), out, stream, qn, kn, (const T*)v, decay,
                     (const float*)nullptr, state, o, cu_q, slots, a);
        return mynah_check_launch("retention_scan (one chunk)");
    }
    // a sequence's chunks are numbered from its last to its first, so the passes go from the last to the first too
    for (int p = (plan.total - 1) / plan.n_pass; p >= 0; p--) {
        a.first = p * plan.n_pass;
        const dim3 grid(plan.n_pass, a.H, plan.cols / JT);
        mynah_launch(retention_local_kernel<T, C, JT>, grid, dim3(RC_THREADS), local, stream, kn, (const T*)v, decay, states, cu_q, a);
        mynah_launch(retention_states_kernel, dim3(ceil_div(d * (plan.cols / 4), RC_THREADS), a.H, a.B), dim3(RC_THREADS), 0, stream,
                     decay, states, state, cu_q, slots, a, C, plan.n_pass);
        mynah_launch(retention_out_kernel<T, C, JT, false>, grid, dim3(RC_THREADS), out, stream, qn, kn, (const T*)v, decay,
                     (const float*)states, state, o, cu_q, slots, a);
        if (mynah_check_launch("retention_scan (chunked)") != 0) return -1;
    }
    return 0;
}

}  // namespace

// 0: every sequence is walked token by token; otherwise those that bring at least this many tokens go chunk by chunk.
static int g_ret_chunk_min = 16;
MYNAH_API int mynah_retention_chunk_min(int n) {
    const int before = g_ret_chunk_min;
    g_ret_chunk_min = n;
    return before;
}

static bool retention_chunked(int dim, int max_q_len) {
    return g_ret_chunk_min > 0 && max_q_len >= g_ret_chunk_min && dim % 32 == 0 && dim <= 256;
}

// Floats of scratch that mynah_retention_scan wants for a step of `rows` rows (0: it walks token by token), and its launches.
MYNAH_API long long mynah_retention_scratch_floats(int rows, int B, int H, int dim, int vd, int max_q_len, int* launches) {
    if (!retention_chunked(dim, max_q_len) || rows <= 0) {
        *launches = 1;
        return 0;
    }
    const RetPlan plan(rows, B, H, dim, vd, max_q_len);
    *launches = plan.launches();
    return plan.floats(H, dim);
}

// qk: rows that hold every head's q from column q_off and every head's k from column k_off; qn, kn: fp32 [T][H*dim].
MYNAH_API int mynah_retention_prep(const void* qk, int ld, int q_off, int k_off, int dtype, float* qn, float* kn,
                                   int T, int H, int dim, const float* cos_t, const float* sin_t, int rot,
                                   int interleaved, int n_pos, float k_scale, const int* tok_seq, const int* tok_pos,
                                   int* status, cudaStream_t stream) {
    if (T == 0) return 0;
    MYNAH_REQUIRE(T > 0 && H > 0 && dim > 0, "retention_prep: bad sizes");
    MYNAH_REQUIRE(rot % 2 == 0 && rot <= dim, "retention_prep: %d rotated dims do not fit a head of %d", rot, dim);
    const RetPrepArgs a{H, dim, ld, q_off, k_off, cos_t ? rot : 0, interleaved, n_pos, k_scale};
    const int size = dtype == MYNAH_BF16 ? 2 : 4;
    const bool vec = dim % 8 == 0 && a.rot % (interleaved ? 8 : 16) == 0 && (ld * size) % 16 == 0 && (q_off * size) % 16 == 0
                     && (k_off * size) % 16 == 0 && (((uintptr_t)qk | (uintptr_t)qn | (uintptr_t)kn) & 15) == 0;
    if (vec && (dtype == MYNAH_F32 || dtype == MYNAH_BF16)) {
        const int y = T < 32768 ? T : 32768;
        const dim3 grid(ceil_div(H * dim / 4, 128), y, ceil_div(T, y));
        if (dtype == MYNAH_F32)
            mynah_launch(retention_prep_vec_kernel<float>, grid, dim3(128), 0, stream, (const float*)qk, qn, kn, cos_t, sin_t, tok_seq,
                         tok_pos, a, T, status);
        else
            mynah_launch(retention_prep_vec_kernel<bf16>, grid, dim3(128), 0, stream, (const bf16*)qk, qn, kn, cos_t, sin_t, tok_seq,
                         tok_pos, a, T, status);
        return mynah_check_launch("retention_prep");
    }
    if (dtype == MYNAH_F32)
        mynah_launch(retention_prep_kernel<float>, dim3(T), dim3(128), 0, stream, (const float*)qk, qn, kn, cos_t, sin_t,
                     tok_seq, tok_pos, a, status);
    else if (dtype == MYNAH_BF16)
        mynah_launch(retention_prep_kernel<bf16>, dim3(T), dim3(128), 0, stream, (const bf16*)qk, qn, kn, cos_t, sin_t,
                     tok_seq, tok_pos, a, status);
    else
        return mynah_fail("retention_prep: unsupported dtype %d", dtype);
    return mynah_check_launch("retention_prep");
}

// v: rows whose columns [v_off + h * vd, ...) are head h's values; decay: fp32 [H]; state: fp32 [n_slots + 1][H][dim][vd];
// o: fp32 [T][H * vd]. max_q_len: no sequence brings more tokens; rows: the step's rows; scratch: mynah_retention_scratch_floats(...)
// floats (null where those are 0, or to have every sequence walked token by token).
MYNAH_API int mynah_retention_scan(const float* qn, const float* kn, const void* v, int ldv, int v_off, int v_dtype,
                                   const float* decay, float* state, int n_slots, float* o, const int* cu_q,
                                   const int* slots, int B, int H, int dim, int vd, int max_q_len, int rows, float* scratch,
                                   cudaStream_t stream) {
    if (B == 0) return 0;
    MYNAH_REQUIRE(B > 0 && H > 0 && dim > 0 && vd > 0, "retention_scan: bad sizes");
    MYNAH_REQUIRE(dim <= 512, "retention_scan: keys of %d values exceed the 512 that the kernel stages", dim);
    MYNAH_REQUIRE(H <= 65535 && B <= 65535, "retention_scan: too many heads or sequences for one launch");
    MYNAH_REQUIRE(v_dtype == MYNAH_F32 || v_dtype == MYNAH_BF16, "retention_scan: unsupported dtype %d", v_dtype);
    int L = 1;
    while (L * RET_RMAX < dim) L <<= 1;
    const int per = ceil_div(dim, L);
    const int JT = RET_THREADS / L;
    const RetArgs a{B, H, dim, vd, n_slots, ldv, v_off, L, per};
    const RetPlan plan(rows, B, H, dim, vd, max_q_len);
    if (retention_chunked(dim, max_q_len) && (plan.one ? ((uintptr_t)state & 15) == 0 : scratch != nullptr) &&
        (((uintptr_t)qn | (uintptr_t)kn | (uintptr_t)scratch) & 15) == 0) {
        const RetChunkArgs ca{H, dim, vd, n_slots, ldv, v_off, B, plan.cols, 0, g_ret_chunk_min, a};
        MYNAH_REQUIRE(plan.cols / plan.JT <= 65535, "retention_scan: too many columns for one launch");
#define RET_CHUNKED(T, C, JT) launch_chunked<T, C, JT>(qn, kn, v, decay, scratch, state, o, cu_q, slots, ca, plan, stream)
        if (v_dtype == MYNAH_F32) return plan.C == 32 ? RET_CHUNKED(float, 32, 64) : plan.JT == 64 ? RET_CHUNKED(float, 64, 64) : RET_CHUNKED(float, 64, 128);
        return plan.C == 32 ? RET_CHUNKED(bf16, 32, 64) : plan.JT == 64 ? RET_CHUNKED(bf16, 64, 64) : RET_CHUNKED(bf16, 64, 128);
#undef RET_CHUNKED
    }
    const size_t smem = walk_floats(RET_THREADS, RET_TB, L, per) * sizeof(float);
    const dim3 grid(ceil_div(vd, JT), H, B);
    if (v_dtype == MYNAH_F32) {
        if (smem > 48 * 1024) cudaFuncSetAttribute(retention_scan_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        mynah_launch(retention_scan_kernel<float>, grid, dim3(RET_THREADS), smem, stream, qn, kn, (const float*)v, decay, state, o, cu_q, slots, a);
    } else if (v_dtype == MYNAH_BF16) {
        if (smem > 48 * 1024) cudaFuncSetAttribute(retention_scan_kernel<bf16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        mynah_launch(retention_scan_kernel<bf16>, grid, dim3(RET_THREADS), smem, stream, qn, kn, (const bf16*)v, decay, state, o, cu_q, slots, a);
    } else
        return mynah_fail("retention_scan: unsupported dtype %d", v_dtype);
    return mynah_check_launch("retention_scan");
}

// A decode step's rows, one a sequence: p [B, ld] holds every head's q, k, v and gate from their columns on; state as above; w [vd]
// in w_dtype; out [B, ldo] in dtype. Keys of up to 128 values, value heads of up to 512 / (lanes a column).
MYNAH_API int mynah_retention_step_supported(int dim, int vd) {
    int L = 1;
    while (L * RET_RMAX < dim) L <<= 1;
    return dim > 0 && dim <= 128 && vd > 0 && L * vd <= 512;
}
// Whether it is the faster form for B rows: a CTA an SM at most, and more than a handful (figures at the kernel). Smaller states move the
// upper end out and leave the lower one without a loss, us against the three launches: 8 heads of 64 1 row 6.5 / 9.1, 64 rows
// 8.1 / 13.2; 32 heads of 32 1 row 7.0 / 8.6, 64 rows 8.6 / 20.9; 64 heads of 128 2 rows 9.6 / 13.2, 4 rows 17.3 / 17.3; within
// the rule it never loses.
MYNAH_API int mynah_retention_step_pays(int B, int H) {
    return (long long)B * H >= 32 && (long long)B * H <= mynah_sm_count();
}
MYNAH_API int mynah_retention_step(const void* p, int ld, int q_off, int k_off, int v_off, int g_off, int dtype, const float* cos_t,
                                   const float* sin_t, int rot, int interleaved, int n_pos, float k_scale, const float* decay,
                                   float* state, int n_slots, const void* w, int w_dtype, float eps, void* out, int ldo, int B, int H,
                                   int dim, int vd, const int* tok_seq, const int* tok_pos, const int* slots, int* status,
                                   cudaStream_t stream) {
    if (B == 0) return 0;
    MYNAH_REQUIRE(B > 0 && H > 0 && B <= 65535 && mynah_retention_step_supported(dim, vd), "retention_step: bad sizes B=%d H=%d dim=%d vd=%d", B, H, dim, vd);
    MYNAH_REQUIRE(rot % 2 == 0 && rot <= dim, "retention_step: %d rotated dims do not fit a head of %d", rot, dim);
    int L = 1;
    while (L * RET_RMAX < dim) L <<= 1;
    const RetStepArgs a{H, dim, vd, n_slots, L, ceil_div(dim, L), ld, q_off, k_off, v_off, g_off, ldo, cos_t ? rot : 0, interleaved, n_pos, k_scale, eps};
    const dim3 grid(H, B), block(ceil_div(L * vd, 32) * 32);
    const VecRef wv{w, w_dtype};
    if (dtype == MYNAH_F32)
        mynah_launch(retention_step_kernel<float>, grid, block, 0, stream, (const float*)p, cos_t, sin_t, decay, state, wv, (float*)out, tok_seq, tok_pos,
                     slots, a, status);
    else if (dtype == MYNAH_BF16)
        mynah_launch(retention_step_kernel<bf16>, grid, block, 0, stream, (const bf16*)p, cos_t, sin_t, decay, state, wv, (bf16*)out, tok_seq, tok_pos,
                     slots, a, status);
    else
        return mynah_fail("retention_step: unsupported dtype %d", dtype);
    return mynah_check_launch("retention_step");
}
