// One page of decode attention on tensor cores: what the per-page kernels of attn_decode_tc.cu and the whole-step kernel
// of decode_layers.cu share (which keys a page shows, the arithmetic of a page's partial result, the tiles' layouts).
// Four warps work on a page together; they may be any aligned four of a CTA.
#pragma once
#include "layout.cuh"
#include "head_prep.cuh"
#include "tcgen05.cuh"

namespace {

constexpr int KEYS = PAGE_TOKENS;     // 64 keys per CTA
constexpr int WARPS = 4;
constexpr int MAX_G = 16;             // query heads per kv head that one MMA tile holds
constexpr int MERGE_MAX_BYTES = KEYS * 64 * 2;   // the merge's weights: (heads per group) * (pages) floats; the smaller K tile holds them

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src, bool valid) {
    const int n = valid ? 16 : 0;     // 0 source bytes: the 16 bytes are zero-filled
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(n));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// The first key that a sequence's newest position (hi - 1) sees. `window` carries either bound: W > 0 keeps the last
// W positions; -C < 0 is a chunk mask, keys from floor((hi - 1) / C) * C on; 0: every key.
__device__ __forceinline__ int first_visible(int hi, int window) {
    if (window > 0) return max(0, hi - window);
    if (window < 0 && hi > 0) return ((hi - 1) / -window) * -window;
    return 0;
}

struct TcArgs {
    int H, KV, ldq;
    int window, S;          // window: see first_visible
    float scale;
    int keep_first = 0;     // with a window (> 0): keys at positions below it are seen whatever their distance; the page
                            // lists must then hold every page of a sequence
    int vdiv = 1;           // kv head g reads value head g / vdiv (the value cache has KV / vdiv heads)
    float softcap = 0.f;    // c > 0: score <- c tanh(score / c), after the scale
    int null_key = 0;       // 1: the softmax has one more term, of score 0 and without a value (the merge adds it)
    float out_scale = 1.f;  // factor on the output rows
    int vdo = 0;            // columns of a head in the output rows; 0: the value head's width
    const float* sink = nullptr;   // null, or the further term's score a query head (the merge adds it)
};

// The pages that a sequence's newest position sees: pages [pg0, pg1) of its window (or of everything), and before them
// `nf` pages that hold kept first tokens and lie wholly before the window.
struct VisiblePages {
    int lo, pg0, pg1, nf;
    __device__ __forceinline__ int count() const { return nf + pg1 - pg0; }
    __device__ __forceinline__ int page(int s) const { return s < nf ? s : (pg0 + s - nf < pg1 ? pg0 + s - nf : -1); }
};
__device__ __forceinline__ VisiblePages visible_pages(int hi, int window, int keep_first) {
    VisiblePages v{0, 0, 0, 0};
    if (hi <= 0) return v;
    v.lo = first_visible(hi, window);
    v.pg0 = v.lo / PAGE_TOKENS;
    v.pg1 = (hi - 1) / PAGE_TOKENS + 1;
    if (window > 0 && keep_first > 0) v.nf = min((keep_first + PAGE_TOKENS - 1) / PAGE_TOKENS, v.pg0);
    return v;
}

// Byte offset of 16-byte chunk c of row r in a tile whose rows hold CH chunks:
// the low three bits of the chunk index are xor-ed with the row, so the eight
// rows of an 8x8 matrix fall into eight different bank groups.
template <int CH> __device__ __forceinline__ int swz(int r, int c) { return (r * CH + (c ^ (r & 7))) * 16; }

// Where 16-byte chunk c of row r of a [64 keys x HD] tile lies in shared memory.
// TileSwz: as the 16-byte asynchronous copies of this file lay it out (rows of HD / 8 chunks).
// TileTma: as a TMA copy with the 128-byte swizzle leaves it: halves of 64 columns one after the other, rows of 128 bytes.
template <int HD> struct TileSwz {
    static __device__ __forceinline__ int off(int r, int c) { return swz<HD / 8>(r, c); }
};
template <int HD> struct TileTma {
    static __device__ __forceinline__ int off(int r, int c) { return (c >> 3) * (KEYS * 128) + r * 128 + (((c & 7) ^ (r & 7)) << 4); }
};
// Who works on a page together: the whole CTA, or the four consumer warps of the streaming kernel (its fifth warp
// feeds them and must not be waited for).
struct SyncCta {
    static __device__ __forceinline__ void sync() { __syncthreads(); }
};
struct SyncConsumers {
    static __device__ __forceinline__ void sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }
};

// One visible page of one (sequence, kv head): what a CTA of the one-shot kernel, or one turn of the persistent
// kernel's loop, works on.
struct PageJob {
    int s, g, b;                      // index among the sequence's visible pages, kv head, sequence
    int page;                         // physical page
    int k_first, k_last;              // rows of the tile in use
    int h_first, h_last;              // rows among them that are not seen (between kept first tokens and the window); none: 1, 0
    __device__ __forceinline__ bool sees(int r) const { return r >= k_first && r <= k_last && !(r >= h_first && r <= h_last); }
    size_t row0;                      // partial of head g*G+i: row0 + i*S
    bool empty;                       // nothing of this page is visible
};

template <int HD>
__device__ __forceinline__ PageJob page_job(int s, int g, int b, const int* __restrict__ kv_len, const PageTable& pt,
                                            const TcArgs& a, int* __restrict__ status, bool reporter) {
    PageJob j;
    j.s = s; j.g = g; j.b = b; j.page = -1; j.k_first = 0; j.k_last = -1; j.h_first = 1; j.h_last = 0;
    const int G = a.H / a.KV;
    const int hi = kv_len[b];
    const VisiblePages vp = visible_pages(hi, a.window, a.keep_first);
    const int lo = vp.lo, kf = a.window > 0 ? a.keep_first : 0;
    int key_begin = 0, key_end = 0;
    if (hi > 0) {
        if (vp.count() > a.S && reporter && s == 0) atomicOr(status, MYNAH_ST_SPLIT_RANGE);
        const int mp = vp.page(s);
        if (mp >= 0) {
            const int p0 = mp * PAGE_TOKENS, win0 = max(lo, p0);    // the page's first key, and its first key inside the window
            key_end = min(hi, p0 + PAGE_TOKENS);
            if (mp < vp.pg0) {                                      // a page of kept first tokens before the window
                key_begin = p0;
                key_end = min(key_end, kf);
            } else if (kf > p0) {                                   // kept tokens and the window meet on this page
                key_begin = p0;
                if (kf < win0) {
                    j.h_first = kf - p0;
                    j.h_last = win0 - p0 - 1;
                }
            } else {
                key_begin = win0;
            }
            j.page = page_of(pt, b, mp * PAGE_TOKENS);
            if (j.page < 0) {
                if (reporter) atomicOr(status, MYNAH_ST_PAGE_RANGE);
                key_end = key_begin;
            }
        }
    }
    j.row0 = ((size_t)b * a.H + (size_t)g * G) * a.S + s;
    j.empty = key_begin >= key_end;
    if (!j.empty) {
        j.k_first = key_begin % PAGE_TOKENS;
        j.k_last = (key_end - 1) % PAGE_TOKENS;
    }
    return j;
}

__device__ __forceinline__ void write_empty_partial(const PageJob& j, const TcArgs& a, float* __restrict__ part_ml) {
    const int G = a.H / a.KV;
    for (int i = threadIdx.x; i < G; i += blockDim.x) {
        part_ml[(j.row0 + (size_t)i * a.S) * 2] = -INFINITY;
        part_ml[(j.row0 + (size_t)i * a.S) * 2 + 1] = 0.f;
    }
}

// The page's K tile, then its V tile, each as its own copy group. Rows that are not visible are zero-filled.
template <int HD, int VD = HD>
__device__ __forceinline__ void issue_page_copies(const PageJob& j, const bf16* __restrict__ k_cache, const bf16* __restrict__ v_cache,
                                                  const TcArgs& a, uint32_t k_base, uint32_t v_base) {
    constexpr int CH = HD / 8, VCH = VD / 8;
    const bf16* k_src = k_cache + ((size_t)j.page * a.KV + j.g) * PAGE_TOKENS * HD;
    const bf16* v_src = v_cache + ((size_t)j.page * (a.KV / a.vdiv) + j.g / a.vdiv) * PAGE_TOKENS * VD;
    for (int i = threadIdx.x; i < KEYS * CH; i += blockDim.x) {
        const int r = i / CH, c = i % CH;
        cp_async_16(k_base + swz<CH>(r, c), k_src + (size_t)r * HD + c * 8, j.sees(r));
    }
    cp_async_commit();
    for (int i = threadIdx.x; i < KEYS * VCH; i += blockDim.x) {
        const int r = i / VCH, c = i % VCH;
        cp_async_16(v_base + swz<VCH>(r, c), v_src + (size_t)r * VD + c * 8, j.sees(r));
    }
    cp_async_commit();
}

// Q as the A operand: rows = query heads of the group (zero beyond G), straight from global memory.
template <int HD>
__device__ __forceinline__ void load_q_fragments(const PageJob& j, const bf16* __restrict__ q, const TcArgs& a, uint32_t (&qa)[HD / 16][4]) {
    const int G = a.H / a.KV;
    const int lane = threadIdx.x & 31;
    const int r0 = lane >> 2, c0 = (lane & 3) * 2;
    const bf16* q0 = q + (size_t)j.b * a.ldq + (size_t)(j.g * G) * HD;
#pragma unroll
    for (int ks = 0; ks < HD / 16; ks++) {
        const int col = ks * 16 + c0;
        qa[ks][0] = r0 < G ? *reinterpret_cast<const uint32_t*>(q0 + (size_t)r0 * HD + col) : 0u;
        qa[ks][1] = r0 + 8 < G ? *reinterpret_cast<const uint32_t*>(q0 + (size_t)(r0 + 8) * HD + col) : 0u;
        qa[ks][2] = r0 < G ? *reinterpret_cast<const uint32_t*>(q0 + (size_t)r0 * HD + col + 8) : 0u;
        qa[ks][3] = r0 + 8 < G ? *reinterpret_cast<const uint32_t*>(q0 + (size_t)(r0 + 8) * HD + col + 8) : 0u;
    }
}

// The page's partial result. Where the K and V fragments come from is the caller's business: k_frag(ks, kb) gives
// the B fragments of this warp's 16 keys for dims [16 ks, 16 ks + 16), v_frag(ks, nt, vb) those of keys
// [16 ks, 16 ks + 16) for this warp's n-tiles nt and nt + 1; before_k() and before_v() run before the first use of
// each (waits and barriers, if the fragments still lie in shared memory). The arithmetic, and so every bit of the
// result, is the same whoever provides them.
// put.o(h, d, v0, v1) takes head h's unnormalised output in columns d and d + 1 (when it runs, red_l holds the four warps'
// shares of the heads' sums), put.ml(h, m, l) a head's maximum and sum.
template <int HD, int VD, class SYNC, class KFRAG, class VFRAG, class BEFORE_K, class BEFORE_V, class PUT>
__device__ __forceinline__ void compute_page_core(const PageJob& job, const uint32_t (&qa)[HD / 16][4], const TcArgs& a,
                                                  KFRAG k_frag, VFRAG v_frag, BEFORE_K before_k, BEFORE_V before_v,
                                                  bf16* p_s, float (*red_m)[MAX_G], float (*red_l)[MAX_G], const PUT& put) {
    constexpr int KSTEPS = HD / 16, NT = VD / 32;
    const int G = a.H / a.KV;
    const int tid = threadIdx.x & 127, warp = tid >> 5, lane = tid & 31;      // among the four warps of this page
    const int k_first = job.k_first, k_last = job.k_last;

    before_k();

    // ---- scores: warp w takes keys [16w, 16w+16): two n-tiles of 8 keys
    float sc[2][4] = {};
#pragma unroll
    for (int ks = 0; ks < KSTEPS; ks++) {
        uint32_t kb[4];
        k_frag(ks, kb);
        mma_bf16(sc[0], qa[ks], kb[0], kb[1]);
        mma_bf16(sc[1], qa[ks], kb[2], kb[3]);
    }
    // C layout: sc[t][0..1] -> head lane/4, keys 16w + 8t + (lane%4)*2 + {0,1}; sc[t][2..3] -> head lane/4 + 8
    const int hrow = lane >> 2;
    float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int t = 0; t < 2; t++)
#pragma unroll
        for (int e = 0; e < 4; e++) {
            const int key = warp * 16 + t * 8 + (lane & 3) * 2 + (e & 1);
            const bool vis = key >= k_first && key <= k_last && !(key >= job.h_first && key <= job.h_last);
            float sv = sc[t][e] * a.scale;
            if (a.softcap > 0.f) sv = a.softcap * tanhf(sv / a.softcap);
            sc[t][e] = vis ? sv : -INFINITY;
            mx[e >> 1] = fmaxf(mx[e >> 1], sc[t][e]);
        }
#pragma unroll
    for (int j = 0; j < 2; j++) {
        mx[j] = fmaxf(mx[j], __shfl_xor_sync(0xffffffffu, mx[j], 1));
        mx[j] = fmaxf(mx[j], __shfl_xor_sync(0xffffffffu, mx[j], 2));
    }
    if ((lane & 3) == 0) {
        red_m[warp][hrow] = mx[0];
        red_m[warp][hrow + 8] = mx[1];
    }
    SYNC::sync();
    float m[2], l[2] = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const int h = hrow + 8 * j;
        m[j] = fmaxf(fmaxf(red_m[0][h], red_m[1][h]), fmaxf(red_m[2][h], red_m[3][h]));   // finite: a visible key exists
    }
    // probabilities: fp32 for the sum, rounded to bf16 for the second product
#pragma unroll
    for (int t = 0; t < 2; t++) {
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const float p0 = expf(sc[t][2 * j] - m[j]), p1 = expf(sc[t][2 * j + 1] - m[j]);   // exp(-inf) = 0
            l[j] += p0 + p1;
            const int h = hrow + 8 * j, key = warp * 16 + t * 8 + (lane & 3) * 2;
            const __nv_bfloat162 pp = __floats2bfloat162_rn(p0, p1);
            // p_s rows hold 64 keys = 8 chunks; same swizzle as the tiles
            *reinterpret_cast<__nv_bfloat162*>(reinterpret_cast<unsigned char*>(p_s) + swz<8>(h, key >> 3) + (key & 7) * 2) = pp;
        }
    }
#pragma unroll
    for (int j = 0; j < 2; j++) {
        l[j] += __shfl_xor_sync(0xffffffffu, l[j], 1);
        l[j] += __shfl_xor_sync(0xffffffffu, l[j], 2);
    }
    if ((lane & 3) == 0) {
        red_l[warp][hrow] = l[0];
        red_l[warp][hrow + 8] = l[1];
    }
    before_v();                                       // (a barrier: the probabilities and the sums are in shared memory)

    // ---- output: warp w takes dims [w*VD/4, (w+1)*VD/4): VD/32 n-tiles of 8, four k-steps of 16 keys
    float oc[NT][4] = {};
    {
        const uint32_t p_base = smem_u32(p_s);
        const int mat = lane >> 3, rr = lane & 7;
#pragma unroll
        for (int ks = 0; ks < KEYS / 16; ks++) {
            uint32_t pa[4];
            // A operand (P, row-major [head][key]): matrices 0: heads 0-7, keys k0..+7; 1: heads 8-15, same keys;
            // 2: heads 0-7, keys +8; 3: heads 8-15, keys +8
            ldmatrix_x4(pa, p_base + swz<8>((mat & 1) * 8 + rr, ks * 2 + (mat >> 1)));
#pragma unroll
            for (int nt = 0; nt < NT; nt += 2) {
                uint32_t vb[4];
                v_frag(ks, nt, vb);
                mma_bf16(oc[nt], pa, vb[0], vb[1]);
                mma_bf16(oc[nt + 1], pa, vb[2], vb[3]);
            }
        }
    }
    // ---- hand the partial over: rows of heads < G
#pragma unroll
    for (int j = 0; j < 2; j++) {
        const int h = hrow + 8 * j;
        if (h < G) {
#pragma unroll
            for (int nt = 0; nt < NT; nt++) put.o(h, warp * (VD / 4) + nt * 8 + (lane & 3) * 2, oc[nt][2 * j], oc[nt][2 * j + 1]);
        }
    }
    if (tid < G) {
        const float ls = (red_l[0][tid] + red_l[1][tid]) + (red_l[2][tid] + red_l[3][tid]);
        const float mm = fmaxf(fmaxf(red_m[0][tid], red_m[1][tid]), fmaxf(red_m[2][tid], red_m[3][tid]));
        put.ml(tid, mm, ls);
    }
}

// The partial result as the per-page kernels leave it: rows of fp32 a head and page, and (maximum, sum) pairs.
template <int VD>
struct PartialRows {
    float *part_o, *part_ml;
    size_t row0;
    int S;
    __device__ __forceinline__ void o(int h, int d, float v0, float v1) const {
        *reinterpret_cast<float2*>(part_o + (row0 + (size_t)h * S) * VD + d) = make_float2(v0, v1);
    }
    __device__ __forceinline__ void ml(int h, float m, float l) const {
        part_ml[(row0 + (size_t)h * S) * 2] = m;
        part_ml[(row0 + (size_t)h * S) * 2 + 1] = l;
    }
};

// The fragments of a page's tiles in shared memory, as compute_page_core wants them.
// K (non-transposed load): matrices 0: keys 0-7 of the warp's 16, dims k0..k0+7; 1: keys 0-7, dims +8; 2: keys 8-15,
// dims k0; 3: keys 8-15, dims +8. V [key][dim] (transposed load): matrices 0: keys k0..+7, dims n0..+7; 1: keys +8,
// same dims; 2: keys k0..+7, dims n0+8; 3: keys +8, dims n0+8.
template <int HD, class TILE>
__device__ __forceinline__ void load_k_frag(uint32_t k_base, int ks, uint32_t (&kb)[4]) {
    const int warp = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31;
    const int mat = lane >> 3, rr = lane & 7;
    ldmatrix_x4(kb, k_base + TILE::off(warp * 16 + (mat >> 1) * 8 + rr, ks * 2 + (mat & 1)));
}
template <int HD, class TILE>
__device__ __forceinline__ void load_v_frag(uint32_t v_base, int ks, int nt, uint32_t (&vb)[4]) {
    const int warp = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31;
    const int mat = lane >> 3, rr = lane & 7;
    ldmatrix_x4_trans(vb, v_base + TILE::off(ks * 16 + (mat & 1) * 8 + rr, warp * (HD / 32) + nt + (mat >> 1)));
}

}  // namespace
