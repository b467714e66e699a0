// What the decode attention of attn_decode_tc.cu (a page a CTA, or a persistent CTA's turn) and that of decode_layers.cu (runs of
// pages within the one launch of a step) share: which pages and keys a sequence's newest position sees, the layout of a page's tile
// as a TMA copy leaves it, and the tensor-core instructions. Their arithmetic is their own.
#pragma once
#include "layout.cuh"

namespace {

constexpr int KEYS = PAGE_TOKENS;     // 64 keys a page

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

// Where 16-byte chunk c of row r of a [64 keys x HD] tile lies in shared memory after a TMA copy with the 128-byte swizzle: halves
// of 64 columns one after the other, rows of 128 bytes.
template <int HD> struct TileTma {
    static __device__ __forceinline__ int off(int r, int c) { return (c >> 3) * (KEYS * 128) + r * 128 + (((c & 7) ^ (r & 7)) << 4); }
};

}  // namespace
