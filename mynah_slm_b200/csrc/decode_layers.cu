// Every layer of a decode step in one launch, for steps of a few rows (up to 8) of the dense design: RMSNorm, grouped-query
// attention over the paged cache, RMSNorm, SwiGLU, with the residual stream in fp32 throughout (mynah-slm
// src/arch_qwen3.c:201-234).
//
// What bounds such a step is the one pass over the weights and the cache (31 MB and up a layer at the 0.6B shape: 5 us),
// but as seven launches a layer it took 29 us at one row: each kernel ends, drains and starts before the next one's loads
// begin. Here one CTA an SM stays for the whole step. A producer warp walks all of the CTA's weights and cache pages in the
// order they are used, copying them by TMA into a ring of shared-memory slots, never waiting for activations: 176 KB an SM
// are under way while the other warps exchange activations.
//
// What the CTAs exchange (a few KB a row and stage) goes through L2 in words of 64 bits, 32 of data and 32 of a tag that
// names the step and the layer. A reader loads what it needs and looks at the tags until they are this stage's: one trip
// where a barrier over the grid takes a fence, a count, a poll and then the load (2 us each, five a layer). No buffer is
// written again before every reader of its last contents has published something that the writer has read: each stage
// (q/k/v, attention, o, gate/up, down) reads all that the stage before it wrote.
//
// A product's unit is eight output rows of the weights: 1,024 outputs make 128 units, so the narrow products still use 128
// SMs without splitting a sum across CTAs. Within the CTA every warp multiplies its 128 of a slot's 1,024 columns
// (mma.sync m16n8k16, two units as the 16 rows, the step's rows as the 8 columns, fp32 sums) and the eight partial sums are
// added in a fixed order. A row's bits do not depend on the other rows. Who owns a column of the residual stream publishes it
// times the norm's gain, and its share of the row's squares; 1/rms is a factor on the finished sums.
//
// Attention takes the sequences' pages as jobs of four warps (attn_page.cuh, the arithmetic of the per-page kernels). The
// group of warps that has a (sequence, kv head)'s newest page merges all of its pages when its own jobs are done, in an order
// that depends on their number only.
//
// All CTAs must be resident at once: the launch is cooperative, and every wait is bounded (status bit 16). Registers: twelve
// warps leave 168 a thread. (Sixteen multiplying warps at 96 spilled, and beside this much shared memory L1 holds no spills:
// 28 us a layer.)
#include "attn_page.cuh"

#include <cuda.h>

namespace {

constexpr int CONSUMERS = 256, CWARPS = CONSUMERS / 32;              // warps that multiply and attend
constexpr int HELPERS = 3;                                           // warps that compute the rows' 1 / rms meanwhile
constexpr int THREADS = CONSUMERS + 32 + HELPERS * 32;               // and the producer warp
constexpr int PAGE_GROUPS = CWARPS / 4;                  // page jobs that a CTA works on at a time
constexpr int KC = 1024, KW = KC / CWARPS, PIECES = KW / 32;         // a slot's columns, a warp's share of them, in pieces of 32
constexpr int UR = 8;                                    // output rows of a unit
constexpr int SLOT_BYTES = UR * KC * 2;                  // eight rows in blocks of 64 columns [block][row][64], or a K or V tile
constexpr int SLOTS = 11;                                // as many as the rest leaves room for
constexpr int TG = 6;                                    // units whose sums a warp holds at a time
constexpr int MAX_LAYERS = 48, MAX_GROUPS = 4, MAX_ROWS = 8;
constexpr uint32_t WAIT_LOOKS = 1u << 22;                // trips to L2 after which a wait is given up (a second and more)
constexpr int TABLE = 64;                                // page jobs of a CTA that are looked up once for all layers
constexpr int BAR_ALL = 5, BAR_NORM = 6;                 // named barriers of the eight warps, and with the helpers (1, 2: a page's four warps)
static_assert(KEYS * 128 * 2 <= SLOT_BYTES && KW % 64 == 0, "a slot holds either kind of tile; a warp takes whole blocks of columns");

struct LayerDesc {                                       // as the host lays them out: 12 words of 64 bits
    const bf16 *w_qkv, *w_o, *w_gu, *w_down;
    const void *gain1, *gain2, *q_gain, *k_gain;
    bf16 *k, *v;
    long long map_row0;                                  // the layer's first row in its group's tensor maps
    long long group;
};
static_assert(sizeof(LayerDesc) == 96, "the host's layout");

struct StepArgs {
    int M, D, H, KV, F, L, S;
    int gain_dtype, qk_dtype, n_pos;
    float eps, qk_eps, scale;
    int window[MAX_GROUPS];
    PageTable pt[MAX_GROUPS];
    const LayerDesc* layers;
    float* x;
    uint64_t *hid, *squares, *qkv, *att, *act;           // tagged words: [rows][columns / 2], squares [rows][D / 8]
    uint64_t *part_o, *part_ml;                          // pages' partial results, tagged: [rows][heads][S][HD], [..][2]
    unsigned* sync;                                      // [0] the last step's tag, [1] CTAs that have left
    const int* kv_len;
    const float *cos_t, *sin_t;
    int* status;
};
struct StepMaps {
    CUtensorMap k[MAX_GROUPS], v[MAX_GROUPS];
    CUtensorMap w[MAX_LAYERS][4];                        // q/k/v, o, gate/up, down as [block of 64 columns][row][64]
};

// a page job's place to work
template <int HD> struct alignas(16) AttnWork {
    bf16 q[MAX_G * (HD + 8)];                            // the group's queries
    bf16 p[MAX_G * KEYS];                                // the probabilities, then the merge's sums
    float red_m[4][MAX_G], red_l[4][MAX_G];
};

template <int HD>
struct Smem {
    unsigned char slots[SLOTS][SLOT_BYTES];
    AttnWork<HD> a[PAGE_GROUPS];
    float sums[2][CWARPS][TG][UR * MAX_ROWS];            // two, used in turn: one barrier a turn is enough
    LayerDesc layers[MAX_LAYERS];
    int2 table[MAX_GROUPS][TABLE];                       // a job's sequence, kv head and page number; the page's place
    unsigned long long full[SLOTS], empty[SLOTS];
    int pg0[MAX_GROUPS][MAX_ROWS], cnt[MAX_GROUPS][MAX_ROWS], cum[MAX_GROUPS][MAX_ROWS + 1];   // pages seen by a sequence; jobs before it
    float inv_rms[MAX_ROWS];
    int hi[MAX_ROWS];
    int abort;
};

struct SyncGroup {
    static __device__ __forceinline__ void sync() { asm volatile("bar.sync %0, 128;" ::"r"(1 + (int)(threadIdx.x >> 7)) : "memory"); }
};
__device__ __forceinline__ void sync_all() { asm volatile("bar.sync %0, %1;" ::"n"(BAR_ALL), "n"(CONSUMERS) : "memory"); }
__device__ __forceinline__ void sync_norm() { asm volatile("bar.sync %0, %1;" ::"n"(BAR_NORM), "n"(CONSUMERS + HELPERS * 32) : "memory"); }
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y), "r"(z) : "memory");
}

// Which part of a product's units this CTA takes: unit cta + i * grid, for i < count.
__device__ __forceinline__ int my_units(int n_units) {
    return (int)blockIdx.x < n_units ? (n_units - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x : 0;
}

// Page jobs are numbered sequence by sequence, kv head by kv head, page by page; a CTA takes a run of them.
struct Job { int b, g, s; };
template <class SM>
__device__ __noinline__ Job find_job(const SM& sm, const PageTable& pt, int grp, int j, int M, int& page) {
    int b = 0;
    while (b + 1 < M && j >= sm.cum[grp][b + 1]) b++;
    const int r = j - sm.cum[grp][b], n = sm.cnt[grp][b];
    const Job job{b, r / n, r % n};
    page = page_of(pt, job.b, (sm.pg0[grp][job.b] + job.s) * PAGE_TOKENS);       // the physical page, -1: none
    return job;
}
template <class SM>
__device__ __forceinline__ Job look_up(const SM& sm, const PageTable& pt, int grp, int j, int j0, int M, int& page) {
    if (j - j0 >= TABLE) return find_job(sm, pt, grp, j, M, page);
    const int2 e = sm.table[grp][j - j0];
    page = e.y;
    return {(int)((unsigned)e.x >> 28), (e.x >> 20) & 255, e.x & 0xfffff};
}
__device__ __forceinline__ int first_job(int jobs, int cta) { return (int)((long long)jobs * cta / gridDim.x); }

// ---- tagged words
__device__ __forceinline__ uint64_t tagged(uint32_t data, uint32_t tag) { return ((uint64_t)tag << 32) | data; }
__device__ __forceinline__ void publish(uint64_t* p, uint32_t data, uint32_t tag) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(tagged(data, tag)) : "memory");
}
__device__ __forceinline__ void publish2(uint64_t* p, uint32_t d0, uint32_t d1, uint32_t tag) {
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(tagged(d0, tag)), "l"(tagged(d1, tag)) : "memory");
}
__device__ __forceinline__ uint64_t peek(const uint64_t* p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void peek2(const uint64_t* p, uint64_t& a, uint64_t& b) {
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ bool has_tag(uint64_t v, uint32_t tag) { return (uint32_t)(v >> 32) == tag; }
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
    const __nv_bfloat162 b = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&b);
}

// ---------------------------------------------------------------- the producer warp

template <int HD>
struct Producer {
    Smem<HD>& sm;
    uint32_t it = 0;
    bool ok = true;
    int lane;

    __device__ __forceinline__ bool wait_empty(uint32_t i) {
        if (ok && i >= SLOTS && !tc5::mbar_wait(tc5::smem_u32(&sm.empty[i % SLOTS]), ((i / SLOTS) & 1) ^ 1)) ok = false;
        ok = __all_sync(0xffffffffu, ok && *(volatile int*)&sm.abort == 0);
        return ok;
    }

    // the slots of one product: units of this CTA in groups of TG tiles, a group's columns outermost
    __device__ __forceinline__ void product(const CUtensorMap* w, int n_units, int K, bool pair, int pair_rows) {
        const int cnt = my_units(n_units), per = pair ? 2 : 1, ug = TG / per;
        for (int u0 = 0; u0 < cnt; u0 += ug) {
            const int nst = min(ug, cnt - u0) * per;
            for (int k0 = 0; k0 < K; k0 += KC) {
                for (int t = 0; t < nst; t++, it++) {
                    if (!wait_empty(it)) return;
                    const int unit = blockIdx.x + (u0 + t / per) * gridDim.x;
                    const int row = unit * UR + (pair ? (t % 2) * pair_rows : 0);
                    if (lane == 0) {                     // (blocks beyond K are filled with zeros)
                        const uint32_t bar = tc5::smem_u32(&sm.full[it % SLOTS]);
                        tc5::mbar_expect_tx(bar, SLOT_BYTES);
                        tma_load_3d(tc5::smem_u32(sm.slots[it % SLOTS]), w, 0, row, k0 / 64, bar);
                    }
                    __syncwarp();
                }
            }
        }
    }

    // the K and V tiles of this CTA's page jobs
    __device__ __forceinline__ void pages(const StepArgs& a, const StepMaps& maps, const LayerDesc& d) {
        const int grp = (int)d.group, J = sm.cum[grp][a.M];
        const int j0 = first_job(J, blockIdx.x), j1 = first_job(J, blockIdx.x + 1);
        for (int jb = j0; jb < j1; jb += 32) {
            int row = -1;                                // every lane finds one job's tile
            if (jb + lane < j1) {
                int page;
                const Job job = look_up(sm, a.pt[grp], grp, jb + lane, j0, a.M, page);
                if (page >= 0) row = (int)d.map_row0 + (page * a.KV + job.g) * PAGE_TOKENS;
            }
            for (int i = 0; i < 32 && jb + i < j1; i++) {
                const int r = __shfl_sync(0xffffffffu, row, i);
#pragma unroll
                for (int kv = 0; kv < 2; kv++, it++) {
                    if (!wait_empty(it)) return;
                    if (lane == 0) {
                        const uint32_t bar = tc5::smem_u32(&sm.full[it % SLOTS]), dst = tc5::smem_u32(sm.slots[it % SLOTS]);
                        if (r >= 0) {
                            const CUtensorMap* m = kv ? &maps.v[grp] : &maps.k[grp];
                            tc5::mbar_expect_tx(bar, KEYS * HD * 2);
#pragma unroll
                            for (int c = 0; c < HD; c += 64) tc5::tma_load_2d(dst + (c / 64) * (KEYS * 128), m, c, r, bar);
                        } else {
                            tc5::mbar_arrive(bar);       // a page that is not there: the slot keeps its turn
                        }
                    }
                    __syncwarp();
                }
            }
        }
    }

    __device__ __forceinline__ void drain() {            // nothing may still be on its way when the CTA ends
        for (uint32_t i = it > SLOTS ? it - SLOTS : 0; i < it; i++) tc5::mbar_wait(tc5::smem_u32(&sm.full[i % SLOTS]), (i / SLOTS) & 1);
    }
};

__device__ __forceinline__ void l2_touch(const void* p, int bytes, int lane) {
    for (int o = lane * 128; o < bytes; o += 32 * 128)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const char*>(p) + o));
}

// ---------------------------------------------------------------- the other warps

enum Result { TO_BF16, ADD_TO_STREAM, TO_SWIGLU };

template <int HD>
struct Worker {
    Smem<HD>& sm;
    const StepArgs& a;
    uint32_t it = 0;                                     // slots taken so far
    int turn = 0;                                        // which of the two buffers of sums is next
    int tid, warp, lane;

    // After `n` fruitless looks (of `limit`): whether to stop waiting, because the limit ran out here or somewhere in this CTA
    // before. (A count, not a clock: it keeps these loops' registers few.)
    __device__ __forceinline__ bool tired(uint32_t n, uint32_t limit) {
        if ((n & 255u) != 255u) return false;
        if (n >= limit) {
            *(volatile int*)&sm.abort = 1;
            atomicOr(a.status, MYNAH_ST_TIMEOUT);
        }
        return *(volatile int*)&sm.abort != 0;
    }
    __device__ __forceinline__ bool is_full(uint32_t i) const {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done) : "r"(tc5::smem_u32(&sm.full[i % SLOTS])), "r"((i / SLOTS) & 1) : "memory");
        return done != 0;
    }
    __device__ __forceinline__ void wait_full(uint32_t i) {
        unsigned long long t0 = 0;                       // (a look may take a hardware wait of its own: a clock, not a count)
        while (!is_full(i)) {
            if (*(volatile int*)&sm.abort != 0) break;
            const unsigned long long now = tc5::now_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > tc5::WAIT_LIMIT_NS) tired(~0u, 0);
        }
        __syncwarp();
    }
    __device__ __forceinline__ bool row_in_use(int m) const { return m < a.M && sm.hi[m] > 0; }

    // One lane's look at one word that is not there yet, until it is: what a long wait costs the others is one sector a warp.
    __device__ __forceinline__ bool watch(const uint64_t* p, bool missing, uint32_t tag) {
        const unsigned who = __ballot_sync(0xffffffffu, missing);
        bool stop = false;
        if (who != 0 && lane == __ffs(who) - 1)
            for (uint32_t n = 0; !has_tag(peek(p), tag); n++)
                if (tired(n, WAIT_LOOKS)) {
                    stop = true;
                    break;
                }
        return __any_sync(0xffffffffu, stop);
    }

    // N times four consecutive words of tagged rows, once they carry the tag; all lanes call it, those without a row (`on`
    // false) get zeros.
    template <int N>
    __device__ __forceinline__ void read_tagged(const uint64_t* const (&p)[N], const bool (&on)[N], uint32_t tag, uint32_t (&f)[N][4]) {
        for (uint32_t n = 0;; n++) {
            const uint64_t* gone = nullptr;
#pragma unroll
            for (int i = 0; i < N; i++) {
                uint64_t v[4] = {(uint64_t)tag << 32, (uint64_t)tag << 32, (uint64_t)tag << 32, (uint64_t)tag << 32};
                if (on[i]) {
                    peek2(p[i], v[0], v[1]);
                    peek2(p[i] + 2, v[2], v[3]);
                }
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    if (!has_tag(v[e], tag)) gone = p[i] + e;
                    f[i][e] = (uint32_t)v[e];
                }
            }
            if (__all_sync(0xffffffffu, gone == nullptr)) break;
            if (n >= 2 && watch(gone, gone != nullptr, tag)) break;
        }
    }

    // 1 / rms of every row from the shares of its columns' owners (by the helper warps, while the others multiply).
    __device__ __forceinline__ void row_scales(int helper, uint32_t tag) {
#pragma unroll 1
        for (int m = helper; m < a.M; m += HELPERS) {
            if (sm.hi[m] <= 0) continue;
            const uint64_t* p = a.squares + (size_t)m * (a.D / UR);
            float ss;
            for (uint32_t n = 0;; n++) {
                const uint64_t* gone = nullptr;
                ss = 0.f;
#pragma unroll 4
                for (int u = lane; u < a.D / UR; u += 32) {
                    const uint64_t v = peek(p + u);
                    if (!has_tag(v, tag)) gone = p + u;
                    ss += __uint_as_float((uint32_t)v);
                }
                if (__all_sync(0xffffffffu, gone == nullptr)) break;
                if (watch(gone, gone != nullptr, tag)) break;
            }
            ss = warp_sum(ss);
            if (lane == 0) sm.inv_rms[m] = 1.0f / sqrtf(ss / (float)a.D + a.eps);
        }
        sync_norm();                                     // (a wait, not an arrival: a helper without rows must not run ahead)
    }

    // The owner's new values of the stream for the next norm: x times the gain in bf16 (pairs of neighbouring lanes) and the
    // squares of a unit's eight columns (lanes of one row). All lanes of a warp call it.
    __device__ __forceinline__ void publish_stream(bool on, float x, float gain, int m, int n, uint32_t tag) {
        const float y = x * gain, y1 = __shfl_down_sync(0xffffffffu, y, 1);
        float q = x * x;
        q += __shfl_xor_sync(0xffffffffu, q, 1);
        q += __shfl_xor_sync(0xffffffffu, q, 2);
        q += __shfl_xor_sync(0xffffffffu, q, 4);
        if (!on) return;
        if ((lane & 1) == 0) publish(a.hid + ((size_t)m * a.D + n) / 2, pack2(y, y1), tag);
        if ((lane & 7) == 0) publish(a.squares + ((size_t)m * a.D + n) / UR, __float_as_uint(q), tag);
    }

    // The stream as the step's embedding left it: every owner publishes its columns.
    __device__ __forceinline__ void first_stream(const void* gain, uint32_t tag) {
        const int n_out = my_units(a.D / UR) * MAX_ROWS * UR;
        for (int i0 = 0; i0 < n_out; i0 += CONSUMERS) {
            const int i = i0 + tid, m = (i / UR) % MAX_ROWS, n = (blockIdx.x + i / (MAX_ROWS * UR) * gridDim.x) * UR + i % UR;
            const bool on = i < n_out && row_in_use(m);
            publish_stream(on, on ? a.x[(size_t)m * a.D + n] : 0.f, on ? VecRef{gain, a.gain_dtype}.at(n) : 0.f, m, n, tag);
        }
    }

    // Tagged rows [M, K] times this CTA's units of the weights. One copy of this code serves the four products of a layer (four
    // copies outgrew the instruction cache).
    struct Product {
        const uint64_t* src;                             // tagged rows, read under `tag`
        uint32_t tag;
        int n_units, K;
        bool normed;                                     // the sums are scaled by the row's 1 / rms
        Result res;
        uint64_t* dst;                                   // tagged rows of width ld; ADD_TO_STREAM: the stream, published
        int ld;                                          // with `gain` unless that is null
        const void* gain;
        uint32_t next;                                   // the tag of what comes out
    };

    // The lane's words of a warp's share of one slot's columns: row lane / 4, as the product's B operand wants them.
    __device__ __forceinline__ void peek_share(const Product& q, int k0, bool on, uint64_t (&v)[PIECES][4]) {
        const int left = min(KC, q.K - k0) - warp * KW;  // columns of this share that exist (a multiple of 64)
        const uint64_t* p = q.src + ((size_t)(lane >> 2) * q.K + k0 + warp * KW) / 2 + (lane & 3);
#pragma unroll
        for (int c = 0; c < PIECES; c++)
#pragma unroll
            for (int e = 0; e < 4; e++) v[c][e] = on && c * 32 < left ? peek(p + c * 16 + e * 4) : (uint64_t)q.tag << 32;
    }

    __device__ __forceinline__ void product(const Product& q) {
        constexpr int PASS = CONSUMERS / (MAX_ROWS * UR), OUTS = (TG + PASS - 1) / PASS;
        const int cnt = my_units(q.n_units), per = q.res == TO_SWIGLU ? 2 : 1, ug = TG / per;
        const int om = (tid / UR) % MAX_ROWS, ou = tid / (MAX_ROWS * UR);        // this thread's outputs: row om, units ou + PASS i
        const bool mine = row_in_use(om), row_on = row_in_use(lane >> 2);
#pragma unroll 1
        for (int u0 = 0; u0 < cnt; u0 += ug) {
            const int nu = min(ug, cnt - u0), nst = nu * per;
            float old[OUTS], gn[OUTS];
            if (q.res == ADD_TO_STREAM) {                // asked for now, needed at the end
#pragma unroll
                for (int o = 0; o < OUTS; o++) {
                    const int u = ou + o * PASS, n = (blockIdx.x + (u0 + u) * gridDim.x) * UR + tid % UR;
                    const bool on = u < nu && mine;
                    old[o] = on ? a.x[(size_t)om * a.D + n] : 0.f;               // (this thread wrote it, or the embedding)
                    gn[o] = on && q.gain != nullptr ? VecRef{q.gain, a.gain_dtype}.at(n) : 0.f;
                }
            }
            // 16-byte pieces j (and 4 + j) of a block of 64 columns: row lane % 8, swizzled by the row
            const int r = lane & 7, j = lane >> 3;
            const uint32_t off = warp * (UR * KW * 2) + r * 128 + ((j ^ r) << 4);
            float acc[TG / 2][4] = {};
            uint64_t v[PIECES][4];
            peek_share(q, 0, row_on, v);
#pragma unroll 1
            for (int k0 = 0; k0 < q.K; k0 += KC) {
                uint32_t f[PIECES][4];
                for (uint32_t n = 0;; n++) {
                    int gone = -1;
#pragma unroll
                    for (int c = 0; c < PIECES; c++)
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            if (!has_tag(v[c][e], q.tag)) gone = c * 16 + e * 4;
                            f[c][e] = (uint32_t)v[c][e];
                        }
                    if (__all_sync(0xffffffffu, gone < 0)) break;
                    if (n >= 2 && watch(q.src + ((size_t)(lane >> 2) * q.K + k0 + warp * KW) / 2 + (lane & 3) + gone, gone >= 0, q.tag)) break;
                    peek_share(q, k0, row_on, v);
                }
                bool ready[TG];
#pragma unroll
                for (int t = 0; t < TG; t++) ready[t] = t < nst && is_full(it + t);
                if (k0 + KC < q.K) peek_share(q, k0 + KC, row_on, v);            // under way while this slot's columns are multiplied
#pragma unroll
                for (int t = 0; t < TG; t += 2) {
                    if (t < nst) {
                        const bool two = t + 1 < nst;
                        uint32_t w0[PIECES][4], w1[PIECES][4] = {};
                        if (!__all_sync(0xffffffffu, ready[t])) wait_full(it);
                        const uint32_t s0 = tc5::smem_u32(sm.slots[it % SLOTS]) + off;
#pragma unroll
                        for (int c = 0; c < PIECES; c++) ldmatrix_x4(w0[c], (s0 + c / 2 * (UR * 128)) ^ (c % 2 * 64));
                        if (two) {
                            if (!__all_sync(0xffffffffu, ready[t + 1])) wait_full(it + 1);
                            const uint32_t s1 = tc5::smem_u32(sm.slots[(it + 1) % SLOTS]) + off;
#pragma unroll
                            for (int c = 0; c < PIECES; c++) ldmatrix_x4(w1[c], (s1 + c / 2 * (UR * 128)) ^ (c % 2 * 64));
                        }
#pragma unroll
                        for (int c = 0; c < PIECES; c++) {
                            const uint32_t lo[4] = {w0[c][0], w1[c][0], w0[c][1], w1[c][1]}, hi[4] = {w0[c][2], w1[c][2], w0[c][3], w1[c][3]};
                            mma_bf16(acc[t / 2], lo, f[c][0], f[c][1]);
                            mma_bf16(acc[t / 2], hi, f[c][2], f[c][3]);
                        }
                        __syncwarp();
                        if (lane == 0) {
                            tc5::mbar_arrive(tc5::smem_u32(&sm.empty[it % SLOTS]));
                            if (two) tc5::mbar_arrive(tc5::smem_u32(&sm.empty[(it + 1) % SLOTS]));
                        }
                        it += two ? 2 : 1;
                    }
                }
            }
            float(*sums)[TG][UR * MAX_ROWS] = sm.sums[turn];
            turn ^= 1;
#pragma unroll
            for (int t = 0; t < TG; t++)
                if (t < nst) {
#pragma unroll
                    for (int e = 0; e < 2; e++)          // a row of the step, a row of the weights
                        sums[warp][t][((lane & 3) * 2 + e) * UR + (lane >> 2)] = acc[t / 2][(t & 1) * 2 + e];
                }
            if (q.normed && u0 == 0) sync_norm();
            else sync_all();
#pragma unroll
            for (int o = 0; o < OUTS; o++) {
                const int u = ou + o * PASS, n = (blockIdx.x + (u0 + u) * gridDim.x) * UR + tid % UR;
                const bool on = u < nu && mine;
                if (!__any_sync(0xffffffffu, on)) continue;
                float s = 0.f, s2 = 0.f;
                if (on) {
                    const float* p = &sums[0][u * per][om * UR + tid % UR];
#pragma unroll
                    for (int w = 0; w < CWARPS; w++) s += p[w * (TG * UR * MAX_ROWS)];
                    if (per == 2) {
#pragma unroll
                        for (int w = 0; w < CWARPS; w++) s2 += p[w * (TG * UR * MAX_ROWS) + UR * MAX_ROWS];
                    }
                    if (q.normed) {
                        s *= sm.inv_rms[om];
                        s2 *= sm.inv_rms[om];
                    }
                }
                if (q.res == ADD_TO_STREAM) {
                    const float x = old[o] + s;
                    if (on) a.x[(size_t)om * a.D + n] = x;
                    if (q.gain != nullptr) publish_stream(on, x, gn[o], om, n, q.next);
                } else {
                    if (per == 2) s = s / (1.0f + expf(-s)) * s2;
                    const float y1 = __shfl_down_sync(0xffffffffu, s, 1);
                    if (on && (lane & 1) == 0) publish(q.dst + ((size_t)om * q.ld + n) / 2, pack2(s, y1), q.next);
                }
            }
        }
    }

    // Where a page's result goes: tagged partial rows, or (a sequence of one visible page) the finished output.
    struct PutPage {
        uint64_t *o_row, *ml_row, *att;                  // of the group's first head
        int S;
        uint32_t tag;
        bool whole;
        const float (*red_l)[MAX_G];
        __device__ __forceinline__ void o(int h, int d, float v0, float v1) const {
            if (whole) {
                const float inv = 1.0f / ((red_l[0][h] + red_l[1][h]) + (red_l[2][h] + red_l[3][h]));
                publish(att + ((size_t)h * HD + d) / 2, pack2(v0 * inv, v1 * inv), tag);
            } else {
                publish2(o_row + (size_t)h * S * HD + d, __float_as_uint(v0), __float_as_uint(v1), tag);
            }
        }
        __device__ __forceinline__ void ml(int h, float m, float l) const {
            if (!whole) publish2(ml_row + (size_t)h * S * 2, __float_as_uint(m), __float_as_uint(l), tag);
        }
    };

    // The n pages of one (sequence, kv head), by the four warps of a group: out[h] = sum_s w_s o_s / sum_s w_s l_s with
    // w_s = exp(m_s - m). 4 / G warps a head (at least one), each adds every so many-th page; their sums are added in order.
    __device__ __forceinline__ void merge(AttnWork<HD>& w, int b, int g, int n, uint32_t tag) {
        constexpr int DL = HD / 32, BATCH = 8;           // a lane's columns; pages whose rows are under way together
        const int G = a.H / a.KV, lw = warp & 3;
        const int wph = G >= 3 ? 1 : 4 / G, hpt = 4 / wph, sub = lw % wph;       // warps a head, heads in one turn
#pragma unroll 1
        for (int h0 = 0; h0 < G; h0 += hpt) {
            const int h = h0 + lw / wph;
            float o[DL] = {}, lsum = 0.f;
            if (h < G) {
                const size_t row = ((size_t)b * a.H + g * G + h) * a.S;
                const uint64_t* ml = a.part_ml + row * 2;
                float m = -INFINITY;
#pragma unroll 1
                for (int s0 = 0; s0 < n; s0 += 32) {     // all pages' maxima and sums, a page a lane
                    const int s = s0 + lane;
                    uint64_t vm = 0, vl = 0;
                    for (uint32_t k = 0;; k++) {
                        if (s < n) peek2(ml + 2 * s, vm, vl);
                        const bool gone = s < n && !(has_tag(vm, tag) && has_tag(vl, tag));
                        if (__all_sync(0xffffffffu, !gone)) break;
                        if (watch(has_tag(vm, tag) ? ml + 2 * s + 1 : ml + 2 * s, gone, tag)) break;
                    }
                    const float pm = s < n ? __uint_as_float((uint32_t)vm) : -INFINITY, pl = __uint_as_float((uint32_t)vl);
                    if (pm > -INFINITY) {
                        const float nm = fmaxf(m, pm);
                        lsum = lsum * expf(m - nm) + pl * expf(pm - nm);
                        m = nm;
                    }
                }
                const float top = warp_max(m);
                lsum = warp_sum(m > -INFINITY ? lsum * expf(m - top) : 0.f);
#pragma unroll 1
                for (int s0 = 0; s0 < n && top > -INFINITY; s0 += 32) {
                    uint64_t vm = 0, vl;
                    if (s0 + lane < n) peek2(ml + 2 * (s0 + lane), vm, vl);
                    const float pm = s0 + lane < n ? __uint_as_float((uint32_t)vm) : -INFINITY;
                    const float e = pm > -INFINITY ? expf(pm - top) : 0.f;       // (0: a page that was not there has no row)
                    const int n1 = min(32, n - s0);
#pragma unroll 1
                    for (int i0 = sub; i0 < n1; i0 += wph * BATCH) {
                        const uint64_t* p = a.part_o + (row + s0 + i0) * HD + lane * DL;
                        float we[BATCH];
#pragma unroll
                        for (int i = 0; i < BATCH; i++) we[i] = i0 + i * wph < n1 ? __shfl_sync(0xffffffffu, e, (i0 + i * wph) & 31) : 0.f;
                        uint64_t q[BATCH][DL];
                        for (uint32_t k = 0;; k++) {
                            const uint64_t* gone = nullptr;
#pragma unroll
                            for (int i = 0; i < BATCH; i++)
#pragma unroll
                                for (int d = 0; d < DL; d += 2) {
                                    q[i][d] = q[i][d + 1] = (uint64_t)tag << 32;
                                    if (we[i] > 0.f) peek2(p + (size_t)i * wph * HD + d, q[i][d], q[i][d + 1]);
                                }
#pragma unroll
                            for (int i = 0; i < BATCH; i++)
#pragma unroll
                                for (int d = 0; d < DL; d++)
                                    if (!has_tag(q[i][d], tag)) gone = p + (size_t)i * wph * HD + d;
                            if (__all_sync(0xffffffffu, gone == nullptr)) break;
                            if (watch(gone, gone != nullptr, tag)) break;
                        }
#pragma unroll
                        for (int i = 0; i < BATCH; i++)
#pragma unroll
                            for (int d = 0; d < DL; d++) o[d] = fmaf(we[i], __uint_as_float((uint32_t)q[i][d]), o[d]);
                    }
                }
            }
            float* part = reinterpret_cast<float*>(w.p); // [4 warps][HD]
            if (wph > 1) {
                SyncGroup::sync();
                if (sub > 0) {
#pragma unroll
                    for (int d = 0; d < DL; d++) part[lw * HD + lane * DL + d] = o[d];
                }
                SyncGroup::sync();
            }
            if (sub == 0 && h < G) {
                for (int p = 1; p < wph; p++)
#pragma unroll
                    for (int d = 0; d < DL; d++) o[d] += part[(lw + p) * HD + lane * DL + d];
                const float inv = lsum > 0.f ? 1.0f / lsum : 0.f;
                uint64_t* dst = a.att + ((size_t)b * a.H * HD + (size_t)(g * G + h) * HD + lane * DL) / 2;
#pragma unroll
                for (int d = 0; d < DL; d += 2) publish(dst + d / 2, pack2(o[d] * inv, o[d + 1] * inv), tag);
            }
        }
        SyncGroup::sync();
    }

    __device__ __forceinline__ void attention(const LayerDesc& d, uint32_t tag) {
        constexpr int KSTEPS = HD / 16, QLD = HD + 8;
        constexpr int LPH = HeadLanes<HD>::LPH, HPW = HeadLanes<HD>::HPW;
        const int grp = (int)d.group, J = sm.cum[grp][a.M], G = a.H / a.KV;
        const int j0 = first_job(J, blockIdx.x), j1 = first_job(J, blockIdx.x + 1);
        const int gi = warp >> 2, lw = warp & 3, ltid = tid & 127, sub = lane / LPH, li = lane % LPH;
        AttnWork<HD>& w = sm.a[gi];
        const TcArgs ta{a.H, a.KV, 0, a.window[grp], a.S, a.scale, 0, 1, 0.f};
        const int NQ = (a.H + 2 * a.KV) * HD;
        const bool rotate = a.cos_t != nullptr, has_gain = d.q_gain != nullptr;
        int pb = -1, pg = -1;                            // the (sequence, kv head) at hand
        bool merges = false;                             // some job of this group is a newest page of several
#pragma unroll 1
        for (int j = j0 + gi; j < j1; j += PAGE_GROUPS) {
            int page;
            const Job job = look_up(sm, a.pt[grp], grp, j, j0, a.M, page);
            const int hi = sm.hi[job.b], pos = hi - 1, n_pages = sm.cnt[grp][job.b];
            const uint64_t* qrow = a.qkv + (size_t)job.b * NQ / 2;
            const int p0 = (sm.pg0[grp][job.b] + job.s) * PAGE_TOKENS, lo = first_visible(hi, a.window[grp]);
            const int r_new = pos >= p0 && pos < p0 + PAGE_TOKENS ? pos - p0 : -1;
            const bool pos_ok = !rotate || pos < a.n_pos;
            if (!pos_ok && ltid == 0) atomicOr(a.status, MYNAH_ST_POS_RANGE);
            merges = merges || (job.s == n_pages - 1 && n_pages > 1);
            // the new key and value, by the fourth warp of the group that has their page; the queries by the first ones
            uint4 ko = make_uint4(0, 0, 0, 0), vn = ko;
            if (r_new >= 0 && lw == 3) {
                float kn[8], gain[8], rc[8], rs[8];
                if (rotate) load_rotation<HD>(a.cos_t, a.sin_t, pos_ok ? pos : 0, lane, rc, rs);
                if (has_gain) load_gain8(VecRef{d.k_gain, a.qk_dtype}, li * 8, gain);
                const uint64_t* p[2] = {qrow + ((size_t)(a.H + job.g) * HD + li * 8) / 2, qrow + ((size_t)(a.H + a.KV + job.g) * HD + li * 8) / 2};
                const bool on[2] = {sub == 0, sub == 0};
                uint32_t raw[2][4];
                read_tagged<2>(p, on, tag, raw);
                Raw8<bf16> r8;
                r8.q[0] = make_uint4(raw[0][0], raw[0][1], raw[0][2], raw[0][3]);
                r8.to_f32(kn);
                vn = make_uint4(raw[1][0], raw[1][1], raw[1][2], raw[1][3]);
                head_norm_rotate<HD>(kn, has_gain, gain, a.qk_eps, rotate, rc, rs, lane);
                ko = make_uint4(pack2(kn[0], kn[1]), pack2(kn[2], kn[3]), pack2(kn[4], kn[5]), pack2(kn[6], kn[7]));
            }
            if (job.b != pb || job.g != pg) {
                pb = job.b;
                pg = job.g;
                if (lw * HPW < G) {                      // uniform over the warp
                    float gain[8], rc[8], rs[8];
                    if (rotate) load_rotation<HD>(a.cos_t, a.sin_t, pos_ok ? pos : 0, lane, rc, rs);
                    if (has_gain) load_gain8(VecRef{d.q_gain, a.qk_dtype}, li * 8, gain);
#pragma unroll 1
                    for (int hb = lw * HPW; hb < G; hb += 4 * HPW) {
                        const uint64_t* p[1] = {qrow + ((size_t)(job.g * G + hb + sub) * HD + li * 8) / 2};
                        const bool on[1] = {hb + sub < G};
                        uint32_t raw[1][4];
                        read_tagged<1>(p, on, tag, raw);
                        Raw8<bf16> r8;
                        r8.q[0] = make_uint4(raw[0][0], raw[0][1], raw[0][2], raw[0][3]);
                        float v[8];
                        r8.to_f32(v);
                        head_norm_rotate<HD>(v, has_gain, gain, a.qk_eps, rotate, rc, rs, lane);
                        if (hb + sub < G) store8<bf16>(w.q + (hb + sub) * QLD + li * 8, v);
                    }
                }
                SyncGroup::sync();
            }
            const uint32_t ik = it + 2 * (uint32_t)(j - j0), iv = ik + 1;
            unsigned char *kt = sm.slots[ik % SLOTS], *vt = sm.slots[iv % SLOTS];
            PageJob pj;
            pj.s = job.s; pj.g = job.g; pj.b = job.b; pj.page = page; pj.h_first = 1; pj.h_last = 0;
            pj.k_first = max(lo, p0) - p0;
            pj.k_last = min(hi, p0 + PAGE_TOKENS) - 1 - p0;
            pj.row0 = ((size_t)job.b * a.H + (size_t)job.g * G) * a.S + job.s;
            pj.empty = page < 0 || !pos_ok;
            const bool mend = !pj.empty && (pj.k_first > 0 || pj.k_last < KEYS - 1 || r_new >= 0);      // uniform over the group
            wait_full(ik);
            wait_full(iv);
            if (mend) {
                // what a page holds outside the visible range may be anything: value rows that meet a probability of zero are
                // cleared (scores of such keys are replaced, not multiplied)
                for (int i = ltid; i < KEYS * (HD / 8); i += 128) {
                    const int r = i / (HD / 8), c = i % (HD / 8);
                    if (r < pj.k_first || r > pj.k_last) *reinterpret_cast<uint4*>(vt + TileTma<HD>::off(r, c)) = make_uint4(0, 0, 0, 0);
                }
                if (r_new >= 0 && lw == 3 && sub == 0) {
                    *reinterpret_cast<uint4*>(kt + TileTma<HD>::off(r_new, li)) = ko;
                    *reinterpret_cast<uint4*>(vt + TileTma<HD>::off(r_new, li)) = vn;
                }
                SyncGroup::sync();
            }
            const PutPage put{a.part_o + pj.row0 * HD, a.part_ml + pj.row0 * 2, a.att + ((size_t)job.b * a.H + (size_t)job.g * G) * HD / 2,
                              a.S, tag, n_pages == 1, w.red_l};
            if (pj.empty) {
                if (page < 0 && ltid == 0) atomicOr(a.status, MYNAH_ST_PAGE_RANGE);
                if (n_pages == 1) {
                    for (int i = ltid; i < G * HD / 2; i += 128) publish(put.att + i, 0, tag);
                } else {
                    for (int i = ltid; i < G; i += 128) put.ml(i, -INFINITY, 0.f);
                }
            } else {
                uint32_t qa[KSTEPS][4];
                const uint32_t q32 = tc5::smem_u32(w.q) + ((lane & 15) * QLD + (lane >> 4) * 8) * 2;     // (rows beyond the group's heads: whatever is there)
#pragma unroll
                for (int ks = 0; ks < KSTEPS; ks++) ldmatrix_x4(qa[ks], q32 + ks * 32);
                const uint32_t kb32 = tc5::smem_u32(kt), vb32 = tc5::smem_u32(vt);
                compute_page_core<HD, HD, SyncGroup>(
                    pj, qa, ta,
                    [&](int ks, uint32_t (&kb)[4]) { load_k_frag<HD, TileTma<HD>>(kb32, ks, kb); },
                    [&](int ks, int nt, uint32_t (&vb)[4]) { load_v_frag<HD, TileTma<HD>>(vb32, ks, nt, vb); },
                    []() {}, []() { SyncGroup::sync(); }, w.p, w.red_m, w.red_l, put);
                if (r_new >= 0 && lw == 3 && sub == 0) {             // the new position's place in the cache
                    const size_t row = (((size_t)page * a.KV + job.g) * PAGE_TOKENS + r_new) * HD + li * 8;
                    *reinterpret_cast<uint4*>(d.k + row) = ko;
                    *reinterpret_cast<uint4*>(d.v + row) = vn;
                }
            }
            if (mend) tc5::fence_async_smem();           // before a copy fills the slots again
            __syncwarp();
            if (lane < CWARPS / 4) {                     // four warps make the arrivals of all that empty a slot
                tc5::mbar_arrive(tc5::smem_u32(&sm.empty[ik % SLOTS]));
                tc5::mbar_arrive(tc5::smem_u32(&sm.empty[iv % SLOTS]));
            }
            SyncGroup::sync();
        }
        it += 2 * (uint32_t)(j1 - j0);
        // Both groups are through with their pages before a warp asks for a slot behind them: a barrier's parity names the right
        // filling only to those who know that the one before has come.
        sync_all();
        if (!merges) return;
        // A merge waits for pages with lower numbers only, and these wait for merges of still lower ones at most.
#pragma unroll 1
        for (int j = j0 + gi; j < j1; j += PAGE_GROUPS) {
            int page;
            const Job job = look_up(sm, a.pt[grp], grp, j, j0, a.M, page);
            const int n_pages = sm.cnt[grp][job.b];
            if (job.s == n_pages - 1 && n_pages > 1) merge(w, job.b, job.g, n_pages, tag);
        }
    }
};

template <int HD>
__global__ void __launch_bounds__(THREADS, 1)
decode_layers_kernel(const __grid_constant__ StepMaps maps, const __grid_constant__ StepArgs a) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    Smem<HD>& sm = *reinterpret_cast<Smem<HD>*>(smem_raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int i = 0; i < SLOTS; i++) {
            tc5::mbar_init(tc5::smem_u32(&sm.full[i]), 1);
            tc5::mbar_init(tc5::smem_u32(&sm.empty[i]), CWARPS);
        }
        sm.abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        tc5::fence_async_smem();
    }
    for (int i = tid; i < a.L * (int)(sizeof(LayerDesc) / 8); i += THREADS)
        reinterpret_cast<unsigned long long*>(sm.layers)[i] = reinterpret_cast<const unsigned long long*>(a.layers)[i];
    if (tid < MAX_ROWS) sm.hi[tid] = tid < a.M ? a.kv_len[tid] : 0;
    __syncthreads();
    if (tid < MAX_GROUPS) {                              // the pages that every sequence sees in each cache group
        int sum = 0;
        for (int b = 0; b < a.M; b++) {
            const VisiblePages vp = visible_pages(sm.hi[b], a.window[tid], 0);
            if (vp.count() > a.S && blockIdx.x == 0 && a.pt[tid].ids != nullptr) atomicOr(a.status, MYNAH_ST_SPLIT_RANGE);
            sm.pg0[tid][b] = vp.pg0;
            sm.cnt[tid][b] = min(vp.count(), a.S);
            sm.cum[tid][b] = sum;
            sum += sm.cnt[tid][b] * a.KV;
        }
        sm.cum[tid][a.M] = sum;
    }
    __syncthreads();
    for (int i = tid; i < MAX_GROUPS * TABLE; i += THREADS) {
        const int g = i / TABLE, J = sm.cum[g][a.M], j = first_job(J, blockIdx.x) + i % TABLE;
        if (a.pt[g].ids != nullptr && j < first_job(J, blockIdx.x + 1)) {
            int page;
            const Job job = find_job(sm, a.pt[g], g, j, a.M, page);
            sm.table[g][i % TABLE] = make_int2((int)((unsigned)job.b << 28) | job.g << 20 | job.s, page);
        }
    }
    __syncthreads();
    const int NQ = (a.H + 2 * a.KV) * HD, NO = a.H * HD;
    const uint32_t base = a.sync[0];
    if (warp == CWARPS) {
        Producer<HD> p{sm};
        p.lane = lane;
#pragma unroll 1
        for (int l = 0; l < a.L && p.ok; l++) {
            const LayerDesc& d = sm.layers[l];
            if (blockIdx.x % 8 == 0) {                   // the gains come from L2 by the time they are needed
                const int gb = a.D * (a.gain_dtype == MYNAH_F32 ? 4 : 2), qb = HD * (a.qk_dtype == MYNAH_F32 ? 4 : 2);
                l2_touch(d.gain1, gb, lane);
                l2_touch(d.gain2, gb, lane);
                if (d.q_gain != nullptr) {
                    l2_touch(d.q_gain, qb, lane);
                    l2_touch(d.k_gain, qb, lane);
                }
            }
#pragma unroll 1
            for (int i = 0; i < 4 && p.ok; i++) {
                p.product(&maps.w[l][i], (i == 0 ? NQ : (i == 2 ? a.F : a.D)) / UR, i == 1 ? NO : (i == 3 ? a.F : a.D), i == 2, a.F);
                if (i == 0 && p.ok) p.pages(a, maps, d);
            }
        }
        if (!p.ok && lane == 0) {
            *(volatile int*)&sm.abort = 1;
            atomicOr(a.status, MYNAH_ST_TIMEOUT);
        }
        p.drain();
    } else {
        Worker<HD> c{sm, a};
        c.tid = tid;
        c.warp = warp;
        c.lane = lane;
        if (warp > CWARPS) {
#pragma unroll 1
            for (int l = 0; l < a.L; l++) {
                const uint32_t t1 = base + 2 * l + 1;
                if (my_units(NQ / UR) > 0) c.row_scales(warp - CWARPS - 1, t1);
                if (my_units(a.F / UR) > 0) c.row_scales(warp - CWARPS - 1, t1 + 1);
            }
        } else {
            c.first_stream(sm.layers[0].gain1, base + 1);
#pragma unroll 1
            for (int l = 0; l < a.L; l++) {
                const LayerDesc& d = sm.layers[l];
                const uint32_t t1 = base + 2 * l + 1, t2 = t1 + 1;
#pragma unroll 1
                for (int i = 0; i < 4; i++) {
                    typename Worker<HD>::Product q;
                    q.src = i == 1 ? a.att : (i == 3 ? a.act : a.hid);
                    q.tag = i < 2 ? t1 : t2;
                    q.n_units = (i == 0 ? NQ : (i == 2 ? a.F : a.D)) / UR;
                    q.K = i == 1 ? NO : (i == 3 ? a.F : a.D);
                    q.normed = i % 2 == 0;
                    q.res = i == 0 ? TO_BF16 : (i == 2 ? TO_SWIGLU : ADD_TO_STREAM);
                    q.dst = i == 0 ? a.qkv : a.act;
                    q.ld = i == 0 ? NQ : a.F;
                    q.gain = i == 1 ? d.gain2 : (l + 1 < a.L ? sm.layers[l + 1].gain1 : nullptr);
                    q.next = i == 0 ? t1 : (i == 3 ? t2 + 1 : t2);
                    c.product(q);
                    if (i == 0) c.attention(d, t1);
                }
            }
        }
    }
    __syncthreads();
    if (tid == 0) {                                      // the last CTA to leave moves the tags on
        unsigned old;
        asm volatile("atom.add.acq_rel.gpu.u32 %0, [%1], 1;" : "=r"(old) : "l"(a.sync + 1) : "memory");
        if (old + 1 == gridDim.x) {
            a.sync[0] += 2 * a.L + 2;
            a.sync[1] = 0;
        }
    }
}

template <int HD>
int launch_step(const StepMaps& maps, const StepArgs& a, int sms, cudaStream_t stream) {
    auto kern = decode_layers_kernel<HD>;
    constexpr int smem = (int)sizeof(Smem<HD>);
    static_assert(smem <= 227 * 1024, "the ring and its companions fit an SM");
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return mynah_fail("decode_layers: %s", cudaGetErrorString(e));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sms);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, kern, maps, a);
    if (e != cudaSuccess) return mynah_fail("decode_layers: %s", cudaGetErrorString(e));
    return mynah_check_launch("decode_layers");
}

// [rows, K] row-major as blocks of 64 columns: (column in the block, row, block), boxes of 64 x 8 rows x 16 blocks, 128-byte
// swizzle (so that the eight rows' pieces of one column lie in different banks).
int weight_map(CUtensorMap* map, const void* base, long long rows, int K) {
    tc5::EncodeTiledFn fn = tc5::encode_fn();
    if (fn == nullptr) return mynah_fail("decode_layers: the driver does not provide cuTensorMapEncodeTiled");
    const cuuint64_t dims[3] = {64, (cuuint64_t)rows, (cuuint64_t)(K / 64)}, strides[2] = {(cuuint64_t)K * 2, 128};
    const cuuint32_t box[3] = {64, UR, KC / 64}, estr[3] = {1, 1, 1};
    const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return mynah_fail("decode_layers: cuTensorMapEncodeTiled failed with code %d", (int)r);
    return 0;
}

}  // namespace

// Sizes that the kernel takes. Products: whole units of eight outputs, columns in whole blocks of 64.
MYNAH_API int mynah_decode_layers_supported(int M, int D, int H, int KV, int HD, int F, int L, int n_groups) {
    if (M < 1 || M > MAX_ROWS || L < 1 || L > MAX_LAYERS || n_groups < 1 || n_groups > MAX_GROUPS) return 0;
    if (HD != 64 && HD != 128) return 0;
    if (KV < 1 || KV > 255 || H < 1 || H % KV != 0 || H / KV > MAX_G) return 0;
    if (D < 64 || F < 64 || D % 64 != 0 || F % 64 != 0) return 0;
    return 1;
}

// One decode step through all layers. layers: L descriptors of 96 bytes on the device; host_layers: the same on the host.
// Per cache group (n_groups of them) eight words: k and v bases, their rows (entries * pages * kv heads * 64), window, and the
// page lists. words: 64-bit words for 8 rows of D / 2 + D / 8 + ((H + 2 KV) HD + H HD + F) / 2; part: 64-bit words for
// 8 * H * S * (HD + 2); sync: two 32-bit words. All three zero before the first launch and kept from step to step.
MYNAH_API int mynah_decode_layers(const void* layers, const void* host_layers, int L, int M, int D, int H, int KV, int HD, int F, int S,
                                  float* x, void* words, void* part, unsigned* sync,
                                  int gain_dtype, float eps, int qk_dtype, float qk_eps, const float* cos_t, const float* sin_t, int n_pos,
                                  const int* kv_len, int n_groups, const long long* group_words, int* status, int sms, cudaStream_t stream) {
    MYNAH_REQUIRE(mynah_decode_layers_supported(M, D, H, KV, HD, F, L, n_groups), "decode_layers: sizes are not supported");
    MYNAH_REQUIRE(S >= 1 && S <= 0xfffff, "decode_layers: %d page splits", S);
    MYNAH_REQUIRE(sms >= 1 && sms <= mynah_sm_count(), "decode_layers: bad CTA count");
    StepMaps maps = {};
    StepArgs a = {};
    a.M = M; a.D = D; a.H = H; a.KV = KV; a.F = F; a.L = L; a.S = S;
    a.gain_dtype = gain_dtype; a.qk_dtype = qk_dtype; a.n_pos = n_pos;
    a.eps = eps; a.qk_eps = qk_eps;
    a.scale = 1.0f / sqrtf((float)HD);
    a.layers = static_cast<const LayerDesc*>(layers);
    a.x = x;
    a.hid = static_cast<uint64_t*>(words);
    a.squares = a.hid + (size_t)MAX_ROWS * (D / 2);
    a.qkv = a.squares + (size_t)MAX_ROWS * (D / UR);
    a.att = a.qkv + (size_t)MAX_ROWS * ((H + 2 * KV) * HD / 2);
    a.act = a.att + (size_t)MAX_ROWS * (H * HD / 2);
    a.part_o = static_cast<uint64_t*>(part);
    a.part_ml = a.part_o + (size_t)MAX_ROWS * H * S * HD;
    a.sync = sync; a.kv_len = kv_len;
    a.cos_t = cos_t; a.sin_t = sin_t; a.status = status;
    for (int g = 0; g < n_groups; g++) {
        const long long* w = group_words + (size_t)g * 8;
        MYNAH_REQUIRE(w[2] > 0 && w[2] <= 0x7fffffffll, "decode_layers: a cache group's rows exceed a tensor map's");
        a.window[g] = (int)w[3];
        a.pt[g] = PageTable{reinterpret_cast<const int*>(w[4]), reinterpret_cast<const int*>(w[5]), reinterpret_cast<const int*>(w[6]), (int)w[7]};
        for (int kv = 0; kv < 2; kv++)
            if (tc5::make_map(kv ? &maps.v[g] : &maps.k[g], reinterpret_cast<const void*>(w[kv]), CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, w[2], HD, HD,
                              KEYS, 64)) return -1;
    }
    const LayerDesc* hl = static_cast<const LayerDesc*>(host_layers);
    for (int l = 0; l < L; l++)
        if (weight_map(&maps.w[l][0], hl[l].w_qkv, (long long)(H + 2 * KV) * HD, D) || weight_map(&maps.w[l][1], hl[l].w_o, D, H * HD)
            || weight_map(&maps.w[l][2], hl[l].w_gu, 2ll * F, D) || weight_map(&maps.w[l][3], hl[l].w_down, D, F)) return -1;
    return HD == 128 ? launch_step<128>(maps, a, sms, stream) : launch_step<64>(maps, a, sms, stream);
}
