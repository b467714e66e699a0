// Every layer of a decode step in one launch, for steps of a few rows (up to 8) of the dense design: RMSNorm, grouped-query
// attention over the paged cache, RMSNorm, SwiGLU, with the residual stream in fp32 throughout (mynah-slm
// src/arch_qwen3.c:201-234).
//
// What bounds such a step is the one pass over the weights and the cache (31 MB and up a layer at the 0.6B shape: 5 us),
// but as seven launches a layer it took 29 us at one row: each kernel ends, drains and starts before the next one's loads
// begin. Here one CTA an SM stays for the whole step. A producer warp walks all of the CTA's weights and cache pages in the
// order they are used, copying them by TMA into a ring of shared-memory slots, never waiting for activations: 160 KB an SM
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
// added in a fixed order. A row's bits do not depend on the other rows of the launch. Who owns a column of the residual stream
// publishes it times the norm's gain, and its share of the row's squares; 1/rms is a factor on the finished sums.
//
// Attention's jobs are runs of two or four pages of a (sequence, kv head), cut by the sequence's own page count, four warps a job:
// each warp keeps its own 16 keys of every page, with a running maximum, and meets the others once a run. The warps that have a
// sequence's newest run merge all of its runs when their own jobs are done, in an order that depends on their number only.
//
// All CTAs must be resident at once: the launch is cooperative, and every wait is bounded (status bit 16). Registers: twelve
// warps leave 168 a thread. (Sixteen multiplying warps at 96 spilled, and beside this much shared memory L1 holds no spills:
// 28 us a layer.)
#include "attn_page.cuh"
#include "head_prep.cuh"
#include "tcgen05.cuh"

#include <cuda.h>

namespace {

constexpr int CONSUMERS = 256, CWARPS = CONSUMERS / 32;              // warps that multiply and attend
constexpr int HELPERS = 3;                                           // warps that compute the rows' 1 / rms meanwhile
constexpr int THREADS = CONSUMERS + 32 + HELPERS * 32;               // and the producer warp
constexpr int PAGE_GROUPS = CWARPS / 4;                  // page jobs that a CTA works on at a time
constexpr int KC = 1024, KW = KC / CWARPS, PIECES = KW / 32;         // a slot's columns, a warp's share of them, in pieces of 32
constexpr int UR = 8;                                    // output rows of a unit
constexpr int SLOT_BYTES = UR * KC * 2;                  // eight rows in blocks of 64 columns [block][row][64], or a K or V tile
constexpr int SLOTS = 10;                                // as many as the rest leaves room for
constexpr int TG = 6;                                    // units whose sums a warp holds at a time
constexpr int MAX_LAYERS = 48, MAX_GROUPS = 4, MAX_ROWS = 8;
constexpr int COPIES = 4, SQUARE_COPIES = 8;             // of what every CTA reads: see publish_pair
// Pages of a job, by the pages that its sequence sees (by nothing else: a sequence's bits must not depend on its company). Short
// runs spread a sequence over more warps, long ones leave fewer partial results to merge. 0.6B shape, us a step with runs of 2 / of
// 4: 5 pages, 1 row 558 / 593, 4 rows 613 / 653; 8 pages, 8 rows 770 / 738; 16 pages, 1 row 588 / 609, 4 rows 648 / 690, 8 rows
// 794 / 844; 24 pages, 1 row 576 / 602, 4 rows 739 / 713, 8 rows 901 / 860; 33 pages, 8 rows 1,029 / 952; 63 pages, 1 row 638 / 635,
// 2 rows 764 / 695; 250 pages, 1 row 1,154 / 958.
constexpr int RUN = 4, RUN_SHIFT = 2, SHORT_RUN_SHIFT = 1, SHORT_PAGES = 16;
constexpr int TABLE = 32;                                // jobs of a CTA that are looked up once for all layers
constexpr int BAR_ALL = 5, BAR_NORM = 6;                 // named barriers of the eight warps, and with the helpers (1, 2: a page's four warps)
static_assert(KEYS * 128 * 2 <= SLOT_BYTES && KW % 64 == 0, "a slot holds either kind of tile; a warp takes whole blocks of columns");
static_assert(SLOTS >= TG, "what is waited for together fits the ring");

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
    int R;                                               // runs of a sequence at most: the pitch of the partial results
    int lg_rows;                                         // M, rounded up to a power of two: its logarithm
    int gain_dtype, qk_dtype, n_pos;
    float eps, qk_eps, scale, inv_d;                     // inv_d: 1 / D
    int window[MAX_GROUPS];
    PageTable pt[MAX_GROUPS];
    const LayerDesc* layers;
    float* x;
    uint64_t *hid, *squares, *qkv, *att, *act;           // tagged words: [copies][rows][columns / 2], squares [copies][rows][D / 8]
    uint64_t *part_o, *part_ml;                          // pages' partial results, tagged: [rows][heads][R][HD], [..][2]
    uint32_t looks, look_mask;                           // trips to L2 after which a wait is given up, and when they are counted
    unsigned* sync;                                      // [0] the last step's tag, [1] CTAs that have left
    const int* kv_len;
    const float *cos_t, *sin_t;
    int* status;
};
struct StepMaps {
    CUtensorMap k[MAX_GROUPS], v[MAX_GROUPS];
    CUtensorMap w[MAX_LAYERS][4];                        // q/k/v, o, gate/up, down as [block of 64 columns][row][64]
};

// a job's place to work
constexpr int HEADS = 8;                                 // query heads per kv head at most: the columns of a product
constexpr int CHUNK = 2;                                 // heads whose outputs the four warps add at a time
template <int HD> struct alignas(16) AttnWork {
    bf16 q[HEADS * (HD + 8)];                            // the group's queries
    float o[4][CHUNK][HD];                               // the warps' outputs, and the merge's sums
    float m[4][HEADS], l[4][HEADS];
};
constexpr int STAGE_PITCH = KW * 2 + 16;                 // bytes of a staged row: eight rows' pieces of 16 bytes in different banks

template <int HD>
struct Smem {
    unsigned char slots[SLOTS][SLOT_BYTES];
    AttnWork<HD> a[PAGE_GROUPS];
    unsigned char stage[CWARPS][MAX_ROWS * STAGE_PITCH]; // a warp's share of the rows at hand
    float sums[2][CWARPS][TG][UR * MAX_ROWS];            // two, used in turn: one barrier a turn is enough
    LayerDesc layers[MAX_LAYERS];
    int table[MAX_GROUPS][TABLE];                        // a job's sequence, kv head and run
    int pages[MAX_GROUPS][TABLE][RUN];                   // the places of its pages, -1: none
    unsigned long long full[SLOTS], empty[SLOTS];
    uint32_t issued;                                     // fillings that the producer has come to: see page_is_full
    int pg0[MAX_GROUPS][MAX_ROWS], cnt[MAX_GROUPS][MAX_ROWS], cum[MAX_GROUPS][MAX_ROWS + 1];   // pages seen by a sequence, jobs before it
    float inv_rms[MAX_ROWS];
    int hi[MAX_ROWS];
    int abort;
};

__device__ __forceinline__ uint32_t transpose8x8(uint32_t r) {       // of 16-bit elements, two a lane
    uint32_t t;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(t) : "r"(r));
    return t;
}
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

// Jobs are numbered sequence by sequence, kv head by kv head, run by run; a CTA takes consecutive ones.
struct Job {
    int b, g, r, p, n;                                   // run r: n pages, from the sequence's visible page p on
};
__host__ __device__ __forceinline__ int run_shift(int pages) { return pages <= SHORT_PAGES ? SHORT_RUN_SHIFT : RUN_SHIFT; }
__host__ __device__ __forceinline__ int runs_of(int pages) {
    const int s = run_shift(pages);
    return (pages + (1 << s) - 1) >> s;
}
template <class SM>
__device__ __noinline__ int find_job(const SM& sm, int grp, int j, int M) {
    int b = 0;
    while (b + 1 < M && j >= sm.cum[grp][b + 1]) b++;
    const int r = j - sm.cum[grp][b], n = runs_of(sm.cnt[grp][b]);
    return (int)((unsigned)b << 28) | (r / n) << 20 | r % n;
}
template <class SM>
__device__ __forceinline__ Job look_up(const SM& sm, int grp, int j, int j0, int M) {
    const int e = j - j0 < TABLE ? sm.table[grp][j - j0] : find_job(sm, grp, j, M);
    Job job{(int)((unsigned)e >> 28), (e >> 20) & 255, e & 0xfffff, 0, 0};
    const int pages = sm.cnt[grp][job.b], s = run_shift(pages);
    job.p = job.r << s;
    job.n = min(1 << s, pages - job.p);
    return job;
}
// The physical page of a run's page i, -1: none.
template <class SM>
__device__ __forceinline__ int page_at(const SM& sm, const PageTable& pt, int grp, const Job& job, int j, int j0, int i) {
    return j - j0 < TABLE ? sm.pages[grp][j - j0][i] : page_of(pt, job.b, (sm.pg0[grp][job.b] + job.p + i) * PAGE_TOKENS);
}
// Runs that a sequence of at most so many visible pages is cut into at most.
inline int most_runs(int pages) { return max(runs_of(min(pages, SHORT_PAGES)), runs_of(pages)); }
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

// A word that every CTA reads is published in several copies, and a CTA reads copy number blockIdx modulo their count: 148 SMs
// at one line of one L2 slice queue for it (a few rows are a few lines, and where these fell decided up to 25% of a step: 0.48
// or 0.58 ms at one row on two GPUs).
__device__ __forceinline__ void publish_copies(uint64_t* p, size_t copy, uint32_t data, uint32_t tag) {
#pragma unroll
    for (int i = 0; i < COPIES; i++) publish(p + i * copy, data, tag);
}
// The same of two neighbouring lanes' values, a lane half of the copies (copy 0: there is one only).
__device__ __forceinline__ void publish_pair(uint64_t* p, size_t copy, bool on, float mine, float other, uint32_t tag) {
    const bool odd = threadIdx.x & 1;
    const uint32_t data = odd ? pack2(other, mine) : pack2(mine, other);
    if (!on || (odd && copy == 0)) return;
    p += odd ? copy : 0;
    publish(p, data, tag);
    if (copy != 0) {
#pragma unroll
        for (int i = 2; i < COPIES; i += 2) publish(p + i * copy, data, tag);
    }
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
        for (int j = j0; j < j1; j++) {
            const Job job = look_up(sm, grp, j, j0, a.M);
            for (int i = 0; i < job.n; i++) {
                const int page = page_at(sm, a.pt[grp], grp, job, j, j0, i);
                const int r = (int)d.map_row0 + (page * a.KV + job.g) * PAGE_TOKENS;
#pragma unroll
                for (int kv = 0; kv < 2; kv++, it++) {
                    if (!wait_empty(it)) return;
                    if (lane == 0) {
                        const uint32_t bar = tc5::smem_u32(&sm.full[it % SLOTS]), dst = tc5::smem_u32(sm.slots[it % SLOTS]);
                        if (page >= 0) {
                            const CUtensorMap* m = kv ? &maps.v[grp] : &maps.k[grp];
                            tc5::mbar_expect_tx(bar, KEYS * HD * 2);
#pragma unroll
                            for (int c = 0; c < HD; c += 64) tc5::tma_load_2d(dst + (c / 64) * (KEYS * 128), m, c, r, bar);
                        } else {
                            tc5::mbar_arrive(bar);       // a page that is not there: the slot keeps its turn
                        }
                        asm volatile("st.release.cta.shared.u32 [%0], %1;" ::"r"(tc5::smem_u32(&sm.issued)), "r"(it + 1) : "memory");
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
    uint32_t live = 0;                                   // the rows in use, a bit each
    int tid, warp, lane;

    __device__ __forceinline__ void give_up() {
        *(volatile int*)&sm.abort = 1;
        atomicOr(a.status, MYNAH_ST_TIMEOUT);
    }
    // After `n` fruitless looks: whether to stop waiting, because the limit ran out here or somewhere in this CTA before. (A
    // count, not a clock: it keeps these loops' registers few.)
    __device__ __forceinline__ bool tired(uint32_t n) {
        if ((n & a.look_mask) != a.look_mask) return false;
        if (n >= a.looks) give_up();
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
    // A barrier's parity tells a filling from the next one, not from the one before: it may be asked only by those who know that
    // the one before is complete. In the products every warp has seen every filling. Among pages a group passes over the other's
    // fillings (which may be still on their way when its own, asked for later, have come), so it first looks whether the producer
    // has come to filling i: the producer has by then seen the slot's last filling read and handed back. (The filling after i
    // cannot come before this group has handed i back. To look at the other group's fillings as well would not do: they may be
    // two fillings past by then.)
    __device__ __forceinline__ bool page_is_full(uint32_t i) const {
        uint32_t n;
        asm volatile("ld.acquire.cta.shared.u32 %0, [%1];" : "=r"(n) : "r"(tc5::smem_u32(&sm.issued)) : "memory");
        return n > i && is_full(i);
    }
    // Until the n slots from number i on are full; a lane looks after a slot (a look may take a hardware wait of its own, so this
    // limit is a clock, not a count).
    template <bool PAGES = false>
    __device__ __forceinline__ void wait_full(uint32_t i, int n) {
        unsigned long long t0 = 0;
        while (!__all_sync(0xffffffffu, lane >= n || (PAGES ? page_is_full(i + lane) : is_full(i + lane)))) {
            const unsigned long long now = tc5::now_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > tc5::WAIT_LIMIT_NS) give_up();
            if (__any_sync(0xffffffffu, *(volatile int*)&sm.abort != 0)) break;
        }
    }
    // This warp is through with the n slots from number i on.
    __device__ __forceinline__ void release(uint32_t i, int n, int arrivals) {
        __syncwarp();
        if (lane < n * arrivals) tc5::mbar_arrive(tc5::smem_u32(&sm.empty[(i + lane / arrivals) % SLOTS]));
    }
    __device__ __forceinline__ bool row_in_use(int m) const { return (live >> m & 1) != 0; }

    // One lane's look at one word that is not there yet, until it is: what a long wait costs the others is one sector a warp.
    __device__ __forceinline__ bool watch(const uint64_t* p, bool missing, uint32_t tag) {
        const unsigned who = __ballot_sync(0xffffffffu, missing);
        bool stop = false;
        if (who != 0 && lane == __ffs(who) - 1)
            for (uint32_t n = 0; !has_tag(peek(p), tag); n++)
                if (tired(n)) {
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

    // 1 / rms of every row from the shares of its columns' owners (by the helper warps, while the others multiply): a helper
    // takes every third row, all of its rows together. One word is watched while nothing has come yet; the rest follows within
    // a microsecond and is looked for by all lanes.
    __device__ __forceinline__ void row_scales(int helper, uint32_t tag) {
        constexpr int ROWS = (MAX_ROWS + HELPERS - 1) / HELPERS;
        float ss[ROWS];
        // (What runs between the last share's arrival and the barrier keeps everybody waiting, and after the attention its code
        // comes from far away: it is kept short.)
        const uint64_t* squares = a.squares + (size_t)(blockIdx.x % SQUARE_COPIES) * MAX_ROWS * (a.D / UR);
        watch(squares + (size_t)helper * (a.D / UR), lane == 0 && row_in_use(helper), tag);
        for (uint32_t n = 0;; n++) {
            uint32_t gone = 0;
#pragma unroll
            for (int i = 0; i < ROWS; i++) ss[i] = 0.f;
#pragma unroll 1
            for (int u = lane * 4; u < a.D / UR; u += 128) {         // (a multiple of eight of them)
#pragma unroll
                for (int i = 0; i < ROWS; i++) {
                    if (!row_in_use(helper + i * HELPERS)) continue;
                    const uint64_t* p = squares + (uint32_t)((helper + i * HELPERS) * (a.D / UR) + u);
                    uint64_t v[4];
                    peek2(p, v[0], v[1]);
                    peek2(p + 2, v[2], v[3]);
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        gone |= (uint32_t)(v[e] >> 32) ^ tag;
                        ss[i] += __uint_as_float((uint32_t)v[e]);
                    }
                }
            }
            if (__all_sync(0xffffffffu, gone == 0)) break;
            if (__any_sync(0xffffffffu, tired(n))) break;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int i = 0; i < ROWS; i++) ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], o);
        // lane i takes the helper's row i; 1 / sqrt by the hardware's estimate and one Newton step: off by 7.4e-8 at most over all
        // exponents (1.0f / sqrtf: 8.9e-8, and a step of one row 508 us for 499). The step would make a NaN of an infinite mean
        // square, where 1 / sqrt is 0.
        float x = ss[0];
#pragma unroll
        for (int i = 1; i < ROWS; i++) x = lane == i ? ss[i] : x;
        x = fmaf(x, a.inv_d, a.eps);
        float y = rsqrtf(x);
        if (x != INFINITY) y = fmaf(0.5f * y, fmaf(-x * y, y, 1.0f), y);
        if (lane < ROWS && row_in_use(helper + lane * HELPERS)) sm.inv_rms[helper + lane * HELPERS] = y;
        sync_norm();                                     // (a wait, not an arrival: a helper without rows must not run ahead)
    }

    // The owner's new values of the stream for the next norm: x times the gain in bf16 (pairs of neighbouring lanes) and the
    // squares of a unit's eight columns (lanes of one row). All lanes of a warp call it.
    __device__ __forceinline__ void publish_stream(bool on, float x, float gain, int m, int n, uint32_t tag) {
        const float y = x * gain, other = __shfl_xor_sync(0xffffffffu, y, 1);
        float q = x * x;
        q += __shfl_xor_sync(0xffffffffu, q, 1);
        q += __shfl_xor_sync(0xffffffffu, q, 2);
        q += __shfl_xor_sync(0xffffffffu, q, 4);
        publish_pair(a.hid + ((uint32_t)(m * a.D + n) >> 1), (size_t)MAX_ROWS * (a.D / 2), on, y, other, tag);
        static_assert(SQUARE_COPIES == UR, "a lane a copy");
        if (on) publish(a.squares + (uint32_t)(((lane & 7) * MAX_ROWS + m) * (a.D / UR) + n / UR), __float_as_uint(q), tag);
    }

    // The stream as the step's embedding left it: every owner publishes its columns.
    __device__ __forceinline__ void first_stream(const void* gain, uint32_t tag) {
        const int n_out = my_units(a.D / UR) * MAX_ROWS * UR;
#pragma unroll 1
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
        uint64_t* dst;                                   // tagged rows of width ld, `copy` words from copy to copy (0: one
        size_t copy;                                     // copy); ADD_TO_STREAM: the stream, published
        int ld;                                          // with `gain` unless that is null
        const void* gain;
        uint32_t next;                                   // the tag of what comes out
    };

    // A warp reads its shares of the rows a stage at a time: as many slots' columns as make eight rows in all (one slot's of
    // eight rows, eight slots' of one row), four columns a lane. Row i of a stage is row i % (1 << lg_rows) of the step, of the
    // stage's slot i >> lg_rows.
    __device__ __forceinline__ const uint64_t* staged(const Product& q, int k0, int i) const {   // null: there is none
        const int m = i & ((1 << a.lg_rows) - 1), k = k0 + (i >> a.lg_rows) * KC + warp * KW + lane * 4;
        return k < q.K && row_in_use(m) ? q.src + ((uint32_t)(m * q.K + k) >> 1) : nullptr;
    }
    __device__ __forceinline__ void peek_stage(const Product& q, int k0, uint64_t (&v)[MAX_ROWS][2]) const {
#pragma unroll
        for (int i = 0; i < MAX_ROWS; i++) {
            const uint64_t* p = staged(q, k0, i);
            v[i][0] = v[i][1] = (uint64_t)q.tag << 32;
            if (p != nullptr) peek2(p, v[i][0], v[i][1]);
        }
    }

    __device__ __forceinline__ void product(const Product& q) {
        const int cnt = my_units(q.n_units), per = q.res == TO_SWIGLU ? 2 : 1, ug = TG / per;
        const int om = (tid / UR) & ((1 << a.lg_rows) - 1), ou = tid >> (3 + a.lg_rows);         // this thread's outputs: row om, units ou, ou + pass ...
        const int pass = (CONSUMERS / UR) >> a.lg_rows, depth = MAX_ROWS >> a.lg_rows;           // (slots' columns in a stage)
        const bool mine = row_in_use(om);
        // 16-byte pieces j (and 4 + j) of a block of 64 columns: row lane % 8, swizzled by the row
        const int r = lane & 7, j = lane >> 3;
        const uint32_t off = warp * (UR * KW * 2) + r * 128 + ((j ^ r) << 4);
        unsigned char* stage = sm.stage[warp];
#pragma unroll 1
        for (int u0 = 0; u0 < cnt; u0 += ug) {
            const int nu = min(ug, cnt - u0), nst = nu * per;
            float old = 0.f, gn = 0.f;
            auto ask = [&](int u) {                      // what an addition to the stream needs of it
                const int n = (blockIdx.x + (u0 + u) * gridDim.x) * UR + tid % UR;
                if (q.res != ADD_TO_STREAM || u >= nu || !mine) return;
                old = a.x[(size_t)om * a.D + n];         // (this thread wrote it, or the embedding)
                gn = q.gain != nullptr ? VecRef{q.gain, a.gain_dtype}.at(n) : 0.f;
            };
            ask(ou);                                     // (asked for now, needed at the end)
            float acc[TG / 2][2][4] = {};                // two chains of products each
            uint64_t v[MAX_ROWS][2];
            peek_stage(q, 0, v);
#pragma unroll 1
            for (int ks0 = 0; ks0 < q.K; ks0 += depth * KC) {
                for (uint32_t n = 0;; n++) {
                    int gone = -1;
#pragma unroll
                    for (int i = 0; i < MAX_ROWS; i++)
                        if (!has_tag(v[i][0], q.tag) || !has_tag(v[i][1], q.tag)) gone = i;
                    if (__all_sync(0xffffffffu, gone < 0)) break;
                    if (n >= 2) {                        // (looking on with all lanes slows the others' copies down)
                        const uint64_t* p = gone >= 0 ? staged(q, ks0, gone) : nullptr;
                        if (gone >= 0 && has_tag(peek(p), q.tag)) p++;
                        if (watch(p, gone >= 0, q.tag)) break;
                    }
                    peek_stage(q, ks0, v);
                }
#pragma unroll
                for (int i = 0; i < MAX_ROWS; i++)
                    *reinterpret_cast<uint2*>(stage + i * STAGE_PITCH + lane * 8) = make_uint2((uint32_t)v[i][0], (uint32_t)v[i][1]);
                __syncwarp();
                if (ks0 + depth * KC < q.K) peek_stage(q, ks0 + depth * KC, v);  // under way while these are multiplied
#pragma unroll 1
                for (int ks = 0; ks < depth && ks0 + ks * KC < q.K; ks++) {
                    uint32_t f[PIECES][4];               // (rows that the step does not have: some other row)
                    const uint32_t s = tc5::smem_u32(stage) + ((ks << a.lg_rows) + min(r, (1 << a.lg_rows) - 1)) * STAGE_PITCH + j * 16;
#pragma unroll
                    for (int c = 0; c < PIECES; c++) ldmatrix_x4(f[c], s + c * 64);
                    wait_full(it, nst);
#pragma unroll
                    for (int t = 0; t < TG; t += 2) {
                        if (t < nst) {
                            const uint32_t s0 = tc5::smem_u32(sm.slots[(it + t) % SLOTS]) + off;
                            // (an odd unit is multiplied with itself: its second half is not looked at)
                            const uint32_t s1 = tc5::smem_u32(sm.slots[(it + (t + 1 < nst ? t + 1 : t)) % SLOTS]) + off;
#pragma unroll
                            for (int c = 0; c < PIECES; c++) {
                                uint32_t w0[4], w1[4];
                                ldmatrix_x4(w0, (s0 + c / 2 * (UR * 128)) ^ (c % 2 * 64));
                                ldmatrix_x4(w1, (s1 + c / 2 * (UR * 128)) ^ (c % 2 * 64));
                                const uint32_t lo[4] = {w0[0], w1[0], w0[1], w1[1]}, hi[4] = {w0[2], w1[2], w0[3], w1[3]};
                                mma_bf16(acc[t / 2][0], lo, f[c][0], f[c][1]);
                                mma_bf16(acc[t / 2][1], hi, f[c][2], f[c][3]);
                            }
                        }
                    }
                    release(it, nst, 1);
                    it += nst;
                }
                __syncwarp();                            // the staged rows have been read
            }
            float(*sums)[TG][UR * MAX_ROWS] = sm.sums[turn];
            turn ^= 1;
#pragma unroll
            for (int t = 0; t < TG; t++)
                if (t < nst) {
#pragma unroll
                    for (int e = 0; e < 2; e++)          // a row of the step, a row of the weights
                        sums[warp][t][((lane & 3) * 2 + e) * UR + (lane >> 2)] = acc[t / 2][0][(t & 1) * 2 + e] + acc[t / 2][1][(t & 1) * 2 + e];
                }
            if (q.normed && u0 == 0) sync_norm();
            else sync_all();
#pragma unroll 1
            for (int u = ou; u - ou < nu; u += pass) {   // (as often in every thread)
                const int n = (blockIdx.x + (u0 + u) * gridDim.x) * UR + tid % UR;
                const bool on = u < nu && mine;
                if (!__any_sync(0xffffffffu, on)) continue;
                if (u != ou) ask(u);
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
                    const float x = old + s;
                    if (on) a.x[(size_t)om * a.D + n] = x;
                    if (q.gain != nullptr) publish_stream(on, x, gn, om, n, q.next);
                } else {
                    if (per == 2) s = s / (1.0f + expf(-s)) * s2;
                    const float other = __shfl_xor_sync(0xffffffffu, s, 1);
                    publish_pair(q.dst + ((uint32_t)(om * q.ld + n) >> 1), q.copy, on, s, other, q.next);
                }
            }
        }
    }

    // The n runs of one (sequence, kv head), by the four warps of a group: out[h] = sum_s w_s o_s / sum_s w_s l_s with
    // w_s = 2^(m_s - m). 4 / G warps a head (at least one), each adds every so many-th run; their sums are added in order.
    __device__ __forceinline__ void merge(AttnWork<HD>& w, int b, int g, int n, uint32_t tag) {
        constexpr int DL = HD / 32, BATCH = 8;           // a lane's columns; runs whose rows are under way together
        const int G = a.H / a.KV, lw = warp & 3;
        const int wph = G >= 3 ? 1 : 4 / G, hpt = 4 / wph, sub = lw % wph;       // warps a head, heads in one turn
#pragma unroll 1
        for (int h0 = 0; h0 < G; h0 += hpt) {
            const int h = h0 + lw / wph;
            float o[DL] = {}, lsum = 0.f;
            if (h < G) {
                const size_t row = ((size_t)b * a.H + g * G + h) * a.R;
                const uint64_t* ml = a.part_ml + row * 2;
                float m = -INFINITY;
#pragma unroll 1
                for (int s0 = 0; s0 < n; s0 += 32) {     // all runs' maxima and sums, a run a lane
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
                        lsum = lsum * exp2f(m - nm) + pl * exp2f(pm - nm);
                        m = nm;
                    }
                }
                const float top = warp_max(m);
                lsum = warp_sum(m > -INFINITY ? lsum * exp2f(m - top) : 0.f);
#pragma unroll 1
                for (int s0 = 0; s0 < n && top > -INFINITY; s0 += 32) {
                    uint64_t vm = 0, vl;
                    if (s0 + lane < n) peek2(ml + 2 * (s0 + lane), vm, vl);
                    const float pm = s0 + lane < n ? __uint_as_float((uint32_t)vm) : -INFINITY;
                    const float e = pm > -INFINITY ? exp2f(pm - top) : 0.f;       // (0: nothing to add)
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
            float* part = &w.o[0][0][0];                 // [4 warps][HD]
            if (wph > 1) {
                SyncGroup::sync();
                if (sub > 0) {
#pragma unroll
                    for (int d = 0; d < DL; d++) part[lw * HD + lane * DL + d] = o[d];
                }
                SyncGroup::sync();
            }
            if (sub == 0 && h < G) {
#pragma unroll 1
                for (int p = 1; p < wph; p++)
#pragma unroll
                    for (int d = 0; d < DL; d++) o[d] += part[(lw + p) * HD + lane * DL + d];
                const float inv = lsum > 0.f ? 1.0f / lsum : 0.f;
                uint64_t* dst = a.att + ((size_t)b * a.H * HD + (size_t)(g * G + h) * HD + lane * DL) / 2;
#pragma unroll
                for (int d = 0; d < DL; d += 2) publish_copies(dst + d / 2, (size_t)MAX_ROWS * (a.H * HD / 2), pack2(o[d] * inv, o[d + 1] * inv), tag);
            }
        }
        SyncGroup::sync();
    }

    __device__ __forceinline__ void attention(const LayerDesc& d, uint32_t tag) {
        constexpr int KSTEPS = HD / 16, NT = HD / 16, QLD = HD + 8;
        constexpr int LPH = HeadLanes<HD>::LPH, HPW = HeadLanes<HD>::HPW;
        const int grp = (int)d.group, J = sm.cum[grp][a.M], G = a.H / a.KV, window = a.window[grp];
        const int j0 = first_job(J, blockIdx.x), j1 = first_job(J, blockIdx.x + 1);
        const int gi = warp >> 2, lw = warp & 3, ltid = tid & 127, sub = lane / LPH, li = lane % LPH;
        const int mat = lane >> 3, rr = lane & 7;
        AttnWork<HD>& w = sm.a[gi];
        const int NQ = (a.H + 2 * a.KV) * HD;
        const bool rotate = a.cos_t != nullptr, has_gain = d.q_gain != nullptr;
        int pb = -1, pg = -1;                            // the (sequence, kv head) at hand
        bool merges = false;                             // some job of this group is a newest run of several
#pragma unroll 1
        for (int j = j0; j < j1; j++) {
            const Job job = look_up(sm, grp, j, j0, a.M);
            if ((j - j0) % PAGE_GROUPS != gi) {          // the other group's
                it += 2 * job.n;
                continue;
            }
            const int hi = sm.hi[job.b], pos = hi - 1, runs = runs_of(sm.cnt[grp][job.b]);
            const uint64_t* qrow = a.qkv + (size_t)job.b * NQ / 2;
            const int first = (sm.pg0[grp][job.b] + job.p) * PAGE_TOKENS, lo = first_visible(hi, window);
            const bool pos_ok = !rotate || pos < a.n_pos;
            if (!pos_ok && ltid == 0) atomicOr(a.status, MYNAH_ST_POS_RANGE);
            merges = merges || (job.r == runs - 1 && runs > 1);
            // The queries (for the first job of a sequence and kv head) and the new key and value: a warp takes every fourth pass
            // of heads, and the key if its place is among the warp's; whose that is begins with the queries last.
            const int at_new = pos - first;
            const bool newest = at_new >= 0 && at_new < job.n * PAGE_TOKENS, fresh = job.b != pb || job.g != pg;
            const int w_new = newest ? (at_new % PAGE_TOKENS) / 16 : 3, i_new = newest && w_new == lw ? at_new / PAGE_TOKENS : -1;
            uint4 ko = make_uint4(0, 0, 0, 0), vn = ko;
            pb = job.b;
            pg = job.g;
#pragma unroll 1
            for (int hb = fresh ? ((lw - w_new - 1) & 3) * HPW : G; hb < G || i_new >= 0; hb += 4 * HPW) {        // uniform over the warp
                const bool is_k = hb >= G;
                const int head = is_k ? a.H + job.g : job.g * G + hb + sub;
                float v[8], gain[8], rc[8], rs[8];
                if (rotate) load_rotation<HD>(a.cos_t, a.sin_t, pos_ok ? pos : 0, lane, rc, rs);
                if (has_gain) load_gain8(VecRef{is_k ? d.k_gain : d.q_gain, a.qk_dtype}, li * 8, gain);
                const uint64_t* p[2] = {qrow + (head * HD + li * 8) / 2, qrow + ((a.H + a.KV + job.g) * HD + li * 8) / 2};
                const bool on[2] = {is_k ? sub == 0 : hb + sub < G, is_k && sub == 0};
                uint32_t raw[2][4];
                read_tagged<2>(p, on, tag, raw);
                Raw8<bf16> r8;
                r8.q[0] = make_uint4(raw[0][0], raw[0][1], raw[0][2], raw[0][3]);
                r8.to_f32(v);
                head_norm_rotate<HD>(v, has_gain, gain, a.qk_eps, rotate, rc, rs, lane);
                const uint4 out = make_uint4(pack2(v[0], v[1]), pack2(v[2], v[3]), pack2(v[4], v[5]), pack2(v[6], v[7]));
                if (is_k) {
                    ko = out;
                    vn = make_uint4(raw[1][0], raw[1][1], raw[1][2], raw[1][3]);
                    break;
                }
                if (on[0]) *reinterpret_cast<uint4*>(w.q + (hb + sub) * QLD + li * 8) = out;
            }
            if (fresh) SyncGroup::sync();
            // ---- the run's pages: this warp's 16 keys of each
            const uint32_t q32 = tc5::smem_u32(w.q) + rr * QLD * 2 + mat * 16;
            float oc[NT][4] = {}, m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll 1
            for (int i = 0; i < job.n; i++, it += 2) {
                const int page = page_at(sm, a.pt[grp], grp, job, j, j0, i), p0 = first + i * PAGE_TOKENS;
                const bool empty = page < 0 || !pos_ok;
                if (page < 0 && ltid == 0) atomicOr(a.status, MYNAH_ST_PAGE_RANGE);
                const int k_first = max(lo, p0) - p0, k_last = min(hi, p0 + PAGE_TOKENS) - 1 - p0;
                const uint32_t ik = it % SLOTS, iv = (it + 1) % SLOTS;
                unsigned char *kt = sm.slots[ik], *vt = sm.slots[iv];
                wait_full<true>(it, 2);
                const bool mend = !empty && (lw * 16 < k_first || lw * 16 + 15 > k_last || i == i_new);      // uniform over the warp
                if (mend) {
                    // what a page holds outside the visible range may be anything: value rows that meet a probability of zero
                    // are cleared (scores of such keys are replaced, not multiplied)
#pragma unroll 1
                    for (int c = lane; c < 16 * (HD / 8); c += 32) {
                        const int row = lw * 16 + c / (HD / 8);
                        if (row < k_first || row > k_last) *reinterpret_cast<uint4*>(vt + TileTma<HD>::off(row, c % (HD / 8))) = make_uint4(0, 0, 0, 0);
                    }
                    if (i == i_new && sub == 0) {
                        *reinterpret_cast<uint4*>(kt + TileTma<HD>::off(at_new % PAGE_TOKENS, li)) = ko;
                        *reinterpret_cast<uint4*>(vt + TileTma<HD>::off(at_new % PAGE_TOKENS, li)) = vn;
                    }
                    __syncwarp();
                }
                if (!empty) {
                    // keys times queries: the warp's 16 keys are the rows, the heads the columns (those beyond the group's hold
                    // whatever is there); element e: key 16 lw + lane / 4 (+ 8 from e = 2 on), head (lane % 4) * 2 + e % 2
                    float sc[2][4] = {};
                    const uint32_t kb32 = tc5::smem_u32(kt), vb32 = tc5::smem_u32(vt);
#pragma unroll
                    for (int ks = 0; ks < KSTEPS; ks += 2) {
                        uint32_t qb[4], k0[4], k1[4];
                        ldmatrix_x4(qb, q32 + ks * 32);
                        ldmatrix_x4(k0, kb32 + TileTma<HD>::off(lw * 16 + (mat & 1) * 8 + rr, ks * 2 + (mat >> 1)));
                        ldmatrix_x4(k1, kb32 + TileTma<HD>::off(lw * 16 + (mat & 1) * 8 + rr, ks * 2 + 2 + (mat >> 1)));
                        mma_bf16(sc[0], k0, qb[0], qb[1]);
                        mma_bf16(sc[1], k1, qb[2], qb[3]);
                    }
                    float top[2] = {-INFINITY, -INFINITY};
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const int key = lw * 16 + (lane >> 2) + (e >> 1) * 8;
                        sc[0][e] = key >= k_first && key <= k_last ? (sc[0][e] + sc[1][e]) * a.scale : -INFINITY;
                        top[e & 1] = fmaxf(top[e & 1], sc[0][e]);
                    }
                    float shrink[2];
#pragma unroll
                    for (int e = 0; e < 2; e++) {
                        top[e] = fmaxf(top[e], __shfl_xor_sync(0xffffffffu, top[e], 4));
                        top[e] = fmaxf(top[e], __shfl_xor_sync(0xffffffffu, top[e], 8));
                        top[e] = fmaxf(m[e], fmaxf(top[e], __shfl_xor_sync(0xffffffffu, top[e], 16)));
                        shrink[e] = m[e] == top[e] ? 1.0f : exp2f(m[e] - top[e]);        // (nothing seen yet: 2^-inf = 0, of zeros)
                        m[e] = top[e];
                        l[e] *= shrink[e];
                        if (top[e] == -INFINITY) top[e] = 0.f;       // no key of this warp is visible: every probability is 0
                    }
                    if (__any_sync(0xffffffffu, shrink[0] != 1.0f || shrink[1] != 1.0f)) {
#pragma unroll
                        for (int nt = 0; nt < NT; nt++)
#pragma unroll
                            for (int e = 0; e < 4; e++) oc[nt][e] *= shrink[e & 1];
                    }
                    // probabilities: fp32 for the sum, bf16 and transposed (a head's keys in a row) for the product
                    uint32_t pr[2];
#pragma unroll
                    for (int t = 0; t < 2; t++) {
                        const float u0 = exp2f(sc[0][2 * t] - top[0]), u1 = exp2f(sc[0][2 * t + 1] - top[1]);
                        l[0] += u0;
                        l[1] += u1;
                        pr[t] = transpose8x8(pack2(u0, u1));
                    }
                    // values (transposed as they are loaded) times probabilities: 16 columns of the heads a product
#pragma unroll
                    for (int nt = 0; nt < NT; nt++) {
                        uint32_t va[4];
                        ldmatrix_x4_trans(va, vb32 + TileTma<HD>::off(lw * 16 + (mat >> 1) * 8 + rr, nt * 2 + (mat & 1)));
                        mma_bf16(oc[nt], va, pr[0], pr[1]);
                    }
                }
                if (mend) tc5::fence_async_smem();       // before a copy fills the slots again
                release(it, 2, CWARPS / 4);              // (four warps make the arrivals of all)
                if (i == i_new && !empty && sub == 0) {  // the new position's place in the cache
                    const size_t row = (((size_t)page * a.KV + job.g) * PAGE_TOKENS + at_new % PAGE_TOKENS) * HD + li * 8;
                    *reinterpret_cast<uint4*>(d.k + row) = ko;
                    *reinterpret_cast<uint4*>(d.v + row) = vn;
                }
            }
            // ---- the four warps' shares together, CHUNK heads at a time
#pragma unroll
            for (int e = 0; e < 2; e++) {
                l[e] += __shfl_xor_sync(0xffffffffu, l[e], 4);
                l[e] += __shfl_xor_sync(0xffffffffu, l[e], 8);
                l[e] += __shfl_xor_sync(0xffffffffu, l[e], 16);
                if (lane < 4) {
                    w.m[lw][lane * 2 + e] = m[e];
                    w.l[lw][lane * 2 + e] = l[e];
                }
            }
            const size_t row0 = ((size_t)job.b * a.H + (size_t)job.g * G) * a.R + job.r;
#pragma unroll 1
            for (int h0 = 0; h0 < G; h0 += CHUNK) {
                if ((lane & 3) == h0 / CHUNK) {
#pragma unroll
                    for (int nt = 0; nt < NT; nt++)
#pragma unroll
                        for (int e = 0; e < 4; e++) w.o[lw][e & 1][nt * 16 + (e >> 1) * 8 + (lane >> 2)] = oc[nt][e];
                }
                SyncGroup::sync();
                const int hc = ltid / (HD / 2), h = h0 + hc, c = ltid % (HD / 2) * 2;
                if (hc < CHUNK && h < G) {
                    const float top = fmaxf(fmaxf(w.m[0][h], w.m[1][h]), fmaxf(w.m[2][h], w.m[3][h]));
                    float o0 = 0.f, o1 = 0.f, sum = 0.f;
#pragma unroll
                    for (int p = 0; p < 4; p++) {
                        const float mp = w.m[p][h], f = mp > -INFINITY ? exp2f(mp - top) : 0.f;
                        const float2 o = *reinterpret_cast<const float2*>(&w.o[p][hc][c]);
                        sum = fmaf(f, w.l[p][h], sum);
                        o0 = fmaf(f, o.x, o0);
                        o1 = fmaf(f, o.y, o1);
                    }
                    if (runs == 1) {                     // all that the sequence sees: finished
                        const float inv = sum > 0.f ? 1.0f / sum : 0.f;
                        publish_copies(a.att + ((size_t)job.b * a.H * HD + (size_t)(job.g * G + h) * HD + c) / 2, (size_t)MAX_ROWS * (a.H * HD / 2),
                                       pack2(o0 * inv, o1 * inv), tag);
                    } else {
                        const size_t row = row0 + (size_t)h * a.R;
                        publish2(a.part_o + row * HD + c, __float_as_uint(o0), __float_as_uint(o1), tag);
                        if (c == 0) publish2(a.part_ml + row * 2, __float_as_uint(top), __float_as_uint(sum), tag);
                    }
                }
                SyncGroup::sync();
            }
        }
        // Both groups are through with their pages before a warp asks for a slot behind them: a barrier's parity names the right
        // filling only to those who know that the one before has come.
        sync_all();
        if (!merges) return;
        // A merge waits for runs with lower numbers only, and these wait for merges of still lower ones at most.
#pragma unroll 1
        for (int j = j0 + gi; j < j1; j += PAGE_GROUPS) {
            const Job job = look_up(sm, grp, j, j0, a.M);
            const int runs = runs_of(sm.cnt[grp][job.b]);
            if (job.r == runs - 1 && runs > 1) merge(w, job.b, job.g, runs, tag);
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
        sm.issued = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        tc5::fence_async_smem();
    }
    for (int i = tid; i < a.L * (int)(sizeof(LayerDesc) / 8); i += THREADS)
        reinterpret_cast<unsigned long long*>(sm.layers)[i] = reinterpret_cast<const unsigned long long*>(a.layers)[i];
    if (tid < MAX_ROWS) {
        int hi = tid < a.M ? a.kv_len[tid] : 0;
        // A row that sees more pages than the launch has splits for is reported and left alone, as a padding row is. (Without its
        // last pages nobody would read its new key and value, and the waits count on everything being read.)
        for (int g = 0; g < MAX_GROUPS; g++)
            if (a.pt[g].ids != nullptr && visible_pages(hi, a.window[g], 0).count() > a.S) {
                if (blockIdx.x == 0) atomicOr(a.status, MYNAH_ST_SPLIT_RANGE);
                hi = 0;
            }
        sm.hi[tid] = hi;
    }
    __syncthreads();
    if (tid < MAX_GROUPS) {                              // the pages that every sequence sees in each cache group
        int sum = 0;
        for (int b = 0; b < a.M; b++) {
            const VisiblePages vp = visible_pages(sm.hi[b], a.window[tid], 0);
            sm.pg0[tid][b] = vp.pg0;
            sm.cnt[tid][b] = vp.count();
            sm.cum[tid][b] = sum;
            sum += runs_of(sm.cnt[tid][b]) * a.KV;
        }
        sm.cum[tid][a.M] = sum;
    }
    __syncthreads();
    for (int i = tid; i < MAX_GROUPS * TABLE; i += THREADS) {
        const int g = i / TABLE, J = sm.cum[g][a.M], j = first_job(J, blockIdx.x) + i % TABLE;
        if (a.pt[g].ids != nullptr && j < first_job(J, blockIdx.x + 1)) {
            sm.table[g][i % TABLE] = find_job(sm, g, j, a.M);
            const Job job = look_up(sm, g, j, first_job(J, blockIdx.x), a.M);
            for (int k = 0; k < job.n; k++) sm.pages[g][i % TABLE][k] = page_of(a.pt[g], job.b, (sm.pg0[g][job.b] + job.p + k) * PAGE_TOKENS);
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
        for (int m = 0; m < a.M; m++) c.live |= sm.hi[m] > 0 ? 1u << m : 0u;
        if (warp > CWARPS) {
#pragma unroll 1
            for (int l = 0; l < a.L; l++) {
                const uint32_t t1 = base + 2 * l + 1;
#pragma unroll 1
                for (int i = 0; i < 2; i++)
                    if (my_units((i == 0 ? NQ : a.F) / UR) > 0) c.row_scales(warp - CWARPS - 1, t1 + i);
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
                    q.src += (size_t)(blockIdx.x % COPIES) * MAX_ROWS * ((i == 1 ? NO : (i == 3 ? a.F : a.D)) / 2);
                    q.tag = i < 2 ? t1 : t2;
                    q.n_units = (i == 0 ? NQ : (i == 2 ? a.F : a.D)) / UR;
                    q.K = i == 1 ? NO : (i == 3 ? a.F : a.D);
                    q.normed = i % 2 == 0;
                    q.res = i == 0 ? TO_BF16 : (i == 2 ? TO_SWIGLU : ADD_TO_STREAM);
                    q.dst = i == 0 ? a.qkv : a.act;
                    q.copy = i == 0 ? 0 : (size_t)MAX_ROWS * (a.F / 2);          // (the queries, keys and values of a head have few readers)
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
    if (e == cudaErrorCooperativeLaunchTooLarge) {       // fewer SMs than CTAs are this process's (or context's) to use
        (void)cudaGetLastError();
        return 1;
    }
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
    if (KV < 1 || KV > 255 || H < 1 || H % KV != 0 || H / KV > HEADS) return 0;
    if (D < 64 || F < 64 || D % 64 != 0 || F % 64 != 0) return 0;
    return 1;
}

// One decode step through all layers. layers: L descriptors of 96 bytes on the device; host_layers: the same on the host.
// Per cache group (n_groups of them) eight words: k and v bases, their rows (entries * pages * kv heads * 64), window, and the
// page lists. words: 64-bit words for 8 rows of 4 (D + H HD + F) / 2 + D + (H + 2 KV) HD / 2; part: 64-bit words for
// M * H * R * (HD + 2), R = most_runs(S), of which there are part_words; sync: two 32-bit words. All three zero before the first launch and kept from step to step.
// looks: trips to L2 that a wait may take (a few tenths of a microsecond each) before it is given up, with MYNAH_ST_TIMEOUT in the
// status, and with it all that its CTA still waits for; the others find what they wait for, if not its values.
// 1: declined, nothing was launched (its CTAs would not all be resident).
MYNAH_API int mynah_decode_layers(const void* layers, const void* host_layers, int L, int M, int D, int H, int KV, int HD, int F, int S,
                                  float* x, void* words, void* part, long long part_words, unsigned* sync,
                                  int gain_dtype, float eps, int qk_dtype, float qk_eps, const float* cos_t, const float* sin_t, int n_pos,
                                  const int* kv_len, int n_groups, const long long* group_words, int* status, int sms, int looks, cudaStream_t stream) {
    MYNAH_REQUIRE(mynah_decode_layers_supported(M, D, H, KV, HD, F, L, n_groups), "decode_layers: sizes are not supported");
    MYNAH_REQUIRE(S >= 1 && S <= 0xfffff, "decode_layers: %d page splits", S);
    MYNAH_REQUIRE(looks >= 0, "decode_layers: a wait of %d looks", looks);
    MYNAH_REQUIRE(sms >= 1 && sms <= mynah_sm_count(), "decode_layers: bad CTA count");
    StepMaps maps = {};
    StepArgs a = {};
    a.M = M; a.D = D; a.H = H; a.KV = KV; a.F = F; a.L = L; a.S = S; a.R = most_runs(S);
    MYNAH_REQUIRE((long long)M * H * a.R * (HD + 2) <= part_words, "decode_layers: %lld words of partial results are too few", part_words);
    a.gain_dtype = gain_dtype; a.qk_dtype = qk_dtype; a.n_pos = n_pos;
    a.eps = eps; a.qk_eps = qk_eps; a.inv_d = 1.0f / (float)D;
    a.scale = (float)(1.4426950408889634 / sqrt((double)HD));        // probabilities are powers of two: score times log2(e)
    while ((1 << a.lg_rows) < M) a.lg_rows++;
    a.layers = static_cast<const LayerDesc*>(layers);
    a.x = x;
    a.hid = static_cast<uint64_t*>(words);
    a.squares = a.hid + (size_t)COPIES * MAX_ROWS * (D / 2);
    a.qkv = a.squares + (size_t)SQUARE_COPIES * MAX_ROWS * (D / UR);
    a.att = a.qkv + (size_t)MAX_ROWS * ((H + 2 * KV) * HD / 2);
    a.act = a.att + (size_t)COPIES * MAX_ROWS * (H * HD / 2);
    a.part_o = static_cast<uint64_t*>(part);
    a.part_ml = a.part_o + (size_t)M * H * a.R * HD;
    a.looks = (uint32_t)looks; a.look_mask = looks >= 255 ? 255 : 0;
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
