// From logits to a token, on the device: penalties, greedy argmax, and
// temperature sampling with top-k, min-p and top-p, in the reference's order
// (mynah-slm src/sampler.c:116-187; penalties :80-106; ring :73-78; the
// generator is splitmix64, :40-46).
//
// The reference sorts the whole vocabulary by (probability descending, id
// ascending) and works on prefixes of that order. Every filter keeps a prefix
// and the draw walks a prefix, so no sort is needed here: a prefix is found by
// a radix search over the bits of the probabilities (three passes of 11, 11
// and 10 bits) with a histogram of counts and of probability mass per digit.
// Mass is summed as 2^-60 fixed point in 64-bit integers: integer sums do not
// depend on the order of the additions, so the same logits and the same
// generator state give the same token in every run.
//
// What bounds a draw is latency: a row of 151,936 logits is 0.6 MB, and what follows its one read is a chain of block and
// cluster barriers. So a draw is one launch (penalties, maximum, exponentials, selection, the walk and the ring), a row is
// read once, into the shared memory of its cluster's CTAs, and every later pass goes over that copy.
#include "common.cuh"

#include <cooperative_groups.h>

namespace {

namespace cg = cooperative_groups;

constexpr int THREADS = 512;
constexpr int WARPS = THREADS / 32;
constexpr int ROW_CTAS = 8;            // CTAs (one cluster) that share a row of a large vocabulary
constexpr int LOADS = 8;               // loads of a row that a thread keeps in flight
constexpr int BINS = 2048;
constexpr int MAX_CAND = 256;          // a top-k of at most this many entries is drawn from a list of candidates

// floor(p * 2^60): for a probability (0 <= p <= 1) a shift of its mantissa, exactly what the product in double gives
__device__ __forceinline__ unsigned long long mass_of(float p) {
    const unsigned int bits = __float_as_uint(p);
    const int e = (int)(bits >> 23);
    if (e > 127) return __double2ull_rd((double)p * 1152921504606846976.0);       // (not a probability: infinite or no number)
    const unsigned long long m = e > 0 ? (bits & 0x7fffffu) | 0x800000u : 0u;      // (a subnormal's product lies below 1)
    const int s = e - 90;                                                          // p = m * 2^(e - 150)
    return s >= 0 ? m << s : (s > -24 ? m >> -s : 0ull);
}

struct Prefix {            // a prefix of the sorted order
    unsigned int value;    // bits of the probability at which it ends
    unsigned int above;    // elements with a larger probability
    unsigned int ties;     // elements equal to `value` that belong to it (by ascending id)
    unsigned long long mass;   // its total mass
};

struct Found {
    unsigned int digit, above, count;                       // the digit, the elements in larger digits, those in it
    unsigned long long mass;                                // mass of the elements in larger digits
};

// Elements of one digit share every bit from `shift` up, their exponent E among them, so where mass_of shifts a mantissa up
// (E >= 90) a digit's mass follows from its count and the sum of the bits below `shift`. That sum is kept in two words, its
// elements' low eleven bits and the rest: adds whose result nobody reads, and none that carries. Where mass_of shifts down,
// or for what is no probability, the words are the low and high half of the masses' own sum (2^-60 fixed point). 64-bit adds
// in shared memory would be compare-and-swap loops that crawl when many warps hit one digit.
struct Histogram {
    unsigned int count[BINS];
    unsigned int lo[BINS], hi[BINS];
};
constexpr int LOW_BITS = 11;
// (a CTA with more than 2^21 elements could overflow the low word: it sums the masses themselves, `span` 0)
constexpr unsigned int SPAN = 128 - 90;
__device__ __forceinline__ bool mass_by_count(unsigned int bits, unsigned int span) { return (bits >> 23) - 90u < span; }

template <int NC>
struct Shared {
    // The row's first maxima a group of threads, of all CTAs: their largest is the row's maximum, and the k-th largest of
    // them is a lower bound of the row's k-th largest element.
    static constexpr int GROUPS = 256, LANES = NC * THREADS / GROUPS;
    __align__(16) float group_v[GROUPS];
    int group_i[GROUPS];
    union {
        Histogram h;
        unsigned long long list[NC][MAX_CAND];              // leading CTA: the candidates of every CTA
    };
    unsigned long long mine[MAX_CAND];                      // this CTA's candidates
    unsigned long long key[MAX_CAND], sorted[MAX_CAND];
    double part_d[NC];                                      // every CTA's sum of exponentials
    unsigned long long part_m[NC];                          // a value a CTA: masses
    unsigned int part_u[NC], part_v[NC];                    // a value a CTA: counts
    Found found;
    unsigned int n_mine, n_key;
    float mx, bound;
    int best, id;
    double red_d[WARPS];
    unsigned long long warp_mass[WARPS];
    unsigned int warp_count[WARPS], scan_u[WARPS];
    int ring[256];
};

struct ArgmaxShared {
    float red_f[32];
    int red_i[32];
};

__device__ __forceinline__ void add_mass(Histogram& h, unsigned int d, unsigned long long m) {
    const unsigned int lo = (unsigned int)m;
    unsigned int hi = (unsigned int)(m >> 32);
    if (lo != 0) {
        const unsigned int old = atomicAdd(&h.lo[d], lo);
        hi += old > 0xffffffffu - lo;                      // the low word wrapped: carry
    }
    if (hi != 0) atomicAdd(&h.hi[d], hi);
}

// A row is shared by NC CTAs (NC = 1, or the ROW_CTAS CTAs of a cluster): CTA r works on the elements
// [r * chunk, (r + 1) * chunk) and the CTAs meet through distributed shared memory. Every CTA of a row runs
// the same code with the same decisions, so the cluster barriers below are reached by all of them.
template <int NC, bool IN_SHARED>
struct RowShare {
    int rank, begin, n;                                     // this CTA's elements: `n` from `begin` on
    float* p;                                               // where it keeps them: shared memory, or the row itself if too long
    bool wide;                                              // more elements a CTA than mass_by_count can add up (never in shared memory)
    __device__ __forceinline__ unsigned int span() const { return IN_SHARED || !wide ? SPAN : 0u; }
    __device__ static int chunk(int V) { return NC == 1 ? V : ((V + NC - 1) / NC + 3) & ~3; }
    __device__ explicit RowShare(int V) {
        rank = NC == 1 ? 0 : (int)cg::this_cluster().block_rank();
        begin = min(V, rank * chunk(V));
        n = min(V, begin + chunk(V)) - begin;
        wide = !IN_SHARED && chunk(V) > 1 << 21;            // the same in every CTA of the row
    }
    __device__ __forceinline__ void sync() const {
        if (NC == 1) __syncthreads();
        else cg::this_cluster().sync();
    }
    template <typename T> __device__ __forceinline__ T* at(T* mine, int r) const {
        return NC == 1 ? mine : cg::this_cluster().map_shared_rank(mine, r);
    }
};

// What a pass of the search goes by: the elements p[i] * scale whose bits under `mask` are `bits`, by their next digit, the bits
// [shift, shift + log2(n_bins)). Three passes: 11, 11 and 10 bits.
struct Digit {
    unsigned int bits, mask;
    int shift, n_bins;
};

// A CTA's slice of the digits over all CTAs of the row: rank r has the r-th slice from the top, its thread t the digits
// [hi - PER + 1, hi], taken from the largest down.
template <int NC>
struct Slice {
    static constexpr int WIDE = BINS / NC, PER = (WIDE + THREADS - 1) / THREADS;
    int hi;
    unsigned int c[PER];
    unsigned long long m[PER];
};

// Counts and masses of a pass. Probabilities crowd into a few digits where the logits do: a warp whose 32 elements fall into
// at most four digits adds each digit up over the warp and lets one lane do the atomics. Counts and masses are integers, so
// the order of the additions does not matter.
template <int NC, bool IN_SHARED>
__device__ __noinline__ void fill_histogram(const RowShare<NC, IN_SHARED>& rs, const Digit dg, float scale, Shared<NC>& sh) {
    for (int i = threadIdx.x; i < BINS; i += THREADS) {
        sh.h.count[i] = 0;
        sh.h.lo[i] = 0;
        sh.h.hi[i] = 0;
    }
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const unsigned int low_mask = (1u << dg.shift) - 1u;
    for (int base0 = 0; base0 < rs.n; base0 += THREADS * LOADS) {             // the same number of turns for every thread
        float vals[LOADS];
#pragma unroll
        for (int u = 0; u < LOADS; u++) {
            const int i = base0 + u * THREADS + (int)threadIdx.x;
            vals[u] = i < rs.n ? rs.p[i] : 0.f;
        }
#pragma unroll
        for (int u = 0; u < LOADS; u++) {
            const int i = base0 + u * THREADS + (int)threadIdx.x;
            if (base0 + u * THREADS >= rs.n) break;               // uniform
            const float v = vals[u] * scale;
            const unsigned int bits = __float_as_uint(v);
            const bool on = i < rs.n && (bits & dg.mask) == dg.bits;
            const unsigned int active = __ballot_sync(0xffffffffu, on);
            if (active == 0u) continue;                           // (most warps, once a prefix is known)
            const unsigned int d = (bits >> dg.shift) & (dg.n_bins - 1);
            // the first element's digit, then the first of what is left: two turns tell a crowd from a spread
            unsigned int left = active;
#pragma unroll
            for (int t = 0; t < 2; t++) {
                if (__popc(left) >= 8) {                          // uniform
                    const int src = __ffs(left) - 1;
                    const unsigned int ds = __shfl_sync(0xffffffffu, d, src);
                    const bool same = ((left >> lane) & 1u) && d == ds;
                    const unsigned int grp = __ballot_sync(0xffffffffu, same);
                    const unsigned int bs = __shfl_sync(0xffffffffu, bits, src);
                    if (__popc(grp) >= 8 && mass_by_count(bs, rs.span())) {
                        const unsigned int low = same ? bits & low_mask : 0u;
                        const unsigned int lo = __reduce_add_sync(0xffffffffu, low & ((1u << LOW_BITS) - 1u));
                        const unsigned int hi = __reduce_add_sync(0xffffffffu, low >> LOW_BITS);
                        if (lane == src) {
                            atomicAdd(&sh.h.count[ds], (unsigned int)__popc(grp));
                            if (lo) atomicAdd(&sh.h.lo[ds], lo);
                            if (hi) atomicAdd(&sh.h.hi[ds], hi);
                        }
                        left &= ~grp;
                    }
                }
            }
            if ((left >> lane) & 1u) {
                atomicAdd(&sh.h.count[d], 1u);
                if (mass_by_count(bits, rs.span())) {
                    const unsigned int low = bits & low_mask, lo = low & ((1u << LOW_BITS) - 1u), hi = low >> LOW_BITS;
                    if (lo) atomicAdd(&sh.h.lo[d], lo);
                    if (hi) atomicAdd(&sh.h.hi[d], hi);
                } else {
                    add_mass(sh.h, d, mass_of(v));
                }
            }
        }
    }
}

// This CTA's slice of a pass over the row. The histograms may be filled again behind find_digit's first barrier.
template <int NC, bool IN_SHARED>
__device__ __forceinline__ Slice<NC> add_up(const RowShare<NC, IN_SHARED>& rs, const Digit dg, float scale, Shared<NC>& sh) {
    fill_histogram<NC, IN_SHARED>(rs, dg, scale, sh);
    rs.sync();                                              // every CTA's histogram is complete
    Slice<NC> s;
    s.hi = dg.n_bins - 1 - (rs.rank * Slice<NC>::WIDE + (int)threadIdx.x * Slice<NC>::PER);
#pragma unroll
    for (int q = 0; q < Slice<NC>::PER; q++) {
        const int d = s.hi - q;
        s.c[q] = 0;
        s.m[q] = 0;
        if ((int)threadIdx.x * Slice<NC>::PER < Slice<NC>::WIDE && d >= 0) {
            unsigned int c[NC], lo[NC], hi[NC];
#pragma unroll
            for (int r = 0; r < NC; r++) {                  // the loads first, all in flight together
                c[r] = *rs.at(&sh.h.count[d], r);
                lo[r] = *rs.at(&sh.h.lo[d], r);
                hi[r] = *rs.at(&sh.h.hi[d], r);
            }
            unsigned long long lows = 0, masses = 0;
#pragma unroll
            for (int r = 0; r < NC; r++) {
                s.c[q] += c[r];
                lows += lo[r] + ((unsigned long long)hi[r] << LOW_BITS);
                masses += ((unsigned long long)hi[r] << 32) | lo[r];
            }
            const unsigned int base = dg.bits | ((unsigned int)d << dg.shift);     // the digit's smallest element
            s.m[q] = mass_by_count(base, rs.span())
                ? ((unsigned long long)((base & 0x7fffffu) | 0x800000u) * s.c[q] + lows) << ((base >> 23) - 90u) : masses;
        }
    }
    return s;
}

// Finds the digit where the running (count, mass), taken from the largest digit down, first satisfies the
// target. by_mass: cum_mass >= target_mass; else cum_count >= target_count. The carried count and mass are those of the
// elements in larger digits of earlier passes. Every thread of every CTA of the row gets the result. A CTA tells the others
// its slice's totals; the one whose slice holds the digit tells them the result: two barriers over the cluster.
template <int NC, bool IN_SHARED>
__device__ __noinline__ Found find_digit(const RowShare<NC, IN_SHARED>& rs, const Slice<NC>& s, bool by_mass, unsigned int target_count,
                                         unsigned long long target_mass, unsigned int carry_count, unsigned long long carry_mass,
                                         Shared<NC>& sh) {
    constexpr int PER = Slice<NC>::PER;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned int cs = 0;
    unsigned long long ms = 0;
#pragma unroll
    for (int q = 0; q < PER; q++) {
        cs += s.c[q];
        ms += s.m[q];
    }
    const unsigned int c_own = cs;
    const unsigned long long m_own = ms;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int ct = __shfl_up_sync(0xffffffffu, cs, o);
        const unsigned long long mt = __shfl_up_sync(0xffffffffu, ms, o);
        if (lane >= o) {
            cs += ct;
            ms += mt;
        }
    }
    if (lane == 31) {
        sh.warp_count[warp] = cs;
        sh.warp_mass[warp] = ms;
    }
    __syncthreads();
    unsigned int c_before = cs - c_own;                     // this slice's elements before the thread's digits
    unsigned long long m_before = ms - m_own;
    for (int w = 0; w < warp; w++) {
        c_before += sh.warp_count[w];
        m_before += sh.warp_mass[w];
    }
    if (threadIdx.x == THREADS - 1) {
        for (int r = 0; r < NC; r++) {
            *rs.at(&sh.part_u[rs.rank], r) = c_before + c_own;
            *rs.at(&sh.part_m[rs.rank], r) = m_before + m_own;
        }
    }
    rs.sync();                                              // every slice's totals are known; the histograms have been read
    auto met = [&](unsigned int cc, unsigned long long mm) {
        return by_mass ? (mm >= target_mass) : (cc >= target_count);
    };
    unsigned int ct = carry_count, c_slice = 0;
    unsigned long long mt = carry_mass, m_slice = 0;
    int owner = -1, last = -1;                              // the slice that meets the target; the lowest with an element
    for (int r = 0; r < NC; r++) {
        if (r == rs.rank) {
            c_slice = ct;
            m_slice = mt;
        }
        const unsigned int cn = ct + sh.part_u[r];
        const unsigned long long mn = mt + sh.part_m[r];
        if (owner < 0 && sh.part_u[r] > 0 && !met(ct, mt) && met(cn, mn)) owner = r;
        if (sh.part_u[r] > 0) last = r;
        ct = cn;
        mt = mn;
    }
    c_before += c_slice;
    m_before += m_slice;
    const bool beyond = owner < 0;                          // target beyond everything (rounding): end at the smallest populated digit
    if (rs.rank == (beyond ? last : owner)) {
#pragma unroll
        for (int q = 0; q < PER; q++) {
            const unsigned int cn = c_before + s.c[q];
            const unsigned long long mn = m_before + s.m[q];
            if (s.c[q] > 0 && (beyond ? cn == ct : !met(c_before, m_before) && met(cn, mn))) {
                const Found f{(unsigned int)(s.hi - q), c_before, s.c[q], m_before};
                for (int r = 0; r < NC; r++) *rs.at(&sh.found, r) = f;
            }
            c_before = cn;
            m_before = mn;
        }
    }
    rs.sync();                                              // the result is there
    return sh.found;                                        // (written again only behind the next search's first barrier)
}

constexpr Digit FIRST_DIGIT{0u, 0u, 21, 2048};

// The smallest prefix of the sorted order whose count reaches target_count
// (by_mass false) or whose mass reaches target_mass (by_mass true). `first`: the row's slice by FIRST_DIGIT.
template <int NC, bool IN_SHARED>
__device__ __noinline__ Prefix find_prefix(const RowShare<NC, IN_SHARED>& rs, const Slice<NC>& first, bool by_mass, unsigned int target_count,
                                           unsigned long long target_mass, Shared<NC>& sh) {
    if (by_mass && target_mass == 0) target_mass = 1;      // a draw of exactly 0 takes the first element
    if (!by_mass && target_count == 0) target_count = 1;
    Found f = find_digit<NC, IN_SHARED>(rs, first, by_mass, target_count, target_mass, 0u, 0ull, sh);
    Digit dg{f.digit << 21, 2047u << 21, 10, 2048};
    f = find_digit<NC, IN_SHARED>(rs, add_up<NC, IN_SHARED>(rs, dg, 1.0f, sh), by_mass, target_count, target_mass, f.above, f.mass, sh);
    dg = Digit{dg.bits | f.digit << 10, dg.mask | 2047u << 10, 0, 1024};
    f = find_digit<NC, IN_SHARED>(rs, add_up<NC, IN_SHARED>(rs, dg, 1.0f, sh), by_mass, target_count, target_mass, f.above, f.mass, sh);
    const unsigned int bits = dg.bits | f.digit, n_eq = f.count;
    // `bits` is the probability at which the prefix ends; n_eq elements have exactly it
    const unsigned long long pm = mass_of(__uint_as_float(bits));
    unsigned int ties;
    if (by_mass) {
        if (pm == 0 || target_mass <= f.mass) ties = 1;
        else {
            const unsigned long long need = target_mass - f.mass;
            const unsigned long long t = (need + pm - 1) / pm;
            ties = (unsigned int)(t < 1 ? 1 : (t > n_eq ? n_eq : t));
        }
    } else {
        ties = target_count > f.above ? target_count - f.above : 1;
        if (ties > n_eq) ties = n_eq;
    }
    if (ties < 1) ties = 1;
    return Prefix{bits, f.above, ties, f.mass + (unsigned long long)ties * pm};
}

// Id of the j-th (1-based) element, by ascending id, whose probability bits equal `value` (-1: there is none).
// The CTAs of a row hold consecutive ranges of ids, so the j-th lies in the first CTA whose running count reaches j.
template <int NC, bool IN_SHARED>
__device__ int nth_equal(const RowShare<NC, IN_SHARED>& rs, unsigned int value, unsigned int j, Shared<NC>& sh) {
    const int per = (rs.n + THREADS - 1) / THREADS;
    const int lo = min(rs.n, (int)threadIdx.x * per), hi = min(rs.n, lo + per);
    unsigned int c = 0;
    for (int i = lo; i < hi; i++) c += __float_as_uint(rs.p[i]) == value;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned int cs = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int t = __shfl_up_sync(0xffffffffu, cs, o);
        if (lane >= o) cs += t;
    }
    if (lane == 31) sh.scan_u[warp] = cs;
    if (threadIdx.x == 0) sh.id = -1;
    __syncthreads();
    unsigned int before = cs - c;                           // equal elements before this thread's range
    for (int w = 0; w < warp; w++) before += sh.scan_u[w];
    if (threadIdx.x == THREADS - 1)
        for (int r = 0; r < NC; r++) *rs.at(&sh.part_v[rs.rank], r) = before + c;       // equal elements in this CTA's range
    rs.sync();
    for (int r = 0; r < rs.rank; r++) before += sh.part_v[r];
    if (c > 0 && before < j && j <= before + c) {
        unsigned int seen = before;
        for (int i = lo; i < hi; i++) {
            if (__float_as_uint(rs.p[i]) == value && ++seen == j) {
                for (int r = 0; r < NC; r++) *rs.at(&sh.id, r) = rs.begin + i;
                break;
            }
        }
    }
    rs.sync();
    return sh.id;                                           // (searched once a draw: id and part_v are not written again)
}

__device__ __forceinline__ double splitmix_uniform(unsigned long long* state) {
    unsigned long long z = (*state += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z = z ^ (z >> 31);
    return (double)(z >> 11) * (1.0 / 9007199254740992.0);
}

struct SampleParams {
    float temp, top_p, min_p;
    int top_k;
};

__device__ __forceinline__ void take_first_max(float& bv, int& bi, float v, int i) {
    if (v > bv || (v == bv && i < bi)) {
        bv = v;
        bi = i;
    }
}

constexpr int ARGMAX_THREADS = 1024;

// First maximum of a row (strict >, lowest index on ties: sampler.c:124-129).
__device__ int block_argmax(const float* __restrict__ row, int V, ArgmaxShared& sh, float* max_out) {
    float bv = -INFINITY;
    int bi = 0x7fffffff;
    for (int i = threadIdx.x; i < V; i += ARGMAX_THREADS) {
        const float v = row[i];
        if (v > bv || (v == bv && i < bi)) {
            bv = v;
            bi = i;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float v2 = __shfl_xor_sync(0xffffffffu, bv, o);
        const int i2 = __shfl_xor_sync(0xffffffffu, bi, o);
        if (v2 > bv || (v2 == bv && i2 < bi)) {
            bv = v2;
            bi = i2;
        }
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) {
        sh.red_f[warp] = bv;
        sh.red_i[warp] = bi;
    }
    __syncthreads();
    bv = sh.red_f[lane];
    bi = sh.red_i[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float v2 = __shfl_xor_sync(0xffffffffu, bv, o);
        const int i2 = __shfl_xor_sync(0xffffffffu, bi, o);
        if (v2 > bv || (v2 == bv && i2 < bi)) {
            bv = v2;
            bi = i2;
        }
    }
    __syncthreads();
    *max_out = bv;
    return bi == 0x7fffffff ? 0 : bi;
}

// The ring of a sequence's recent tokens (all null: none is kept). Rows are `stride` apart; the window in use is
// params[7] <= stride.
struct Ring {
    int* tokens;
    int* n;
    int* head;
    int stride;
};

// ring[slot][head] = token; head advances; the count saturates at the window.
__device__ __forceinline__ void accept_token(const Ring& ring, int slot, int window, int token) {
    const int head = ring.head[slot] % window;
    ring.tokens[(size_t)slot * ring.stride + head] = token;
    ring.head[slot] = (head + 1) % window;
    if (ring.n[slot] < window) ring.n[slot]++;
}

// One of the reference's turns over an entry of the ring: a token that sits there c times takes it c times (sampler.c:80-106).
__device__ __forceinline__ float penalise(float l, float repeat, float freq, float presence, int count) {
    if (repeat != 1.0f) l = l > 0.f ? l / repeat : l * repeat;
    l -= freq * (float)count;
    l -= presence;
    return l;
}

// The walk over at most MAX_CAND candidates by one CTA (sampler.c:146-186): sh.key[0, n_key) are probability bits above,
// ~id below, each key once. A key's place in the order (probability descending, id ascending) is the number of larger keys;
// one warp then walks the places, 32 at a time: min-p, top-p, the kept mass and the drawn place are prefixes in the same
// integer arithmetic as the general search's. Returns the drawn id (-1: no candidate) to lane 0 of warp 0.
template <int NC>
__device__ int draw_from_keys(Shared<NC>& sh, unsigned int n_key, const SampleParams& sp, float p_best, double u) {
    constexpr int TPK = THREADS / MAX_CAND;                 // threads a key
    const unsigned int t = threadIdx.x / TPK, part = threadIdx.x % TPK;
    unsigned int place = 0;
    const unsigned long long own = t < n_key ? sh.key[t] : 0ull;
    if (t < n_key)
        for (unsigned int j = part; j < n_key; j += TPK) place += sh.key[j] > own;
#pragma unroll
    for (int o = TPK / 2; o > 0; o >>= 1) place += __shfl_xor_sync(0xffffffffu, place, o);
    if (t < n_key && part == 0) sh.sorted[place] = own;
    __syncthreads();
    if (threadIdx.x >= 32) return -1;
    const unsigned int lane = threadIdx.x;
    const unsigned int n_c = min(n_key, (unsigned int)sp.top_k);
    constexpr int TURNS = MAX_CAND / 32;
    unsigned long long cum[TURNS], carry = 0;               // running masses; place i is lane i % 32 of turn i / 32
    unsigned int above_floor = 0;
    const float floor_p = sp.min_p * p_best;
#pragma unroll
    for (int k = 0; k < TURNS; k++) {
        cum[k] = 0;
        if (k * 32u < n_c) {                                // uniform
            const unsigned int i = k * 32 + lane;
            const float p = i < n_c ? __uint_as_float((unsigned int)(sh.sorted[i] >> 32)) : 0.f;
            unsigned long long m = i < n_c ? mass_of(p) : 0ull;
            above_floor += __popc(__ballot_sync(0xffffffffu, i < n_c && p >= floor_p));
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long x = __shfl_up_sync(0xffffffffu, m, o);
                if ((int)lane >= o) m += x;
            }
            cum[k] = carry + m;
            carry = __shfl_sync(0xffffffffu, cum[k], 31);
        }
    }
    unsigned int n = n_c;
    if (sp.min_p > 0.f) n = min(n, max(above_floor, 1u));
    // the first place below n whose running mass reaches the target (n: none)
    auto first = [&](unsigned long long target) {
        unsigned int at = n;
#pragma unroll
        for (int k = TURNS - 1; k >= 0; k--) {
            if (k * 32u < n) {
                const unsigned int b = __ballot_sync(0xffffffffu, k * 32 + lane < n && cum[k] >= target);
                if (b) at = k * 32 + __ffs(b) - 1;
            }
        }
        return at;
    };
    if (sp.top_p < 1.0f) {
        unsigned long long target = __double2ull_ru((double)sp.top_p * 1152921504606846976.0);
        if (target == 0) target = 1;
        const unsigned int at = first(target);
        if (at < n) n = at + 1;
    }
    if (n < 1) n = 1;
    unsigned long long total = 0;
#pragma unroll
    for (int k = 0; k < TURNS; k++) {
        const unsigned long long x = __shfl_sync(0xffffffffu, cum[k], (n - 1) & 31);
        if (k == (int)((n - 1) >> 5)) total = x;
    }
    unsigned long long target = __double2ull_ru(u * (double)total);
    if (target > total) target = total;
    if (target == 0) target = 1;
    unsigned int pick = first(target);
    if (pick >= n) pick = n - 1;                            // (only through rounding: the last kept one)
    return n_c > 0 ? (int)(0xffffffffu - (unsigned int)sh.sorted[pick]) : -1;
}

// One CTA a row, or for a large vocabulary the ROW_CTAS CTAs of a cluster (NC), each with a consecutive part of
// the row: penalties, the maximum, exponentials and their sum, the draw, the accepted token into the ring.
//
// A small top-k (sampler.c:132-186, the same decisions in another order): the maxima of groups of threads are at hand from the
// row's maximum, and the k-th largest of them bounds the row's k-th largest from below, so the pass that forms the
// exponentials also lists everything that can be among the k largest probabilities (equal ones included: a bound with a
// margin above rounding). The leading CTA sorts that list and walks it. Two barriers over the cluster. The bound is used while
// k is at most half the groups (then about 0.7 entries a group are expected above it); beyond that, and for rows with many
// equal logits, the leading bits of the k-th largest are searched by count, and if even those leave more than MAX_CAND entries
// (many equal logits) the whole k-th probability and the id up to which its equals belong.
// Everything else goes through find_prefix.
// Measured (151,936 logits a row; us a draw on the device for 1, 8 and 64 rows; before: a launch for the maximum and one for
// each kind of draw, passes over the row in L2): top-k 20 48, 50, 200 -> 17, 17, 48; top-p 0.95 alone 156, 158, 757 -> 76, 77, 212;
// temperature alone 70, 70, 326 -> 58, 59, 160. 512 threads a CTA, so that two share an SM: with 1,024 (whose registers fill
// it) 64 rows took 63 us with top-k 20 and 496 with top-p, one row 15 instead of 17. A cluster a row at 32,000 logits: 12 us
// against 18 at one row, but 45 against 19 at 64 and 268 against 86 with top-p: one CTA a row below 32,768.
template <int NC, bool IN_SHARED>
__global__ void __launch_bounds__(THREADS)
sample_kernel(float* __restrict__ logits, int V, int ld, const float* __restrict__ params, unsigned long long* __restrict__ rng,
              const int* __restrict__ slots, int* __restrict__ out, Ring ring) {
    extern __shared__ __align__(16) unsigned char smem[];
    Shared<NC>& sh = *reinterpret_cast<Shared<NC>*>(smem);
    constexpr int GROUPS = Shared<NC>::GROUPS, LANES = Shared<NC>::LANES;      // groups of LANES lanes
    // another CTA's shared memory may be written once that CTA runs: arrive here, wait before the first such write
    if (NC > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    griddep_launch();
    griddep_wait();
    const SampleParams sp{params[0], params[1], params[2], (int)params[3]};
    const float repeat = params[4], freq = params[5], presence = params[6];
    const int window = ring.tokens != nullptr ? min((int)params[7], ring.stride) : 0;
    const int b = NC == 1 ? blockIdx.x : blockIdx.x / NC;
    float* row = logits + (size_t)b * ld;
    const int slot = slots ? slots[b] : b;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    RowShare<NC, IN_SHARED> rs(V);
    if (slot < 0) {                          // padding row (all CTAs of the row leave)
        if (NC > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (threadIdx.x == 0 && rs.rank == 0) out[b] = 0;
        return;
    }
    unsigned long long state = rng[slot];                   // (written by the leading CTA, behind the last barrier of all CTAs)
    if (threadIdx.x == 0) {
        sh.n_mine = 0;
        sh.n_key = 0;
    }
    // ---- the row, and each thread's first maximum
    rs.p = IN_SHARED ? reinterpret_cast<float*>(smem + sizeof(Shared<NC>)) : row + rs.begin;
    const float* from = row + rs.begin;
    float bv = -INFINITY;
    int bi = 0x7fffffff;
    auto scan = [&](const float* src, bool keep) {
        for (int base0 = 0; base0 < rs.n; base0 += THREADS * LOADS) {
            float vals[LOADS];
#pragma unroll
            for (int u = 0; u < LOADS; u++) {
                const int i = base0 + u * THREADS + (int)threadIdx.x;
                vals[u] = i < rs.n ? src[i] : -INFINITY;
            }
#pragma unroll
            for (int u = 0; u < LOADS; u++) {
                const int i = base0 + u * THREADS + (int)threadIdx.x;
                if (i < rs.n) {
                    take_first_max(bv, bi, vals[u], rs.begin + i);
                    if (keep) rs.p[i] = vals[u];
                }
            }
        }
    };
    if ((ld & 3) == 0 && (reinterpret_cast<uintptr_t>(logits) & 15) == 0) {   // (begin is a multiple of 4)
        constexpr int LOADS4 = 5;
        const int n4 = rs.n / 4;
        const float4* from4 = reinterpret_cast<const float4*>(from);
        for (int base0 = 0; base0 < n4; base0 += THREADS * LOADS4) {
            float4 v[LOADS4];
#pragma unroll
            for (int u = 0; u < LOADS4; u++) {
                const int j = base0 + u * THREADS + (int)threadIdx.x;
                if (j < n4) v[u] = IN_SHARED ? __ldcs(from4 + j) : from4[j];
            }
#pragma unroll
            for (int u = 0; u < LOADS4; u++) {
                const int j = base0 + u * THREADS + (int)threadIdx.x;
                if (j < n4) {
                    const int i = rs.begin + 4 * j;
                    take_first_max(bv, bi, v[u].x, i);
                    take_first_max(bv, bi, v[u].y, i + 1);
                    take_first_max(bv, bi, v[u].z, i + 2);
                    take_first_max(bv, bi, v[u].w, i + 3);
                    if (IN_SHARED) reinterpret_cast<float4*>(rs.p)[j] = v[u];
                }
            }
        }
        for (int i = 4 * n4 + (int)threadIdx.x; i < rs.n; i += THREADS) {
            const float x = from[i];
            if (IN_SHARED) rs.p[i] = x;
            take_first_max(bv, bi, x, rs.begin + i);
        }
    } else {
        scan(from, IN_SHARED);
    }
    if (window > 0 && !(repeat == 1.0f && freq == 0.0f && presence == 0.0f)) {       // sampler.c:81-84
        const int n = min(ring.n[slot], min(window, 256));
        const int* r = ring.tokens + (size_t)slot * ring.stride;
        if ((int)threadIdx.x < n) sh.ring[threadIdx.x] = r[threadIdx.x];
        __syncthreads();                                    // the ring is there, and so is the row
        if ((int)threadIdx.x < n) {
            const int tok = sh.ring[threadIdx.x], at = tok - rs.begin;
            int count = 0, before = 0;
            for (int k = 0; k < n; k++) {
                count += sh.ring[k] == tok;
                before += k < (int)threadIdx.x && sh.ring[k] == tok;
            }
            if (before == 0 && tok >= 0 && at >= 0 && at < rs.n) {       // one thread a token, in the CTA that holds it
                float l = rs.p[at];
                for (int k = 0; k < count; k++) l = penalise(l, repeat, freq, presence, count);
                rs.p[at] = l;
                row[tok] = l;
            }
        }
        __syncthreads();
        bv = -INFINITY;
        bi = 0x7fffffff;
        scan(rs.p, false);
    }
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) {
        const float v2 = __shfl_xor_sync(0xffffffffu, bv, o);
        const int i2 = __shfl_xor_sync(0xffffffffu, bi, o);
        take_first_max(bv, bi, v2, i2);
    }
    if (NC > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    const int group = rs.rank * (THREADS / LANES) + (int)threadIdx.x / LANES;
    if (lane % LANES < NC) {                                // a lane a CTA
        *rs.at(&sh.group_v[group], lane % LANES) = bv;
        *rs.at(&sh.group_i[group], lane % LANES) = bi;
    }
    rs.sync();                                              // the maxima of all groups are in every CTA
    // ---- the row's first maximum (warp 0), the k-th largest of the groups' maxima (all warps)
    const bool small_k = sp.temp > 0.f && sp.top_k > 0 && sp.top_k <= MAX_CAND && sp.top_k < V;
    const bool bounded = small_k && sp.top_k <= GROUPS / 2;
    if (warp == 0) {
        float v = -INFINITY;
        int at = 0x7fffffff;
        for (int k = lane; k < GROUPS; k += 32) take_first_max(v, at, sh.group_v[k], sh.group_i[k]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float v2 = __shfl_xor_sync(0xffffffffu, v, o);
            const int i2 = __shfl_xor_sync(0xffffffffu, at, o);
            take_first_max(v, at, v2, i2);
        }
        if (lane == 0) {
            sh.mx = v;
            sh.best = at == 0x7fffffff ? 0 : at;
        }
    }
    if (bounded) {
        constexpr int TPG = THREADS / GROUPS;               // threads a group's value
        const int g = threadIdx.x / TPG, part = threadIdx.x % TPG;
        const float own = sh.group_v[g];
        int place = 0;
#pragma unroll 4
        for (int k = part; k < GROUPS / 4; k += TPG) {
            const float4 v = reinterpret_cast<const float4*>(sh.group_v)[k];
            place += (v.x > own || (v.x == own && 4 * k < g)) + (v.y > own || (v.y == own && 4 * k + 1 < g))
                   + (v.z > own || (v.z == own && 4 * k + 2 < g)) + (v.w > own || (v.w == own && 4 * k + 3 < g));
        }
#pragma unroll
        for (int o = TPG / 2; o > 0; o >>= 1) place += __shfl_xor_sync(0xffffffffu, place, o);
        if (part == 0 && place == sp.top_k - 1) sh.bound = own;
    }
    __syncthreads();
    const float mx = sh.mx;
    const int best = sh.best;
    const bool leading = rs.rank == 0;
    if (sp.temp <= 0.f) {
        if (threadIdx.x == 0 && leading) {
            out[b] = best;
            if (window > 0) accept_token(ring, slot, window, best);
        }
        return;
    }
    // Everything whose exponential is at least `least` is listed. Probabilities are the exponentials times a rounded factor:
    // those equal to the k-th largest come from exponentials within 2^-22 of its own, and expf is within 2^-22 of being
    // monotonic; the margin is 2^-20. Below 1e-20 a product could be subnormal and merge more: the search by count then.
    const float bound_e = bounded ? expf((sh.bound - mx) / sp.temp) : 0.f;
    const bool listing = bounded && bound_e >= 1e-20f;
    const float least = bound_e * (1.0f - 9.5367431640625e-7f);
    // ---- p_i = expf((l_i - max) / temp) * (float)(1 / sum), the sum in double (sampler.c:132-143)
    double part = 0.0;
    for (int base0 = 0; base0 < rs.n; base0 += THREADS * LOADS) {
        float vals[LOADS];
#pragma unroll
        for (int u = 0; u < LOADS; u++) {
            const int i = base0 + u * THREADS + (int)threadIdx.x;
            vals[u] = i < rs.n ? rs.p[i] : 0.f;
        }
#pragma unroll
        for (int u = 0; u < LOADS; u++) {
            const int i = base0 + u * THREADS + (int)threadIdx.x;
            if (i < rs.n) {
                const float e = expf((vals[u] - mx) / sp.temp);
                rs.p[i] = e;
                part += (double)e;                          // in index order within a thread
                if (listing && e >= least) {
                    const unsigned int at = atomicAdd(&sh.n_mine, 1u);
                    if (at < (unsigned int)MAX_CAND)
                        sh.mine[at] = ((unsigned long long)__float_as_uint(e) << 32) | (0xffffffffu - (unsigned int)(rs.begin + i));
                }
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    if (lane == 0) sh.red_d[warp] = part;
    __syncthreads();
    const unsigned int n_mine = sh.n_mine;
    if (warp == 0) {
        double mine = lane < WARPS ? sh.red_d[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mine += __shfl_xor_sync(0xffffffffu, mine, o);
        if (lane < NC) {                                    // a lane a CTA
            *rs.at(&sh.part_d[rs.rank], lane) = mine;
            *rs.at(&sh.part_u[rs.rank], lane) = n_mine;
        }
    } else if (listing && threadIdx.x - 32 < min(n_mine, (unsigned int)MAX_CAND)) {
        *rs.at(&sh.list[rs.rank][threadIdx.x - 32], 0) = sh.mine[threadIdx.x - 32];
    }
    rs.sync();                                              // sums and counts are in every CTA, the lists in the leading one
    double sum = 0.0;
    unsigned int listed = 0;
    for (int r = 0; r < NC; r++) {                          // in the CTAs' order: the same value in each of them
        sum += sh.part_d[r];
        listed += min(sh.part_u[r], (unsigned int)MAX_CAND + 1u);
    }
    const float inv = (float)(1.0 / sum);
    const float p_best = expf((mx - mx) / sp.temp) * inv;
    const double u = splitmix_uniform(&state);
    int id = -1;
    if (small_k && listing && listed <= (unsigned int)MAX_CAND && inv > 0.f) {
        if (!leading) return;                               // (the leading CTA reads its own memory only from here on)
        if (threadIdx.x < listed) {
            int r = 0;
            unsigned int at = threadIdx.x;
            while (at >= sh.part_u[r]) at -= sh.part_u[r++];
            const unsigned long long k = sh.list[r][at];
            const float p = __uint_as_float((unsigned int)(k >> 32)) * inv;
            sh.key[threadIdx.x] = ((unsigned long long)__float_as_uint(p) << 32) | (unsigned int)k;
        }
        __syncthreads();
        id = draw_from_keys<NC>(sh, listed, sp, p_best, u);
    } else if (small_k) {
        // One pass over the probabilities (the stored exponentials times inv) finds the leading eleven bits of the k-th
        // largest, a second one, where those leave a long list, eleven more. Everything with those bits or larger ones holds the k
        // largest; when that is a short list it is gathered.
        Found lead = find_digit<NC, IN_SHARED>(rs, add_up<NC, IN_SHARED>(rs, FIRST_DIGIT, inv, sh), false, (unsigned int)sp.top_k, 0ull, 0u, 0ull, sh);
        unsigned int lead_bits = lead.digit;
        int lead_shift = FIRST_DIGIT.shift;
        if (lead.above + lead.count > (unsigned int)MAX_CAND) {                         // the same in every CTA of the row
            const Digit next{lead.digit << 21, 2047u << 21, 10, 2048};
            lead = find_digit<NC, IN_SHARED>(rs, add_up<NC, IN_SHARED>(rs, next, inv, sh), false, (unsigned int)sp.top_k, 0ull, lead.above, lead.mass, sh);
            lead_bits = lead_bits << 11 | lead.digit;
            lead_shift = next.shift;
        }
        const bool short_list = lead.above + lead.count <= (unsigned int)MAX_CAND;
        Prefix topk{0u, 0u, 0u, 0ull};
        int id_bound = -1;
        float gather_scale = inv;
        if (!short_list) {
            for (int i = threadIdx.x; i < rs.n; i += THREADS) rs.p[i] *= inv;
            __syncthreads();                                // this CTA's part holds probabilities
            topk = find_prefix<NC, IN_SHARED>(rs, add_up<NC, IN_SHARED>(rs, FIRST_DIGIT, 1.0f, sh), false, (unsigned int)sp.top_k, 0ull, sh);
            id_bound = nth_equal<NC, IN_SHARED>(rs, topk.value, topk.ties, sh);
            gather_scale = 1.0f;
        }
        unsigned int* cnt = rs.at(&sh.n_key, 0);
        unsigned long long* keys = rs.at(&sh.key[0], 0);
        for (int i = threadIdx.x; i < rs.n; i += THREADS) {
            const unsigned int bits = __float_as_uint(rs.p[i] * gather_scale);    // probabilities are not negative: bits order as values
            const bool take = short_list ? (bits >> lead_shift) >= lead_bits : (bits > topk.value || (bits == topk.value && rs.begin + i <= id_bound));
            if (take) {
                const unsigned int at = atomicAdd(cnt, 1u);
                if (at < (unsigned int)MAX_CAND) keys[at] = ((unsigned long long)bits << 32) | (0xffffffffu - (unsigned int)(rs.begin + i));
            }
        }
        rs.sync();                                          // the list is complete
        if (!leading) return;
        id = draw_from_keys<NC>(sh, min(sh.n_key, (unsigned int)MAX_CAND), sp, p_best, u);
    } else {
        unsigned long long mass_part = 0;                   // the mass of this thread's probabilities (integers: any order)
        unsigned int c = 0;
        const float floor_p = sp.min_p * p_best;
        for (int i = threadIdx.x; i < rs.n; i += THREADS) {
            const float pr = rs.p[i] * inv;
            rs.p[i] = pr;
            mass_part += mass_of(pr);
            c += pr >= floor_p;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            mass_part += __shfl_xor_sync(0xffffffffu, mass_part, o);
            c += __shfl_xor_sync(0xffffffffu, c, o);
        }
        if (lane == 0) {
            sh.warp_mass[warp] = mass_part;
            sh.scan_u[warp] = c;
        }
        __syncthreads();                                    // this CTA's part holds probabilities
        if (warp == 0) {
            unsigned long long m = lane < WARPS ? sh.warp_mass[lane] : 0ull;
            unsigned int n = lane < WARPS ? sh.scan_u[lane] : 0u;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                m += __shfl_xor_sync(0xffffffffu, m, o);
                n += __shfl_xor_sync(0xffffffffu, n, o);
            }
            if (lane < NC) {
                *rs.at(&sh.part_m[rs.rank], lane) = m;
                *rs.at(&sh.part_v[rs.rank], lane) = n;
            }
        }
        rs.sync();
        unsigned long long row_mass = 0;
        unsigned int n_floor = 0;
        for (int r = 0; r < NC; r++) {
            row_mass += sh.part_m[r];
            n_floor += sh.part_v[r];
        }
        // the kept prefix: top-k, then min-p, then top-p (sampler.c:146-175)
        unsigned int n = (unsigned int)V;
        if (sp.top_k > 0 && (unsigned int)sp.top_k < n) n = (unsigned int)sp.top_k;
        if (sp.min_p > 0.f) n = min(n, max(n_floor, 1u));
        // mass of the kept prefix, then the draw r = U * total and the walk (sampler.c:178-186); with nothing cut off it is
        // the row's mass, and a prefix that top-p ends is the one its search has found
        const Slice<NC> first = add_up<NC, IN_SHARED>(rs, FIRST_DIGIT, 1.0f, sh);       // (both searches begin with it)
        Prefix kept{0u, 0u, 0u, row_mass};
        bool found = false;
        if (sp.top_p < 1.0f) {
            const unsigned long long target = __double2ull_ru((double)sp.top_p * 1152921504606846976.0);
            const Prefix pp = find_prefix<NC, IN_SHARED>(rs, first, true, 0u, target, sh);
            const unsigned int np = pp.above + pp.ties;
            if (np <= n) {
                n = np;
                kept = pp;
                found = true;
            }
        }
        if (n < 1) n = 1;
        if (!found && n < (unsigned int)V) kept = find_prefix<NC, IN_SHARED>(rs, first, false, n, 0ull, sh);
        const double r = u * (double)kept.mass;
        unsigned long long target = __double2ull_ru(r);
        if (target > kept.mass) target = kept.mass;
        const Prefix hit = find_prefix<NC, IN_SHARED>(rs, first, true, 0u, target, sh);
        const unsigned int rank = hit.above + hit.ties;     // 1-based place in the sorted order
        const bool within = rank <= n;                      // (beyond only through rounding: the last kept one)
        id = nth_equal<NC, IN_SHARED>(rs, within ? hit.value : kept.value, within ? hit.ties : kept.ties, sh);
        if (!leading) return;
    }
    if (threadIdx.x == 0) {
        const int token = id >= 0 ? id : best;
        out[b] = token;
        rng[slot] = state;
        if (window > 0) accept_token(ring, slot, window, token);
    }
}

__global__ void __launch_bounds__(ARGMAX_THREADS)
argmax_kernel(const float* __restrict__ logits, int V, int ld, int* __restrict__ out) {
    __shared__ ArgmaxShared sh;
    griddep_launch();
    griddep_wait();
    float mx;
    const int best = block_argmax(logits + (size_t)blockIdx.x * ld, V, sh, &mx);
    if (threadIdx.x == 0) out[blockIdx.x] = best;
}

}  // namespace

MYNAH_API int mynah_argmax(const float* logits, int B, int V, int ld, int* out, cudaStream_t stream) {
    if (B == 0) return 0;
    MYNAH_REQUIRE(B > 0 && V > 0 && ld >= V, "argmax: bad sizes B=%d V=%d ld=%d", B, V, ld);
    mynah_launch(argmax_kernel, dim3(B), dim3(ARGMAX_THREADS), 0, stream, logits, V, ld, out);
    return mynah_check_launch("argmax");
}

// One draw a row of logits [B, ld], in one launch: penalties from the ring, the draw, the token into the ring. The logits
// may be overwritten (by penalised values, and by what is left of the search where a row does not fit shared memory). params
// (device): temp, top_p, min_p, top_k, repeat, freq, presence, window as floats; they are read on the device so that a
// captured step serves every setting. rng: one 64-bit generator state per slot; slots [B] maps rows to slots (null: row b is
// slot b; a negative slot marks a padding row). out [B] receives the token ids. ring, ring_n, ring_head: the slots' rings,
// `stride` <= 256 entries a row, or null: then no penalty is taken and nothing is accepted.
MYNAH_API int mynah_sample(float* logits, int B, int V, int ld, const float* params,
                           unsigned long long* rng, const int* slots, int* out,
                           int* ring, int* ring_n, int* ring_head, int stride, cudaStream_t stream) {
    if (B == 0) return 0;
    MYNAH_REQUIRE(B > 0 && V > 0 && ld >= V, "sample: bad sizes B=%d V=%d ld=%d", B, V, ld);
    MYNAH_REQUIRE(params != nullptr && rng != nullptr, "sample: parameters and generator states are required");
    MYNAH_REQUIRE(B <= 65535, "sample: too many rows");
    MYNAH_REQUIRE((ring == nullptr) == (ring_n == nullptr) && (ring == nullptr) == (ring_head == nullptr)
                      && (ring == nullptr || (stride > 0 && stride <= 256)), "sample: bad ring");
    const Ring rings{ring, ring_n, ring_head, stride};
    // A cluster a row from this vocabulary size on (see the kernel), whatever the batch: a row's draw does not depend on its
    // company. A row stays where it is when its CTAs' shared memory cannot hold it, or when it would leave an SM to one CTA while the step has
    // more CTAs than SMs (262,144 logits, us a draw from shared memory / where they are: 8 rows top-k 20 23 / 25, top-p 116 / 132; 32 rows
    // 62 / 40 and 338 / 203; 256 rows greedy 204 / 155, top-k 20 412 / 315, top-p 2,076 / 1,560).
    const bool cluster = V >= ROW_CTAS * 4096;
    const size_t own = cluster ? sizeof(Shared<ROW_CTAS>) : sizeof(Shared<1>);
    const size_t part = sizeof(float) * (size_t)(cluster ? ((V + ROW_CTAS - 1) / ROW_CTAS + 3) & ~3 : V);
    const bool in_shared = own + part <= 113 * 1024 || (own + part <= 227 * 1024 && B * (cluster ? ROW_CTAS : 1) <= mynah_sm_count());
    const size_t smem = own + (in_shared ? part : 0);
    auto kernel = cluster ? (in_shared ? sample_kernel<ROW_CTAS, true> : sample_kernel<ROW_CTAS, false>) : (in_shared ? sample_kernel<1, true> : sample_kernel<1, false>);
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return mynah_fail("sample: %s", cudaGetErrorString(e));
    if (!cluster) {
        mynah_launch(kernel, dim3(B), dim3(THREADS), smem, stream, logits, V, ld, params, rng, slots, out, rings);
        return mynah_check_launch("sample");
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)B * ROW_CTAS);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ROW_CTAS;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    e = cudaLaunchKernelEx(&cfg, kernel, logits, V, ld, params, rng, slots, out, rings);
    if (e != cudaSuccess) return mynah_fail("sample: %s", cudaGetErrorString(e));
    return mynah_check_launch("sample");
}

namespace {
// After a sampled decode step: the sampled token becomes the sequence's next
// input, one position further on.
__global__ void decode_advance_kernel(int* __restrict__ tokens, const int* __restrict__ sampled,
                                      int* __restrict__ tok_pos, int* __restrict__ kv_len,
                                      const int* __restrict__ slots, int B) {
    griddep_launch();
    griddep_wait();
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= B || slots[b] < 0) return;
    tokens[b] = sampled[b];
    tok_pos[b] += 1;
    kv_len[b] += 1;
}
}  // namespace

MYNAH_API int mynah_decode_advance(int* tokens, const int* sampled, int* tok_pos, int* kv_len, const int* slots,
                                   int B, cudaStream_t stream) {
    if (B == 0) return 0;
    mynah_launch(decode_advance_kernel, dim3(ceil_div(B, 64)), dim3(64), 0, stream, tokens, sampled, tok_pos, kv_len, slots, B);
    return mynah_check_launch("decode_advance");
}
