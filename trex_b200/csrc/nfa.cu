// Family (c): Boolean NFA with up to 64 states, bit-parallel on uint64 masks.
//
// Semantics (reference src/nfa_matrices.py:133-157 simulate_nfa and
// cuda/nfa_tc_evolution.cu:683-745 nfa_bitpar_v4_kernel): the state is the
// set of active NFA states; one symbol c maps it to
//     s' = OR over active sources j of col[c][j]      (= min(T[c] s, 1))
// where col[c][j] is the destination mask of source j (epsilon closure
// folded in). A byte >= sigma is either skipped (the C engine) or rejects
// the string (Python simulate_nfa). Outputs: the final mask and accept flag
// (s & accept_mask != 0; a rejected string has the empty mask).
//
// Design: "four Russians" tables. For every symbol c the T source bits are
// cut into G groups of nearly equal width (T mod G of them one bit wider) and
// tbl[c][g][v] holds the OR of the columns of the set bits of v, so a step is G
// table lookups ORed together. Symbol index sigma is an extra table: the
// identity (skip) or all zeros (reject), so bytes >= sigma need no branch.
// T = 64, or 32 / 16 for automata of that many states, whose masks and entries
// are 32-bit words. G is the smallest number of groups (of at most 8 bits) whose
// tables fit in shared memory: a step is bound by the shared-memory wavefronts
// of its lookups (about five a warp lookup of random 64-bit entries), so each
// group less is that share of the time. 64 states, 20 symbols: 9 groups (one of
// 8 bits, eight of 7) take the memory that ten 7-bit groups took: 262144 strings of
// 4096 bytes 5.83 -> 5.37 ms (184 -> 200 Gchar/s). Larger alphabets than fit at 16
// groups read 8-bit tables from global memory through L1.
// One persistent CTA per SM, a thread per string; threads take strings from
// an atomic counter and walk them in 16-byte windows.
//
// Long strings of small batches are cut into units walked side by side (a
// string of 64 KiB alone would keep one thread busy for milliseconds while the
// SMs idle). Unit j > 0 starts kNfaWarm bytes early from the set of all states:
// the set shrinks towards the true one, and for automata whose sets do not
// depend on the distant past it is the true one at the cut (the unit's guess).
// Each unit's thread, at its end, compares its set with the next unit's guess
// and reports; the last reporter of a string whose guesses all hold writes the
// last unit's set. Where a guess fails, the string is walked again from there
// by one thread (for unit 0, whose set is always the true one, by its own
// thread at once), which jumps to a unit's end when it meets the unit's guess or its
// checkpoint. Nobody waits for anybody. Exact for every NFA. 2048 log-normal
// strings (median 2 KiB, longest 64 KiB), 64 states, 20 symbols: 7.7 -> 0.17 ms. An automaton whose
// guesses never hold (permutations) pays for the looks at every unit: one string of 64 KiB, 10 / 20 /
// 60 symbols, 3.39 / 3.61 / 4.88 ms, uncut 3.09 / 3.30 / 4.66; 2000 strings of 4 KiB 0.34 ms, uncut 2.7.
#include <algorithm>
#include <cstring>
#include <new>
#include <vector>

#include "trex_internal.cuh"

namespace trex {

constexpr int kNfaThreads = 1024;
constexpr size_t kNfaSmemBudget = 220 * 1024;

// Group g of T bits in G groups: width, first bit, first table entry.
__host__ __device__ constexpr int nfa_width(int T, int G, int g) { return T / G + (g < T % G ? 1 : 0); }
__host__ __device__ constexpr int nfa_shift(int T, int G, int g) { return g * (T / G) + (g < T % G ? g : T % G); }
__host__ __device__ constexpr int nfa_first(int T, int G, int g) {
    int e = 0;
    for (int k = 0; k < g; ++k) e += 1 << nfa_width(T, G, k);
    return e;
}
__host__ __device__ constexpr int nfa_table_entries(int T, int G) { return nfa_first(T, G, G); }
// Entries of symbol c are stored at v ^ swizzle(c): with dense states many
// lanes look up the same v for different symbols, and every table starts on
// the same bank; the XOR sends them to different banks (pairs of 64-bit entries).
template <int T>
__host__ __device__ constexpr uint32_t nfa_swizzle(uint32_t c) {
    return T > 32 ? (c ^ (c >> 4)) & 15u : (c ^ (c >> 5)) & 31u;
}
// Masks and table entries of T states.
template <int T> struct NfaWord { using type = uint64_t; };
template <> struct NfaWord<32> { using type = uint32_t; };
template <> struct NfaWord<16> { using type = uint32_t; };

struct NfaParams {
    const uint8_t *data;
    int64_t total_bytes;
    const int64_t *offsets;
    int64_t n;
    const void *tables;       // (sigma + 1) x entries of the layout
    int sigma;
    uint64_t start_mask, accept_mask;
    uint64_t *final_mask;
    uint8_t *accept;
    int32_t *accept_i32;
    unsigned long long *head;
    uint32_t *err;
    struct NfaUnit *units;    // units of cut strings (null: no string is cut)
    const uint32_t *n_units;
    int64_t seg;              // bytes of a unit
    uint32_t max_units;
    uint64_t all_states;
};

constexpr int kNfaWarm = 64;            // warm-up bytes of a unit
constexpr int kNfaCheck = 128;          // checkpoint, bytes into a unit
constexpr int64_t kNfaMinSeg = 512;
constexpr int kNfaUnitsPerSm = 64;
enum : uint32_t { kUnitGuess = 1u, kUnitDone = 2u, kUnitBroken = 4u };   // Broken: the next guess fails
struct NfaUnit {
    uint64_t guess, exit, check;   // sets at the cut, at the end, at the checkpoint
    uint32_t str, word;            // string, low half; its next 8 bits << 24 | index << 8 | flags
    __device__ int64_t string() const { return (int64_t)(((uint64_t)(word >> 24) << 32) | str); }
    __device__ uint32_t index() const { return (word >> 8) & 0xFFFFu; }
    // unit 0 has no guess: the string's reports (low half) and failed guesses
    __device__ uint32_t *reports() { return reinterpret_cast<uint32_t *>(&guess); }
    __device__ uint32_t *broken() { return reinterpret_cast<uint32_t *>(&guess) + 1; }
};

// Units of string [a, b): the cuts lie seg bytes apart on 16-byte aligned addresses.
__device__ __forceinline__ int64_t nfa_cut0(const uint8_t *d, int64_t a) {
    return a + (int64_t)((16u - ((uint32_t)(uintptr_t)(d + a) & 15u)) & 15u);
}
__device__ __forceinline__ uint32_t nfa_units_of(const uint8_t *d, int64_t a, int64_t b, int64_t seg) {
    const int64_t c = nfa_cut0(d, a);
    return b - c <= seg ? 1u : (uint32_t)min((b - c - 1) / seg + 1, (int64_t)(1 << 24));
}

// Lists the units of every string cut into several (a warp writes a string's records together).
__global__ void nfa_units_kernel(NfaParams P, uint32_t *n_units) {
    const uint32_t FULL = 0xffffffffu, lane = threadIdx.x & 31u;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x / 32);
    for (int64_t base = ((int64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5)) * 32; base < P.n;
         base += warps * 32) {
        uint32_t k = 1u;
        if (base + lane < P.n) {
            const int64_t a = P.offsets[base + lane], b = P.offsets[base + lane + 1];
            if (!(a < 0 || b < a || b > P.total_bytes)) k = nfa_units_of(P.data, a, b, P.seg);
        }
        uint32_t cut = __ballot_sync(FULL, k > 1u);
        while (cut) {
            const int l = __ffs(cut) - 1;
            cut &= cut - 1u;
            const uint32_t ks = __shfl_sync(FULL, k, l);
            uint32_t at = 0u;
            // (saturating: more units than records means no string is cut)
            if (lane == 0) {
                at = *(volatile uint32_t *)n_units;
                if (at <= P.max_units) at = atomicAdd(n_units, min(ks, P.max_units + 1u));
            }
            at = __shfl_sync(FULL, at, 0);
            if (at > P.max_units || at + ks > P.max_units) continue;
            for (uint32_t j = lane; j < ks; j += 32u)
                P.units[at + j] = NfaUnit{0, 0, 0, (uint32_t)(base + l), (uint32_t)((uint64_t)(base + l) >> 32) << 24 | j << 8};
        }
    }
}

template <int T, int G>
__device__ __forceinline__ typename NfaWord<T>::type nfa_step(const typename NfaWord<T>::type *tbl,
                                                              typename NfaWord<T>::type s, uint32_t byte,
                                                              int sigma) {
    const uint32_t sym = min(byte, (uint32_t)sigma);
    const typename NfaWord<T>::type *t = tbl + (size_t)sym * nfa_table_entries(T, G);
    const uint32_t x = nfa_swizzle<T>(sym);
    typename NfaWord<T>::type acc = 0;
#pragma unroll
    for (int g = 0; g < G; ++g) {
        const uint32_t m = (1u << nfa_width(T, G, g)) - 1u;
        acc |= t[nfa_first(T, G, g) + (((uint32_t)(s >> nfa_shift(T, G, g)) ^ x) & m)];
    }
    return acc;
}

// Walks bytes [p, b) from set s in 16-byte windows.
template <int T, int G>
__device__ __forceinline__ typename NfaWord<T>::type nfa_walk(const typename NfaWord<T>::type *tbl, int sigma,
                                                              const uint8_t *d, int64_t p, int64_t b,
                                                              typename NfaWord<T>::type s) {
    while (p < b && (((uintptr_t)(d + p)) & 15u)) s = nfa_step<T, G>(tbl, s, __ldg(d + p++), sigma);
    if (b - p >= 16) {
        uint4 v = ld_stream16(d + p);
        while (true) {
            const bool more = b - p >= 32;
            uint4 nv = make_uint4(0, 0, 0, 0);
            if (more) nv = ld_stream16(d + p + 16);
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int k2 = 0; k2 < 16; ++k2) s = nfa_step<T, G>(tbl, s, (w[k2 >> 2] >> (8 * (k2 & 3))) & 0xffu, sigma);
            p += 16;
            if (!more) break;
            v = nv;
        }
    }
    while (p < b) s = nfa_step<T, G>(tbl, s, __ldg(d + p++), sigma);
    return s;
}

__device__ __forceinline__ void nfa_write(uint64_t *final_mask, uint8_t *accept, int32_t *accept_i32, int64_t i,
                                          uint64_t s, uint64_t accept_mask) {
    const bool ok = (s & accept_mask) != 0;
    if (final_mask) final_mask[i] = s;
    if (accept) accept[i] = ok ? 1 : 0;
    if (accept_i32) accept_i32[i] = ok ? 1 : 0;
}

// Threads take strings first .. first + n - 1 from the counter *head; results go to index i of
// the output arrays.
template <int T, int G>
__device__ __forceinline__ void nfa_walk_queue(const typename NfaWord<T>::type *tbl, int sigma, uint64_t start_mask,
                                               uint64_t accept_mask, const uint8_t *d, int64_t total_bytes,
                                               const int64_t *offsets, int64_t first, int64_t n,
                                               unsigned long long *head, uint32_t *err, uint64_t *final_mask,
                                               uint8_t *accept, int32_t *accept_i32) {
    using W = typename NfaWord<T>::type;
    while (true) {
        const unsigned long long k = atomicAdd(head, 1ull);
        if (k >= (unsigned long long)n) break;
        const int64_t i = first + (int64_t)k;
        const int64_t a = offsets[i], b = offsets[i + 1];
        if (a < 0 || b < a || b > total_bytes) {
            atomicOr(err, 1u);
            continue;
        }
        const W s = nfa_walk<T, G>(tbl, sigma, d, a, b, (W)start_mask);
        nfa_write(final_mask, accept, accept_i32, i, s, accept_mask);
    }
}

// The same with cut strings: the units first, then the strings that are not cut.
template <int T, int G>
__device__ __forceinline__ void nfa_walk_units(const NfaParams &P, const typename NfaWord<T>::type *tbl) {
    using W = typename NfaWord<T>::type;
    uint32_t U = *P.n_units;
    U = U > P.max_units ? 0u : U;
    // as many warps a CTA as there is work for, so that few units spread over the SMs
    const int64_t lanes = (int64_t)gridDim.x * 32;
    if ((int64_t)(threadIdx.x >> 5) >= ((int64_t)U + P.n + lanes - 1) / lanes) return;
    while (true) {
        const unsigned long long q = atomicAdd(P.head, 1ull);
        if (q >= (unsigned long long)P.n + U) break;
        NfaUnit *u = q < U ? P.units + q : nullptr;   // the unit walked
        const int64_t i = u ? u->string() : (int64_t)q - U;
        const int64_t a = P.offsets[i], b = P.offsets[i + 1];
        if (a < 0 || b < a || b > P.total_bytes) {
            if (!u) atomicOr(P.err, 1u);
            continue;
        }
        const uint32_t k = U ? nfa_units_of(P.data, a, b, P.seg) : 1u;
        if (!u && k > 1u) continue;
        const int64_t c0 = nfa_cut0(P.data, a);
        uint32_t j = u ? u->index() : 0u;
        NfaUnit *const u0 = u - j;
        auto cut = [&](uint32_t x) { return x == 0u ? a : x >= k ? b : c0 + (int64_t)x * P.seg; };
        // stage 0: the warm-up; 1: to the checkpoint; 2: to the unit's end
        bool truth = false;   // this thread walks the string again with its true set
        int stage = j ? 0 : 1;
        int64_t p = cut(j) - (j ? kNfaWarm : 0);
        W s = j ? (W)P.all_states : (W)P.start_mask;
        for (;;) {
            const int64_t b1 = cut(j + 1u);
            const int64_t stop = !u || stage == 2 ? b1 : stage == 0 ? cut(j) : min(b1, cut(j) + kNfaCheck);
            s = nfa_walk<T, G>(tbl, P.sigma, P.data, p, stop, s);
            p = stop;
            if (!u) break;
            volatile NfaUnit *r = u;
            if (stage == 0) {
                r->guess = s;
                __threadfence();
                atomicOr(&u->word, kUnitGuess);
            } else if (stage == 1 && !truth) {
                r->check = s;
            } else if (stage == 1 && p < b1 && (r->word & kUnitDone)) {
                // walking unit j again: where the sets are equal at the checkpoint, its end is known
                __threadfence();
                if (r->check == (uint64_t)s) {
                    s = (W)r->exit;
                    p = b1;
                    stage = 2;
                }
            }
            if (stage < 2) {
                ++stage;
                continue;
            }
            // ---- the end of unit j
            if (!truth) {
                r->exit = s;
                __threadfence();
                uint32_t flags = kUnitDone;
                if (j + 1u < k) {
                    volatile NfaUnit *x = u + 1;
                    const bool known = (x->word & kUnitGuess) != 0u;
                    __threadfence();
                    if (!known || x->guess != (uint64_t)s) flags |= kUnitBroken;
                }
                atomicOr(&u->word, flags);
                if ((flags & kUnitBroken) && j == 0u) {
                    truth = true;   // this set is the true one: walk on
                } else {
                    if (flags & kUnitBroken) atomicAdd(u0->broken(), 1u);
                    __threadfence();
                    if (atomicAdd(u0->reports(), 1u) + 1u != k) break;
                    // the last reporter of the string: its units are all done
                    __threadfence();
                    if (*(volatile uint32_t *)u0->broken() == 0u) {
                        s = (W)((volatile NfaUnit *)(u0 + (k - 1u)))->exit;
                        nfa_write(P.final_mask, P.accept, P.accept_i32, i, s, P.accept_mask);
                        break;
                    }
                    for (j = 0u; !(((volatile NfaUnit *)(u0 + j))->word & kUnitBroken); ++j) {}
                    s = (W)((volatile NfaUnit *)(u0 + j))->exit;   // true: every guess before held
                    truth = true;
                }
            }
            // the true set at the end of unit j: past the units whose guess it is
            while (++j < k && s != 0) {   // (the empty set stays empty)
                r = u0 + j;
                if ((r->word & (kUnitGuess | kUnitDone)) != (kUnitGuess | kUnitDone)) break;
                __threadfence();
                if (r->guess != (uint64_t)s) break;
                s = (W)r->exit;
            }
            if (j >= k || s == 0) {
                nfa_write(P.final_mask, P.accept, P.accept_i32, i, s, P.accept_mask);
                break;
            }
            u = u0 + j;
            stage = 1;
            p = cut(j);
        }
        if (!u) nfa_write(P.final_mask, P.accept, P.accept_i32, i, s, P.accept_mask);
    }
}

// Copies an automaton's tables into shared memory (16 bytes at a time; the device tables are
// padded to that).
extern __shared__ __align__(16) uint8_t s_nfa_tbl[];
template <int T, int G>
__device__ __forceinline__ const typename NfaWord<T>::type *nfa_tables_in(const void *tables, int sigma) {
    using W = typename NfaWord<T>::type;
    const int n16 = (int)(((size_t)(sigma + 1) * nfa_table_entries(T, G) * sizeof(W) + 15) / 16);
    const uint4 *src = static_cast<const uint4 *>(tables);
    uint4 *dst = reinterpret_cast<uint4 *>(s_nfa_tbl);
    // asynchronous copies: all of a thread's pieces in flight at once
    for (int i = threadIdx.x; i < n16; i += blockDim.x)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                     :: "r"((uint32_t)__cvta_generic_to_shared(dst + i)), "l"(src + i) : "memory");
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    return reinterpret_cast<const W *>(s_nfa_tbl);
}

template <int T, int G, bool SMEM>
__global__ void __launch_bounds__(kNfaThreads, 1) nfa_bitpar_kernel(NfaParams P) {
    const typename NfaWord<T>::type *tbl = static_cast<const typename NfaWord<T>::type *>(P.tables);
    if constexpr (SMEM) tbl = nfa_tables_in<T, G>(P.tables, P.sigma);
    nfa_walk_units<T, G>(P, tbl);
}

// Many automata in one launch (a serving batch: strings grouped by automaton). Group g
// owns CTAs cta_first[g] .. cta_first[g+1] - 1 and strings first[g] .. first[g] +
// count[g] - 1; each CTA loads its group's tables and its threads take the group's
// strings, so the groups run side by side instead of one launch after another.
constexpr int kNfaMultiMax = 64;
struct NfaMultiParams {
    const uint8_t *data;
    int64_t total_bytes;
    const int64_t *offsets;
    uint64_t *final_mask;
    uint8_t *accept;
    int32_t *accept_i32;
    unsigned long long *heads;   // one counter a group
    uint32_t *err;
    int n_groups;
    const void *tables[kNfaMultiMax];
    uint64_t start_mask[kNfaMultiMax], accept_mask[kNfaMultiMax];
    int64_t first[kNfaMultiMax], count[kNfaMultiMax];
    int32_t cta_first[kNfaMultiMax + 1];
    int32_t sigma[kNfaMultiMax];
};

template <int T, int G, bool SMEM>
__global__ void __launch_bounds__(kNfaThreads, 1) nfa_bitpar_multi_kernel(const __grid_constant__ NfaMultiParams P) {
    int g = 0;
    while (g + 1 < P.n_groups && (int)blockIdx.x >= P.cta_first[g + 1]) ++g;
    const int sigma = P.sigma[g];
    const typename NfaWord<T>::type *tbl = static_cast<const typename NfaWord<T>::type *>(P.tables[g]);
    if constexpr (SMEM) tbl = nfa_tables_in<T, G>(P.tables[g], sigma);
    nfa_walk_queue<T, G>(tbl, sigma, P.start_mask[g], P.accept_mask[g], P.data, P.total_bytes, P.offsets,
                      P.first[g], P.count[g], P.heads + g, P.err, P.final_mask, P.accept,
                      P.accept_i32);
}

// The table layouts, fewest lookups a byte first for each T.
struct NfaLayout {
    int T, G;
    bool smem;
    void (*run)(NfaParams);
    void (*run_multi)(NfaMultiParams);
};
#define TREX_NFA_LAYOUT(T, G, SMEM) \
    NfaLayout{T, G, SMEM, nfa_bitpar_kernel<T, G, SMEM>, nfa_bitpar_multi_kernel<T, G, SMEM>}
static const NfaLayout kNfaLayouts[] = {
    TREX_NFA_LAYOUT(16, 2, true),  TREX_NFA_LAYOUT(32, 4, true),  TREX_NFA_LAYOUT(32, 5, true),
    TREX_NFA_LAYOUT(32, 6, true),  TREX_NFA_LAYOUT(32, 7, true),
    TREX_NFA_LAYOUT(64, 8, true),  TREX_NFA_LAYOUT(64, 9, true),  TREX_NFA_LAYOUT(64, 10, true),
    TREX_NFA_LAYOUT(64, 11, true), TREX_NFA_LAYOUT(64, 12, true), TREX_NFA_LAYOUT(64, 13, true),
    TREX_NFA_LAYOUT(64, 16, true), TREX_NFA_LAYOUT(64, 8, false)};
#undef TREX_NFA_LAYOUT
static size_t nfa_table_bytes(const NfaLayout &L, int sigma) {
    return ((size_t)(sigma + 1) * nfa_table_entries(L.T, L.G) * (L.T > 32 ? 8 : 4) + 15) & ~size_t(15);
}

}  // namespace trex

struct trex_nfa {
    int n_states = 0, sigma = 0;
    const trex::NfaLayout *lay = nullptr;   // table layout and its kernels
    uint64_t start_mask = 0, accept_mask = 0;
    uint8_t *d_tables = nullptr;   // one allocation: tables, d_misc, d_units
    size_t table_bytes = 0;   // a multiple of 16
    void *d_misc = nullptr;   // head counter, error word, number of units
    trex::NfaUnit *d_units = nullptr;
    uint32_t max_units = 0;   // a cut string has over seg bytes, so at most 2 total / seg units
    int n_sms = 0;
    std::vector<uint64_t> cols;   // host copy: sigma x 64 destination masks
    int unknown_rejects = 0;
};

namespace trex {

// The first layout that holds the states and whose tables fit in shared memory (the last one
// stays in global memory).
static const NfaLayout *nfa_choose_layout(int n_states, int sigma) {
    const NfaLayout *l = kNfaLayouts;
    while (l->T < n_states || (l->smem && nfa_table_bytes(*l, sigma) > kNfaSmemBudget)) ++l;
    return l;
}

// The tables of a layout, in its entry type.
template <int T>
static void nfa_build_tables(const std::vector<uint64_t> &cols, int sigma, int G, int unknown_rejects, uint8_t *out) {
    using W = typename NfaWord<T>::type;
    const int E = nfa_table_entries(T, G);
    W *t = reinterpret_cast<W *>(out);
    for (int c = 0; c <= sigma; ++c) {
        for (int g = 0; g < G; ++g) {
            const int width = nfa_width(T, G, g), first = nfa_first(T, G, g), src0 = nfa_shift(T, G, g);
            const int x = (int)(nfa_swizzle<T>((uint32_t)c) & ((1u << width) - 1u));
            for (int v = 0; v < (1 << width); ++v) {
                uint64_t acc = 0;
                for (int bit = 0; bit < width; ++bit) {
                    if (!((v >> bit) & 1)) continue;
                    if (c < sigma) acc |= cols[(size_t)c * 64 + src0 + bit];
                    else if (!unknown_rejects) acc |= 1ull << (src0 + bit);   // identity: skip the byte
                }
                t[(size_t)c * E + first + (v ^ x)] = (W)acc;
            }
        }
    }
}

int nfa_run(trex_nfa *nfa, const uint8_t *data, const int64_t *offsets, int64_t n,
            int64_t total_bytes, uint64_t *final_mask, uint8_t *accept, int32_t *accept_i32,
            cudaStream_t stream, uint32_t **err_out) {
    if (!nfa) return TREX_ERR_NOT_INIT;
    if (n < 0 || total_bytes < 0 || (n > 0 && !offsets) || (total_bytes > 0 && !data))
        return TREX_ERR_ARG;
    if (n == 0) return TREX_OK;
    unsigned long long *head = static_cast<unsigned long long *>(nfa->d_misc);
    uint32_t *err = reinterpret_cast<uint32_t *>(head + 1);
    TREX_CUDA(cudaMemsetAsync(nfa->d_misc, 0, 16, stream));
    NfaParams P;
    P.data = data;
    P.total_bytes = total_bytes;
    P.offsets = offsets;
    P.n = n;
    P.tables = nfa->d_tables;
    P.sigma = nfa->sigma;
    P.start_mask = nfa->start_mask;
    P.accept_mask = nfa->accept_mask;
    P.final_mask = final_mask;
    P.accept = accept;
    P.accept_i32 = accept_i32;
    P.head = head;
    P.err = err;
    // Units: two warps of lookups keep an SM's shared memory busy, so a string is cut only where
    // it holds more than 1/64 of an SM's share of the batch (262144 x 4096 bytes: no string is
    // cut, and only the listing kernel is added, 3 us); at least kNfaMinSeg bytes, so that the
    // warm-up is at most an eighth of a unit.
    P.units = nfa->d_units;
    P.n_units = err + 1;
    P.max_units = nfa->max_units;
    P.seg = std::max(kNfaMinSeg, (total_bytes / ((int64_t)nfa->n_sms * kNfaUnitsPerSm) + 15) & ~(int64_t)15);
    P.all_states = nfa->n_states == 64 ? ~0ull : (1ull << nfa->n_states) - 1;
    profile_kernel_begin(stream);   // (the listing kernel is part of the run)
    if (total_bytes > P.seg) {
        const int ugrid = (int)std::min<int64_t>((n + 255) / 256, (int64_t)nfa->n_sms);
        nfa_units_kernel<<<ugrid, 256, 0, stream>>>(P, err + 1);
        TREX_CHECK_LAUNCH();
    }
    const size_t smem = nfa->lay->smem ? nfa->table_bytes : 0;
    // a thread a string: a few strings need one CTA, so that batches of several
    // automata launched on separate streams run side by side
    const int grid = (int)std::max<int64_t>(
        1, std::min<int64_t>(nfa->n_sms, std::max((n + 31) / 32, total_bytes / (32 * P.seg))));
    nfa->lay->run<<<grid, kNfaThreads, smem, stream>>>(P);
    TREX_CHECK_LAUNCH();
    profile_kernel_end(stream);
    if (err_out) *err_out = err;
    return TREX_OK;
}

int nfa_run_multi(trex_nfa *const *nfas, int n_groups, const int64_t *group_first, const uint8_t *data,
                  const int64_t *offsets, int64_t total_bytes, uint64_t *final_mask, uint8_t *accept,
                  int32_t *accept_i32, void *scratch, cudaStream_t st) {
    if (n_groups < 1 || n_groups > kNfaMultiMax || !nfas || !group_first || !scratch) return TREX_ERR_ARG;
    if (group_first[0] != 0) return TREX_ERR_ARG;
    for (int g = 0; g < n_groups; ++g)
        if (!nfas[g] || group_first[g + 1] < group_first[g]) return TREX_ERR_ARG;
    const int64_t n = group_first[n_groups];
    if (total_bytes < 0 || (n > 0 && !offsets) || (total_bytes > 0 && !data)) return TREX_ERR_ARG;
    TREX_CUDA(cudaMemsetAsync(scratch, 0, 8 * (size_t)(n_groups + 1), st));
    if (n == 0) return TREX_OK;
    unsigned long long *heads = static_cast<unsigned long long *>(scratch);
    uint32_t *err = reinterpret_cast<uint32_t *>(heads + n_groups);
    // one launch per table layout (bits a lookup; tables in shared or global memory)
    bool taken[kNfaMultiMax] = {};
    int used_heads = 0;
    for (int g0 = 0; g0 < n_groups; ++g0) {
        if (taken[g0]) continue;
        const NfaLayout *lay = nfas[g0]->lay;
        NfaMultiParams P{};
        P.data = data;
        P.total_bytes = total_bytes;
        P.offsets = offsets;
        P.final_mask = final_mask;
        P.accept = accept;
        P.accept_i32 = accept_i32;
        P.heads = heads + used_heads;
        P.err = err;
        int k = 0, ctas = 0;
        size_t smem = 0;
        for (int g = g0; g < n_groups; ++g) {
            const trex_nfa *h = nfas[g];
            if (taken[g] || h->lay != lay) continue;
            taken[g] = true;
            const int64_t cnt = group_first[g + 1] - group_first[g];
            if (cnt == 0) continue;
            P.tables[k] = h->d_tables;
            P.start_mask[k] = h->start_mask;
            P.accept_mask[k] = h->accept_mask;
            P.sigma[k] = h->sigma;
            P.first[k] = group_first[g];
            P.count[k] = cnt;
            P.cta_first[k] = ctas;
            // a thread a string, as in a single-automaton run
            ctas += (int)std::max<int64_t>(1, std::min<int64_t>(h->n_sms, (cnt + 31) / 32));
            smem = std::max(smem, h->table_bytes);
            ++k;
        }
        if (k == 0) continue;
        P.n_groups = k;
        P.cta_first[k] = ctas;
        used_heads += k;
        lay->run_multi<<<ctas, kNfaThreads, lay->smem ? smem : 0, st>>>(P);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) {
            set_last_error("trex_nfa_run_multi", e);
            return TREX_ERR_CUDA;
        }
    }
    return TREX_OK;
}

}  // namespace trex

extern "C" {

int trex_nfa_create(int n_states, int sigma, const uint64_t *cols, uint64_t start_mask,
                    uint64_t accept_mask, int unknown_rejects, trex_nfa **out) {
    using namespace trex;
    if (!out) return TREX_ERR_ARG;
    *out = nullptr;
    if (n_states < 1 || n_states > 64 || sigma < 0 || sigma > 255 || (sigma > 0 && !cols))
        return TREX_ERR_ARG;
    trex_nfa *nfa = new (std::nothrow) trex_nfa();
    if (!nfa) return TREX_ERR_OOM;
    nfa->n_states = n_states;
    nfa->sigma = sigma;
    nfa->unknown_rejects = unknown_rejects ? 1 : 0;
    const uint64_t keep = n_states == 64 ? ~0ull : ((1ull << n_states) - 1);
    nfa->start_mask = start_mask & keep;
    nfa->accept_mask = accept_mask & keep;
    nfa->cols.assign((size_t)sigma * 64, 0);
    for (int c = 0; c < sigma; ++c)
        for (int j = 0; j < n_states; ++j) nfa->cols[(size_t)c * 64 + j] = cols[(size_t)c * 64 + j] & keep;
    nfa->lay = nfa_choose_layout(n_states, sigma);
    nfa->table_bytes = nfa_table_bytes(*nfa->lay, sigma);
    std::vector<uint8_t> t(nfa->table_bytes);
    if (nfa->lay->T == 64) nfa_build_tables<64>(nfa->cols, sigma, nfa->lay->G, nfa->unknown_rejects, t.data());
    else if (nfa->lay->T == 32) nfa_build_tables<32>(nfa->cols, sigma, nfa->lay->G, nfa->unknown_rejects, t.data());
    else nfa_build_tables<16>(nfa->cols, sigma, nfa->lay->G, nfa->unknown_rejects, t.data());
    nfa->n_sms = sm_count();
    if (nfa->n_sms <= 0) {
        delete nfa;
        set_last_error_msg("trex_nfa_create: no CUDA device");
        return TREX_ERR_SHAPE;
    }
    nfa->max_units = std::min(65535u, 2u * (uint32_t)nfa->n_sms * kNfaUnitsPerSm + 64u);   // (16-bit index)
    const size_t misc_off = (nfa->table_bytes + 255) & ~size_t(255);
    cudaError_t e;
    if ((e = cudaMalloc(&nfa->d_tables, misc_off + 256 + sizeof(NfaUnit) * nfa->max_units)) != cudaSuccess ||
        (e = cudaMemcpy(nfa->d_tables, t.data(), t.size(), cudaMemcpyHostToDevice)) != cudaSuccess) {
        set_last_error("trex_nfa_create", e);
        cudaFree(nfa->d_tables);
        delete nfa;
        return e == cudaErrorMemoryAllocation ? TREX_ERR_OOM : TREX_ERR_CUDA;
    }
    nfa->d_misc = nfa->d_tables + misc_off;
    nfa->d_units = reinterpret_cast<NfaUnit *>(nfa->d_tables + misc_off + 256);
    if (nfa->lay->smem) {
        // the attribute is per kernel: raised to what any automaton of the layout can need
        for (const void *f : {(const void *)nfa->lay->run, (const void *)nfa->lay->run_multi}) {
            if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kNfaSmemBudget)) == cudaSuccess)
                continue;
            set_last_error("trex_nfa_create: cudaFuncSetAttribute", e);
            cudaFree(nfa->d_tables);
            delete nfa;
            return TREX_ERR_CUDA;
        }
    }
    *out = nfa;
    return TREX_OK;
}

void trex_nfa_destroy(trex_nfa *nfa) {
    if (!nfa) return;
    cudaFree(nfa->d_tables);
    delete nfa;
}

int trex_nfa_run(trex_nfa *nfa, const uint8_t *data, const int64_t *offsets, int64_t n_strings,
                 int64_t total_bytes, uint64_t *final_mask, uint8_t *accept, int32_t *accept_i32,
                 void *stream) {
    return trex::nfa_run(nfa, data, offsets, n_strings, total_bytes, final_mask, accept, accept_i32,
                         static_cast<cudaStream_t>(stream), nullptr);
}

int trex_nfa_run_multi(trex_nfa *const *nfas, int n_groups, const int64_t *group_first,
                       const uint8_t *data, const int64_t *offsets, int64_t total_bytes,
                       uint64_t *final_mask, uint8_t *accept, int32_t *accept_i32, void *scratch,
                       void *stream) {
    return trex::nfa_run_multi(nfas, n_groups, group_first, data, offsets, total_bytes, final_mask, accept,
                               accept_i32, scratch, static_cast<cudaStream_t>(stream));
}

int trex_nfa_error(trex_nfa *nfa, int32_t *err_out) {
    if (!nfa || !err_out) return TREX_ERR_ARG;
    uint32_t v = 0;
    TREX_CUDA(cudaMemcpy(&v, static_cast<uint8_t *>(nfa->d_misc) + 8, 4, cudaMemcpyDeviceToHost));
    *err_out = (int32_t)v;
    return TREX_OK;
}

}  // extern "C"

// ---- reference C ABI: nfa_tc_engine_* (cuda/nfa_tc_evolution.cu:936-1015) -----------------
namespace trex {
struct RefNfaEngine {
    trex_nfa *nfa = nullptr;
    uint8_t *d_data = nullptr;
    int64_t *d_off64 = nullptr;
    int32_t *d_off32 = nullptr;
    int32_t *d_res = nullptr;
    int64_t max_chars = 0, max_b = 0;
    cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};
    bool ready = false;
    void destroy() {
        trex_nfa_destroy(nfa);
        cudaFree(d_data);
        cudaFree(d_off64);
        cudaFree(d_off32);
        cudaFree(d_res);
        for (auto &x : ev)
            if (x) cudaEventDestroy(x);
        *this = RefNfaEngine();
    }
};
static RefNfaEngine g_ref_nfa;
__global__ void nfa_widen_kernel(const int32_t *in, int64_t *out, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        out[i] = in[i];
}
}  // namespace trex

extern "C" {

int nfa_tc_engine_init(const float *T_matrices, const float *accept_mask, const float *start_vec,
                       int n, int sigma, int max_B, int max_L) {
    using namespace trex;
    RefNfaEngine &E = g_ref_nfa;
    E.destroy();
    if (!T_matrices || !accept_mask || !start_vec || max_B < 0 || max_L < 0) return TREX_ERR_ARG;
    if (n < 1 || n > 64 || sigma < 1 || sigma > 255) return TREX_ERR_SHAPE;
    // T[c][dst][src] > 0.5 is an edge (reference float_to_bitpar, nfa_tc_evolution.cu:632-644)
    std::vector<uint64_t> cols((size_t)sigma * 64, 0);
    for (int c = 0; c < sigma; ++c)
        for (int dst = 0; dst < n; ++dst)
            for (int src = 0; src < n; ++src)
                if (T_matrices[((size_t)c * n + dst) * n + src] > 0.5f) cols[(size_t)c * 64 + src] |= 1ull << dst;
    uint64_t sm = 0, am = 0;
    for (int i = 0; i < n; ++i) {
        if (start_vec[i] > 0.5f) sm |= 1ull << i;
        if (accept_mask[i] > 0.5f) am |= 1ull << i;
    }
    int rc = trex_nfa_create(n, sigma, cols.data(), sm, am, 0, &E.nfa);
    if (rc) return rc;
    E.max_b = max_B;
    E.max_chars = (int64_t)max_B * max_L;
    cudaError_t e;
    if ((e = cudaMalloc(&E.d_data, std::max<int64_t>(E.max_chars, 16))) != cudaSuccess ||
        (e = cudaMalloc(&E.d_off64, (max_B + 1) * 8)) != cudaSuccess ||
        (e = cudaMalloc(&E.d_off32, (max_B + 1) * 4)) != cudaSuccess ||
        (e = cudaMalloc(&E.d_res, std::max(max_B, 1) * 4)) != cudaSuccess) {
        set_last_error("nfa_tc_engine_init", e);
        E.destroy();
        return TREX_ERR_OOM;
    }
    for (auto &x : E.ev) TREX_CUDA(cudaEventCreate(&x));
    E.ready = true;
    return TREX_OK;
}

int nfa_tc_engine_dispatch(const uint8_t *raw_concat, const int *offsets, int *results, int B,
                           int total_chars, float *kernel_ms, float *total_ms) {
    using namespace trex;
    RefNfaEngine &E = g_ref_nfa;
    if (!E.ready) return TREX_ERR_NOT_INIT;
    if (B < 0 || total_chars < 0 || (B > 0 && (!offsets || !results))) return TREX_ERR_ARG;
    if (B > E.max_b || total_chars > E.max_chars) return TREX_ERR_CAPACITY;
    if (kernel_ms) *kernel_ms = 0.f;
    if (total_ms) *total_ms = 0.f;
    if (B == 0) return TREX_OK;
    cudaStream_t st = 0;
    TREX_CUDA(cudaEventRecord(E.ev[0], st));
    if (total_chars) TREX_CUDA(cudaMemcpyAsync(E.d_data, raw_concat, total_chars, cudaMemcpyHostToDevice, st));
    TREX_CUDA(cudaMemcpyAsync(E.d_off32, offsets, (size_t)(B + 1) * 4, cudaMemcpyHostToDevice, st));
    nfa_widen_kernel<<<std::min(1024, (B + 256) / 256), 256, 0, st>>>(E.d_off32, E.d_off64, B + 1);
    TREX_CHECK_LAUNCH();
    TREX_CUDA(cudaEventRecord(E.ev[1], st));
    uint32_t *err = nullptr;
    int rc = nfa_run(E.nfa, E.d_data, E.d_off64, B, total_chars, nullptr, nullptr, E.d_res, st, &err);
    if (rc) return rc;
    TREX_CUDA(cudaEventRecord(E.ev[2], st));
    TREX_CUDA(cudaMemcpyAsync(results, E.d_res, (size_t)B * 4, cudaMemcpyDeviceToHost, st));
    uint32_t h_err = 0;
    TREX_CUDA(cudaMemcpyAsync(&h_err, err, 4, cudaMemcpyDeviceToHost, st));
    TREX_CUDA(cudaEventRecord(E.ev[3], st));
    TREX_CUDA(cudaEventSynchronize(E.ev[3]));
    if (kernel_ms) TREX_CUDA(cudaEventElapsedTime(kernel_ms, E.ev[1], E.ev[2]));
    if (total_ms) TREX_CUDA(cudaEventElapsedTime(total_ms, E.ev[0], E.ev[3]));
    return h_err ? TREX_ERR_ARG : TREX_OK;
}

void nfa_tc_engine_destroy(void) { trex::g_ref_nfa.destroy(); }

}  // extern "C"
