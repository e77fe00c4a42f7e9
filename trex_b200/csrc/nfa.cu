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
};

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

// Threads take strings first .. first + n - 1 from the counter *head and walk them
// in 16-byte windows; results go to index i of the output arrays.
template <int T, int G>
__device__ __forceinline__ void nfa_walk_queue(const typename NfaWord<T>::type *tbl, int sigma, uint64_t start_mask,
                                               uint64_t accept_mask, const uint8_t *d, int64_t total_bytes,
                                               const int64_t *offsets, int64_t first, int64_t n,
                                               unsigned long long *head, uint32_t *err, uint64_t *final_mask,
                                               uint8_t *accept, int32_t *accept_i32) {
    while (true) {
        const unsigned long long k = atomicAdd(head, 1ull);
        if (k >= (unsigned long long)n) break;
        const int64_t i = first + (int64_t)k;
        const int64_t a = offsets[i], b = offsets[i + 1];
        if (a < 0 || b < a || b > total_bytes) {
            atomicOr(err, 1u);
            continue;
        }
        using W = typename NfaWord<T>::type;
        W s = (W)start_mask;
        int64_t p = a;
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
        const bool ok = (s & (W)accept_mask) != 0;
        if (final_mask) final_mask[i] = s;
        if (accept) accept[i] = ok ? 1 : 0;
        if (accept_i32) accept_i32[i] = ok ? 1 : 0;
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
    for (int i = threadIdx.x; i < n16; i += blockDim.x) dst[i] = src[i];
    __syncthreads();
    return reinterpret_cast<const W *>(s_nfa_tbl);
}

template <int T, int G, bool SMEM>
__global__ void __launch_bounds__(kNfaThreads, 1) nfa_bitpar_kernel(NfaParams P) {
    const typename NfaWord<T>::type *tbl = static_cast<const typename NfaWord<T>::type *>(P.tables);
    if constexpr (SMEM) tbl = nfa_tables_in<T, G>(P.tables, P.sigma);
    nfa_walk_queue<T, G>(tbl, P.sigma, P.start_mask, P.accept_mask, P.data, P.total_bytes, P.offsets, 0, P.n,
                      P.head, P.err, P.final_mask, P.accept, P.accept_i32);
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
    uint8_t *d_tables = nullptr;
    size_t table_bytes = 0;   // a multiple of 16
    void *d_misc = nullptr;   // head counter + error word
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
    const size_t smem = nfa->lay->smem ? nfa->table_bytes : 0;
    // a thread a string: a few strings need one CTA, so that batches of several
    // automata launched on separate streams run side by side
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(nfa->n_sms, (n + 31) / 32));
    profile_kernel_begin(stream);
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
    cudaError_t e;
    if ((e = cudaMalloc(&nfa->d_tables, t.size())) != cudaSuccess ||
        (e = cudaMalloc(&nfa->d_misc, 16)) != cudaSuccess ||
        (e = cudaMemcpy(nfa->d_tables, t.data(), t.size(), cudaMemcpyHostToDevice)) != cudaSuccess) {
        set_last_error("trex_nfa_create", e);
        cudaFree(nfa->d_tables);
        cudaFree(nfa->d_misc);
        delete nfa;
        return e == cudaErrorMemoryAllocation ? TREX_ERR_OOM : TREX_ERR_CUDA;
    }
    if (nfa->lay->smem) {
        // the attribute is per kernel: raised to what any automaton of the layout can need
        for (const void *f : {(const void *)nfa->lay->run, (const void *)nfa->lay->run_multi}) {
            if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kNfaSmemBudget)) == cudaSuccess)
                continue;
            set_last_error("trex_nfa_create: cudaFuncSetAttribute", e);
            cudaFree(nfa->d_tables);
            cudaFree(nfa->d_misc);
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
    cudaFree(nfa->d_misc);
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
