// Small batches of the ragged DFA path in one launch (included by dfa_batch.cu).
//
// A batch of a few MiB is bound by latency: the planning, walking and chaining
// launches cost several times its walk, and its strings occupy a fraction of the
// lanes. Here nothing is planned: strings are dealt to the warps of the GPU, and
// a warp walks a string with all its lanes. Lane l takes the l-th share of the
// string's 32-byte windows and starts warm_bytes(N) earlier from state 0 (the
// speculation of the ragged kernel); then each lane compares its guess with lane
// l - 1's end state, and lanes that guessed wrong walk their share again from
// that state until all agree, which is exact for every automaton (lane l is right
// after at most l rounds). Automata of at most 16 states that do not agree after
// kSmallRounds rounds (permutations) map all their states over each share
// instead. Several short strings of a warp are walked side by side, a string a
// lane. Strings above kSmallLongBytes are cut into pieces of 1024 windows, which
// the CTAs take in turn and walk the same way with all their lanes (every CTA
// finds the same pieces in the offsets it checks anyway); the CTA that reports a
// string's last piece compares the pieces' guesses with their predecessors' end
// states in order, walking again those that do not match.
// The byte maps are read unreplicated from shared memory: building a replicated
// table would cost more than the bank conflicts of the short walks.
#pragma once

namespace trex {

constexpr int kSmallThreads = 1024;
constexpr int64_t kSmallBytes = 8ll << 20;       // bytes walked (see dfa_set_run_ex)
constexpr int64_t kSmallStrings = 131072;
constexpr int64_t kSmallMapBytes = 128 * 1024;   // byte maps kept in shared memory
constexpr int64_t kSmallLongBytes = 16 * 1024;
constexpr uint32_t kSmallPieceWindows = kSmallThreads;
constexpr int kSmallRounds = 3;
constexpr int kSmallLong = 512;   // long strings (more, from overlapping offsets: a warp walks each)

// A byte map in shared memory (offset into g_dfa_tbl) or, for large sets, global memory.
template <bool SMEM>
struct SmallMap {
    const uint8_t *g;
    uint32_t off, n;
    __device__ __forceinline__ uint32_t next(uint32_t c, uint32_t s) const {
        if constexpr (SMEM) return g_dfa_tbl[off + c * n + s];
        else return __ldg(g + c * n + s);
    }
};

// A string as windows of 32 aligned bytes: [w, w + 32 nw), its bytes [lo, hi).
struct SmallView {
    const uint8_t *lo, *hi, *w;
    uint32_t nw;
};
__device__ __forceinline__ SmallView small_view(const RaggedParams &P, int64_t a, int64_t b) {
    SmallView v;
    v.lo = P.data + a;
    v.hi = P.data + b;
    v.w = reinterpret_cast<const uint8_t *>((uintptr_t)v.lo & ~(uintptr_t)31);
    v.nw = (uint32_t)((v.hi - v.w + 31) >> 5);
    return v;
}

// Walks windows [k0, k1) from state s: the end state (low byte) and the state at the start of
// window kc (second byte; s when kc is not among them). Lanes may have different ranges. One copy
// of the unrolled walk for all callers (not inlined: the instruction cache).
template <class M>
__device__ __noinline__ uint32_t small_walk(M map, const uint8_t *lo, const uint8_t *hi, const uint8_t *w,
                                            uint32_t k0, uint32_t k1, uint32_t kc, uint32_t s) {
    uint4 a = make_uint4(0u, 0u, 0u, 0u), b = a;
    uint32_t guess = s;
    w += 32 * (size_t)k0;
    if (k0 < k1) load_window(w, lo, hi, a, b);
    for (uint32_t k = k0; k < k1; ++k, w += 32) {
        if (k == kc) guess = s;
        const uint32_t x[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        if (k + 1 < k1) load_window(w + 32, lo, hi, a, b);
        const uint32_t m = bit_range(w < lo ? (int)(lo - w) : 0, w + 32 > hi ? (int)(hi - w) : 32);
        if (m == 0xffffffffu) {
#pragma unroll
            for (int j = 0; j < 32; ++j) s = map.next((x[j >> 2] >> (8 * (j & 3))) & 0xffu, s);
        } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                const uint32_t t = map.next((x[j >> 2] >> (8 * (j & 3))) & 0xffu, s);
                s = (m >> j) & 1u ? t : s;
            }
        }
    }
    return s | (guess << 8);
}

// One string (not empty) by the whole warp; its final state, in every lane.
template <class M>
__device__ __forceinline__ uint32_t small_warp(const RaggedParams &P, const M &map, uint32_t N, int64_t a,
                                               int64_t b, uint32_t start) {
    const uint32_t FULL = 0xffffffffu, lane = threadIdx.x & 31u;
    const SmallView v = small_view(P, a, b);
    const uint32_t per = (v.nw + 31u) / 32u, used = (v.nw + per - 1u) / per;
    const uint32_t k0 = min(v.nw, lane * per), k1 = min(v.nw, k0 + per);
    const uint32_t warm = (uint32_t)(warm_bytes((int)N, 224) / 32);
    const uint32_t ks = k0 > warm ? k0 - warm : 0u;
    const uint32_t both = small_walk(map, v.lo, v.hi, v.w, ks, k1, k0, ks == 0u ? start : 0u);
    uint32_t fin = both & 0xffu, guess = both >> 8;
    for (int round = 0;; ++round) {
        const uint32_t prev = __shfl_up_sync(FULL, fin, 1);
        const bool wrong = lane > 0u && lane < used && guess != prev;
        if (!__any_sync(FULL, wrong)) break;
        if (round >= kSmallRounds && N <= (uint32_t)kSmallDfaStates) {
            // every lane maps all states over its share; the maps are applied in order
            uint32_t st[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) st[j] = (uint32_t)j;
            const uint8_t *p = v.w + 32 * (size_t)k0, *e = v.w + 32 * (size_t)k1;
            p = p < v.lo ? v.lo : p;
            e = e > v.hi ? v.hi : e;
            for (; p < e; ++p) {
                const uint32_t c = __ldg(p);
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    if ((uint32_t)j < N) st[j] = map.next(c, st[j]);
            }
            uint64_t f = 0;
#pragma unroll
            for (int j = 0; j < 16; ++j) f |= (uint64_t)st[j] << (4 * j);
            uint32_t s = start;
            for (uint32_t l = 0; l < used; ++l) s = (uint32_t)(__shfl_sync(FULL, f, (int)l) >> (4 * s)) & 15u;
            return s;
        }
        if (wrong) {
            guess = prev;
            fin = small_walk(map, v.lo, v.hi, v.w, k0, k1, 0xffffffffu, prev) & 0xffu;
        }
    }
    return __shfl_sync(FULL, fin, (int)(used - 1u));
}

// Windows [w0, w1) of a string by the whole CTA, a window a thread (every thread calls it): the end
// state (low byte) and the state it started from, in every thread. entry < 0: guessed with a
// warm-up (the true start state when it reaches the string's first byte).
template <class M>
__device__ __forceinline__ uint32_t small_piece(const RaggedParams &P, const M &map, uint32_t N, const SmallView &v,
                                                uint32_t w0, uint32_t w1, uint32_t start, int entry, uint64_t *s_map) {
    const uint32_t t = threadIdx.x, used = w1 - w0;
    const uint32_t k0 = min(w1, w0 + t), k1 = min(w1, k0 + 1u);
    const uint32_t warm = (uint32_t)(warm_bytes((int)N, 224) / 32);
    const uint32_t first = entry >= 0 ? w0 : 0u;   // the first window whose entry state is known
    const uint32_t ks = k0 > first + warm ? k0 - warm : first;
    const uint32_t both = small_walk(map, v.lo, v.hi, v.w, k0 < k1 ? ks : k1, k1, k0,
                                     ks == first ? (entry >= 0 ? (uint32_t)entry : start) : 0u);
    uint32_t fin = both & 0xffu, guess = both >> 8;
    for (int round = 0;; ++round) {
        __syncthreads();
        s_map[t] = fin | (guess << 8);
        __syncthreads();
        const uint32_t prev = t > 0u ? (uint32_t)s_map[t - 1u] & 0xffu : 0u;
        const bool wrong = t > 0u && t < used && guess != prev;
        if (!__syncthreads_or(wrong)) break;
        if (round >= kSmallRounds && N <= (uint32_t)kSmallDfaStates) {
            // every lane maps all states over its window; the maps are applied in order
            uint32_t st[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) st[j] = (uint32_t)j;
            const uint8_t *p = v.w + 32 * (size_t)k0, *e = v.w + 32 * (size_t)k1;
            p = p < v.lo ? v.lo : p;
            e = e > v.hi ? v.hi : e;
            for (; p < e; ++p) {
                const uint32_t c = __ldg(p);
#pragma unroll
                for (int j = 0; j < 16; ++j)
                    if ((uint32_t)j < N) st[j] = map.next(c, st[j]);
            }
            uint64_t f = 0;
#pragma unroll
            for (int j = 0; j < 16; ++j) f |= (uint64_t)st[j] << (4 * j);
            const uint32_t g0 = ((uint32_t)s_map[0] >> 8) & 0xffu;
            __syncthreads();
            s_map[t] = f;
            __syncthreads();
            uint32_t s = g0;
            for (uint32_t l = 0; l < used; ++l) s = (uint32_t)(s_map[l] >> (4 * s)) & 15u;
            __syncthreads();
            return s | (g0 << 8);
        }
        if (wrong) {
            guess = prev;
            fin = small_walk(map, v.lo, v.hi, v.w, k0, k1, 0xffffffffu, prev) & 0xffu;
        }
    }
    const uint32_t s = ((uint32_t)s_map[used - 1u] & 0xffu) | ((uint32_t)s_map[0] & 0xff00u);
    __syncthreads();
    return s;
}

// Warp g of the launch (g = CTA + CTAs * warp, so that few strings spread over the SMs) takes
// strings g, g + W, g + 2 W, ... of the W warps. cnt (a zeroed report counter a long string) and
// rec (a record a piece) are only used when the batch can hold a long string.
template <bool SMEM>
__global__ void __launch_bounds__(kSmallThreads, 1) dfa_small_kernel(RaggedParams P, uint32_t *cnt, uint32_t *rec) {
    __shared__ uint64_t s_map[kSmallThreads];
    __shared__ uint32_t s_found[kSmallLong], s_long[kSmallLong], s_first[kSmallLong + 1];
    __shared__ uint32_t s_n_long, s_last;
    const uint32_t FULL = 0xffffffffu, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_n_long = 0u;
    if constexpr (SMEM) {
        const uint4 *src = reinterpret_cast<const uint4 *>(P.tmaps);
        uint4 *dst = reinterpret_cast<uint4 *>(g_dfa_tbl);
        for (uint32_t i = threadIdx.x; i < P.fix_tm_bytes / 16u; i += kSmallThreads) dst[i] = src[i];
    }
    __syncthreads();
    // Malformed strings get no result. Well-formed offsets do not overlap; when some string is
    // malformed, the others may, and a batch that would need more work items than the planned
    // path has room for is refused whole, as there. CTA 0 writes the error word.
    const int64_t n_off = P.multi_n > 0 ? P.multi_n : P.n;
    bool bad = false, bad_id = false;
    for (int64_t i = threadIdx.x; i < n_off; i += kSmallThreads) {
        const int64_t a = P.offsets[i], b = P.offsets[i + 1];
        const bool bi = a < 0 || b < a || b > P.total_bytes;
        bad |= bi;
        if (!bi && b - a > kSmallLongBytes) {
            const uint32_t k = atomicAdd(&s_n_long, 1u);
            if (k < (uint32_t)kSmallLong) s_found[k] = (uint32_t)i;
        }
        if (blockIdx.x == 0 && P.dfa_id && P.multi_n == 0) {
            const int d = P.dfa_id[i];
            bad_id |= !bi && (d < 0 || d >= P.n_dfas);   // (a string with malformed offsets raises only that bit)
        }
    }
    uint32_t err = 0u;
    if (__syncthreads_or(bad)) {
        uint64_t items = 0;
        for (int64_t i = threadIdx.x; i < P.n; i += kSmallThreads) {
            const StringIn in = load_string(P.offsets, P.dfa_id, i, P.n, P.multi_n);
            if (in.a < 0 || in.b < in.a || in.b > P.total_bytes || in.d < 0 || in.d >= P.n_dfas) continue;
            items += item_geom(in.b - in.a, in.a, P.desc[in.d].n_states, P.seg_len, P.base_mis).k;
        }
        s_map[threadIdx.x] = items;
        __syncthreads();
        for (int o = kSmallThreads / 2; o > 0; o >>= 1) {
            if ((int)threadIdx.x < o) s_map[threadIdx.x] += s_map[threadIdx.x + o];
            __syncthreads();
        }
        err = kErrBadOffsets | (s_map[0] > (uint64_t)P.max_items ? kErrCapacity : 0u);
        __syncthreads();
    }
    if (blockIdx.x == 0) {
        if (__syncthreads_or(bad_id)) err |= kErrBadDfaId;
        if (threadIdx.x == 0) *P.err = err;
    }
    if (err & kErrCapacity) return;
    // the long strings in order, and each one's first piece (the same in every CTA)
    const uint32_t n_long = s_n_long <= (uint32_t)kSmallLong && !(err & kErrBadOffsets) ? s_n_long : 0u;
    if (n_long != 0u) {
        for (uint32_t i = threadIdx.x; i < n_long; i += kSmallThreads) {
            const uint32_t mine = s_found[i];
            uint32_t before = 0u;
            for (uint32_t j = 0; j < n_long; ++j) before += s_found[j] < mine;
            s_long[before] = mine;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            uint32_t run = 0u;
            for (uint32_t i = 0; i < n_long; ++i) {
                s_first[i] = run;
                run += (small_view(P, P.offsets[s_long[i]], P.offsets[s_long[i] + 1]).nw + kSmallPieceWindows - 1u) /
                       kSmallPieceWindows;
            }
            s_first[n_long] = run;
        }
        __syncthreads();
    }
    auto map_of = [&](const DfaDesc &D) {
        return SmallMap<SMEM>{P.tmaps + D.tmap_off, (uint32_t)D.tmap_off, (uint32_t)D.n_states};
    };
    const int64_t warps = (int64_t)gridDim.x * (kSmallThreads / 32);
    const int64_t g = (int64_t)blockIdx.x + (int64_t)gridDim.x * warp;
    for (int64_t base = g; base < P.n; base += warps * 32) {
        // up to 32 strings, one a lane
        const int64_t i = base + warps * lane;
        const uint32_t mine = (uint32_t)min((int64_t)32, (P.n - base + warps - 1) / warps);
        int64_t len = -1, a = 0;
        int d = 0;
        if (i < P.n) {
            const StringIn in = load_string(P.offsets, P.dfa_id, i, P.n, P.multi_n);
            if (!(in.a < 0 || in.b < in.a || in.b > P.total_bytes || in.d < 0 || in.d >= P.n_dfas) &&
                !(n_long != 0u && in.b - in.a > kSmallLongBytes)) {
                a = in.a;
                len = in.b - in.a;
                d = in.d;
            }
        }
        // strings of at most 64 bytes for each string of the warp: a string a lane (walking them
        // one by one with all lanes costs a warm-up each)
        const bool alone = len >= 0 && len <= 64 * (int64_t)mine;
        if (alone) {
            const DfaDesc &D = P.desc[d];
            const SmallView v = small_view(P, a, a + len);
            const uint32_t s = small_walk(map_of(D), v.lo, v.hi, v.w, 0u, len ? v.nw : 0u, 0xffffffffu,
                                          (uint32_t)D.start) & 0xffu;
            write_result(P, (uint32_t)i, s, D.accept_off);
        }
        __syncwarp();
        uint32_t left = __ballot_sync(FULL, len >= 0 && !alone);
        while (left) {
            const int l = __ffs(left) - 1;
            left &= left - 1u;
            const int64_t sa = __shfl_sync(FULL, a, l), sl = __shfl_sync(FULL, len, l);
            const DfaDesc &D = P.desc[__shfl_sync(FULL, d, l)];
            const uint32_t s = small_warp(P, map_of(D), (uint32_t)D.n_states, sa, sa + sl, (uint32_t)D.start);
            if (lane == 0) write_result(P, (uint32_t)(base + warps * l), s, D.accept_off);
        }
    }
    if (n_long == 0u) return;
    // ---- long strings: pieces in turn (multi-pattern runs: every automaton's pieces)
    const uint32_t pieces = s_first[n_long], every = P.multi_n > 0 ? (uint32_t)P.n_dfas : 1u;
    for (uint32_t p = blockIdx.x; p < pieces * every; p += gridDim.x) {
        const uint32_t q = p % pieces;
        uint32_t x = 0;   // the last long string whose first piece is at most q
        for (uint32_t step = 256u; step > 0u; step >>= 1)
            if (x + step < n_long && s_first[x + step] <= q) x += step;
        const uint32_t k = s_first[x + 1u] - s_first[x], j = q - s_first[x];
        const int64_t i = (int64_t)s_long[x] + (int64_t)(p / pieces) * P.multi_n;
        const StringIn in = load_string(P.offsets, P.dfa_id, i, P.n, P.multi_n);
        if (in.d < 0 || in.d >= P.n_dfas) continue;   // flagged above
        const DfaDesc &D = P.desc[in.d];
        const uint32_t N = (uint32_t)D.n_states, start = (uint32_t)D.start;
        const SmallView v = small_view(P, in.a, in.b);
        uint32_t r = small_piece(P, map_of(D), N, v, j * kSmallPieceWindows, min(v.nw, (j + 1u) * kSmallPieceWindows),
                                 start, -1, s_map);
        if (k == 1u) {
            if (threadIdx.x == 0) write_result(P, (uint32_t)i, r & 0xffu, D.accept_off);
            continue;
        }
        uint32_t *const rs = rec + (p - j);
        if (threadIdx.x == 0) {
            *(volatile uint32_t *)(rs + j) = r;
            __threadfence();
            s_last = atomicAdd(cnt + (p / pieces) * n_long + x, 1u) + 1u == k;
            __threadfence();
        }
        __syncthreads();
        if (!s_last) continue;
        // every piece is recorded: chain them
        uint32_t s = start;
        for (uint32_t j0 = 0; j0 < k; j0 += kSmallThreads) {
            __syncthreads();
            if (j0 + threadIdx.x < k) s_map[threadIdx.x] = *(volatile uint32_t *)(rs + j0 + threadIdx.x);
            __syncthreads();
            const uint32_t n_rec = min(k - j0, (uint32_t)kSmallThreads);
            for (uint32_t l = 0; l < n_rec;) {
                const uint32_t w = (uint32_t)s_map[l];
                if ((w >> 8) == s) {
                    s = w & 0xffu;
                    ++l;
                    continue;
                }
                // a wrong guess: the piece again from its true state (small_piece uses s_map)
                const uint32_t jj = j0 + l;
                s = small_piece(P, map_of(D), N, v, jj * kSmallPieceWindows, min(v.nw, (jj + 1u) * kSmallPieceWindows),
                                start, (int)s, s_map) & 0xffu;
                ++l;
                if (l + threadIdx.x < n_rec) s_map[l + threadIdx.x] = *(volatile uint32_t *)(rs + j0 + l + threadIdx.x);
                __syncthreads();
            }
        }
        if (threadIdx.x == 0) write_result(P, (uint32_t)i, s, D.accept_off);
        __syncthreads();
    }
}

}  // namespace trex
