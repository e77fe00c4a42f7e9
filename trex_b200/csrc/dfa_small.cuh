// Small batches of the ragged DFA path in one launch (included by dfa_batch.cu).
//
// A batch of a few MiB (and a set whose byte maps fit beside each other in shared memory:
// from L2 a step takes 430 cycles) is bound by latency: the planning, walking and chaining
// launches cost several times its walk, and its strings occupy a fraction of the
// lanes. Here nothing is planned: strings are dealt to the warps of the GPU, and
// a warp walks a string with all its lanes. Lane l takes the l-th share of the
// string's 32-byte windows and starts warm_bytes(N) earlier from state 0 (the
// speculation of the ragged kernel); then each lane compares its guess with lane
// l - 1's end state, and lanes that guessed wrong walk their share again from
// that state until all agree, which is exact for every automaton. Where most of them
// are still wrong after kSmallRounds rounds (permutations never agree, and would
// take a round a lane), every lane maps all states over its share and the maps are
// applied in order (N <= 16), or the string is walked by one lane beside the warp's
// others.
// Several short strings of a warp are walked side by side from the start, a string
// a lane. Strings above kSmallLongBytes are cut into pieces of 1024 windows, which
// the CTAs take in turn and walk the same way with all their lanes (every CTA
// finds the same pieces in the offsets it checks anyway); a piece whose lanes do
// not agree is recorded as the map of all states over it. The CTA that reports a
// string's last piece chains them: it applies the maps, and walks again the pieces
// whose guessed entry state was wrong.
// One launch against planned, us, automata that never synchronise, 8 / 24 / 256 states: 30
// strings of 256 KiB 90 / 154 / 756 against 1969 / 9362 / 8014, 200 of 40000 bytes 121 / 206 / 1086
// against 487 / 1582 / 1205, 8000 of 1000 bytes 87 / 91 / 81 against 97 / 114 / 153.
// The byte maps are read unreplicated from shared memory: building a replicated
// table would cost more than the bank conflicts of the short walks.
#pragma once

namespace trex {

constexpr int kSmallThreads = 1024;
constexpr int64_t kSmallBytes = 8ll << 20;       // bytes walked (see dfa_set_run_ex)
constexpr int64_t kSmallStrings = 131072;
constexpr int64_t kSmallMapBytes = 200 * 1024;   // byte maps, kept in shared memory
constexpr int64_t kSmallLongBytes = 16 * 1024;
constexpr uint32_t kSmallPieceWindows = kSmallThreads;
constexpr int kSmallRounds = 3;
constexpr int kSmallLane = 2048;    // bytes one lane walks in less time than a warp's maps of several strings
constexpr int kSmallMaxPieces = (int)(kSmallBytes / (32 * kSmallPieceWindows)) + 2;   // of one string
constexpr int kSmallLong = 512;   // long strings (more, from overlapping offsets: a warp walks each)

// A byte map in shared memory (offset into g_dfa_tbl).
struct SmallMap {
    uint32_t off, n;
    __device__ __forceinline__ uint32_t next(uint32_t c, uint32_t s) const { return g_dfa_tbl[off + c * n + s]; }
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
__device__ __noinline__ uint32_t small_walk(SmallMap map, const uint8_t *lo, const uint8_t *hi, const uint8_t *w,
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

// Whether the lanes' chains do not meet: n_wrong lanes after kSmallRounds rounds, of `open` that the start
// state has not reached yet. Chains that never meet leave (N - 1) / N of them wrong; a random automaton's
// about 3% for up to 64 states, 8% for 128, 28% for 256, but one string of thousands with many more
// sets the time of the launch, so the limits lie well above.
__device__ __forceinline__ bool small_hopeless(int round, uint32_t n_wrong, int open, uint32_t N) {
    return round == kSmallRounds && open > 4 && 8 * (int)n_wrong > open * (N < 4u ? 0 : N <= 16u ? 3 : N <= 128u ? 4 : 6);
}

// One string (not empty) by the whole warp; its final state, in every lane, or kSmallOpen where the
// lanes do not agree and one lane is to walk it (`lone`: this automaton and string have no better way).
constexpr uint32_t kSmallOpen = 0xffffffffu;
__device__ __noinline__ uint32_t small_warp(SmallMap map, uint32_t N, SmallView v, uint32_t start, bool lone) {
    const uint32_t FULL = 0xffffffffu, lane = threadIdx.x & 31u;
    const uint32_t per = (v.nw + 31u) / 32u, used = (v.nw + per - 1u) / per;
    const uint32_t k0 = min(v.nw, lane * per), k1 = min(v.nw, k0 + per);
    const uint32_t warm = (uint32_t)(warm_bytes((int)N, 224) / 32);
    const uint32_t ks = k0 > warm ? k0 - warm : 0u;
    const uint32_t both = small_walk(map, v.lo, v.hi, v.w, ks, k1, k0, ks == 0u ? start : 0u);
    uint32_t fin = both & 0xffu, guess = both >> 8;
    const int guessed = __popc(__ballot_sync(FULL, lane < used && ks > 0u));
    for (int round = 0;; ++round) {
        const uint32_t prev = __shfl_up_sync(FULL, fin, 1);
        const bool wrong = lane > 0u && lane < used && guess != prev;
        const uint32_t n_wrong = (uint32_t)__popc(__ballot_sync(FULL, wrong));
        if (n_wrong == 0u) break;
        if (small_hopeless(round, n_wrong, guessed - round, N)) {
            if (lone) return kSmallOpen;
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

// The map of all states over windows [w0, w1) of a string by the whole CTA (every thread calls it),
// in s_map[0 .. N - 1]: thread (share, state) walks one share of the windows from one state, with as
// many shares as 1024 threads give; then N threads apply the shares' maps in order.
__device__ __forceinline__ void small_piece_map(const SmallMap &map, uint32_t N, const SmallView &v, uint32_t w0, uint32_t w1,
                                                uint64_t *s_map) {
    const uint32_t t = threadIdx.x;
    uint32_t width = 8u;
    while (width < N) width <<= 1;
    const uint32_t shares = kSmallThreads / width, each = (w1 - w0 + shares - 1u) / shares;
    const uint32_t k0 = min(w1, w0 + (t / width) * each), k1 = min(w1, k0 + each), from = t & (width - 1u);
    const uint32_t to = from < N ? small_walk(map, v.lo, v.hi, v.w, k0, k1, 0xffffffffu, from) & 0xffu : 0u;
    __syncthreads();
    s_map[t] = to;
    __syncthreads();
    uint32_t s = t;
    if (t < N)
        for (uint32_t l = 0; l < shares; ++l) s = (uint32_t)s_map[l * width + s];
    __syncthreads();
    if (t < N) s_map[t] = s;
    __syncthreads();
}

// Windows [w0, w1) of a string by the whole CTA, a window a thread (every thread calls it): the end
// state (low byte) and the state it started from, in every thread; with kSmallIsMap the map of all
// states is in s_map instead. entry < 0: guessed with a warm-up (the true start state when it
// reaches the string's first byte).
constexpr uint32_t kSmallIsMap = 1u << 16;
__device__ __noinline__ uint32_t small_piece(SmallMap map, uint32_t N, SmallView v, uint32_t w0, uint32_t w1,
                                             uint32_t start, int entry, uint64_t *s_map) {
    const uint32_t t = threadIdx.x, used = w1 - w0;
    const uint32_t k0 = min(w1, w0 + t), k1 = min(w1, k0 + 1u);
    // (the piece's own entry warms up longer: a wrong one costs the whole CTA a walk)
    const uint32_t warm = (uint32_t)(warm_bytes((int)N, 224) / 32) * (t > 0u ? 1u : N <= 64u ? 2u : 4u);
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
        const uint32_t n_wrong = (uint32_t)__syncthreads_count(wrong);
        if (n_wrong == 0u) break;
        // (chains of N states meet within N bytes in the mean, a round is 32: 16 + N / 2 rounds are far
        // more than random automata take, where one wrong lane a round could go on for 1023)
        if (small_hopeless(round, n_wrong, (int)used - round, N) || round >= 16 + (int)(N / 2u)) {
            small_piece_map(map, N, v, w0, w1, s_map);
            return kSmallIsMap;
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
// strings g, g + W, g + 2 W, ... of the W warps. cnt (a zeroed report counter a long string), rec (a
// record a piece) and maps (256 bytes a piece) are only used when the batch can hold a long string.
__global__ void __launch_bounds__(kSmallThreads, 1) dfa_small_kernel(RaggedParams P, uint32_t *cnt, uint32_t *rec,
                                                                    uint8_t *maps) {
    __shared__ uint64_t s_map[kSmallThreads];
    __shared__ uint32_t s_found[kSmallLong], s_long[kSmallLong], s_first[kSmallLong + 1];
    __shared__ uint32_t s_rec[kSmallMaxPieces];
    __shared__ uint32_t s_n_long, s_last;
    const uint32_t FULL = 0xffffffffu, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_n_long = 0u;
    {
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
        return SmallMap{(uint32_t)D.tmap_off, (uint32_t)D.n_states};
    };
    // (strings, bytes and offsets of a batch of this path fit in 32 bits)
    const uint32_t warps = gridDim.x * (uint32_t)(kSmallThreads / 32), n = (uint32_t)P.n;
    for (uint32_t base = blockIdx.x + gridDim.x * warp; base < n; base += warps * 32u) {
        // up to 32 strings, one a lane
        const uint32_t i = base + warps * lane, mine = min(32u, (n - base + warps - 1u) / warps);
        int len = -1, a = 0, d = 0;
        if (i < n) {
            const StringIn in = load_string(P.offsets, P.dfa_id, i, P.n, P.multi_n);
            if (!(in.a < 0 || in.b < in.a || in.b > P.total_bytes || in.d < 0 || in.d >= P.n_dfas) &&
                !(n_long != 0u && in.b - in.a > kSmallLongBytes)) {
                a = (int)in.a;
                len = (int)(in.b - in.a);
                d = in.d;
            }
        }
        // Strings of up to `most` windows go to a lane each, side by side, the others to all lanes, one
        // after the other: a share and a warm-up each, counted twice, because 32 lanes' lookups take more
        // of the SM than one's. The limit is the length of one of the strings (or 0) with the least sum.
        uint32_t nw = 0u, each = 0u;
        if (len >= 0) {
            nw = ((uint32_t)len + 31u) / 32u;
            each = 2u * ((nw + 31u) / 32u + (uint32_t)(warm_bytes(P.desc[d].n_states, 224) / 32));
        }
        uint32_t all = 0u, sum = nw;
        for (uint32_t j = 0; j < mine; ++j) {
            const uint32_t x = __shfl_sync(FULL, nw, (int)j), y = __shfl_sync(FULL, each, (int)j);
            all += y;
            sum += x > nw ? y : 0u;
        }
        const uint32_t least = __reduce_min_sync(FULL, len >= 0 ? sum : 0xffffffffu);
        const uint32_t most = least > all ? 0u : __reduce_max_sync(FULL, len >= 0 && sum == least ? nw : 0u);
        const bool alone = len >= 0 && nw <= most;
        uint32_t lanes = __ballot_sync(FULL, alone), left = __ballot_sync(FULL, len >= 0 && !alone);
        int open = -1;   // an automaton whose lanes did not agree
        while (left) {
            const int l = __ffs(left) - 1;
            left &= left - 1u;
            const int sa = __shfl_sync(FULL, a, l), sl = __shfl_sync(FULL, len, l), sd = __shfl_sync(FULL, d, l);
            const DfaDesc &D = P.desc[sd];
            const bool lone = (mine > 1u && sl <= kSmallLane) || D.n_states > kSmallDfaStates;
            const uint32_t s = lone && sd == open ? kSmallOpen
                                                  : small_warp(map_of(D), (uint32_t)D.n_states, small_view(P, sa, sa + sl),
                                                               (uint32_t)D.start, lone);
            if (s == kSmallOpen) {
                open = sd;
                lanes |= 1u << l;
            } else if (lane == 0) {
                write_result(P, base + warps * (uint32_t)l, s, D.accept_off);
            }
        }
        if ((lanes >> lane) & 1u) {
            const DfaDesc &D = P.desc[d];
            const SmallView v = small_view(P, a, a + len);
            const uint32_t s = small_walk(map_of(D), v.lo, v.hi, v.w, 0u, len ? v.nw : 0u, 0xffffffffu,
                                          (uint32_t)D.start) & 0xffu;
            write_result(P, i, s, D.accept_off);
        }
        __syncwarp();
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
        uint32_t r = small_piece(map_of(D), N, v, j * kSmallPieceWindows, min(v.nw, (j + 1u) * kSmallPieceWindows),
                                 start, -1, s_map);
        if (k == 1u) {
            if (threadIdx.x == 0)
                write_result(P, (uint32_t)i, r == kSmallIsMap ? (uint32_t)s_map[start] : r & 0xffu, D.accept_off);
            __syncthreads();
            continue;
        }
        uint32_t *const rs = rec + (p - j);
        uint8_t *const ms = maps + 256 * (size_t)(p - j);
        if (r == kSmallIsMap && threadIdx.x < N)
            *(volatile uint8_t *)(ms + 256 * (size_t)j + threadIdx.x) = (uint8_t)s_map[threadIdx.x];
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) {
            *(volatile uint32_t *)(rs + j) = r;
            __threadfence();
            s_last = atomicAdd(cnt + (p / pieces) * n_long + x, 1u) + 1u == k;
            __threadfence();
        }
        __syncthreads();
        if (!s_last) continue;
        // every piece is recorded: chain them
        for (uint32_t l = threadIdx.x; l < k; l += kSmallThreads) s_rec[l] = *(volatile uint32_t *)(rs + l);
        __syncthreads();
        uint32_t s = start;
        for (uint32_t l = 0; l < k; ++l) {
            const uint32_t w = s_rec[l];
            if (w & kSmallIsMap) {
                s = *(volatile uint8_t *)(ms + 256 * (size_t)l + s);
            } else if ((w >> 8) == s) {
                s = w & 0xffu;
            } else {   // a wrong guess: the piece again from its true state
                const uint32_t again = small_piece(map_of(D), N, v, l * kSmallPieceWindows,
                                                   min(v.nw, (l + 1u) * kSmallPieceWindows), start, (int)s, s_map);
                s = again == kSmallIsMap ? (uint32_t)s_map[s] : again & 0xffu;
                __syncthreads();
            }
        }
        if (threadIdx.x == 0) write_result(P, (uint32_t)i, s, D.accept_off);
        __syncthreads();
    }
}

}  // namespace trex
