// Tensor-core forms of the 64-state NFA for alphabets of up to 28 symbols: every
// warp keeps one symbol's table in its registers and the strings come to it
// (included by pnfa.cu).
//
// s' = T[c] s needs the strings of one MMA to share a symbol. Here the 64 x 64
// table of a symbol is a warp's A operand (mma.sync m16n8k16: 64 registers a
// thread; m16n8k32 for int8: 32), loaded once for the whole launch; the states
// stay in shared memory, a row a slot, and all strings of the CTA advance one
// symbol a step. A step's strings are in lists by symbol: the symbol's warp takes
// eight strings of its list at a time as the N = 8 columns of 16 MMAs (8 for
// int8), rounds the results into the strings' rows and appends each string to the
// next step's list of the symbol it reads next. One barrier of all warps
// separates the steps; nothing is sorted, planned or staged. Every 16 steps
// (a block) each slot's thread takes the next 16 symbols of its string, writes
// the result of a string that ended and gives its slot the next string.
//
// Bound by the chain of a group's dependent steps (list entry, state row, MMAs, rounding, store,
// append) with five warps a scheduler to hide it: 65536 strings x 2048 symbols, 20 symbols, BF16
// take 7.03 ms, of which the MMAs' issue (2 cycles each on an SM) is 1.9 ms. tcgen05.mma needs 128
// rows of A, two symbols' tables, throws half of every product away and brings it back through
// TMEM: that form, with a step's strings sorted by symbol pair, took 20.65 ms. With mbarriers
// between the warps of a symbol instead of one barrier a step it took 12.1 ms: a warp that polls takes
// issue slots and the shared-memory pipe from those that work.
#pragma once

namespace trex {

constexpr int kSyWarps = 20;            // 5 a scheduler: 96 registers a thread
constexpr int kSyThreads = 32 * kSyWarps;
constexpr int kSyMaxSigma = 28;
constexpr int kSyMaxSlots = 512;        // a thread keeps one or two (11 to 15 symbols launch fewer threads)
constexpr int kSyBlk = 16;              // steps a block
constexpr uint32_t kSyEnd = 0xFFu;      // symbol after a string's last
// a slot: free, walking a string, or its string ended and the result is to be written
enum : uint32_t { kSlFree = 0u, kSlLive = 1u, kSlEnded = 2u };

struct SyParams {
    const uint8_t *data;
    int64_t total_bytes;
    const int64_t *offsets;
    int64_t n;
    const uint16_t *T16;   // [sigma][64][64] row-major in the operand type (probabilistic forms)
    const float *T32;      // [sigma][64][64] (Boolean forms: a nonzero entry is an edge)
    const uint4 *start_img;   // start vector in the operand type, a state row
    const float *acc;         // [64] accept weights
    const float *rsym;        // [sigma] growth bound a symbol
    float start_max;
    int sigma, rep;           // rep warps a symbol take alternate groups of its list
    int slots, cap_shift;     // slots a CTA; log2 of a list's entries
    int resc;                 // steps between rescales, 1 or 4 (power-of-two scaling is exact, so only the
                              // range matters: 4 for BF16 with growth <= 16 a step, else 1)
    uint32_t state_off, sym_off, raw_off, list_off, rows_off;
    long long wait_cycles;
    double ll_empty;
    double *loglik;
    uint8_t *accept;
    int32_t *accept_i32;
    unsigned long long *queue;
    uint32_t *err;
};

// A slot's string.
struct alignas(16) SyRec {
    const uint8_t *p, *e;   // next byte, end of the string
    int32_t E;              // exponent sum
    float m;                // max |s| (left for a rescale)
    int32_t seq;
    float dot;              // accept-weighted sum of an ended string
};

// Shared memory: control words; records [slots]; uint8 state of a slot [slots]; symbols [2
// blocks][16][slots]; raw bytes [slots][32]; lists uint16 [2][sigma][1 << cap_shift]; state rows.
constexpr uint32_t kSyLive = 0, kSyLate = 8;   // uint32 [2] each (parity of the block, of the meeting)
constexpr uint32_t kSyCnt = 32;                              // uint32 [3][32]: list lengths
constexpr uint32_t kSyAcc = kSyCnt + 3 * 128;                // float [64]
constexpr uint32_t kSyStart = kSyAcc + 256;                  // uint4 [8]
constexpr uint32_t kSyRecs = kSyStart + 128;
// bytes between state rows: 16 more than a row, so that rows of any slots spread over the banks
template <int KIND>
__host__ __device__ constexpr uint32_t sy_row_bytes() { return KIND == 2 ? 64u + 16u : 128u + 16u; }

// ---- shared memory by byte offset
extern __shared__ __align__(16) uint8_t sy_smem[];
template <class T>
__device__ __forceinline__ T &sy_at(uint32_t off) {
    return *reinterpret_cast<T *>(sy_smem + off);
}
__device__ __forceinline__ uint32_t sy_umax2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("max.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

// d = a b + c
template <int KIND>
__device__ __forceinline__ void sy_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1,
                                       float c0, float c1, float c2, float c3) {
    if constexpr (KIND == 2) {
        int32_t i[4];
        asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
            : "=r"(i[0]), "=r"(i[1]), "=r"(i[2]), "=r"(i[3])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(__float_as_int(c0)),
              "r"(__float_as_int(c1)), "r"(__float_as_int(c2)), "r"(__float_as_int(c3)));
#pragma unroll
        for (int k = 0; k < 4; ++k) d[k] = __int_as_float(i[k]);
    } else if constexpr (KIND == 1) {
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
            : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
    } else {
        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
            : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c0), "f"(c1), "f"(c2), "f"(c3));
    }
}
// The table times the eight columns, K tiles [k0, k0 + NK): b holds their states.
template <int KIND, int K0, int NK>
__device__ __forceinline__ void sy_tiles(float (&d)[4][4], const uint32_t (&a)[4][KIND == 2 ? 2 : 4][4], const uint4 b) {
    const uint32_t w[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int k = 0; k < NK; ++k)
#pragma unroll
        for (int mt = 0; mt < 4; ++mt) {
            if (K0 + k == 0) sy_mma<KIND>(d[mt], a[mt][0], w[0], w[1], 0.f, 0.f, 0.f, 0.f);
            else sy_mma<KIND>(d[mt], a[mt][K0 + k], w[2 * k], w[2 * k + 1], d[mt][0], d[mt][1], d[mt][2], d[mt][3]);
        }
}

// All warps of the CTA meet (meeting k of the launch); false for all of them when the meeting
// before took some warp longer than the wait limit (the error bit is set). Flags of alternate
// meetings, so that every warp reads the same value: a flag is set after meeting k - 1 and read
// after meeting k. A hardware barrier: a warp that polls an mbarrier takes the shared-memory
// pipe from the warps it waits for, one parked on it wakes thousands of cycles late.
__device__ __forceinline__ bool sy_meet(const SyParams &P, uint32_t k) {
    const long long t0 = clock64();
    __syncthreads();
    const bool go = sy_at<volatile uint32_t>(kSyLate + 4u * ((k & 1u) ^ 1u)) == 0u;
    if (clock64() - t0 > P.wait_cycles) {
        sy_at<volatile uint32_t>(kSyLate + 4u * (k & 1u)) = 1u;
        if ((threadIdx.x & 31u) == 0u) atomicOr(P.err, kPnErrTimeout);
    }
    return go;
}

// ---- a slot's string (by the slot's thread) ----------------------------------------------------
__device__ __forceinline__ SyRec &sy_rec(uint32_t slot) { return sy_at<SyRec>(kSyRecs + 32u * slot); }

// The 32 aligned bytes around p (the 16 at p lie in them) into the slot's raw buffer; bytes
// outside the batch are not read. ASYNC: with cp.async where the 16-byte pieces lie inside it.
template <bool ASYNC>
__device__ __forceinline__ void sy_fetch(const SyParams &P, uint32_t slot, const uint8_t *p, const uint8_t *e) {
    const uint8_t *a = reinterpret_cast<const uint8_t *>(reinterpret_cast<uintptr_t>(p) & ~(uintptr_t)15);
    const uint8_t *const hi = P.data + P.total_bytes;
    const uint32_t dst = P.raw_off + 32u * slot;
#pragma unroll
    for (int k = 0; k < 2; ++k, a += 16) {
        if (a >= e) break;
        if (a >= P.data && a + 16 <= hi) {
            if constexpr (ASYNC)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" :: "r"(pn_smem_u32(sy_smem + dst + 16u * k)), "l"(a)
                             : "memory");
            else
                sy_at<uint4>(dst + 16u * k) = __ldg(reinterpret_cast<const uint4 *>(a));
        } else {
            for (int j = 0; j < 16; ++j)
                if (a + j >= P.data && a + j < hi) sy_at<uint8_t>(dst + 16u * k + j) = __ldg(a + j);
        }
    }
}

// The next 16 symbols of a slot's string from its raw buffer (which holds the bytes at p) into
// block half `half` of the symbol buffer; kSyEnd after the last. Bytes >= sigma are skipped.
// Returns the first symbol and moves p.
__device__ __forceinline__ uint32_t sy_symbols(const SyParams &P, uint32_t slot, uint32_t half, const uint8_t *&p,
                                               const uint8_t *e) {
    const uint32_t dst = P.sym_off + half * (uint32_t)(kSyBlk * P.slots) + slot;
    const uint32_t stride = (uint32_t)P.slots;
    const int left = (int)min((int64_t)kSyBlk, (int64_t)(e - p));
    const uint32_t at = (uint32_t)(reinterpret_cast<uintptr_t>(p) & 15u);
    const uint32_t src = P.raw_off + 32u * slot + (at & ~3u);
    uint32_t w[4], bad = 0u;
    {
        uint32_t x = sy_at<uint32_t>(src);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t y = k < 3 || (at & 3u) ? sy_at<uint32_t>(src + 4u * (k + 1)) : 0u;
            w[k] = __funnelshift_r(x, y, (at & 3u) * 8u);
            x = y;
            // bytes past the end count as the end symbol
            const int in = left - 4 * k;
            const uint32_t keep = in >= 4 ? 0xFFFFFFFFu : in <= 0 ? 0u : (1u << (8 * in)) - 1u;
            bad |= __vcmpgeu4(w[k], (uint32_t)P.sigma * 0x01010101u) & keep;
            w[k] |= ~keep;
        }
    }
    if (bad == 0u) {
#pragma unroll
        for (int j = 0; j < kSyBlk; ++j) sy_at<uint8_t>(dst + j * stride) = (uint8_t)(w[j >> 2] >> (8 * (j & 3)));
        p += left;
        return w[0] & 0xFFu;
    }
    int count = 0;
    uint32_t first = kSyEnd;
    while (count < kSyBlk && p < e) {
        const uint32_t c = __ldg(p++);
        if (c >= (uint32_t)P.sigma) continue;
        if (count == 0) first = c;
        sy_at<uint8_t>(dst + count * stride) = (uint8_t)c;
        ++count;
    }
    for (; count < kSyBlk; ++count) sy_at<uint8_t>(dst + count * stride) = (uint8_t)kSyEnd;
    return first;
}

// Appends a slot to the list of symbol c (cnt: the lengths of that step's lists).
__device__ __forceinline__ void sy_append(const SyParams &P, uint32_t cnt, uint32_t list, uint32_t c, uint32_t slot) {
    const uint32_t pos = atomicAdd(&sy_at<uint32_t>(cnt + 4u * c), 1u);
    sy_at<uint16_t>(list + 2u * ((c << P.cap_shift) + pos)) = (uint16_t)slot;
}

// Start of block b, by the slot's thread: the result of a string that ended; then the symbols of
// block b + 1 for a string that goes on, or the next string with the symbols of blocks b and
// b + 1. Returns whether the slot holds a string. Not inlined: the tables stay in registers.
template <int KIND>
__device__ __noinline__ bool sy_block(const SyParams &P, uint32_t slot, uint32_t b, uint32_t cnt, uint32_t list) {
    SyRec &S = sy_rec(slot);
    uint8_t &state = sy_at<uint8_t>(P.state_off + slot);
    asm volatile("cp.async.wait_all;" ::: "memory");   // this thread's own copies
    if (state == kSlLive) {
        const uint8_t *p = S.p, *const e = S.e;
        sy_symbols(P, slot, (b + 1u) & 1u, p, e);
        S.p = p;
        sy_fetch<true>(P, slot, p, e);
        return true;
    }
    if (state == kSlEnded) {
        const double dot = (double)S.dot;
        pn_write_result(P.loglik, P.accept, P.accept_i32, (int64_t)S.seq,
                        dot > 0.0 ? log(dot) + (double)S.E * 0.69314718055994530942 : -INFINITY);
        state = kSlFree;
    }
    for (;;) {
        // (a look first: free slots do not count the queue on for ever)
        if (*reinterpret_cast<volatile unsigned long long *>(P.queue) >= (unsigned long long)P.n) return false;
        const unsigned long long idx = atomicAdd(P.queue, 1ull);
        if (idx >= (unsigned long long)P.n) return false;
        const int64_t p0 = P.offsets[idx], p1 = P.offsets[idx + 1];
        if (p0 < 0 || p1 < p0 || p1 > P.total_bytes) {
            atomicOr(P.err, kPnErrOffsets);
            continue;
        }
        const uint8_t *p = P.data + p0, *const e = P.data + p1;
        sy_fetch<false>(P, slot, p, e);
        const uint32_t c = sy_symbols(P, slot, b & 1u, p, e);
        if (c == kSyEnd) {
            pn_write_result(P.loglik, P.accept, P.accept_i32, (int64_t)idx, P.ll_empty);
            continue;
        }
        sy_fetch<false>(P, slot, p, e);
        sy_symbols(P, slot, (b + 1u) & 1u, p, e);
        sy_fetch<true>(P, slot, p, e);
        S.p = p;
        S.e = e;
        S.E = 0;
        S.m = P.start_max;
        S.seq = (int32_t)idx;
        state = kSlLive;
        const uint32_t row = P.rows_off + slot * sy_row_bytes<KIND>();
        for (uint32_t k = 0; k < sy_row_bytes<KIND>() - 16u; k += 16u) sy_at<uint4>(row + k) = sy_at<uint4>(kSyStart + k);
        sy_append(P, cnt, list, c, slot);
        return true;
    }
}

// The A operand of symbol c: row 16 mt + 8 h + r of the MMA is destination state 8 r + 2 mt + h
// (so that a thread's results of one string are eight adjacent states), K position
// 16 kt + 8 hk + 2 q + i source state 16 q + 4 kt + 2 hk + i (so that a thread's B operand is
// sixteen adjacent states); int8: 32 kt + 16 hk + 4 q + i is 16 q + 8 kt + 4 hk + i.
template <int KIND>
__device__ __forceinline__ void sy_load_table(const SyParams &P, int c,
                                              uint32_t (&a)[4][KIND == 2 ? 2 : 4][4]) {
    const int lane = threadIdx.x & 31, r = lane >> 2, q = lane & 3;
#pragma unroll
    for (int mt = 0; mt < 4; ++mt)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const size_t o = ((size_t)c * 64 + 8 * r + 2 * mt + h) * 64 + 16 * q;
            if constexpr (KIND >= 2) {
#pragma unroll
                for (int w = 0; w < (KIND == 2 ? 4 : 8); ++w) {
                    uint32_t x = 0u;
                    if constexpr (KIND == 2) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) x |= (__ldg(P.T32 + o + 4 * w + i) != 0.f ? 1u : 0u) << (8 * i);
                    } else {
                        x = (__ldg(P.T32 + o + 2 * w) != 0.f ? 0x3F80u : 0u) |
                            (__ldg(P.T32 + o + 2 * w + 1) != 0.f ? 0x3F800000u : 0u);
                    }
                    a[mt][w >> 1][h + 2 * (w & 1)] = x;
                }
            } else {
                const uint4 *src = reinterpret_cast<const uint4 *>(P.T16 + o);
                const uint4 u = __ldg(src), v = __ldg(src + 1);
                const uint32_t w[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
#pragma unroll
                for (int k = 0; k < 8; ++k) a[mt][k >> 1][h + 2 * (k & 1)] = w[k];
            }
        }
}

// Up to eight strings of a list (entries at `ent`, nv of them) one step on: t the step, R the
// growth bound of their symbol. SCALE: this step rescales by the maxima that the step before
// left; MAX: this step leaves them. Columns past the group repeat its last string (the same
// values are written again). Beside the table's 64 registers there is room for the sixteen
// results and one half of the states, so everything else is read from shared memory when it is
// needed.
template <int KIND, bool SCALE, bool MAX>
__device__ __forceinline__ void sy_group(const SyParams &P, const uint32_t (&a)[4][KIND == 2 ? 2 : 4][4], uint32_t ent,
                                         uint32_t nv, float R, uint32_t t) {
    constexpr bool I8 = KIND == 2, BOOL = KIND >= 2, FP16 = KIND == 1;
    constexpr uint32_t ROW = sy_row_bytes<KIND>();
    const uint32_t FULL = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u, r = lane >> 2, q = lane & 3u;
    float d[4][4];
    {
        // B: sixteen states of column r
        const uint32_t row = P.rows_off + (uint32_t)sy_at<uint16_t>(ent + 2u * min(r, nv - 1u)) * ROW + (I8 ? 16u : 32u) * q;
        if constexpr (I8) {
            sy_tiles<KIND, 0, 2>(d, a, sy_at<uint4>(row));
        } else {
            const uint4 u = sy_at<uint4>(row);
            sy_tiles<KIND, 0, 2>(d, a, u);
            const uint4 v = sy_at<uint4>(row + 16u);
            sy_tiles<KIND, 2, 2>(d, a, v);
        }
    }
    // this lane's results: states 8r .. 8r + 7 of columns 2q and 2q + 1
    const uint32_t slot0 = sy_at<uint16_t>(ent + 2u * min(2u * q, nv - 1u));
    const uint32_t slot1 = sy_at<uint16_t>(ent + 2u * min(2u * q + 1u, nv - 1u));
    // lanes 0-7 keep string 2q + (r & 1) of the group: its next symbol
    const bool own = lane < 8u && 2u * q + (r & 1u) < nv;
    const uint32_t slot = (r & 1u) ? slot1 : slot0;
    const uint32_t nc = sy_at<uint8_t>(P.sym_off + ((t + 1u) % (2u * kSyBlk)) * (uint32_t)P.slots + slot);
    if constexpr (BOOL) {
#pragma unroll
        for (int mt = 0; mt < 4; ++mt)
#pragma unroll
            for (int i = 0; i < 4; ++i)
                d[mt][i] = (I8 ? __float_as_int(d[mt][i]) != 0 : d[mt][i] > 0.f) ? 1.f : 0.f;
    } else if constexpr (SCALE) {
        // 2^-f for each column (exact), f the exponent of max |s| R
        const int f0 = min(max(pn_ceil_exp(sy_rec(slot0).m * R), -125), 125);
        const int f1 = min(max(pn_ceil_exp(sy_rec(slot1).m * R), -125), 125);
        const float s0 = pn_pow2(-f0), s1 = pn_pow2(-f1);
#pragma unroll
        for (int mt = 0; mt < 4; ++mt) {
            d[mt][0] *= s0;
            d[mt][2] *= s0;
            d[mt][1] *= s1;
            d[mt][3] *= s1;
        }
        __syncwarp();   // (the maxima are read before MAX writes the next ones)
        if (own) sy_rec(slot).E += (r & 1u) ? f1 : f0;
    }
    if (__any_sync(FULL, nc == kSyEnd)) {   // a string's last symbol: the accept-weighted sum of its state
        float dot0 = 0.f, dot1 = 0.f;
#pragma unroll
        for (int mt = 0; mt < 4; ++mt) {
            const float2 w = sy_at<float2>(kSyAcc + 4u * (8u * r + 2u * mt));
            dot0 = fmaf(w.x, d[mt][0], dot0);
            dot0 = fmaf(w.y, d[mt][2], dot0);
            dot1 = fmaf(w.x, d[mt][1], dot1);
            dot1 = fmaf(w.y, d[mt][3], dot1);
        }
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) {
            dot0 += __shfl_xor_sync(FULL, dot0, o);
            dot1 += __shfl_xor_sync(FULL, dot1, o);
        }
        if (own && nc == kSyEnd) {
            sy_rec(slot).dot = (r & 1u) ? dot1 : dot0;
            sy_at<uint8_t>(P.state_off + slot) = (uint8_t)kSlEnded;
        }
    }
    uint32_t x0[4], x1[4];
#pragma unroll
    for (int mt = 0; mt < 4; ++mt) {
        if constexpr (I8) {
            x0[mt] = (d[mt][0] != 0.f ? 1u : 0u) | (d[mt][2] != 0.f ? 0x100u : 0u);
            x1[mt] = (d[mt][1] != 0.f ? 1u : 0u) | (d[mt][3] != 0.f ? 0x100u : 0u);
        } else {
            x0[mt] = pn_pack2<FP16>(d[mt][0], d[mt][2]);
            x1[mt] = pn_pack2<FP16>(d[mt][1], d[mt][3]);
        }
    }
    // (every lane has read its column: the products need all lanes' states)
    if constexpr (I8) {
        sy_at<uint2>(P.rows_off + slot0 * ROW + 8u * r) = make_uint2(x0[0] | (x0[1] << 16), x0[2] | (x0[3] << 16));
        sy_at<uint2>(P.rows_off + slot1 * ROW + 8u * r) = make_uint2(x1[0] | (x1[1] << 16), x1[2] | (x1[3] << 16));
    } else {
        sy_at<uint4>(P.rows_off + slot0 * ROW + 16u * r) = make_uint4(x0[0], x0[1], x0[2], x0[3]);
        sy_at<uint4>(P.rows_off + slot1 * ROW + 16u * r) = make_uint4(x1[0], x1[1], x1[2], x1[3]);
    }
    if constexpr (MAX) {
        // max |s| of the rounded states: |x| of 16-bit floats orders like the integer of its low
        // 15 bits; both columns in one register
        constexpr uint32_t ABS = 0x7FFF7FFFu;
        const uint32_t m0 = sy_umax2(sy_umax2(x0[0] & ABS, x0[1] & ABS), sy_umax2(x0[2] & ABS, x0[3] & ABS));
        const uint32_t m1 = sy_umax2(sy_umax2(x1[0] & ABS, x1[1] & ABS), sy_umax2(x1[2] & ABS, x1[3] & ABS));
        uint32_t m2 = sy_umax2(__byte_perm(m0, m1, 0x5410), __byte_perm(m0, m1, 0x7632));
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) m2 = sy_umax2(m2, __shfl_xor_sync(FULL, m2, o));
        const uint32_t mh = (r & 1u) ? m2 >> 16 : m2 & 0xFFFFu;
        if (own) sy_rec(slot).m = FP16 ? __half2float(__ushort_as_half((unsigned short)mh)) : __uint_as_float(mh << 16);
    }
    if (own && nc != kSyEnd)
        sy_append(P, kSyCnt + 128u * ((t + 1u) % 3u), P.list_off + ((t + 1u) & 1u) * ((2u << P.cap_shift) * (uint32_t)P.sigma),
                  nc, slot);
}

// A warp's groups of step t; mine: its symbol, and the first group it takes of the symbol's list
// (in the upper half).
template <int KIND, bool RELOAD, bool SCALE, bool MAX>
__device__ __forceinline__ void sy_groups(const SyParams &P, uint32_t (&a)[4][KIND == 2 ? 2 : 4][4], uint32_t t,
                                          uint32_t mine) {
    for (uint32_t c = mine & 0xFFFFu; c < (uint32_t)P.sigma; c += blockDim.x >> 5) {
        int n = (int)sy_at<uint32_t>(kSyCnt + 128u * (t % 3u) + 4u * c);
        if (RELOAD && n != 0) sy_load_table<KIND>(P, (int)c, a);
        const float R = SCALE ? __ldg(P.rsym + c) : 0.f;
        const uint32_t first = RELOAD ? 0u : mine >> 16, step = RELOAD ? 8u : 8u * (uint32_t)P.rep;
        uint32_t ent = P.list_off + (2u << P.cap_shift) * ((t & 1u) * (uint32_t)P.sigma + c) + 2u * first;
        for (n -= (int)first; n > 0; n -= (int)step, ent += 2u * step)
            sy_group<KIND, SCALE, MAX>(P, a, ent, (uint32_t)min(8, n), R, t);
        if (!RELOAD) break;
    }
}

// SEVERAL: alphabets of more symbols than warps. Two int8 tables take the registers of one in 16
// bits, so a warp keeps both (8192 strings x 512, 20 / 21 / 28 symbols: 0.53 / 0.83 / 0.91 ms; loading
// each table at every step, 12.0 / 14.5 for 21 / 28); in the 16-bit forms it loads its symbols' tables in
// turn at every step (BF16 0.73 / 2.09 / 2.35, FP16 0.84 / 2.14 / 2.41).
template <int KIND, bool SEVERAL>
__global__ void __launch_bounds__(kSyThreads, 1) pnfa_sym_kernel(const __grid_constant__ SyParams P) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    for (uint32_t i = threadIdx.x; i < kSyAcc / 4; i += blockDim.x) sy_at<uint32_t>(4u * i) = 0u;
    for (uint32_t i = threadIdx.x; i < 64u; i += blockDim.x) sy_at<float>(kSyAcc + 4u * i) = P.acc[i];
    if (threadIdx.x < 8) sy_at<uint4>(kSyStart + 16u * threadIdx.x) = P.start_img[threadIdx.x];
    for (uint32_t s = threadIdx.x; s < (uint32_t)P.slots; s += blockDim.x) sy_at<uint8_t>(P.state_off + s) = (uint8_t)kSlFree;
    __syncthreads();
    constexpr bool BOTH = SEVERAL && KIND == 2, RELOAD = SEVERAL && !BOTH;
    uint32_t a[4][KIND == 2 ? 2 : 4][4], a2[4][KIND == 2 ? 2 : 4][4];   // (a2: with BOTH)
    const uint32_t mine = warp % (uint32_t)P.sigma | ((8u * (warp / (uint32_t)P.sigma)) << 16);
    if (!RELOAD) sy_load_table<KIND>(P, (int)(mine & 0xFFFFu), a);
    if (BOTH && warp + kSyWarps < (uint32_t)P.sigma) sy_load_table<KIND>(P, (int)(warp + kSyWarps), a2);
    for (uint32_t t = 0;; ++t) {
        // meetings before this step's: one a step and one a block
        if (t % kSyBlk == 0u) {
            const uint32_t blk = t / kSyBlk, live = kSyLive + 4u * (blk & 1u);
            bool has = false;
            for (uint32_t s = threadIdx.x; s < (uint32_t)P.slots; s += blockDim.x)
                has |= sy_block<KIND>(P, s, blk, kSyCnt + 128u * (t % 3u),
                                      P.list_off + (t & 1u) * ((2u << P.cap_shift) * (uint32_t)P.sigma));
            if (__any_sync(0xffffffffu, has) && lane == 0u) sy_at<volatile uint32_t>(live) = 1u;
            if (!sy_meet(P, t + blk)) break;
            if (sy_at<volatile uint32_t>(live) == 0u) break;
            // (the other parity's flag was last read before the previous block's steps)
            if (threadIdx.x == 0) sy_at<volatile uint32_t>(kSyLive + 4u * ((blk & 1u) ^ 1u)) = 0u;
        }
        // (the lengths of the step after the next: read by nobody in this step)
        if (threadIdx.x < 32u) sy_at<uint32_t>(kSyCnt + 128u * ((t + 2u) % 3u) + 4u * lane) = 0u;
        if (KIND >= 2) {
            sy_groups<KIND, RELOAD, false, false>(P, a, t, mine);
            if constexpr (BOTH) sy_groups<KIND, false, false, false>(P, a2, t, warp + kSyWarps);
        } else if (P.resc == 1) {
            sy_groups<KIND, RELOAD, true, true>(P, a, t, mine);
        } else {
            const uint32_t x = t & (uint32_t)(P.resc - 1);
            if (x == 0u) sy_groups<KIND, RELOAD, true, false>(P, a, t, mine);
            else if (x + 1u == (uint32_t)P.resc) sy_groups<KIND, RELOAD, false, true>(P, a, t, mine);
            else sy_groups<KIND, RELOAD, false, false>(P, a, t, mine);
        }
        if (!sy_meet(P, t + t / kSyBlk + 1u)) break;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
}

}  // namespace trex
