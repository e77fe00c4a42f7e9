// FP32 form of the 64-state NFA for alphabets of up to 20 symbols: every warp keeps one
// symbol's table on the SM and the strings come to it (included by pnfa.cu).
//
// The plain kernel (a warp a string, the table of every symbol read through L1 for every
// string) is bound by those reads: 16 KB a symbol, each row's piece from another line. Here a
// warp owns a symbol: six of the sixteen four-column pieces of its FP32 table in registers (48
// a thread: rows `lane` and `lane` + 32), the rest in shared memory, so that 20 tables (320 KB)
// fit on an SM, and reads them once for up to four strings. The states stay in shared memory,
// a row a slot. A string waits in the ring of its next symbol; the symbol's warp takes up to
// four strings of its ring, writes their next states and puts each in the ring of the symbol it
// reads next. Slots of ended strings go to one more ring, whose entries a warp without work
// turns into log-likelihoods and refills with the next strings of the batch. No step is common
// to all strings, so there are no barriers and no sorting. The products of a row are added in
// the plain kernel's order, k = 0 .. 63, and the state is rescaled by the exponent of max |s'|
// at every step, as there: the states are the same bits.
//
// 8192 strings x 512, 20 symbols: 16.7 -> 1.72 ms (0.26 -> 2.4 Gchar/s), the shared-memory pipe
// 83% busy (80 wavefronts of table a group, 16 of states a string).
#pragma once

namespace trex {

constexpr int kRiWarps = 20;            // 5 a scheduler: 96 registers a thread
constexpr int kRiThreads = 32 * kRiWarps;
constexpr int kRiMaxSlots = 512;
constexpr uint32_t kRiNone = 0xFFFFu;
constexpr int kRiReg = 6, kRiGroup = 4;
constexpr uint32_t kRiTblBytes = (16 - kRiReg) * 64 * 16;   // a symbol's part in shared memory
constexpr uint32_t kRiRowBytes = 256 + 16;   // a state row; 16 more, so that rows spread over the banks

// Record of a slot's string, 32 bytes of shared memory: next byte to read, end of the string
// (addresses), exponent sum (64 bits), string index, accept-weighted sum of an ended string.
constexpr uint32_t kRiRecBytes = 32, kRiRecP = 0, kRiRecE = 16, kRiRecDot = 28;

struct RiParams {
    const uint8_t *data;
    int64_t total_bytes;
    const int64_t *offsets;
    int64_t n;
    const float *T32;         // [sigma][64][64]
    const uint4 *start_img;   // [64] start vector, a state row
    const float *acc;         // [64] accept weights
    int sigma, rep, n_rings;  // rep rings a symbol: ring c + sigma * (slot * rep >> rep_shift)
    int grid, slots, ring_cap, rep_shift;
    uint32_t recs_off, rows_off, tbl_off;
    long long wait_cycles;
    double ll_empty;
    double *loglik;
    uint8_t *accept;
    int32_t *accept_i32;
    unsigned long long *queue;
    uint32_t *err;
};

// Shared memory: control words, rings (n_rings, then that of ended slots), records, state rows,
// tables.
constexpr uint32_t kRiTails = 0;                        // uint32 [kRiWarps + 1]
constexpr uint32_t kRiBusy = 4 * (kRiWarps + 1);        // lanes that look for a string or skip its bytes
constexpr uint32_t kRiEndHead = 128, kRiLock = 132, kRiLive = 136, kRiDone = 140;
constexpr uint32_t kRiAcc = 144;                        // float [64]
constexpr uint32_t kRiStart = kRiAcc + 256;             // uint4 [16]
constexpr uint32_t kRiRings = kRiStart + 256;           // uint16 [n_rings + 1][ring_cap]

// ---- 32-bit shared addresses (a generic pointer would take two registers)
extern __shared__ __align__(16) uint8_t ri_smem[];
__device__ __forceinline__ uint32_t ri_base() { return pn_smem_u32(ri_smem); }
__device__ __forceinline__ uint32_t ri_ld32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t ri_ld16(uint32_t a) {
    uint16_t v;
    asm volatile("ld.volatile.shared.u16 %0, [%1];" : "=h"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint2 ri_ld64(uint32_t a) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ uint4 ri_ld128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void ri_ldp(uint32_t a, const uint8_t *&p, const uint8_t *&e) {
    asm volatile("ld.shared.v2.u64 {%0,%1}, [%2];" : "=l"(p), "=l"(e) : "r"(a) : "memory");
}
__device__ __forceinline__ void ri_stp(uint32_t a, const uint8_t *p) {
    asm volatile("st.shared.u64 [%0], %1;" :: "r"(a), "l"(p) : "memory");
}
__device__ __forceinline__ void ri_st16(uint32_t a, uint32_t v) {
    asm volatile("st.volatile.shared.u16 [%0], %1;" :: "r"(a), "h"((uint16_t)v) : "memory");
}
__device__ __forceinline__ void ri_st32(uint32_t a, uint32_t v) {
    asm volatile("st.volatile.shared.u32 [%0], %1;" :: "r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void ri_st64(uint32_t a, uint32_t x, uint32_t y) {
    asm volatile("st.shared.v2.u32 [%0], {%1,%2};" :: "r"(a), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void ri_st128(uint32_t a, uint4 v) {
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" :: "r"(a), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ uint32_t ri_add32(uint32_t a, uint32_t v) {
    uint32_t o;
    asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(o) : "r"(a), "r"(v) : "memory");
    return o;
}
__device__ __forceinline__ void ri_fence() { asm volatile("fence.acq_rel.cta;" ::: "memory"); }
// Address of entry `pos` of ring `ring`.
__device__ __forceinline__ uint32_t ri_entry(const RiParams &P, uint32_t ring, uint32_t pos) {
    return ri_base() + kRiRings + 2u * (ring * (uint32_t)P.ring_cap + (pos & (uint32_t)(P.ring_cap - 1)));
}
// The ring in which slot waits for symbol c.
__device__ __forceinline__ uint32_t ri_ring_of(const RiParams &P, uint32_t c, uint32_t slot) {
    return c + (uint32_t)P.sigma * ((slot * (uint32_t)P.rep) >> P.rep_shift);
}
// Puts a slot in a ring, after its row and record were written (by this thread, or by its warp
// before a __syncwarp): the fence makes them visible to the warp that finds the entry. A ring
// holds as many entries as there are slots and a slot is in one ring at a time, so an entry is
// read before its place is used again.
__device__ __forceinline__ void ri_push(const RiParams &P, uint32_t ring, uint32_t slot) {
    ri_fence();
    const uint32_t pos = ri_add32(ri_base() + kRiTails + 4u * ring, 1u);
    ri_st16(ri_entry(P, ring, pos), slot);
}
// The entries at the front of a ring: this lane's entry (lanes below `most`); returns how many.
__device__ __forceinline__ uint32_t ri_poll(const RiParams &P, uint32_t ring, uint32_t head, uint32_t most,
                                            uint32_t &ent) {
    const uint32_t lane = threadIdx.x & 31u;
    ent = kRiNone;
    if (lane < most) ent = ri_ld16(ri_entry(P, ring, head + lane));
    const uint32_t got = __ballot_sync(0xffffffffu, ent != kRiNone);
    return got == 0xffffffffu ? 32u : (uint32_t)__ffs(~got) - 1u;
}

// The first byte below sigma of [p, e), or e: four bytes at a time to a 64-byte line, then a line a
// step, so that a long run of skipped bytes does not take a round trip a byte.
__device__ __forceinline__ const uint8_t *ri_skip(const uint8_t *p, const uint8_t *e, uint32_t sigma) {
    const uint32_t sig4 = sigma * 0x01010101u;
    while (p < e && (reinterpret_cast<uintptr_t>(p) & 3u)) {
        if (__ldg(p) < sigma) return p;
        ++p;
    }
    while (e - p >= 4) {
        if ((reinterpret_cast<uintptr_t>(p) & 63u) == 0u) {
            for (; e - p >= 64; p += 64) {
                uint32_t in = 0u;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint4 v = __ldg(reinterpret_cast<const uint4 *>(p) + k);
                    in |= __vcmpltu4(v.x, sig4) | __vcmpltu4(v.y, sig4) | __vcmpltu4(v.z, sig4) | __vcmpltu4(v.w, sig4);
                }
                if (in) break;
            }
            if (e - p < 4) break;
        }
        const uint32_t in = __vcmpltu4(__ldg(reinterpret_cast<const uint32_t *>(p)), sig4);
        if (in) return p + ((__ffs(in) - 1) >> 3);
        p += 4;
    }
    while (p < e && __ldg(p) >= sigma) ++p;
    return p;
}

// Gives a slot the next string of the batch: its record, its start row and its first ring.
// Strings without symbols get their result at once; false when the batch has no more strings.
__device__ __forceinline__ bool ri_refill(const RiParams &P, uint32_t slot) {
    bool found = false;
    ri_add32(ri_base() + kRiBusy, 1u);
    for (;;) {
        const unsigned long long idx = atomicAdd(P.queue, 1ull);
        if (idx >= (unsigned long long)P.n) break;
        const int64_t p0 = P.offsets[idx], p1 = P.offsets[idx + 1];
        if (p0 < 0 || p1 < p0 || p1 > P.total_bytes) {
            atomicOr(P.err, kPnErrOffsets);
            continue;
        }
        const uint8_t *p = P.data + p0, *const e = P.data + p1;
        uint32_t c = p < e ? __ldg(p) : 255u;
        if (c >= (uint32_t)P.sigma && p < e && (p = ri_skip(p + 1, e, (uint32_t)P.sigma)) < e) c = __ldg(p);
        if (p == e) {
            pn_write_result(P.loglik, P.accept, P.accept_i32, (int64_t)idx, P.ll_empty);
            continue;
        }
        const uint32_t rec = ri_base() + P.recs_off + slot * kRiRecBytes;
        ri_stp(rec + kRiRecP, p + 1);
        ri_stp(rec + kRiRecP + 8u, e);
        ri_st128(rec + kRiRecE, make_uint4(0u, 0u, (uint32_t)idx, 0u));
        const uint32_t row = ri_base() + P.rows_off + slot * kRiRowBytes;
        for (uint32_t k = 0; k < kRiRowBytes - 16u; k += 16u) ri_st128(row + k, ri_ld128(ri_base() + kRiStart + k));
        ri_push(P, ri_ring_of(P, c, slot), slot);
        found = true;
        break;
    }
    ri_add32(ri_base() + kRiBusy, 0xffffffffu);
    return found;
}

// The ended slots, up to 32 at a time (the calling warp holds the lock): results, next strings.
// The last slot without a string ends the kernel's work.
__device__ __noinline__ void ri_feed(const RiParams &P) {
    const uint32_t FULL = 0xffffffffu, lane = threadIdx.x & 31u;
    const uint32_t head = ri_ld32(ri_base() + kRiEndHead);
    uint32_t slot;
    const uint32_t cnt = ri_poll(P, (uint32_t)P.n_rings, head, 32u, slot);
    bool retired = false;
    if (lane < cnt) {
        ri_fence();
        ri_st16(ri_entry(P, (uint32_t)P.n_rings, head + lane), kRiNone);
    }
    // every place is free before a slot goes on: its string can end and come back to one of them
    // (with as many slots as places)
    __syncwarp();
    if (lane < cnt) {
        const uint4 w = ri_ld128(ri_base() + P.recs_off + slot * kRiRecBytes + kRiRecE);
        const double dot = (double)__uint_as_float(w.w);
        const int64_t E = (int64_t)(((uint64_t)w.y << 32) | w.x);
        pn_write_result(P.loglik, P.accept, P.accept_i32, (int64_t)w.z,
                        dot > 0.0 ? log(dot) + (double)E * 0.69314718055994530942 : -INFINITY);
        retired = !ri_refill(P, slot);
    }
    const uint32_t gone = (uint32_t)__popc(__ballot_sync(FULL, retired));
    if (lane == 0) {
        ri_st32(ri_base() + kRiEndHead, head + cnt);
        if (gone && ri_add32(ri_base() + kRiLive, 0u - gone) == gone) ri_st32(ri_base() + kRiDone, 1u);
        ri_fence();
        ri_st32(ri_base() + kRiLock, 0u);
    }
    __syncwarp();
}
// Feeds when slots are waiting (at least `least`) and no other warp does.
__device__ __forceinline__ bool ri_try_feed(const RiParams &P, uint32_t least) {
    const uint32_t tail = ri_ld32(ri_base() + kRiTails + 4u * (uint32_t)P.n_rings);
    if (tail - ri_ld32(ri_base() + kRiEndHead) < least) return false;
    uint32_t got = 0u;
    if ((threadIdx.x & 31u) == 0u)
        asm volatile("atom.shared.cas.b32 %0, [%1], 0, 1;" : "=r"(got) : "r"(ri_base() + kRiLock) : "memory");
    if (__shfl_sync(0xffffffffu, got, 0) != 0u) return false;
    ri_fence();
    ri_feed(P);
    return true;
}

// A wait without work: true when nothing moved in any ring for the limit of clock cycles while no lane was
// looking for a string or skipping bytes of one, which ends by itself (all lanes call it; mark and t0
// carry over between calls).
__device__ __forceinline__ bool ri_stalled(const RiParams &P, uint32_t &mark, long long &t0) {
    const uint32_t lane = threadIdx.x & 31u;
    if (__any_sync(0xffffffffu, clock64() - t0 <= P.wait_cycles)) return false;
    const uint32_t v = (int)lane <= P.n_rings ? ri_ld32(ri_base() + kRiTails + 4u * lane) : 0u;
    const uint32_t sum = __reduce_add_sync(0xffffffffu, v);
    const bool busy = __any_sync(0xffffffffu, ri_ld32(ri_base() + kRiBusy) != 0u);
    if (sum == mark && !busy) return true;
    mark = sum;
    t0 = clock64();
    return false;
}

// Waits for entries of a ring (up to `most`), feeding ended slots meanwhile; 0 when the work is
// done (or the wait gave up).
__device__ __forceinline__ uint32_t ri_wait(const RiParams &P, uint32_t ring, uint32_t head, uint32_t most, uint32_t &ent) {
    uint32_t cnt, mark = 0xFFFFFFFFu;   // (no sum yet)
    long long t0 = 0;
    ri_try_feed(P, 32u);
    while ((cnt = ri_poll(P, ring, head, most, ent)) == 0u) {
        if (ri_ld32(ri_base() + kRiDone)) return 0u;
        if (ri_try_feed(P, 1u)) continue;
        if (t0 == 0) t0 = clock64();
        if (ri_stalled(P, mark, t0)) {
            if ((threadIdx.x & 31u) == 0u) {
                atomicOr(P.err, kPnErrTimeout);
                ri_st32(ri_base() + kRiDone, 1u);
            }
            return 0u;
        }
    }
    return cnt;
}

// Clears the control words, copies the small tables in and gives every slot its first string.
__device__ __forceinline__ void ri_init(const RiParams &P) {
    uint32_t *w = reinterpret_cast<uint32_t *>(ri_smem);
    for (uint32_t i = threadIdx.x; i < kRiAcc / 4; i += blockDim.x) w[i] = 0u;
    for (int i = threadIdx.x; i < (P.n_rings + 1) * P.ring_cap / 2; i += blockDim.x) w[kRiRings / 4 + i] = 0xFFFFFFFFu;
    for (int i = threadIdx.x; i < 64; i += blockDim.x) reinterpret_cast<float *>(ri_smem + kRiAcc)[i] = P.acc[i];
    if (threadIdx.x < 16) reinterpret_cast<uint4 *>(ri_smem + kRiStart)[threadIdx.x] = P.start_img[threadIdx.x];
    __syncthreads();
    if (threadIdx.x == 0) w[kRiLive / 4] = (uint32_t)P.slots;
    __syncthreads();
    for (uint32_t slot = threadIdx.x; slot < (uint32_t)P.slots; slot += blockDim.x)
        if (!ri_refill(P, slot) && ri_add32(ri_base() + kRiLive, 0xffffffffu) == 1u) ri_st32(ri_base() + kRiDone, 1u);
    __syncwarp();
}

// One group's products: row `lane` and row `lane` + 32 of the table times the states of G strings.
template <int G>
__device__ __forceinline__ void ri_products(const float4 (&t)[2][kRiReg], uint32_t tbl, const uint32_t (&row)[kRiGroup],
                                              float (&a)[kRiGroup][2]) {
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
    for (int g = 0; g < G; ++g) a[g][0] = a[g][1] = 0.f;
#pragma unroll
    for (int k = 0; k < 16; ++k) {
        float4 t0, t1;
        if (k < kRiReg) {
            t0 = t[0][k < kRiReg ? k : 0];
            t1 = t[1][k < kRiReg ? k : 0];
        } else {
            const uint32_t at = tbl + (uint32_t)(k - kRiReg) * 1024u + lane * 16u;
            const uint4 u = ri_ld128(at), v = ri_ld128(at + 512u);
            t0 = make_float4(__uint_as_float(u.x), __uint_as_float(u.y), __uint_as_float(u.z), __uint_as_float(u.w));
            t1 = make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
        }
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const uint4 x = ri_ld128(row[g] + 16u * k);
            a[g][0] = fmaf(t0.x, __uint_as_float(x.x), a[g][0]);
            a[g][0] = fmaf(t0.y, __uint_as_float(x.y), a[g][0]);
            a[g][0] = fmaf(t0.z, __uint_as_float(x.z), a[g][0]);
            a[g][0] = fmaf(t0.w, __uint_as_float(x.w), a[g][0]);
            a[g][1] = fmaf(t1.x, __uint_as_float(x.x), a[g][1]);
            a[g][1] = fmaf(t1.y, __uint_as_float(x.y), a[g][1]);
            a[g][1] = fmaf(t1.z, __uint_as_float(x.z), a[g][1]);
            a[g][1] = fmaf(t1.w, __uint_as_float(x.w), a[g][1]);
        }
    }
}

__global__ void __launch_bounds__(kRiThreads, 1) pnfa_fp32_kernel(const __grid_constant__ RiParams P) {
    const uint32_t FULL = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    // pieces 6 .. 15 of every table: [symbol][piece][row] float4
    for (int i = threadIdx.x; i < P.sigma * (16 - kRiReg) * 64; i += blockDim.x) {
        const int c = i / ((16 - kRiReg) * 64), rest = i % ((16 - kRiReg) * 64);
        const int k = kRiReg + rest / 64, r = rest % 64;
        *reinterpret_cast<float4 *>(ri_smem + P.tbl_off + 16 * (size_t)i) =
            __ldg(reinterpret_cast<const float4 *>(P.T32 + ((size_t)c * 64 + r) * 64) + k);
    }
    const uint32_t ring = warp, c = ring % (uint32_t)P.sigma;
    float4 t[2][kRiReg];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int k = 0; k < kRiReg; ++k)
            t[h][k] = __ldg(reinterpret_cast<const float4 *>(P.T32 + ((size_t)c * 64 + 32 * h + lane) * 64) + k);
    ri_init(P);   // (its barriers also cover the tables)
    const uint32_t tbl = ri_base() + P.tbl_off + c * kRiTblBytes;
    uint32_t head = 0u;
    for (;;) {
        uint32_t ent;
        const uint32_t cnt = ri_wait(P, ring, head, kRiGroup, ent);
        if (cnt == 0u) return;
        ri_fence();
        if (lane < cnt) ri_st16(ri_entry(P, ring, head + lane), kRiNone);
        head += cnt;
        const bool own = lane < cnt;   // lanes 0 .. cnt - 1 keep the records
        const uint32_t rec = ri_base() + P.recs_off + (own ? ent : 0u) * kRiRecBytes;
        uint32_t nc = 255u;
        if (own) {
            const uint8_t *p, *e;
            ri_ldp(rec + kRiRecP, p, e);
            if (p < e) nc = __ldg(p);
        }
        uint32_t row[kRiGroup];
#pragma unroll
        for (int g = 0; g < kRiGroup; ++g)
            row[g] = ri_base() + P.rows_off + __shfl_sync(FULL, ent, g < (int)cnt ? g : 0) * kRiRowBytes;
        float a[kRiGroup][2];
        if (cnt == 1u) ri_products<1>(t, tbl, row, a);
        else if (cnt == 2u) ri_products<2>(t, tbl, row, a);
        else ri_products<4>(t, tbl, row, a);
        bool ending = false;
        if (own) {   // the symbol after this one (bytes >= sigma are skipped)
            const uint8_t *p, *e;
            ri_ldp(rec + kRiRecP, p, e);
            bool found = p < e && nc < (uint32_t)P.sigma;
            if (p < e) ++p;
            if (!found && p < e) {
                // (a byte at a time: reading lines here, or calling a function that does, costs registers
                // and 3% of the time of every batch)
                ri_add32(ri_base() + kRiBusy, 1u);
                while (!found && p < e) {
                    nc = __ldg(p++);
                    found = nc < (uint32_t)P.sigma;
                }
                ri_add32(ri_base() + kRiBusy, 0xffffffffu);
            }
            ending = !found;
            ri_stp(rec + kRiRecP, p);
        }
        const uint32_t ends = __ballot_sync(FULL, ending);
#pragma unroll
        for (int g = 0; g < kRiGroup; ++g) {
            if (g >= (int)cnt) break;
            // frexp exponent of max|s'|, then the exact scale (NaN as the plain kernel's fmaxf: ignored)
            const uint32_t mb = __reduce_max_sync(
                FULL, __float_as_uint(fmaxf(fmaxf(fabsf(a[g][0]), fabsf(a[g][1])), 0.f)));
            float m = __uint_as_float(mb), s0 = 0.f, s1 = 0.f;
            if (m > 0.f) {
                uint32_t bits = mb;
                int pre = 0;
                if (((bits >> 23) & 0xFFu) == 0) {   // subnormal: lift by 2^64 first
                    m *= 18446744073709551616.0f;
                    bits = __float_as_uint(m);
                    pre = 64;
                }
                const int e = (int)((bits >> 23) & 0xFFu) - 126 - pre;
                const int e1 = max(min(e, 126), -126);   // scale by 2^-e in (at most) two exact steps
                const float sc1 = pn_pow2(-e1);
                s0 = a[g][0] * sc1;
                s1 = a[g][1] * sc1;
                if (e != e1) {
                    const float sc2 = pn_pow2(-(e - e1));
                    s0 *= sc2;
                    s1 *= sc2;
                }
                if ((int)lane == g) {
                    const uint2 w = ri_ld64(rec + kRiRecE);
                    const int64_t E = (int64_t)(((uint64_t)w.y << 32) | w.x) + e;
                    ri_st64(rec + kRiRecE, (uint32_t)E, (uint32_t)((uint64_t)E >> 32));
                }
            }
            __syncwarp();   // every lane has read the row
            if ((ends >> g) & 1u) {
                float d = s0 * __uint_as_float(ri_ld32(ri_base() + kRiAcc + 4u * lane)) +
                          s1 * __uint_as_float(ri_ld32(ri_base() + kRiAcc + 4u * lane + 128u));
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(FULL, d, o);
                if ((int)lane == g) ri_st32(rec + kRiRecDot, __float_as_uint(d));
            } else {
                ri_st32(row[g] + 4u * lane, __float_as_uint(s0));
                ri_st32(row[g] + 4u * lane + 128u, __float_as_uint(s1));
            }
        }
        __syncwarp();
        if (own) ri_push(P, ending ? (uint32_t)P.n_rings : ri_ring_of(P, nc, ent), ent);
        __syncwarp();
    }
}

}  // namespace trex
