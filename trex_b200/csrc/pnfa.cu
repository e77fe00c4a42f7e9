// Family (d): probabilistic NFA (weighted automaton, HMM forward pass) with up
// to 64 states.
//
// Semantics (reference cuda/nfa_tc_evolution.cu:456-561 nfa_prob_v5_tc_kernel,
// :572-610 nfa_prob_v6_cuda_kernel): T[c] is a real 64 x 64 matrix in the
// T[dst][src] convention; the state starts at the start vector and symbol c
// maps it to s' = T[c] s; a string's result is dot(s_L, accept). The
// reference returns only dot > 0.5; this engine returns the natural
// log-likelihood log(dot) in FP64 and that flag. Bytes >= sigma are skipped
// (the reference kernels leave the state unchanged for them).
//
// Range: every step renormalises s by an exact power of two 2^-f and adds the
// integer f to the string's exponent E, so log-likelihood = log(dot) + E ln 2.
//
// Plain form (FP32, CUDA cores): a warp per string, lane l owns states l and
// l + 32, T[c] rows read through L1; f = the frexp exponent of the step's
// max |s'|, the rule of the FP64 oracle.
//
// Tensor forms (BF16, FP16, Boolean): alphabets of up to four symbols keep a string on
// each TMEM lane and fold the symbol into K (tcgen05, below); larger ones keep a symbol's
// table in each warp's registers and bring the strings to it (mma.sync, pnfa_sym.cuh). FP32:
// tables on the SM (pnfa_fp32.cuh), or through L1 for alphabets that do not fit. The
// low-latency forms with 16-bit tables are at the end.
// A wait at an mbarrier or a ring is bounded, a meeting at a hardware barrier is timed afterwards
// (its warps never wait for another CTA); one that ran out or took too long sets the error word
// (bit 2) and ends the run.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <vector>

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "trex_internal.cuh"

namespace trex {

constexpr int kPnStates = 64;
constexpr uint32_t kPnSmemCap = 232448;
constexpr uint32_t kPnErrOffsets = 1u, kPnErrTimeout = 4u;
// The drain of committed MMAs before the TMEM is freed always waits up to the
// default limit (an MMA still writing TMEM must not outlive the allocation);
// the hand-off waits use the run's own limit.
constexpr long long kPnDrainCycles = kDefaultMbarCycles;

__host__ __device__ inline uint32_t pn_align16(uint32_t x) { return (x + 15u) & ~15u; }

// ---- small device helpers -------------------------------------------------------------------
__device__ __forceinline__ uint32_t pn_smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void pn_tc_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void pn_tc_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void pn_fence_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ bool pn_mbar_test(uint32_t addr, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(done) : "r"(addr), "r"(parity) : "memory");
    return done != 0;
}
// The same without the pause that the hardware may take before it answers.
__device__ __forceinline__ bool pn_mbar_look(uint32_t addr, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(done) : "r"(addr), "r"(parity) : "memory");
    return done != 0;
}
// The warp waits for the completion of the phase with the given parity; bounded, the same result
// in all lanes. A limit shorter than the hardware's pause starts with a look, so that it holds (the
// look costs a tile of a few int8 strings up to a tenth of its time).
__device__ __forceinline__ bool ln_wait(uint32_t addr, uint32_t parity, volatile uint32_t *abort_flag,
                                        uint32_t *err, long long limit) {
    bool ok = true;
    const long long t0 = clock64();
    for (bool done = limit < 1000 ? pn_mbar_look(addr, parity) : pn_mbar_test(addr, parity); !done;
         done = pn_mbar_test(addr, parity)) {
        if (*abort_flag) { ok = false; break; }
        if (clock64() - t0 > limit) {
            atomicOr(err, kPnErrTimeout);
            *abort_flag = 1u;
            ok = false;
            break;
        }
    }
    return __all_sync(0xffffffffu, ok);
}

__device__ __forceinline__ void pn_write_result(double *loglik, uint8_t *accept, int32_t *accept_i32,
                                                int64_t seq, double ll) {
    if (loglik) loglik[seq] = ll;
    const int a = ll > -0.69314718055994530942;   // dot > 0.5
    if (accept) accept[seq] = (uint8_t)a;
    if (accept_i32) accept_i32[seq] = a;
}

// exponent f with x < 2^f for a finite positive float x (x >= 2^-126); 0 for x == 0
__device__ __forceinline__ int pn_ceil_exp(float x) {
    const uint32_t e = (__float_as_uint(x) >> 23) & 0xFFu;
    if (e == 0) return 0;
    return (int)e - 126;
}
__device__ __forceinline__ float pn_pow2(int f) {   // 2^f, |f| <= 126
    return __uint_as_float((uint32_t)(127 + f) << 23);
}

template <bool FP16>
__device__ __forceinline__ uint16_t pn_to16(float v) {
    if constexpr (FP16) return __half_as_ushort(__float2half_rn(v));
    else return __bfloat16_as_ushort(__float2bfloat16_rn(v));
}

// two values rounded to the operand type, packed low/high
template <bool FP16>
__device__ __forceinline__ uint32_t pn_pack2(float lo, float hi) {
    if constexpr (FP16) {
        const __half2 h = __floats2half2_rn(lo, hi);
        return *reinterpret_cast<const uint32_t *>(&h);
    } else {
        const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<const uint32_t *>(&h);
    }
}

__device__ __forceinline__ void pn_tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
        "%14,%15,%16};"
        :: "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]),
           "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]),
           "r"(r[14]), "r"(r[15])
        : "memory");
}

// ---- strings on TMEM lanes (alphabets of at most four symbols) -------------------------------
// Each of four tiles of 128 strings keeps one string on each TMEM lane: the string's state is
// row m of the tile's A operand, K = 64 * sigma, with the 64 states in the K range of the
// string's next symbol and zeros in the other range; B (shared memory) stacks the tables,
// B[n][64 c + q] = T_c[n][q]. One MMA chain (M = 128, N = 64) then gives every string the
// product with its own symbol, D[m][n] = (T_c s_m)[n], with no sorting of strings by symbol.
// The epilogue is thread-local (thread = TMEM lane = string): it reads its 64 states, finds
// their maximum and rescales by an exact power of two, rounds them to the operand type and
// writes its next A row with tcgen05.st; at the string's end it forms the log-likelihood and
// takes the next string from the queue.
//
// Bound by the latency of a tile's step, about 2500 cycles (the 512 TMEM columns hold no more
// strings): 262144 strings x 2048 symbols, 2 symbols, FP16 take 10.70 ms (20.27 with a warp of its
// own to issue the products, and two hand-offs a step). A step has one hand-off: the four warps of
// a tile meet at a hardware barrier, which also tells whether any string is left, an elected thread
// of the first issues the products, and the next symbol is found while they run; a tcgen05.commit
// brings the result (a bounded wait).
constexpr int kLnTiles = 4;
constexpr int kLnEpiWarps = 4 * kLnTiles;   // tile T: warps 4T .. 4T + 3 (lane quadrants 0-3)
constexpr int kLnThreads = 32 * kLnEpiWarps;
constexpr int kLnMaxSigma = 4;
constexpr uint32_t kLnLbo = 1024;           // B: bytes between 16-byte K columns (64 rows x 16 B)

struct LnParams {
    const uint8_t *data;
    int64_t total_bytes;
    const int64_t *offsets;
    int64_t n;
    const uint16_t *T16;   // [sigma][64][64] row-major in the operand type (probabilistic forms)
    const float *T32;      // [sigma][64][64] (Boolean forms: a nonzero entry is an edge)
    const float *start;    // [64]
    const float *acc;      // [64] accept weights (Boolean forms: 0/1)
    int sigma;
    int tiles;             // tiles in flight: as many of kLnTiles as fit in the 512 TMEM columns
    uint32_t a_cols;       // TMEM columns of a tile's A (32 sigma, int8: 16 sigma); D follows
    uint32_t tile_cols;    // a_cols + 64, rounded up to 32
    int resc;              // steps between rescales (1 for FP16 operands)
    long long wait_cycles;
    double ll_empty;
    double *loglik;
    uint8_t *accept;
    int32_t *accept_i32;
    unsigned long long *queue;
    uint32_t *err;
};

// A string's symbols: aligned 8-byte words of the batch, the next word loaded while this one
// is used; bytes >= sigma are skipped.
struct LnSym {
    uintptr_t p, e;        // next byte, end of the string (addresses)
    uintptr_t cw;          // address of the word in `cur`
    uint64_t cur, nxt;
};
__device__ __forceinline__ uint64_t ln_word(uintptr_t w, uintptr_t lo, uintptr_t hi) {
    if (w >= lo && w + 8 <= hi) return __ldg(reinterpret_cast<const unsigned long long *>(w));
    uint64_t v = 0;
    for (int k = 0; k < 8; ++k)
        if (w + k >= lo && w + k < hi) v |= (uint64_t)__ldg(reinterpret_cast<const uint8_t *>(w + k)) << (8 * k);
    return v;
}
// next symbol < sigma of the string, or -1 at its end
__device__ __forceinline__ int ln_next(LnSym &s, int sigma, uintptr_t lo, uintptr_t hi) {
    while (s.p < s.e) {
        const uintptr_t w = s.p & ~(uintptr_t)7;
        if (w != s.cw) {
            s.cur = (s.cw != 0 && w == s.cw + 8) ? s.nxt : ln_word(w, lo, hi);
            s.cw = w;
            s.nxt = ln_word(w + 8, lo, hi);
        }
        const int b = (int)((s.cur >> (8 * (s.p & 7))) & 0xffu);
        ++s.p;
        if (b < sigma) return b;
    }
    return -1;
}
// The next string from the queue (index and byte range); seq = -1 when the queue is empty.
// Not inlined: a rare path, kept out of the epilogue's registers.
struct LnRange {
    int64_t seq, a, b;
};
__device__ __noinline__ LnRange ln_take(const LnParams &P) {
    while (true) {
        const unsigned long long idx = atomicAdd(P.queue, 1ull);
        if (idx >= (unsigned long long)P.n) return LnRange{-1, 0, 0};
        const int64_t a = P.offsets[idx], b = P.offsets[idx + 1];
        if (a < 0 || b < a || b > P.total_bytes) {
            atomicOr(P.err, kPnErrOffsets);
            continue;
        }
        return LnRange{(int64_t)idx, a, b};
    }
}
__device__ __noinline__ void ln_empty(const LnParams &P, int64_t seq) {
    pn_write_result(P.loglik, P.accept, P.accept_i32, seq, P.ll_empty);
}

// A finished string: log-likelihood from the accept-weighted sum of its last state and its
// exponent sum.
__device__ __noinline__ void ln_finish(const LnParams &P, int64_t seq, float dot, int E) {
    const double ll = dot > 0.f ? log((double)dot) + (double)E * 0.69314718055994530942 : -INFINITY;
    pn_write_result(P.loglik, P.accept, P.accept_i32, seq, ll);
}

// Waits for this thread's TMEM loads; r is named so that nothing reads it before.
__device__ __forceinline__ void ln_tmem_wait32(uint32_t *r) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                 "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]),
                 "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]),
                 "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
                 :: "memory");
}
// The 128 threads of tile T meet; whether any of them passed true.
__device__ __forceinline__ bool ln_tile_any(int T, bool v) {
    uint32_t any;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %2, 0;\n\t"
        "barrier.cta.red.or.pred p, %1, 128, q;\n\tselp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(any) : "r"(T + 1), "r"((uint32_t)v) : "memory");
    return any != 0u;
}
__device__ __forceinline__ bool ln_elect() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0u;
}
// max(a, |b|, |c|), a >= 0 (a NaN is passed over)
__device__ __forceinline__ float ln_max_abs3(float a, float b, float c) {
    float m;
    asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(c));
    return m;
}

__device__ __forceinline__ void ln_tmem_ld32(uint32_t taddr, uint32_t *r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,"
        "%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
          "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
          "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr) : "memory");
}

// KIND: 0 = BF16, 1 = FP16 operands (kind::f16, FP32 sums, rescaled by exact powers of two);
// 2 = Boolean 0/1 int8 (kind::i8, int32 sums); 3 = Boolean 0/1 BF16. The Boolean forms
// threshold every product to {0, 1} (exact).
template <int KIND>
__global__ void __launch_bounds__(kLnThreads, 1) pnfa_lane_kernel(const __grid_constant__ LnParams P) {
    constexpr bool I8 = KIND == 2, BOOL = KIND >= 2, FP16 = KIND == 1;
    __shared__ __align__(1024) uint8_t s_b[64 * 64 * kLnMaxSigma * 2];
    __shared__ __align__(8) uint64_t s_bar[kLnTiles];   // a tile's products are complete
    __shared__ uint32_t s_tmem, s_abort;
    __shared__ float s_acc[64], s_start[64];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int sig = P.sigma;
    const int K = 64 * sig;
    // B: row n = destination state, K index 64 c + q (symbol c, source state q); 16-byte K
    // columns kLnLbo bytes apart, rows 16 bytes apart inside 8-row core matrices
    if constexpr (I8) {
        for (int t = threadIdx.x; t < 64 * (K / 16); t += blockDim.x) {
            const int n = t & 63, kc = t >> 6;
            uint32_t w[4] = {0u, 0u, 0u, 0u};
            for (int j = 0; j < 16; ++j) {
                const int k = 16 * kc + j;
                if (P.T32[((size_t)(k >> 6) * 64 + n) * 64 + (k & 63)] != 0.f) w[j >> 2] |= 1u << (8 * (j & 3));
            }
            *reinterpret_cast<uint4 *>(s_b + kc * kLnLbo + (n >> 3) * 128 + (n & 7) * 16) =
                make_uint4(w[0], w[1], w[2], w[3]);
        }
    } else {
        for (int t = threadIdx.x; t < 64 * (K / 8); t += blockDim.x) {
            const int n = t & 63, kc = t >> 6;
            uint32_t w[4];
            for (int j = 0; j < 4; ++j) {
                const int k = 8 * kc + 2 * j;   // k and k + 1 belong to the same symbol
                const size_t o = ((size_t)(k >> 6) * 64 + n) * 64 + (k & 63);
                uint32_t lo16, hi16;
                if constexpr (BOOL) {
                    lo16 = P.T32[o] != 0.f ? 0x3F80u : 0u;   // BF16 1.0
                    hi16 = P.T32[o + 1] != 0.f ? 0x3F80u : 0u;
                } else {
                    lo16 = P.T16[o];
                    hi16 = P.T16[o + 1];
                }
                w[j] = lo16 | (hi16 << 16);
            }
            *reinterpret_cast<uint4 *>(s_b + kc * kLnLbo + (n >> 3) * 128 + (n & 7) * 16) =
                make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
    if (threadIdx.x < 64) {
        s_acc[threadIdx.x] = P.acc[threadIdx.x];
        s_start[threadIdx.x] = P.start[threadIdx.x];
    }
    if (threadIdx.x == 0) {
        s_abort = 0u;
        for (int T = 0; T < kLnTiles; ++T)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(pn_smem_u32(&s_bar[T])));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(pn_smem_u32(&s_tmem)), "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    pn_fence_async_smem();   // B, written by these stores, is read by the tensor cores
    pn_tc_before();
    __syncthreads();
    pn_tc_after();
    const uint32_t tbase = *reinterpret_cast<volatile uint32_t *>(&s_tmem);
    volatile uint32_t *abort_flag = &s_abort;
    if ((warp >> 2) < P.tiles) {   // fewer tiles for larger alphabets
        // (broadcast, so that the operands of the MMAs are known to be the same in all lanes)
        const int T = __shfl_sync(0xffffffffu, warp >> 2, 0), qd = __shfl_sync(0xffffffffu, warp & 3, 0);
        const uint32_t tile = __shfl_sync(0xffffffffu, tbase, 0) + (uint32_t)T * P.tile_cols;
        const uint32_t tA = tile + ((uint32_t)(32 * qd) << 16), tD = tA + P.a_cols;
        const uint32_t bar_full = pn_smem_u32(&s_bar[T]);
        const uint32_t fmt = KIND == 1 ? 0u : 1u;
        const uint32_t idesc = I8 ? ((2u << 4) | ((64u >> 3) << 17) | ((128u >> 4) << 24))
                                  : ((1u << 4) | (fmt << 7) | (fmt << 10) | ((64u >> 3) << 17) |
                                     ((128u >> 4) << 24));
        const uint32_t sb = pn_smem_u32(s_b);
        const uint64_t desc0 = (uint64_t)(((sb >> 4) & 0x3FFFu) | ((kLnLbo >> 4) << 16)) |
                               ((uint64_t)((128u >> 4) | (1u << 14)) << 32);
        const uintptr_t lo = reinterpret_cast<uintptr_t>(P.data), hi = lo + (uintptr_t)P.total_bytes;
        LnSym sy{0, 0, 0, 0, 0};
        int64_t seq = -1;
        int c = 0, E = 0, since = 0;
        // the next string with its first symbol in c (strings with no symbol get their result
        // at once); false when the queue is empty
        auto fetch = [&]() -> bool {
            while (true) {
                const LnRange r = ln_take(P);
                if (r.seq < 0) return false;
                sy.p = lo + (uintptr_t)r.a;
                sy.e = lo + (uintptr_t)r.b;
                sy.cw = 0;
                c = ln_next(sy, sig, lo, hi);
                if (c >= 0) {
                    seq = r.seq;
                    return true;
                }
                ln_empty(P, r.seq);
            }
        };
        bool live = fetch();
        const uint32_t FULL = 0xffffffffu;
        uint32_t d[64];   // this string's states: a row of D
        auto d_value = [&](uint32_t w) -> float {
            if constexpr (I8) return w != 0u ? 1.f : 0.f;
            else if constexpr (BOOL) return __uint_as_float(w) > 0.f ? 1.f : 0.f;
            else return __uint_as_float(w);
        };
        // this string's A row: the states in the K range of symbol c, zeros in the other ranges
        // (tcgen05.st is warp-wide; each thread supplies its own row)
        auto store_row = [&]() {
            if constexpr (I8) {
                uint32_t r[16];
#pragma unroll
                for (int k = 0; k < 16; ++k) {
                    // four path counts (at most 64 each) as bytes, then 1 for each that is not 0
                    const uint32_t w = __byte_perm(__byte_perm(d[4 * k], d[4 * k + 1], 0x0040),
                                                   __byte_perm(d[4 * k + 2], d[4 * k + 3], 0x0040), 0x5410);
                    r[k] = ((w + 0x7F7F7F7Fu) >> 7) & 0x01010101u;
                }
                for (int h = 0; h < sig; ++h) {
                    uint32_t q[16];
#pragma unroll
                    for (int k = 0; k < 16; ++k) q[k] = h == c ? r[k] : 0u;
                    pn_tmem_st16(tA + 16u * (uint32_t)h, q);
                }
            } else {
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    uint32_t r[16];
#pragma unroll
                    for (int k = 0; k < 16; ++k)
                        r[k] = pn_pack2<FP16>(d_value(d[32 * j + 2 * k]), d_value(d[32 * j + 2 * k + 1]));
                    for (int h = 0; h < sig; ++h) {
                        uint32_t q[16];
#pragma unroll
                        for (int k = 0; k < 16; ++k) q[k] = h == c ? r[k] : 0u;
                        pn_tmem_st16(tA + 32u * (uint32_t)h + 16u * (uint32_t)j, q);
                    }
                }
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            pn_tc_before();
        };
        // d becomes the start vector (zeros without a string) where `fresh`
        auto start_row = [&](bool fresh) {
#pragma unroll
            for (int i = 0; i < 64; ++i) {
                const float s0 = s_start[i];
                const uint32_t w = !live ? 0u : I8 ? (s0 != 0.f ? 1u : 0u)
                                              : __float_as_uint(BOOL ? (s0 != 0.f ? 1.f : 0.f) : s0);
                if (fresh) d[i] = w;
            }
        };
#pragma unroll
        for (int i = 0; i < 64; ++i) d[i] = 0u;
        start_row(true);
        __syncwarp();
        store_row();
        uint32_t ph = 0u;
        bool failed = false, pend = false;
        for (;;) {
            if (!ln_tile_any(T, live)) break;
            if (failed) continue;   // (the other warps of the tile give up at their next wait)
            pn_tc_after();
            if (qd == 0) {
                // One K chain (4 sigma K16 or 2 sigma K32 steps), issued by an elected thread with
                // the steps unrolled: 37-43 cycles an MMA (M = 128, N = 64, K = 16 takes 32); a loop
                // under `lane == 0` took 103-109.
                if (ln_elect()) {
                    // K step kk: B 2 kLnLbo bytes further (+128 in the descriptor's start field,
                    // which stays below 2^14 for shared addresses), A 8 TMEM columns further
                    constexpr int KS = I8 ? 2 : 4;
                    for (int h = 0; h < sig; ++h) {
#pragma unroll
                        for (int k = 0; k < KS; ++k) {
                            const uint32_t kk = (uint32_t)(KS * h + k);
                            const uint64_t desc = desc0 + (uint64_t)(128u * kk);
                            const uint32_t ta = tile + 8u * kk, td = tile + P.a_cols;
                            const uint32_t acc = kk > 0u;
                            if constexpr (I8)
                                asm volatile(
                                    "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                                    "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
                                    :: "r"(td), "r"(ta), "l"(desc), "r"(idesc), "r"(acc) : "memory");
                            else
                                asm volatile(
                                    "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                                    "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                                    :: "r"(td), "r"(ta), "l"(desc), "r"(idesc), "r"(acc) : "memory");
                        }
                    }
                    asm volatile(
                        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                        :: "r"(bar_full) : "memory");
                }
                __syncwarp();
            }
            pend = true;
            // while the products run: what comes after this symbol
            const int nc = live ? ln_next(sy, sig, lo, hi) : -1;
            const bool ending = live && nc < 0;
            bool resc_now = false;
            if (live && !ending) {
                c = nc;
                if (!BOOL && ++since >= P.resc) {
                    since = 0;
                    resc_now = true;
                }
            }
            if (!ln_wait(bar_full, ph, abort_flag, P.err, P.wait_cycles)) {
                failed = true;
                live = false;
                continue;
            }
            ph ^= 1u;
            pend = false;
            pn_tc_after();
            // D row = this string's state after its symbol
            ln_tmem_ld32(tD, d);
            ln_tmem_ld32(tD + 32u, d + 32);
            ln_tmem_wait32(d);
            ln_tmem_wait32(d + 32);
            const bool any_end = __any_sync(FULL, ending);
            if (any_end) {   // a string's last symbol: the accept-weighted sum of its state
                float dot = 0.f;
#pragma unroll
                for (int i = 0; i < 64; ++i) dot = fmaf(s_acc[i], d_value(d[i]), dot);
                if (ending) {   // the string's log-likelihood, then the next string
                    ln_finish(P, seq, dot, E);
                    live = fetch();
                    E = 0;
                    since = 0;
                }
                __syncwarp();
            }
            if (!BOOL && __any_sync(FULL, resc_now)) {   // exact power-of-two rescale by the row's maximum
                float m = 0.f;
#pragma unroll
                for (int i = 0; i < 64; i += 2) m = ln_max_abs3(m, __uint_as_float(d[i]), __uint_as_float(d[i + 1]));
                const int f = resc_now ? min(max(pn_ceil_exp(m), -125), 125) : 0;
                const float sc = pn_pow2(-f);
                E += f;
#pragma unroll
                for (int i = 0; i < 64; ++i) d[i] = __float_as_uint(__uint_as_float(d[i]) * sc);
            }
            if (!live) c = 0;
            // (the row of a lane without a string stays zero)
            if (any_end) start_row(ending);
            __syncwarp();
            store_row();
        }
        // a product committed but not read must be complete before the TMEM is freed
        if (qd == 0 && pend && lane == 0) {
            const long long t0 = clock64();
            while (!pn_mbar_test(bar_full, ph)) {
                if (clock64() - t0 > kPnDrainCycles) { atomicOr(P.err, kPnErrTimeout); break; }
            }
        }
        __syncwarp();
    }
    pn_tc_before();
    __syncthreads();
    pn_tc_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tbase), "r"(512));
}

// ---- plain FP32 form -------------------------------------------------------------------------
struct PnPlainParams {
    const uint8_t *data;
    int64_t total_bytes;
    const int64_t *offsets;
    int64_t n;
    const float *T;         // [sigma][64][64]
    const float *start;     // [64]
    const float *acc;       // [64]
    int sigma;
    double ll_empty;
    double *loglik;
    uint8_t *accept;
    int32_t *accept_i32;
    unsigned long long *queue;
    uint32_t *err;
};

constexpr int kPnPlainWarps = 8;

__global__ void __launch_bounds__(kPnPlainWarps * 32) pnfa_plain_kernel(PnPlainParams P) {
    __shared__ __align__(16) float sv[kPnPlainWarps][64];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    float *v = sv[w];
    for (;;) {
        unsigned long long idx = 0;
        if (lane == 0) idx = atomicAdd(P.queue, 1ull);
        idx = __shfl_sync(0xffffffffu, idx, 0);
        if (idx >= (unsigned long long)P.n) break;
        const int64_t p0 = P.offsets[idx], p1 = P.offsets[idx + 1];
        if (p0 < 0 || p1 < p0 || p1 > P.total_bytes) {
            if (lane == 0) atomicOr(P.err, kPnErrOffsets);
            continue;
        }
        float s0 = P.start[lane], s1 = P.start[lane + 32];
        int64_t E = 0;
        for (int64_t base = p0; base < p1; base += 32) {
            const int64_t pl = base + lane;
            const uint32_t mybyte = pl < p1 ? P.data[pl] : 255u;
            const int nb = (int)min((int64_t)32, p1 - base);
            for (int k = 0; k < nb; ++k) {
                const uint32_t c = __shfl_sync(0xffffffffu, mybyte, k);
                if (c >= (uint32_t)P.sigma) continue;
                v[lane] = s0;
                v[lane + 32] = s1;
                __syncwarp();
                const float4 *r0 = reinterpret_cast<const float4 *>(P.T + ((size_t)c * 64 + lane) * 64);
                const float4 *r1 = reinterpret_cast<const float4 *>(P.T + ((size_t)c * 64 + lane + 32) * 64);
                const float4 *vv = reinterpret_cast<const float4 *>(v);
                float a0 = 0.f, a1 = 0.f;
#pragma unroll
                for (int q = 0; q < 16; ++q) {
                    const float4 x = vv[q];
                    const float4 t0 = __ldg(r0 + q), t1 = __ldg(r1 + q);
                    a0 = fmaf(t0.x, x.x, a0); a0 = fmaf(t0.y, x.y, a0);
                    a0 = fmaf(t0.z, x.z, a0); a0 = fmaf(t0.w, x.w, a0);
                    a1 = fmaf(t1.x, x.x, a1); a1 = fmaf(t1.y, x.y, a1);
                    a1 = fmaf(t1.z, x.z, a1); a1 = fmaf(t1.w, x.w, a1);
                }
                __syncwarp();
                float m = fmaxf(fabsf(a0), fabsf(a1));
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
                if (m > 0.f) {
                    // frexp exponent of m: m = mant * 2^e, mant in [0.5, 1)
                    uint32_t bits = __float_as_uint(m);
                    int pre = 0;
                    if (((bits >> 23) & 0xFFu) == 0) {   // subnormal: lift by 2^64 first
                        m *= 18446744073709551616.0f;
                        bits = __float_as_uint(m);
                        pre = 64;
                    }
                    const int e = (int)((bits >> 23) & 0xFFu) - 126 - pre;
                    // scale by 2^-e in (at most) two exact steps
                    const int e1 = max(min(e, 126), -126);
                    const float sc1 = pn_pow2(-e1);
                    s0 = a0 * sc1;
                    s1 = a1 * sc1;
                    if (e != e1) {
                        const float sc2 = pn_pow2(-(e - e1));
                        s0 *= sc2;
                        s1 *= sc2;
                    }
                    E += e;
                } else {
                    s0 = 0.f;
                    s1 = 0.f;
                }
            }
        }
        float d = s0 * P.acc[lane] + s1 * P.acc[lane + 32];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        if (lane == 0) {
            const double ll = d > 0.f ? log((double)d) + (double)E * 0.69314718055994530942 : -INFINITY;
            pn_write_result(P.loglik, P.accept, P.accept_i32, (int64_t)idx, ll);
        }
    }
}

// CUDA-core form with 16-bit tables in shared memory (modes BF16_CC / FP16_CC):
// the low-latency chain. The transition tables of all symbols (sigma x 8 KB)
// are copied into shared memory once per CTA, so a step reads no global
// memory; the state stays in FP32. Four warps advance one string: thread
// (o, h) = (gt / 2, gt % 2) of the group forms the dot product of row o of
// T[c] with states 32h .. 32h + 31 (four independent FMA chains of eight),
// the two halves meet by one shuffle and the new state goes to the other of
// two state buffers, so a step costs one named barrier of the group. Rows are
// stored with their 16-byte chunks permuted by (o & 3), so the eight lanes of
// a quarter-warp read eight different chunks (no bank conflicts), and the two
// state halves sit 144 bytes apart for the same reason. Every `resc` steps
// the group finds max|s| (warp maxima through shared memory) and the next
// step scales by the exact power of two 2^-f and adds f to the exponent sum,
// as the plain kernel does every step (power-of-two scaling is exact, so only
// the rounding of the products differs between the forms). CTA = four groups
// = four strings in flight; the per-step latency is far below the
// tensor-core kernel's (which advances many strings per step): the form for
// few strings, long ones included (serving).
template <bool FP16>
__device__ __forceinline__ float pn_h2f(uint32_t h) {
    if constexpr (FP16) return __half2float(__ushort_as_half((unsigned short)h));
    else return __uint_as_float(h << 16);
}

constexpr int kChainThreads = 128;   // one string per group of four warps
constexpr int kChainGroups = 4;      // strings per CTA
struct ChainShared {
    float s[2][72];        // the state, double-buffered; state i at i + (i >= 32 ? 4 : 0)
    float wmax[2][4];      // warp maxima of a check step (by its parity)
    float red[4];
    unsigned long long idx;
    uint32_t pad[2];
};
constexpr uint32_t kChainSharedBytes = kChainGroups * (uint32_t)sizeof(ChainShared);

__device__ __forceinline__ void pn_group_bar(int g) {
    asm volatile("bar.sync %0, %1;" :: "r"(g + 1), "r"(kChainThreads) : "memory");
}
__device__ __forceinline__ int pn_sidx(int i) { return i + (i >= 32 ? 4 : 0); }

template <bool FP16>
__global__ void __launch_bounds__(kChainThreads * kChainGroups, 1)
pnfa_chain_kernel(PnPlainParams P, const uint16_t *T16, int resc) {
    extern __shared__ __align__(16) uint8_t pn_ch_smem[];
    const uint32_t FULL = 0xffffffffu;
    const int g = threadIdx.x / kChainThreads, gt = threadIdx.x % kChainThreads;
    const int lane = threadIdx.x & 31, wg = gt >> 5;
    const int o = gt >> 1, h = gt & 1, sw = o & 3;
    uint4 *tbl = reinterpret_cast<uint4 *>(pn_ch_smem);   // [sigma][64 rows][8 chunks], chunk p at p ^ (row & 3)
    ChainShared *cs = reinterpret_cast<ChainShared *>(pn_ch_smem + (size_t)P.sigma * 8192) + g;
    {
        const uint4 *src = reinterpret_cast<const uint4 *>(T16);
        const int chunks = P.sigma * 64 * 8;
        for (int i = threadIdx.x; i < chunks; i += blockDim.x) {
            const int row = i >> 3, p = i & 7;
            tbl[(row << 3) | (p ^ (row & 3))] = src[i];
        }
        __syncthreads();
    }
    const float acc_o = gt < 64 ? P.acc[gt] : 0.f;
    const float start_o = gt < 64 ? P.start[gt] : 0.f;
    for (;;) {
        if (gt == 0) cs->idx = atomicAdd(P.queue, 1ull);
        pn_group_bar(g);
        const unsigned long long idx = cs->idx;
        if (idx >= (unsigned long long)P.n) break;
        const int64_t p0 = P.offsets[idx], p1 = P.offsets[idx + 1];
        if (p0 < 0 || p1 < p0 || p1 > P.total_bytes) {
            if (gt == 0) atomicOr(P.err, kPnErrOffsets);
            pn_group_bar(g);
            continue;
        }
        if (gt < 64) cs->s[0][pn_sidx(gt)] = start_o;
        pn_group_bar(g);
        int cur = 0;          // the buffer holding the state
        int64_t E = 0;
        bool any = false;     // some symbol was applied
        bool pend = false;    // the previous step was a check step
        uint32_t par = 0;     // parity of the step
        int chk = resc;       // steps to the next check step
        for (int64_t base = p0; base < p1; base += 32) {
            const int64_t pl = base + lane;
            const uint32_t byte = pl < p1 ? P.data[pl] : 255u;
            uint32_t m = __ballot_sync(FULL, byte < (uint32_t)P.sigma);
            while (m) {
                const int src = __ffs(m) - 1;
                m &= m - 1;
                const uint32_t c = __shfl_sync(FULL, byte, src);
                const uint4 *row = tbl + ((c * 64 + o) << 3);
                float sc = 1.f;
                if (pend) {   // the maxima of the previous step's outputs: exact power-of-two scale
                    const float4 w4 = *reinterpret_cast<const float4 *>(cs->wmax[par ^ 1u]);
                    const float mx = fmaxf(fmaxf(w4.x, w4.y), fmaxf(w4.z, w4.w));
                    const uint32_t eb = (__float_as_uint(mx) >> 23) & 0xFFu;
                    if (mx > 0.f && eb != 0) {
                        const int f = min(max((int)eb - 126, -125), 125);
                        sc = pn_pow2(-f);
                        E += f;
                    }
                    pend = false;
                }
                const float4 *sv = reinterpret_cast<const float4 *>(&cs->s[cur][h * 36]);
                float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint4 t = row[(4 * h + k) ^ sw];   // states 32h + 8k .. + 7 of row o
                    const float4 x0 = sv[2 * k], x1 = sv[2 * k + 1];
                    a0 = fmaf(pn_h2f<FP16>(t.x & 0xFFFFu), x0.x, a0);
                    a1 = fmaf(pn_h2f<FP16>(t.x >> 16), x0.y, a1);
                    a2 = fmaf(pn_h2f<FP16>(t.y & 0xFFFFu), x0.z, a2);
                    a3 = fmaf(pn_h2f<FP16>(t.y >> 16), x0.w, a3);
                    a0 = fmaf(pn_h2f<FP16>(t.z & 0xFFFFu), x1.x, a0);
                    a1 = fmaf(pn_h2f<FP16>(t.z >> 16), x1.y, a1);
                    a2 = fmaf(pn_h2f<FP16>(t.w & 0xFFFFu), x1.z, a2);
                    a3 = fmaf(pn_h2f<FP16>(t.w >> 16), x1.w, a3);
                }
                float sum = (a0 + a1) + (a2 + a3);
                sum += __shfl_xor_sync(FULL, sum, 1);
                sum *= sc;
                if (--chk == 0) {   // a check step: this group's max|s'|
                    float mx = fabsf(sum);
#pragma unroll
                    for (int d = 2; d < 32; d <<= 1) mx = fmaxf(mx, __shfl_xor_sync(FULL, mx, d));
                    if (lane == 0) cs->wmax[par][wg] = mx;
                    pend = true;
                    chk = resc;
                }
                if (h == 0) cs->s[cur ^ 1][pn_sidx(o)] = sum;
                cur ^= 1;
                par ^= 1u;
                any = true;
                pn_group_bar(g);
            }
        }
        if (!any) {
            if (gt == 0) pn_write_result(P.loglik, P.accept, P.accept_i32, (int64_t)idx, P.ll_empty);
        } else {
            float d = gt < 64 ? cs->s[cur][pn_sidx(gt)] * acc_o : 0.f;
#pragma unroll
            for (int k = 16; k > 0; k >>= 1) d += __shfl_xor_sync(FULL, d, k);
            if (lane == 0) cs->red[wg] = d;
            pn_group_bar(g);
            if (gt == 0) {
                const float dot = (cs->red[0] + cs->red[1]) + (cs->red[2] + cs->red[3]);
                const double ll = dot > 0.f ? log((double)dot) + (double)E * 0.69314718055994530942 : -INFINITY;
                pn_write_result(P.loglik, P.accept, P.accept_i32, (int64_t)idx, ll);
            }
        }
        pn_group_bar(g);   // the slot (idx, red) is free again
    }
}

}  // namespace trex

#include "pnfa_fp32.cuh"
#include "pnfa_sym.cuh"

// ---- handle -----------------------------------------------------------------------------------
struct trex_pnfa {
    int n_states = 0, sigma = 0, n_sms = 0;
    double ll_empty = 0.0, ll_empty_bool = 0.0;
    // tensor-core tables: [bf16, fp16, Boolean 0/1 in bf16, Boolean 0/1 in int8]
    float start_max16[4] = {0.f, 0.f, 0.f, 0.f};
    float *d_T32 = nullptr, *d_start32 = nullptr, *d_acc = nullptr, *d_acc_bool = nullptr;
    uint16_t *d_T16[2] = {nullptr, nullptr};   // [sigma][64][64] row-major: bf16, fp16
    float *d_rsym[4] = {nullptr, nullptr, nullptr, nullptr};
    uint4 *d_simg[4] = {nullptr, nullptr, nullptr, nullptr};
    uint8_t *d_misc = nullptr;   // [0,8) queue, [8,12) error word
    // steps between the rescale checks of the chain kernel per 16-bit table type: 4
    // when the tables' growth bound allows (max |T s| / max |s| <= 16 a step, so five
    // unchecked steps stay far inside FP32), else every step
    int chain_resc[2] = {1, 1};
    int tc_resc = 1;   // the tensor-core kernel's rescale period for BF16 operands (same bound)
    int sm_limit = 0;  // launches size their grids for at most this many SMs (0: all)
};

namespace trex {

static uint16_t pn_host16(float x, bool fp16) {
    if (fp16) {
        const __half h = __float2half_rn(x);
        return __half_as_ushort(h);
    }
    const __nv_bfloat16 b = __float2bfloat16_rn(x);
    return __bfloat16_as_ushort(b);
}
static float pn_host16_to_f(uint16_t v, bool fp16) {
    if (fp16) return __half2float(__ushort_as_half(v));
    return __bfloat162float(__ushort_as_bfloat16(v));
}

static void pn_free(trex_pnfa *h) {
    cudaFree(h->d_T32);
    cudaFree(h->d_T16[0]);
    cudaFree(h->d_T16[1]);
    cudaFree(h->d_start32);
    cudaFree(h->d_acc);
    cudaFree(h->d_acc_bool);
    for (int k = 0; k < 4; ++k) {
        cudaFree(h->d_rsym[k]);
        cudaFree(h->d_simg[k]);
    }
    cudaFree(h->d_misc);
}

static int64_t pn_sms(const trex_pnfa *h) {
    return h->sm_limit > 0 ? std::min(h->sm_limit, h->n_sms) : h->n_sms;
}

// Tables, rings, slots and shared-memory layout of a run of pnfa_fp32_kernel: one CTA an SM, the
// strings spread over all SMs, as many slots a CTA as it has strings or fit beside the tables.
static RiParams ri_params(const trex_pnfa *h, int64_t n) {
    RiParams Q{};
    Q.T32 = h->d_T32;
    Q.start_img = reinterpret_cast<const uint4 *>(h->d_start32);
    Q.acc = h->d_acc;
    Q.ll_empty = h->ll_empty;
    Q.wait_cycles = mbar_wait_cycles();
    Q.sigma = h->sigma;
    Q.rep = std::max(1, kRiWarps / h->sigma);
    Q.n_rings = Q.sigma * Q.rep;
    Q.grid = (int)std::max<int64_t>(1, std::min<int64_t>(n, pn_sms(h)));
    Q.slots = (int)std::min<int64_t>((n + Q.grid - 1) / Q.grid, kRiMaxSlots);
    for (;; --Q.slots) {
        Q.rep_shift = 5;
        while ((1 << Q.rep_shift) < Q.slots) ++Q.rep_shift;
        Q.ring_cap = 1 << Q.rep_shift;
        Q.recs_off = pn_align16(kRiRings + (uint32_t)(Q.n_rings + 1) * (uint32_t)Q.ring_cap * 2u);
        Q.rows_off = Q.recs_off + (uint32_t)Q.slots * kRiRecBytes;
        Q.tbl_off = Q.rows_off + (uint32_t)Q.slots * kRiRowBytes;
        if (Q.tbl_off + (uint32_t)Q.sigma * kRiTblBytes <= kPnSmemCap) return Q;
    }
}

}  // namespace trex

extern "C" {

int trex_pnfa_create(int n_states, int sigma, const float *T, const float *start, const float *accept,
                     trex_pnfa **out) {
    using namespace trex;
    if (!out) return TREX_ERR_ARG;
    *out = nullptr;
    if (n_states < 1 || n_states > kPnStates || sigma < 1 || sigma > 255 || !T || !start || !accept)
        return TREX_ERR_ARG;
    trex_pnfa *h = new (std::nothrow) trex_pnfa();
    if (!h) return TREX_ERR_OOM;
    h->n_states = n_states;
    h->sigma = sigma;
    h->n_sms = sm_count();
    if (h->n_sms <= 0) {
        delete h;
        set_last_error_msg("trex_pnfa_create: no CUDA device");
        return TREX_ERR_SHAPE;
    }
    const int N = n_states;
    // padded FP32 copies (states >= n_states are zero: they never gain mass)
    std::vector<float> T32((size_t)sigma * 64 * 64, 0.f), s32(64, 0.f), a32(64, 0.f);
    for (int c = 0; c < sigma; ++c)
        for (int d = 0; d < N; ++d)
            for (int q = 0; q < N; ++q) T32[((size_t)c * 64 + d) * 64 + q] = T[((size_t)c * N + d) * N + q];
    double dot = 0.0;
    for (int i = 0; i < N; ++i) {
        s32[i] = start[i];
        a32[i] = accept[i];
        dot += (double)start[i] * (double)accept[i];
    }
    h->ll_empty = dot > 0.0 ? std::log(dot) : -INFINITY;
    // Boolean form: every nonzero entry is an edge (1), start and accept are sets
    std::vector<float> Tb(T32.size()), sb(64), ab(64);
    for (size_t i = 0; i < T32.size(); ++i) Tb[i] = T32[i] != 0.f ? 1.f : 0.f;
    int nacc = 0;
    for (int i = 0; i < 64; ++i) {
        sb[i] = s32[i] != 0.f ? 1.f : 0.f;
        ab[i] = a32[i] != 0.f ? 1.f : 0.f;
        nacc += sb[i] != 0.f && ab[i] != 0.f;
    }
    h->ll_empty_bool = nacc ? std::log((double)nacc) : -INFINITY;
    std::vector<float> rs[4];
    std::vector<uint4> simg[4];
    for (int k = 0; k < 3; ++k) {
        const bool fp16 = k == 1;
        const std::vector<float> &Tk = k == 2 ? Tb : T32;
        const std::vector<float> &sk = k == 2 ? sb : s32;
        rs[k].assign(sigma, 0.f);
        for (int c = 0; c < sigma; ++c) {
            double rmax = 0.0;
            for (int d = 0; d < 64; ++d) {
                double rsum = 0.0;
                for (int q = 0; q < 64; ++q)
                    rsum += std::fabs((double)pn_host16_to_f(pn_host16(Tk[((size_t)c * 64 + d) * 64 + q], fp16), fp16));
                rmax = std::max(rmax, rsum);
            }
            // a little above the largest row sum: bounds max|T s| / max|s| through FP32 rounding
            rs[k][c] = (float)(rmax * (1.0 + 1.0 / 64));
        }
        simg[k].assign(8, make_uint4(0, 0, 0, 0));
        float smax = 0.f;
        for (int i = 0; i < 64; ++i) {
            const uint16_t v = pn_host16(sk[i], fp16);
            smax = std::max(smax, std::fabs(pn_host16_to_f(v, fp16)));
            uint32_t *w = reinterpret_cast<uint32_t *>(&simg[k][i >> 3]);
            w[(i & 7) >> 1] |= (uint32_t)v << (16 * (i & 1));
        }
        h->start_max16[k] = smax;
        if (k < 2) {
            float rmax = 0.f;
            for (int c = 0; c < sigma; ++c) rmax = std::max(rmax, rs[k][c]);
            h->chain_resc[k] = rmax <= 16.f ? 4 : 1;
            if (k == 0) h->tc_resc = h->chain_resc[0];
        }
    }
    {   // int8 Boolean form
        rs[3] = rs[2];
        simg[3].assign(8, make_uint4(0, 0, 0, 0));   // a state row of bytes
        uint8_t *b = reinterpret_cast<uint8_t *>(simg[3].data());
        for (int i = 0; i < 64; ++i) b[i] = sb[i] != 0.f ? 1 : 0;
        h->start_max16[3] = 1.f;
    }
    cudaError_t e = cudaSuccess;
    auto up = [&](void **dst, const void *src, size_t bytes) {
        if (e != cudaSuccess) return;
        if ((e = cudaMalloc(dst, std::max<size_t>(bytes, 16))) != cudaSuccess) return;
        if (bytes) e = cudaMemcpy(*dst, src, bytes, cudaMemcpyHostToDevice);
    };
    up((void **)&h->d_T32, T32.data(), T32.size() * 4);
    for (int k = 0; k < 2; ++k) {
        std::vector<uint16_t> t16(T32.size());
        for (size_t i = 0; i < T32.size(); ++i) t16[i] = pn_host16(T32[i], k == 1);
        up((void **)&h->d_T16[k], t16.data(), t16.size() * 2);
    }
    up((void **)&h->d_start32, s32.data(), 256);
    up((void **)&h->d_acc, a32.data(), 256);
    up((void **)&h->d_acc_bool, ab.data(), 256);
    for (int k = 0; k < 4; ++k) {
        up((void **)&h->d_rsym[k], rs[k].data(), rs[k].size() * 4);
        up((void **)&h->d_simg[k], simg[k].data(), 8 * sizeof(uint4));
    }
    if (e == cudaSuccess) e = cudaMalloc(&h->d_misc, 16);
    if (e == cudaSuccess) e = cudaMemset(h->d_misc, 0, 16);
    // the attribute is per kernel: raised to what any handle can need
    for (const void *f :
         {(const void *)pnfa_sym_kernel<0, false>, (const void *)pnfa_sym_kernel<0, true>,
          (const void *)pnfa_sym_kernel<1, false>, (const void *)pnfa_sym_kernel<1, true>,
          (const void *)pnfa_sym_kernel<2, false>, (const void *)pnfa_sym_kernel<2, true>,
          (const void *)pnfa_sym_kernel<3, false>, (const void *)pnfa_sym_kernel<3, true>,
          (const void *)pnfa_fp32_kernel, (const void *)pnfa_chain_kernel<false>, (const void *)pnfa_chain_kernel<true>})
        if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPnSmemCap);
    if (e != cudaSuccess) {
        set_last_error("trex_pnfa_create", e);
        pn_free(h);
        delete h;
        return e == cudaErrorMemoryAllocation ? TREX_ERR_OOM : TREX_ERR_CUDA;
    }
    *out = h;
    return TREX_OK;
}

void trex_pnfa_destroy(trex_pnfa *h) {
    if (!h) return;
    trex::pn_free(h);
    delete h;
}

int trex_pnfa_run(trex_pnfa *h, int mode, const uint8_t *data, const int64_t *offsets,
                  int64_t n_strings, int64_t total_bytes, double *loglik, uint8_t *accept,
                  int32_t *accept_i32, void *stream) {
    using namespace trex;
    if (!h) return TREX_ERR_NOT_INIT;
    if (n_strings < 0 || total_bytes < 0 || n_strings >= (int64_t)1 << 31) return TREX_ERR_ARG;
    if (mode < TREX_PNFA_BF16 || mode > TREX_PNFA_BOOL8) return TREX_ERR_ARG;
    if (n_strings == 0) return TREX_OK;
    if (!offsets || (total_bytes > 0 && !data)) return TREX_ERR_ARG;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    unsigned long long *queue = reinterpret_cast<unsigned long long *>(h->d_misc);
    uint32_t *err = reinterpret_cast<uint32_t *>(h->d_misc + 8);
    TREX_CUDA(cudaMemsetAsync(h->d_misc, 0, 16, st));
    if (mode == TREX_PNFA_FP32 || mode == TREX_PNFA_BF16_CC || mode == TREX_PNFA_FP16_CC) {
        PnPlainParams Q;
        Q.data = data;
        Q.total_bytes = total_bytes;
        Q.offsets = offsets;
        Q.n = n_strings;
        Q.T = h->d_T32;
        Q.start = h->d_start32;
        Q.acc = h->d_acc;
        Q.sigma = h->sigma;
        Q.ll_empty = h->ll_empty;
        Q.loglik = loglik;
        Q.accept = accept;
        Q.accept_i32 = accept_i32;
        Q.queue = queue;
        Q.err = err;
        if (mode != TREX_PNFA_FP32) {
            const size_t smem = (size_t)h->sigma * 64 * 64 * 2 + kChainSharedBytes;
            if (smem > kPnSmemCap) {
                set_last_error_msg("trex_pnfa_run: the shared-memory CUDA-core form takes at most 28 symbols");
                return TREX_ERR_SHAPE;
            }
            // one CTA an SM (the tables fill its shared memory), four strings at a time each
            const int grid = (int)std::max<int64_t>(
                1, std::min<int64_t>((n_strings + kChainGroups - 1) / kChainGroups, pn_sms(h)));
            const bool fp16 = mode == TREX_PNFA_FP16_CC;
            profile_kernel_begin(st);
            if (fp16)
                pnfa_chain_kernel<true><<<grid, kChainThreads * kChainGroups, smem, st>>>(Q, h->d_T16[1],
                                                                                          h->chain_resc[1]);
            else
                pnfa_chain_kernel<false><<<grid, kChainThreads * kChainGroups, smem, st>>>(Q, h->d_T16[0],
                                                                                           h->chain_resc[0]);
            profile_kernel_end(st);
            TREX_CHECK_LAUNCH();
            return TREX_OK;
        }
        // alphabets whose tables fit on an SM: strings in rings by symbol (20 symbols, 8192 strings x 512:
        // 1.72 ms against 16.7; 64 x 512 0.59 against 2.3, one string of 4096 4.4 against 6.5); larger ones
        // read every table through L1 and L2
        if (h->sigma <= kRiWarps) {
            RiParams S = ri_params(h, n_strings);
            S.data = data;
            S.total_bytes = total_bytes;
            S.offsets = offsets;
            S.n = n_strings;
            S.loglik = loglik;
            S.accept = accept;
            S.accept_i32 = accept_i32;
            S.queue = queue;
            S.err = err;
            profile_kernel_begin(st);
            pnfa_fp32_kernel<<<S.grid, 32 * S.n_rings, S.tbl_off + (uint32_t)S.sigma * kRiTblBytes, st>>>(S);
            profile_kernel_end(st);
            TREX_CHECK_LAUNCH();
            return TREX_OK;
        }
        const int64_t warps = std::min<int64_t>(n_strings, pn_sms(h) * 64);
        const int grid = (int)std::max<int64_t>(1, (warps + kPnPlainWarps - 1) / kPnPlainWarps);
        profile_kernel_begin(st);
        pnfa_plain_kernel<<<grid, kPnPlainWarps * 32, 0, st>>>(Q);
        profile_kernel_end(st);
        TREX_CHECK_LAUNCH();
        return TREX_OK;
    }
    // Strings on TMEM lanes up to four symbols: at four, 262144 x 512 take 4.26 / 4.65 / 2.53 ms (BF16,
    // FP16, int8) there and 7.11 / 8.94 / 5.30 with lists by symbol; above, A's columns (32 a symbol)
    // leave room for fewer tiles and B outgrows its 32 KB. (The other side: below some ten thousand
    // strings the lists spread them over more SMs, 512 x 2048 at four symbols 2.37 / 2.61 / 2.46 ms on
    // lanes, 1.76 / 1.98 / 1.21 in lists; 32768 x 512 0.65 / 0.71 / 0.68 and 1.07 / 1.29 / 0.79.)
    if (h->sigma <= kLnMaxSigma) {
        const int k = mode == TREX_PNFA_FP16 ? 1 : mode == TREX_PNFA_BOOL8 ? 2 : mode == TREX_PNFA_BOOL ? 3 : 0;
        LnParams Q;
        Q.data = data;
        Q.total_bytes = total_bytes;
        Q.offsets = offsets;
        Q.n = n_strings;
        Q.T16 = h->d_T16[k == 1 ? 1 : 0];
        Q.T32 = h->d_T32;
        Q.start = h->d_start32;
        Q.acc = k >= 2 ? h->d_acc_bool : h->d_acc;
        Q.sigma = h->sigma;
        Q.a_cols = (uint32_t)(k == 2 ? 16 : 32) * (uint32_t)h->sigma;
        Q.tile_cols = (Q.a_cols + 64u + 31u) & ~31u;
        Q.tiles = (int)std::min<uint32_t>((uint32_t)kLnTiles, 512u / Q.tile_cols);
        Q.resc = k == 0 ? h->tc_resc : 1;
        Q.wait_cycles = mbar_wait_cycles();
        Q.ll_empty = k >= 2 ? h->ll_empty_bool : h->ll_empty;
        Q.loglik = loglik;
        Q.accept = accept;
        Q.accept_i32 = accept_i32;
        Q.queue = queue;
        Q.err = err;
        // one CTA an SM (it owns the 512 TMEM columns), 128 strings in flight a tile
        const int64_t per_cta = (int64_t)Q.tiles * 128;
        const int grid = (int)std::max<int64_t>(
            1, std::min<int64_t>((n_strings + per_cta - 1) / per_cta, pn_sms(h)));
        profile_kernel_begin(st);
        if (k == 1) pnfa_lane_kernel<1><<<grid, kLnThreads, 0, st>>>(Q);
        else if (k == 2) pnfa_lane_kernel<2><<<grid, kLnThreads, 0, st>>>(Q);
        else if (k == 3) pnfa_lane_kernel<3><<<grid, kLnThreads, 0, st>>>(Q);
        else pnfa_lane_kernel<0><<<grid, kLnThreads, 0, st>>>(Q);
        profile_kernel_end(st);
        TREX_CHECK_LAUNCH();
        return TREX_OK;
    }
    if (h->sigma > kSyMaxSigma) {
        set_last_error_msg("trex_pnfa_run: the tensor-core form takes at most 28 symbols");
        return TREX_ERR_SHAPE;
    }
    const int k = mode == TREX_PNFA_FP16 ? 1 : mode == TREX_PNFA_BOOL ? 2 : mode == TREX_PNFA_BOOL8 ? 3 : 0;
    SyParams Q;
    Q.data = data;
    Q.total_bytes = total_bytes;
    Q.offsets = offsets;
    Q.n = n_strings;
    Q.T16 = h->d_T16[k == 1 ? 1 : 0];
    Q.T32 = h->d_T32;
    Q.start_img = h->d_simg[k];
    Q.acc = k >= 2 ? h->d_acc_bool : h->d_acc;
    Q.sigma = h->sigma;
    Q.rep = std::max(1, kSyWarps / h->sigma);
    Q.rsym = h->d_rsym[k];
    Q.start_max = h->start_max16[k];
    Q.resc = k == 0 ? h->tc_resc : 1;
    Q.wait_cycles = mbar_wait_cycles();
    Q.ll_empty = k >= 2 ? h->ll_empty_bool : h->ll_empty;
    Q.loglik = loglik;
    Q.accept = accept;
    Q.accept_i32 = accept_i32;
    Q.queue = queue;
    Q.err = err;
    // one CTA an SM (its registers hold the tables), the strings spread over all SMs
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(n_strings, pn_sms(h)));
    const uint32_t row = k == 3 ? sy_row_bytes<2>() : sy_row_bytes<0>();
    uint32_t smem = 0;
    for (Q.slots = (int)std::min<int64_t>((n_strings + grid - 1) / grid, kSyMaxSlots);; --Q.slots) {
        const uint32_t n = (uint32_t)Q.slots;
        Q.cap_shift = 3;
        while ((1 << Q.cap_shift) < Q.slots) ++Q.cap_shift;
        Q.state_off = kSyRecs + n * (uint32_t)sizeof(SyRec);
        Q.sym_off = Q.state_off + n;
        Q.raw_off = pn_align16(Q.sym_off + 2u * kSyBlk * n);
        Q.list_off = Q.raw_off + 32u * n;
        Q.rows_off = pn_align16(Q.list_off + (4u << Q.cap_shift) * (uint32_t)Q.sigma);
        smem = Q.rows_off + n * row;
        if (smem <= kPnSmemCap) break;
    }
    const int threads = 32 * std::min(kSyWarps, Q.sigma * Q.rep);
    profile_kernel_begin(st);
    const bool several = Q.sigma > kSyWarps;
    void (*const f)(SyParams) = k == 1   ? (several ? pnfa_sym_kernel<1, true> : pnfa_sym_kernel<1, false>)
                                : k == 2 ? (several ? pnfa_sym_kernel<3, true> : pnfa_sym_kernel<3, false>)
                                : k == 3 ? (several ? pnfa_sym_kernel<2, true> : pnfa_sym_kernel<2, false>)
                                         : (several ? pnfa_sym_kernel<0, true> : pnfa_sym_kernel<0, false>);
    f<<<grid, threads, smem, st>>>(Q);
    profile_kernel_end(st);
    TREX_CHECK_LAUNCH();
    return TREX_OK;
}

int trex_pnfa_set_sm_limit(trex_pnfa *pnfa, int max_sms) {
    if (!pnfa || max_sms < 0) return TREX_ERR_ARG;
    pnfa->sm_limit = max_sms;
    return TREX_OK;
}

int trex_pnfa_error(trex_pnfa *h, int32_t *err_out) {
    if (!h || !err_out) return TREX_ERR_ARG;
    uint32_t v = 0;
    TREX_CUDA(cudaMemcpy(&v, h->d_misc + 8, 4, cudaMemcpyDeviceToHost));
    *err_out = (int32_t)v;
    return TREX_OK;
}

}  // extern "C"
