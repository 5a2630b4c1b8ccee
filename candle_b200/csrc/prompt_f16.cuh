// Shared parts of the f16 prompt kernels (prompt_kq.cu: Q4_K / Q6_K with one activation scale per 256 elements;
// prompt_b32.cu: formats with an activation scale per 32 elements).
//
// Both run the quantized product on `tcgen05.mma kind::f16` with INTEGERS in f16: int8 activations, and weight codes times
// their integer sub-scales, are whole numbers of at most 11 significant bits, so every product is exact and the f32
// accumulator holds the exact integer sum as long as no partial sum passes 2^24: each kernel says how it sees to that.  Against
// int8 operands this saves the second weight plane (Q4_K) and the int -> float conversions of the epilogue.
//
// Operand A (M = 128 weight rows) lives in TENSOR MEMORY: a producer thread owns one row = one TMEM lane, expands its GGUF
// bytes in registers and stores them with `tcgen05.st`.  Through shared memory the same operand would cost a write and, per
// MMA, a read of 4 KiB: at N = 128 the two operands' reads alone would fill the 128 B/clk shared-memory pipe.  Operand B
// (N = up to 128 tokens, any multiple of 16, so a ragged tile pays only for the tokens it has) comes pre-tiled from the
// quantize kernel with bulk copies.  The accumulator lane is then the weight row, so 32 lanes store 32 consecutive outputs.
// Measured rate of this form (one CTA per SM): 16.4 / 32.3 / 64.4 clocks per MMA at N = 32 / 64 / 128, the nominal rate; with
// A in shared memory 40 / 48 / 64, so small token tiles need the tensor-memory form.
#pragma once
#include "common.cuh"
#include "tcgen05.cuh"
#include "tensor_map.cuh"

namespace cq_prompt {
using namespace cq_tc;

constexpr int kRows = 128;         // weight rows per CTA tile (MMA M = TMEM lanes)
constexpr int kTokMax = 128;       // tokens per CTA tile (MMA N), at most

// Issuing.  An MMA takes its descriptors and addresses from uniform registers.  Computed by one diverged thread they sit in vector
// registers and are moved over one by one, ~115 clocks per MMA (measured: 2300 clocks of issue per 256 k-elements, where the
// MMAs of 128 tokens last 1090).  So the whole warp runs the issuing loop on values the compiler can keep uniform - loop
// counters, kernel arguments, constants, and a tile's token count passed through a warp reduction - and one elected lane
// executes the instruction.  A shared-memory descriptor is kept as its low word: address / 16 and, in the upper half, the
// distance / 16 between the two 16-byte halves of a K step, which for a tile of n tokens is n; the next K step is 2 n further.
// Hand-offs are kept coarse: a wait that has to be woken costs 110 - 190 clocks, a commit 45 to issue and 180 until it is seen.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ uint32_t uniform(uint32_t v) { return __reduce_max_sync(0xffffffffu, v); }      // the same in every lane
__device__ __forceinline__ uint64_t desc_of(uint32_t lo) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"((128u >> 4) | (1u << 14)));      // 8-row groups 128 bytes apart; sm_100 descriptor
    return r;
}
// D[128 rows][n tokens] (+)= A[tmem: 128 x 16 f16] * B[smem: n x 16 f16]
template <bool ACC> __device__ __forceinline__ void mma_f16_ts(uint32_t tmem_d, uint32_t tmem_a, uint32_t desc_b, uint32_t idesc) {
    if constexpr (ACC)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.b32 p, 0, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                     ::"r"(tmem_d), "r"(tmem_a), "l"(desc_of(desc_b)), "r"(idesc) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, 0, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                     ::"r"(tmem_d), "r"(tmem_a), "l"(desc_of(desc_b)), "r"(idesc) : "memory");
}
// the same with A in shared memory, into a fresh accumulator
__device__ __forceinline__ void mma_f16_ss(uint32_t tmem_d, uint32_t desc_a, uint32_t desc_b, uint32_t idesc) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, 0, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "l"(desc_of(desc_a)), "l"(desc_of(desc_b)), "r"(idesc) : "memory");
}
// kind::f16 instruction descriptor: D = f32, A = B = f16, both K-major, M = 128, N = n.
__device__ __forceinline__ uint32_t idesc_f16(int n) { return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kRows >> 4) << 24); }

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t *v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
}
// 8 N columns of 16 lanes: value 4 j + 2 s + e of a thread is lane 8 s + lane / 4, column 8 j + 2 (lane % 4) + e.
template <int N> __device__ __forceinline__ void tmem_ld_16x256b(uint32_t taddr, uint32_t *v) {
    static_assert(N == 2 || N == 4, "");
    if constexpr (N == 2)
        asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]) : "r"(taddr) : "memory");
    else
        asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                     : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
                       "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Bounded wait like wait_or_abort; between two looks at the barrier the warp sleeps, since fourteen waiting warps that poll took more than half of all issue
// slots, from the producers above all.  The votes keep the loop free of divergence, and the expected case falls through.  The bound counts looks, 2^23
// sleeps of 64 ns, and so the loop tests and does not try: a try may suspend the warp for a time of its own, any number of which is no bound.  A clock
// would do, too, but every wait is copied into its place - calls do not go with changed register budgets - and the longer code cost 3 - 5 % of Q6_K
// and Q8_0 prompts (14336 -> 4096, 512 tokens 140 us -> 145; 4096 -> 4096, 333 tokens 64.7 -> 67.7).
// There is no per-lane form: every role goes on to warp-wide instructions, so its warp decides as one whether a wait gave up (lanes
// that left at different places would meet at different warp-wide instructions, which need not end).
__device__ __forceinline__ bool wait_warp(uint64_t *bar, unsigned parity, volatile int *abort_flag) {
    if (__builtin_expect(__all_sync(0xffffffffu, cq_mbar_try_wait(bar, parity)), 1)) return true;
#pragma unroll 1
    for (unsigned n = 0; n < (1u << 23); ++n) {
        __nanosleep(64);
        if (__all_sync(0xffffffffu, cq_mbar_test_wait(bar, parity))) return true;
        if ((n & 1023u) == 1023u && __any_sync(0xffffffffu, *abort_flag)) return false;
    }
    *abort_flag = 1;
    return false;
}
// One arrival per warp: barriers count warps, not threads.
__device__ __forceinline__ void arrive_warp(uint64_t *bar, int lane) {
    __syncwarp();
    asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.s32 p, %1, 0;\n\t@p mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}" ::"r"(cq_smem_u32(bar)), "r"(lane) : "memory");
}

// Register budgets per warpgroup (kernels of 640 threads = 96 registers each at launch, 61,440 in all): the two epilogue
// warpgroups go up to 128, the two producer warpgroups down to 88, the one of the issuing and loading warps to 48:
// 256 * 128 + 256 * 88 + 128 * 48 = 61,440.
constexpr int kRegsEpi = 128, kRegsProd = 88, kRegsMisc = 48;
template <int N> __device__ __forceinline__ void regs_up() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void regs_down() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

// (x & M) | C and (x & M) ^ C: written in C with two constants they became two instructions each
template <uint32_t M, uint32_t C> __device__ __forceinline__ uint32_t and_or(uint32_t x) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(x), "n"(M), "n"(C));
    return r;
}
template <uint32_t M, uint32_t C> __device__ __forceinline__ uint32_t and_xor(uint32_t x) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0x6A;" : "=r"(r) : "r"(x), "n"(M), "n"(C));
    return r;
}
template <uint32_t M> __device__ __forceinline__ uint32_t and_or(uint32_t x, uint32_t c) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(x), "n"(M), "r"(c));
    return r;
}

// two f32 operations per instruction; each half rounds like the scalar operation
__device__ __forceinline__ uint64_t pack2(uint32_t lo, uint32_t hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ uint64_t pack2f(float lo, float hi) { return pack2(__float_as_uint(lo), __float_as_uint(hi)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float lo2(uint64_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi2(uint64_t v) { return __uint_as_float((uint32_t)(v >> 32)); }

__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<uint32_t *>(&h); }
__device__ __forceinline__ __half2 bits_h2(uint32_t b) { return *reinterpret_cast<__half2 *>(&b); }
__device__ __forceinline__ uint32_t hfma2_bits(uint32_t a, __half2 b, __half2 c) { return h2_bits(__hfma2(bits_h2(a), b, c)); }

// K runs in groups of four with the middle two swapped (elements 0, 2, 1, 3): masking a word of four codes gives the
// pairs (byte 0, byte 2) and (byte 1, byte 3), which is what lies in one 32-bit TMEM cell.  Both operands use this order.

// Eight consecutive activations of one lane; `vec`: the row is 16-byte aligned.
__device__ __forceinline__ void load8(const float *p, bool vec, float (&e)[8]) {
    if (vec) {
        const float4 a = *reinterpret_cast<const float4 *>(p), b = *reinterpret_cast<const float4 *>(p + 4);
        e[0] = a.x; e[1] = a.y; e[2] = a.z; e[3] = a.w; e[4] = b.x; e[5] = b.y; e[6] = b.z; e[7] = b.w;
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) e[i] = p[i];
    }
}
template <typename T> __device__ __forceinline__ void load8(const T *p, bool vec, float (&e)[8]) {      // 16-bit types
    if (vec) {
        const uint4 a = *reinterpret_cast<const uint4 *>(p);
        const T *h = reinterpret_cast<const T *>(&a);
#pragma unroll
        for (int i = 0; i < 8; ++i) e[i] = cq_elem_to_float(h, i);
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) e[i] = cq_elem_to_float(p, i);
    }
}
// eight integral floats of at most 2048 as f16 in the operands' K order
__device__ __forceinline__ uint4 pack_q8(const float (&q)[8]) {
    return make_uint4(h2_bits(__floats2half2_rn(q[0], q[2])), h2_bits(__floats2half2_rn(q[1], q[3])), h2_bits(__floats2half2_rn(q[4], q[6])),
                      h2_bits(__floats2half2_rn(q[5], q[7])));
}
// eight small integers, the same
__device__ __forceinline__ uint4 pack_q8(const int (&q)[8]) {
    auto pr = [](int a, int b) { return h2_bits(__halves2half2(__short2half_rn((short)a), __short2half_rn((short)b))); };
    return make_uint4(pr(q[0], q[2]), pr(q[1], q[3]), pr(q[4], q[6]), pr(q[5], q[7]));
}

// Eight tokens x 32 weight rows of a warp as a 16-bit kind: v[i] are a thread's values of row 8 i + lane / 4, tokens 2 (lane % 4) and the next (the 16x256b
// layout).  `dst`: row 0 of the first token; `rows`: how many of the 32 are stored; `tokens`: how many of the eight.
__device__ __forceinline__ uint32_t pair_16bit(uint64_t v, int kind) {
    if (kind == CQ_F16) return h2_bits(__halves2half2(__float2half(lo2(v)), __float2half(hi2(v))));
    const __nv_bfloat162 b = __halves2bfloat162(__float2bfloat16(lo2(v)), __float2bfloat16(hi2(v)));
    return *reinterpret_cast<const uint32_t *>(&b);
}
// Rows a multiple of 16 bytes apart: 8 x 8 transposes leave a thread with rows 8 i + 2 (lane % 4), + 1 of token lane / 4, a 4 x 4 transpose over four lanes with
// eight rows of it, so a token's 32 rows go out as 64 contiguous bytes.  (Stored as they lie, in 16-byte pieces of half a sector, the 2048 x 14336
// outputs of a bf16 prompt took 25 us more than twice the bytes as f32.)
__device__ __forceinline__ void store_rows32_wide(const uint64_t (&v)[4], int kind, uint16_t *dst, int64_t stride, int rows, int tokens) {
    const int lane = threadIdx.x & 31;
    uint32_t r[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r[i]) : "r"(pair_16bit(v[i], kind)));
#pragma unroll
    for (int m = 1; m < 4; m <<= 1) {           // swap bit log2 m of the register number with that of the lane
        const bool up = lane & m;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (!(i & m)) {
                const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? r[i] : r[i | m], m);
                if (up) r[i] = got; else r[i | m] = got;
            }
    }
    const int row = 8 * (lane & 3), tok = lane >> 2;
    if (row < rows && tok < tokens) *reinterpret_cast<uint4 *>(dst + tok * stride + row) = make_uint4(r[0], r[1], r[2], r[3]);     // rows: a multiple of eight
}
// Any distance: a lane per row, so that a token's rows go out as one run.  (Pieces of two bytes after the transposes above: 4 x the sectors, Q4_K
// 6144 -> 12108, 320 tokens f16 83 us; this 70.)
__device__ __forceinline__ void store_rows32_any(const uint64_t (&v)[4], int kind, uint16_t *dst, int64_t stride, int rows, int tokens) {
    const int lane = threadIdx.x & 31;
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = pair_16bit(v[i], kind);
#pragma unroll
    for (int c = 0; c < 4; ++c) {               // tokens 2 c and 2 c + 1 of row `lane`
        uint32_t got[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) got[i] = __shfl_sync(0xffffffffu, w[i], 4 * (lane & 7) + c);
        const uint32_t x = lane & 16 ? (lane & 8 ? got[3] : got[2]) : (lane & 8 ? got[1] : got[0]);
        if (lane < rows && 2 * c < tokens) dst[2 * c * stride + lane] = (uint16_t)x;
        if (lane < rows && 2 * c + 1 < tokens) dst[(2 * c + 1) * stride + lane] = (uint16_t)(x >> 16);
    }
}

// What a kernel stores, one instantiation each (the code of the others between the loops of a tile costs them 5 - 10 % in instruction fetches):
// f32 or 16-bit rows of tokens (a multiple of 16 bytes apart, or not), or f32 rows of (token, expert) pairs.
enum { kStoreF32, kStore16, kStore16Any, kStorePairs };
inline bool rows_16_bytes_apart(const void *out, int stride) { return ((uintptr_t)out & 15) == 0 && stride % 8 == 0; }

// ---- tiles --------------------------------------------------------------------------------------------------
// The jobs of a grouped (expert-indexed) launch; null `tiles` = dense.
struct GroupInfo {
    const int *tiles;                  // [max_tiles][4]: expert, first job, valid rows, first blob row; then the number of tiles in use
    const int32_t *sorted_token_ids;
    const float *topk_weights;
    long long expert_rows;             // weight rows per expert
    int topk, row_per_pair;            // input row of a pair: the pair itself, or pair / topk
};

// Tokens are cut into `ntt` tiles of `tt` (a multiple of 16, at most 128).  The activation blobs of (tile, 256-element chunk)
// follow each other, their rows padded to a multiple of 16.
struct Tiling {
    int tokens, tt, ntt;
    __host__ __device__ int rows(int t) const {
        const int left = tokens - t * tt;
        return ((left < tt ? left : tt) + 15) / 16 * 16;
    }
};

struct TileCtx {
    int row0;           // first weight row inside the matrix (of the expert)
    long long wrow0;    // the same counted from the start of the weights
    long long blob_row; // rows of activation blobs before this tile
    int t, valid, n, job0;
};
// Tile number -> row tile and token tile; `ntt` token tiles are in use.
__device__ __forceinline__ void tile_ctx(int tile, int ntt, const Tiling &tl, const GroupInfo &gi, TileCtx &c) {
    c.t = tile % ntt;
    c.row0 = (tile / ntt) * kRows;
    c.wrow0 = c.row0;
    c.job0 = 0;
    if (gi.tiles) {
        const int4 ti = *reinterpret_cast<const int4 *>(gi.tiles + 4 * c.t);
        c.valid = ti.z;
        c.wrow0 += ti.x * gi.expert_rows;
        c.job0 = ti.y;
        c.blob_row = ti.w;
    } else {
        c.blob_row = (long long)c.t * tl.tt;
        const int left = tl.tokens - c.t * tl.tt;
        c.valid = left < tl.tt ? left : tl.tt;
    }
    c.n = (c.valid + 15) / 16 * 16;
}

// Number of token tiles for `nrt` row tiles.  Results do not depend on it.  A tile's time per chunk is affine in its tokens, `fixed`
// tokens' worth of it whatever they are (expanding 128 weight rows and the hand-offs); the launch takes as many rounds of `sms`
// tiles as it needs.  Q4_K on B200: 0.68 us + 4.5 ns per token, hence 150.
inline Tiling plan_tiling(int tokens, int nrt, int sms, int fixed, int tok_max = kTokMax) {
    Tiling best{tokens, 16, 0};
    long long best_cost = -1;
    for (int ntt = (tokens + tok_max - 1) / tok_max; ntt <= (tokens + 15) / 16; ++ntt) {
        const int tt = ((tokens + ntt - 1) / ntt + 15) / 16 * 16;
        if ((tokens + tt - 1) / tt != ntt) continue;
        const long long rounds = ((long long)nrt * ntt + sms - 1) / sms;
        const long long cost = rounds * (tt + fixed);
        if (best_cost < 0 || cost < best_cost) { best_cost = cost; best.tt = tt; best.ntt = ntt; }
        if (rounds > 64) break;          // many rounds: smaller tiles only repeat the expansion
    }
    return best;
}

inline int sm_count() { return cq_sm_count(); }

// ---- raw weight bytes: (128 rows, one 256-element chunk) -> shared memory ---------------------------------------
// One tiled TMA copy when rows are whole multiples of 16 bytes apart; else (Q6_K rows of K % 2048 != 0 and the like) two warps copy
// 16-byte pieces with cp.async, a lane per piece and two rows per warp step, from the 16-byte boundary below each row's chunk - a bulk copy
// per row was three times slower than the whole int8 kernel, and splitting a running piece number into row and piece made Q6_K of
// K = 2304 .. 14080 up to 30 % slower than this (128 experts, K = 1792 -> 768, 512 pairs: 157 us, now 125).  In shared memory row r starts
// at r * kPitch, the chunk a few bytes behind it when it does not start on such a boundary.  CB: bytes of a chunk.
constexpr int kRawThreads = 64;
template <int CB> struct Raw {
    static constexpr bool kAligned = CB % 16 == 0;
    static constexpr int kNeed = kAligned ? CB : (CB + 14 + 15) / 16 * 16;       // 16-byte window that covers the chunk
    // pitch: an odd number of 16-byte units, so that eight lanes' 16-byte reads of one column fall into different banks
    static constexpr int kPitch = (kNeed / 16) % 2 ? kNeed : kNeed + 16;
    static_assert(kAligned || kNeed <= 256, "one unit per thread");
    static constexpr int kBytes = kRows * kPitch;
    // Pieces reach at most the last 16-byte unit that holds a byte of the chunk, rows past the matrix repeat its last one.
    // `bar` counts kRawThreads; `w` points at the chunk of the tile's first row, `rows_left` rows are in memory from there.
    static __device__ __forceinline__ void load_rows(uint8_t *dst, const uint8_t *w, int rows_left, uint32_t row_bytes, int thread, uint64_t *bar) {
        // 16 threads per row (one 16-byte unit each), four rows at a time
        const int u = thread & 15;
        if (16 * u < kNeed) {
            uint32_t to = cq_smem_u32(dst) + (uint32_t)((thread >> 4) * kPitch + 16 * u);
            const uint8_t *p = w + (size_t)(uint32_t)min(thread >> 4, rows_left - 1) * row_bytes, *last = w + (size_t)(uint32_t)(rows_left - 1) * row_bytes;
#pragma unroll 8
            for (int i = 0; i < kRows / 4; ++i) {
                const uintptr_t src = ((uintptr_t)p & ~(uintptr_t)15) + 16 * u;
                if (src < (uintptr_t)p + CB) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to), "l"(src) : "memory");
                to += 4 * kPitch;
                p += 4 * (size_t)row_bytes;
                if (p > last) p = last;
            }
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(cq_smem_u32(bar)) : "memory");
    }
};

}  // namespace cq_prompt
