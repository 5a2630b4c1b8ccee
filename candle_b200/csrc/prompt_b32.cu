// Prompt-phase quantized GEMM for activations with one scale per 32 elements, on tcgen05.mma kind::f16 (prompt_f16.cuh):
//   Q8_0, Q4_0                            BlockQ8_0 activations, candle's CPU arithmetic (k_quants.rs:294-311, 720-738)
//   Q4_1, Q5_0, Q5_1, Q2_K, Q3_K, Q5_K     Q8_1 activations, the arithmetic of the decode kernels (mmvq_gguf.cu:208-334, 357-381,
//                                          492-531; gemv_chunks.cuh), the same arithmetic at every row count
//
// Both sides of a product carry a scale per 32 elements, so nothing beyond the integer sub-scales of a K-quant can be folded
// into the operands: every 32-element block is two K = 16 steps into a FRESH accumulator slot, exact (sums below 2^24: at most
// 16 * 63 * 127 * 32), and the epilogue adds the scaled slots to f32 running sums, two values per instruction.
//
// What moved out of the epilogue, whose instructions per block bound the kernel before:
//   * The minimum part of the formats that have one.  Codes are CENTRED (signed) in the operand - q - 8, q - 16, sc (q - 16), sc (2 q - 3), sc (q - 4) - and
//     what the shift and the minimum contribute together is a sum over a chunk of (coefficient of the weights) x (sum of the activations):
//         Q5_K  sum_g (16 d sc_g - dmin m_g) s_g     Q2_K  sum_j (1.5 d sc_j - dmin m_j) s_j, per 16 elements     Q5_0  sum_g -16 d_g (t_g - s_g)
//     with s = d_a sum q8 and t the f16 sum of the inputs that Q8_1 stores.  Coefficients and sums are f32; each is split exactly into three
//     bf16 parts, hi, mid and lo, and the six products of parts down to 2^-16 are K steps of the tensor core.  It cuts sums off where an f32 addition
//     rounds, a bias that adds up over the chunks of one-signed data, so hi hi has an accumulator of its own and hi no more than 7 bits: its sums of 8 or 16
//     products fit 24 bits, up to terms 2^-7 of the largest, and the other five products are small enough for a cut not to matter; the two sums are
//     added in f32.  The large parts of d q and the minimum cancel in the coefficient and not in sums of thousands.  2-norm error against 64
//     bits, K = 4096, a minimum added per block in f32 / here:  weights around zero, normal activations Q5_K 8.8e-8 / 5.7e-8, Q2_K 7.2e-8 / 5.5e-8, Q5_0
//     6.7e-8 / 6.5e-8; no minimum and activations of one sign Q5_K 2.5e-8 / 2.5e-8, Q2_K 3.2e-8 / 3.1e-8 (4.9e-8 and 5.3e-8 with all products in one
//     accumulator).  Larger only where every code of a block is its lowest and its
//     scale is not zero, which no quantizer writes (Q5_K 6.0e-8 / 6.7e-8).  It costs 7 % (Q5_K
//     4096 -> 14336, 512 tokens 237 us -> 253).  Not for Q4_1 and Q5_1, whose stored sum can be most of the result: their codes stay unsigned and a
//     block's two parts meet in the epilogue.
//   * A super-block format has one d per 256 elements: a block is then ONE fma per value, sum += d_a I, and d is applied per chunk.
//   * The accumulators are read with the 16x256b shape of tcgen05.ld: a thread holds four rows x two columns of each eight columns, so one
//     8-byte shared load of token scales serves eight values (a 16-byte load served four with a row per lane: a broadcast takes as long as the
//     bytes it delivers, 1.2 loads of 16 bytes a clock and SM).
//
// Summation: Q8_0 / Q4_0 add block after block, as the kernel behind cq_prefill32_gemm does (the same f32 operations, the same
// bits).  The decode kernels, which the Q8_1 formats use otherwise, sum by a balanced tree; a plain chain of K / 32 additions would
// lose precision against that, so the blocks of a 256-element chunk are added first and the chunks with a compensated sum.
//
// Mapping as in prompt_kq.cu: tiles of 128 weight rows x up to 64 tokens (the compensated sums take three registers per value),
// warps 0-7 epilogue, 8-15 producers (two sets of four, a weight row per thread, the sets take turns), 16 MMA issuer, 17 loader, 18-19
// raw bytes where there is no tensor map; tensor memory: three accumulator slots of two blocks (128 columns each), which the minimum sums of a chunk take
// like a fifth pair, and operand A in three buffers of two blocks.  The roles hand over two blocks at a time; where no minimum sums are between
// them, slots and buffers go together and one commit tells both the producers and the epilogue.  Every wait is bounded as there.
//
// bf16 results of Q5_0, Q5_K, Q2_K and Q3_K that QMatMul.forward returns come from PLAIN sums: unsigned codes, d and the minimum in the terms of each block, in f32.
// Sums in the other order differ by 1e-7 of them, and a few in 100 000 bf16 results then round to the neighbouring value, 2^-8 to 2^-7 of it away; bf16
// results keep their bits instead, for 14 - 59 % more time (512 tokens below: Q5_K 325 us, Q2_K 418, Q5_0 351, Q3_K 296).  Before this mapping: 468, 579, 482, 475.
//
// Measured (B200, quantizer included, f32; before this mapping -> now): 4096 -> 14336, 512 tokens Q5_K 493 us -> 253, Q2_K 263, Q5_0 306, Q3_K 259, Q4_1 337, Q5_1 350,
// Q4_0 226, Q8_0 212; Q8_0 4096 -> 4096, 333 tokens 88 -> 65.  A chunk of 256 elements takes about 2.2 us and 11 ns per token, 11 - 13 thousand warp
// instructions at 2.3 a clock; two tensor-core steps of a block are 64 clocks.
// Tried: tiles of 128 tokens with one producer set (Q5_K 327), the group's first warp polling for the others (534: branches and barrier reads outweigh
// the polls), a branch on the tile's tokens inside the block loop (312: the compiler then moves every running sum).
#include "../../include/candle_q_b200.h"
#include "prompt_f16.cuh"

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace {
using namespace cq_prompt;

constexpr int kEpiWarps = 8, kProdWarps = 8;     // producers: two sets of four
constexpr int kMmaWarp = kEpiWarps + kProdWarps, kLoadWarp = kMmaWarp + 1, kRawWarp = kMmaWarp + 2;
constexpr int kThreads = (kEpiWarps + kProdWarps + 4) * 32;      // the last two: raw bytes without a tensor map
constexpr int kTok = 64;                         // tokens per tile, at most
constexpr int kSlots = 3;                        // accumulator slots of two blocks
constexpr int kStagesT = 4;                      // token stages of half a chunk
constexpr int kRawStages = 3;                    // chunks of raw weight bytes
constexpr int kFixedTokens = 180;                // plan_tiling: 2.1 us + 11 ns per token and chunk
// registers: 640 threads x 96 at launch = 256 * 144 + 256 * 72 + 128 * 48
constexpr int kRegsEpi32 = 144, kRegsProd32 = 72, kRegsMisc32 = 48;

__device__ int g_prompt_b32_timeout_flag = 0;

// kSum: the activations' sums of the minimum part: none; s per 32 (Q5_K) or 16 (Q2_K) elements, t - s (Q5_0), which meet their coefficients on the tensor
// core; t (Q4_1, Q5_1), which meets the minima in the epilogue.  PLAIN: all of them in the epilogue, with unsigned codes and a block's d in its own
// term; no difference for Q8_0, Q4_0, Q4_1 and Q5_1.  kTerm: the terms of a block are added up apart from the running sum: d_a d_w I and m_w s are both large and nearly
// cancel for weights around zero; added to the running sum one after the other they left two to four times the decode kernels' error against 64 bits (2-norm, K = 4096,
// activations of one sign: Q4_1 2.2e-7 for 7.6e-8, Q5_1 2.6e-7 for 7.7e-8; now 6.7e-8 and 6.9e-8).  Q5_K stays below the decode kernel's error without.
enum { kNoSum, kSum32, kSum16, kDelta, kTermSum, kPlain32, kPlain16 };
template <int SUM, bool Q81, bool BLOCK, bool TERM = false> struct FmtOf {
    static constexpr bool kQ81 = Q81, kBlockScale = BLOCK, kTerm = TERM;
    static constexpr int kSum = SUM, kMins = SUM == kTermSum || SUM == kPlain32 ? 1 : SUM == kPlain16 ? 2 : 0;       // minima of a block in the epilogue
};
template <int WTYPE, bool PLAIN> struct Fmt : FmtOf<kNoSum, false, true> {};       // Q8_0, Q4_0
template <bool PLAIN> struct Fmt<CQ_Q4_1, PLAIN> : FmtOf<kTermSum, true, true, true> {};
template <bool PLAIN> struct Fmt<CQ_Q5_1, PLAIN> : FmtOf<kTermSum, true, true, true> {};
template <> struct Fmt<CQ_Q5_0, false> : FmtOf<kDelta, true, true> {};
template <> struct Fmt<CQ_Q5_0, true> : FmtOf<kTermSum, true, true, true> {};
template <> struct Fmt<CQ_Q5_K, false> : FmtOf<kSum32, true, false> {};
template <> struct Fmt<CQ_Q5_K, true> : FmtOf<kPlain32, true, false> {};
template <> struct Fmt<CQ_Q2_K, false> : FmtOf<kSum16, true, false> {};
template <> struct Fmt<CQ_Q2_K, true> : FmtOf<kPlain16, true, false, true> {};
template <bool PLAIN> struct Fmt<CQ_Q3_K, PLAIN> : FmtOf<kNoSum, true, false> {};

constexpr int sums_of(int sum) { return sum == kSum32 || sum == kDelta ? 8 : sum == kSum16 ? 16 : 0; }   // coefficients per chunk
constexpr int kColA = 384;                       // tensor memory column of operand A
// f16 values; scales, and sums where the epilogue takes them; planes of bf16 sums (lo, mid, hi where finite, zeros where two planes make a K step, hi) of one
// token and chunk
constexpr int float_bytes(int sum) { return sum == kTermSum || sum == kPlain32 ? 64 : sum == kPlain16 ? 96 : 32; }
constexpr int planes_of(int sum) { return sums_of(sum) == 8 ? 5 : sums_of(sum) / 4; }
constexpr int sum_bytes(int sum) { return planes_of(sum) * 2 * sums_of(sum); }
constexpr int tok_bytes(int sum) { return 512 + float_bytes(sum) + sum_bytes(sum); }
template <int WTYPE> constexpr int chunk_bytes() { return 256 / cq_block_elems(WTYPE) * cq_type_size(WTYPE); }
template <int WTYPE, bool PLAIN> struct Smem {
    using F = Fmt<WTYPE, PLAIN>;
    static constexpr int kSums = sums_of(F::kSum);
    static constexpr int kStageT = 16 * kTok * 16, kAux = kTok * (float_bytes(F::kSum) + sum_bytes(F::kSum));
    static constexpr int kScales = F::kBlockScale ? 8 : 1, kRingW = kRows * 4 * (kScales + 8 * F::kMins);      // d of the rows, then minima, of one chunk
    static constexpr int kCoef = 3 * kRows * 2 * kSums;                              // planes lo, hi, mid of the coefficients
    static constexpr int kBytes = 1024 + kStagesT * kStageT + 4 * kAux + 4 * kRingW + 2 * kCoef + kRawStages * Raw<chunk_bytes<WTYPE>()>::kBytes + 16;
};

// a = hi + mid + lo, exactly (bf16 of 7, 8 and 8 bits, and the signs of the rests), b in the upper halves; a value that is not finite has only its first part.
// (NaNs are results of f32 operations, with all bits set.)
__device__ __forceinline__ void split3(float a, float b, uint32_t &hi, uint32_t &mid, uint32_t &lo) {
    auto pair = [](float x, float y) { const __nv_bfloat162 v = __floats2bfloat162_rn(x, y); return *reinterpret_cast<const uint32_t *>(&v); };
    const bool fa = fabsf(a) <= 3.3e38f, fb = fabsf(b) <= 3.3e38f;
    const uint32_t ha = (__float_as_uint(a) + (fa ? 0x10000u : 0u)) & 0xFFFE0000u, hb = (__float_as_uint(b) + (fb ? 0x10000u : 0u)) & 0xFFFE0000u;
    const float ra = fa ? __fsub_rn(a, __uint_as_float(ha)) : 0.0f, rb = fb ? __fsub_rn(b, __uint_as_float(hb)) : 0.0f;
    hi = __byte_perm(ha, hb, 0x7632);
    mid = pair(ra, rb);
    lo = pair(__fsub_rn(ra, __uint_as_float(mid << 16)), __fsub_rn(rb, __uint_as_float(mid & 0xFFFF0000u)));
}

// ---- activations ---------------------------------------------------------------------------------------------------
// One warp per (token, chunk of 256), 8 tokens of one chunk per block, through shared memory (see prompt_kq.cu).
template <typename T, bool Q81, int SUM>
__global__ void __launch_bounds__(256) quantize_kernel(const T *__restrict__ x, uint8_t *__restrict__ y, int k, Tiling tl) {
    constexpr int kPitch = 8 * 16 + 16, kPlane = sums_of(SUM) / 8, kPlanes = planes_of(SUM), kSlabs = 32 + kPlanes * kPlane, kFloats = float_bytes(SUM) / 4;
    __shared__ __align__(16) uint8_t sm[kSlabs * kPitch];
    __shared__ float sv[kFloats][8];    // [value][token]: scales of the blocks, then sums
    cq_pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nch = k / 256;
    const int c = blockIdx.x % nch, g = blockIdx.x / nch, per_tile = tl.tt / 8;
    const int t = g / per_tile, row0 = (g % per_tile) * 8, row = row0 + warp;
    const int rows = tl.rows(t);
    if (row0 >= rows) return;           // block-uniform
    const int64_t tok = (int64_t)t * tl.tt + row;
    float e[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) e[i] = 0.0f;
    if (row < rows && tok < tl.tokens) load8(x + tok * k + c * 256 + lane * 8, ((uintptr_t)x & 15) == 0, e);
    float amax = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(e[i]));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    const float d = __fdiv_rn(amax, 127.0f);
    int q[8];
    if constexpr (Q81) {                // mmvq_gguf.cu:811-911
#pragma unroll
        for (int i = 0; i < 8; ++i) q[i] = (amax == 0.0f) ? 0 : (int)(int8_t)roundf(__fdiv_rn(e[i], d));
    } else {                            // k_quants.rs:658-687
        const float id = d != 0.0f ? __fdiv_rn(1.0f, d) : 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float r = roundf(__fmul_rn(e[i], id));
            r = fminf(fmaxf(r, -128.0f), 127.0f);
            q[i] = (int)r;
        }
    }
    const float dh = __half2float(__float2half_rn(d));
    *reinterpret_cast<uint4 *>(sm + lane * kPitch + warp * 16) = pack_q8(q);
    const int b = lane >> 2;
    if ((lane & 3) == 0) sv[b][warp] = dh;
    if constexpr (SUM != kNoSum) {
        int si = q[0] + q[1] + q[2] + q[3] + q[4] + q[5] + q[6] + q[7];
        si += __shfl_xor_sync(0xffffffffu, si, 1);
        if constexpr (SUM != kSum16 && SUM != kPlain16) si += __shfl_xor_sync(0xffffffffu, si, 2);
        const float s = __fmul_rn(dh, (float)si);
        [[maybe_unused]] auto put = [&](int j, float v) {        // sum j of the chunk: element j % 8 of slab j / 8 of each plane
            uint32_t hi, mid, lo;
            split3(v, 0.0f, hi, mid, lo);
            uint8_t *p = sm + (32 + (j >> 3)) * kPitch + warp * 16 + 2 * (j & 7);
            const uint16_t plane[5] = {(uint16_t)lo, (uint16_t)mid, (uint16_t)((hi & 0x7F80u) == 0x7F80u ? 0 : hi), (uint16_t)(kPlanes == 5 ? 0 : hi), (uint16_t)hi};
#pragma unroll
            for (int i = 0; i < kPlanes; ++i) *reinterpret_cast<uint16_t *>(p + i * kPlane * kPitch) = plane[i];
        };
        if constexpr (SUM == kSum16) { if ((lane & 1) == 0) put(lane >> 1, s); }
        else if constexpr (SUM == kSum32) { if ((lane & 3) == 0) put(b, s); }
        else if constexpr (SUM == kPlain16) { if ((lane & 1) == 0) sv[8 + 8 * ((lane >> 1) & 1) + b][warp] = s; }
        else if constexpr (SUM == kPlain32) { if ((lane & 3) == 0) sv[8 + b][warp] = s; }
        else {
            // t: the f16-rounded sum of the inputs, added in the order of a 32-lane xor butterfly over the block (16, 8, 4, 2, 1)
            float u[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) u[i] = __fadd_rn(e[i], __shfl_xor_sync(0xffffffffu, e[i], 2));
#pragma unroll
            for (int i = 0; i < 8; ++i) u[i] = __fadd_rn(u[i], __shfl_xor_sync(0xffffffffu, u[i], 1));
            const float t0 = __fadd_rn(__fadd_rn(u[0], u[4]), __fadd_rn(u[2], u[6])), t1 = __fadd_rn(__fadd_rn(u[1], u[5]), __fadd_rn(u[3], u[7]));
            const float ts = __half2float(__float2half_rn(__fadd_rn(t0, t1)));
            if ((lane & 3) == 0) {
                if constexpr (SUM == kDelta) put(b, __fsub_rn(ts, s));
                else sv[8 + b][warp] = ts;
            }
        }
    }
    __syncthreads();
    uint8_t *blob = y + ((size_t)t * tl.tt * nch + (size_t)c * rows) * tok_bytes(SUM);
    for (int i = threadIdx.x; i < kSlabs * 8; i += 256) {
        const int slab = i >> 3;
        *reinterpret_cast<uint4 *>(blob + (size_t)rows * (slab < 32 ? slab * 16 : slab * 16 + 4 * kFloats) + (size_t)(row0 + (i & 7)) * 16) =
            *reinterpret_cast<const uint4 *>(sm + slab * kPitch + (i & 7) * 16);
    }
    if (threadIdx.x < kFloats * 8)
        *reinterpret_cast<float *>(blob + (size_t)rows * 512 + ((size_t)(threadIdx.x >> 3) * rows + row0 + (threadIdx.x & 7)) * 4) = sv[threadIdx.x >> 3][threadIdx.x & 7];
}

// ---- producers: chunk ch = 0..3 covers blocks 2 ch (cells 0-15) and 2 ch + 1 (cells 16-31) -----------------------------

// 32-bit word at byte offset OFF (even) of a row chunk held as 16-byte vectors from vector V0 on
template <int OFF, int V0, int NV> __device__ __forceinline__ uint32_t word_at(const uint4 (&v)[NV]) {
    constexpr int w = OFF / 4 - 4 * V0;
    auto get = [&](int i) -> uint32_t { const uint4 &q = v[i >> 2]; return (i & 3) == 0 ? q.x : (i & 3) == 1 ? q.y : (i & 3) == 2 ? q.z : q.w; };
    if constexpr (OFF % 4 == 0) return get(w);
    else return __funnelshift_r(get(w), get(w + 1), 16);
}
__device__ __forceinline__ float h16(uint32_t w) { return __half2float(__ushort_as_half((unsigned short)(w & 0xFFFFu))); }
// pairs (byte 0, byte 2) and (byte 1, byte 3) of a word of small unsigned codes, minus `off`, as f16
__device__ __forceinline__ void codes4(uint32_t w, float off, uint32_t &a, uint32_t &b) {
    const __half2 o = __float2half2_rn(1024.0f + off);
    a = h2_bits(__hsub2(bits_h2(and_or<0x00FF00FFu, 0x64006400u>(w)), o));
    b = h2_bits(__hsub2(bits_h2(and_or<0x00FF00FFu, 0x64006400u>(w >> 8)), o));
}
__device__ __forceinline__ __half2 twice(uint32_t v) { return __hsub2(bits_h2(v * 0x00010001u | 0x64006400u), bits_h2(0x64006400u)); }   // v < 1024
// The SUMS coefficients c(j) of a row: planes lo, hi, mid of SUMS / 8 slabs of 128 rows x 16 bytes
template <int SUMS, typename C> __device__ __forceinline__ void put_coefs(uint8_t *row, C &&c) {
#pragma unroll
    for (int slab = 0; slab < SUMS / 8; ++slab) {
        uint32_t hi[4], mid[4], lo[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) split3(c(8 * slab + 2 * i), c(8 * slab + 2 * i + 1), hi[i], mid[i], lo[i]);
        uint4 *p = reinterpret_cast<uint4 *>(row + slab * kRows * 16);
        p[0] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        p[SUMS / 8 * kRows] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        p[2 * (SUMS / 8) * kRows] = make_uint4(mid[0], mid[1], mid[2], mid[3]);
    }
}

template <int WTYPE, bool PLAIN> struct Expand;

// the 32-element block formats: their chunk is a whole number of 16-byte vectors
template <int WTYPE, bool PLAIN> struct ExpandBlock {
    static constexpr int kBlk = cq_type_size(WTYPE);
    static constexpr bool kHasM = WTYPE == CQ_Q4_1 || WTYPE == CQ_Q5_1, kFive = WTYPE == CQ_Q5_0 || WTYPE == CQ_Q5_1;
    const uint8_t *p;
    __device__ __forceinline__ void header(const uint8_t *rr, int) { p = rr; }
    __device__ __forceinline__ void scales(float *dst) const {          // [8 blocks][128 rows] d, then the same of the minima
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            const float d = h16(cq_lds_u16(p + b * kBlk));
            dst[b * kRows] = d;
            if constexpr (kHasM) dst[(8 + b) * kRows] = h16(cq_lds_u16(p + b * kBlk + 2));
            else if constexpr (WTYPE == CQ_Q5_0 && PLAIN) dst[(8 + b) * kRows] = __fmul_rn(-16.0f, d);
        }
    }
    __device__ __forceinline__ void coef(uint8_t *row) const {
        if constexpr (WTYPE == CQ_Q5_0) put_coefs<8>(row, [&](int b) { return __fmul_rn(-16.0f, h16(cq_lds_u16(p + b * kBlk))); });
    }
    template <int B, int V0, int NV> __device__ __forceinline__ void block(const uint4 (&v)[NV], uint32_t *o) const {
        constexpr int off = B * kBlk, qs = off + 2 + (kHasM ? 2 : 0) + (kFive ? 4 : 0);
        if constexpr (WTYPE == CQ_Q8_0) {
            auto four = [&](auto ic) {
                constexpr int i = decltype(ic)::value;
                const uint32_t w = word_at<qs + 4 * i, V0>(v);
                const __half2 c = __float2half2_rn(1152.0f);        // int8 + 128 in the mantissa of 1024
                o[2 * i] = h2_bits(__hsub2(bits_h2(and_xor<0x00FF00FFu, 0x64806480u>(w)), c));
                o[2 * i + 1] = h2_bits(__hsub2(bits_h2(and_xor<0x00FF00FFu, 0x64806480u>(w >> 8)), c));
            };
            four(std::integral_constant<int, 0>{}); four(std::integral_constant<int, 1>{}); four(std::integral_constant<int, 2>{});
            four(std::integral_constant<int, 3>{}); four(std::integral_constant<int, 4>{}); four(std::integral_constant<int, 5>{});
            four(std::integral_constant<int, 6>{}); four(std::integral_constant<int, 7>{});
        } else {
            uint32_t qh = 0;
            if constexpr (kFive) qh = word_at<qs - 4, V0>(v);
            auto four = [&](auto ic) {          // elements 4 i .. and 16 + 4 i ..
                constexpr int i = decltype(ic)::value;
                const uint32_t w = word_at<qs + 4 * i, V0>(v);
                uint32_t lo = w & 0x0F0F0F0Fu, hi = (w >> 4) & 0x0F0F0F0Fu;
                if constexpr (kFive) {          // bit e of qh -> bit 4 of element e
                    lo |= ((((qh >> (4 * i)) & 0xFu) * 0x00204081u) & 0x01010101u) << 4;
                    hi |= ((((qh >> (16 + 4 * i)) & 0xFu) * 0x00204081u) & 0x01010101u) << 4;
                }
                constexpr float minus = WTYPE == CQ_Q4_0 ? 8.0f : WTYPE == CQ_Q5_0 && !PLAIN ? 16.0f : 0.0f;
                codes4(lo, minus, o[2 * i], o[2 * i + 1]);
                codes4(hi, minus, o[8 + 2 * i], o[8 + 2 * i + 1]);
            };
            four(std::integral_constant<int, 0>{}); four(std::integral_constant<int, 1>{});
            four(std::integral_constant<int, 2>{}); four(std::integral_constant<int, 3>{});
        }
    }
    template <int CH> __device__ __forceinline__ void pair(uint32_t (&o)[32]) const {
        constexpr int v0 = 2 * CH * kBlk / 16, nv = (2 * (CH + 1) * kBlk + 15) / 16 - v0;
        uint4 v[nv + 1];
#pragma unroll
        for (int i = 0; i < nv; ++i) v[i] = *reinterpret_cast<const uint4 *>(p + 16 * (v0 + i));
        v[nv] = make_uint4(0u, 0u, 0u, 0u);       // word_at may name (not use) the word after the last
        block<2 * CH, v0>(v, o);
        block<2 * CH + 1, v0>(v, o + 16);
    }
    __device__ __forceinline__ void chunk(int ch, uint32_t (&o)[32]) const {
        if (ch == 0) pair<0>(o);
        else if (ch == 1) pair<1>(o);
        else if (ch == 2) pair<2>(o);
        else pair<3>(o);
    }
};
template <bool PLAIN> struct Expand<CQ_Q8_0, PLAIN> : ExpandBlock<CQ_Q8_0, PLAIN> {};
template <bool PLAIN> struct Expand<CQ_Q4_0, PLAIN> : ExpandBlock<CQ_Q4_0, PLAIN> {};
template <bool PLAIN> struct Expand<CQ_Q4_1, PLAIN> : ExpandBlock<CQ_Q4_1, PLAIN> {};
template <bool PLAIN> struct Expand<CQ_Q5_0, PLAIN> : ExpandBlock<CQ_Q5_0, PLAIN> {};
template <bool PLAIN> struct Expand<CQ_Q5_1, PLAIN> : ExpandBlock<CQ_Q5_1, PLAIN> {};

// Super-block formats.  A code of b bits goes to the top of the mantissa, or near it, so that scale times (code - middle) is one fma whose
// addend, -(base + middle) * scale, is exact in f16 (PLAIN: no middle); one copy of the code for all of a chunk's four pairs (see prompt_kq.cu).

// Q5_K: Q4_K with the fifth bits of sub-block g in bit g of 32 bytes.  Code q in bits 4-8: the value 64 + q.
template <bool PLAIN> struct Expand<CQ_Q5_K, PLAIN> {
    const uint8_t *p;
    uint32_t sc[2], mn[2], dm;
    __device__ __forceinline__ void header(const uint8_t *rr, int) {
        p = rr;
        const uint4 h = *reinterpret_cast<const uint4 *>(p);
        dm = h.x;
        sc[0] = h.y & 0x3F3F3F3Fu; mn[0] = h.z & 0x3F3F3F3Fu;
        sc[1] = (h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u);
        mn[1] = ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u);
    }
    __device__ __forceinline__ void scales(float *dst) const {
        *dst = __low2float(bits_h2(dm));
        if constexpr (PLAIN) {
            const float dmin = __high2float(bits_h2(dm));
#pragma unroll
            for (int g = 0; g < 8; ++g) dst[(1 + g) * kRows] = -__fmul_rn(dmin, (float)((mn[g >> 2] >> (8 * (g & 3))) & 0xFFu));
        }
    }
    __device__ __forceinline__ void coef(uint8_t *row) const {
        const float d16 = __fmul_rn(16.0f, __low2float(bits_h2(dm))), dmin = __high2float(bits_h2(dm));
        auto c = [&](int g) {       // 16 d sc is exact
            const float s = (float)((sc[g >> 2] >> (8 * (g & 3))) & 0xFFu), m = (float)((mn[g >> 2] >> (8 * (g & 3))) & 0xFFu);
            return __fmaf_rn(-dmin, m, __fmul_rn(d16, s));
        };
        put_coefs<8>(row, c);
    }
    __device__ __forceinline__ void chunk(int ch, uint32_t (&o)[32]) const {
        const uint4 a = *reinterpret_cast<const uint4 *>(p + 48 + 32 * ch), b = *reinterpret_cast<const uint4 *>(p + 64 + 32 * ch);
        const uint4 ha = *reinterpret_cast<const uint4 *>(p + 16), hb = *reinterpret_cast<const uint4 *>(p + 32);
        const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}, h[8] = {ha.x, ha.y, ha.z, ha.w, hb.x, hb.y, hb.z, hb.w};
        const uint32_t s16 = (ch & 2 ? sc[1] : sc[0]) >> (16 * (ch & 1));
        const __half2 s0 = twice(s16 & 0xFFu), s1 = twice((s16 >> 8) & 0xFFu);
        const __half2 base = __float2half2_rn(PLAIN ? -64.0f : -80.0f), c0 = __hmul2(s0, base), c1 = __hmul2(s1, base);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t he = h[i] << (7 - 2 * ch), ho = h[i] >> (2 * ch);        // fifth bits 2 ch + 1 | 2 ch in bit 8
            o[2 * i] = hfma2_bits(and_or<0x00F000F0u>(w[i] << 4, and_or<0x01000100u, 0x54005400u>(he << 1)), s0, c0);
            o[2 * i + 1] = hfma2_bits(and_or<0x00F000F0u>(w[i] >> 4, and_or<0x01000100u, 0x54005400u>(ho)), s0, c0);
            o[16 + 2 * i] = hfma2_bits(and_or<0x00F000F0u>(w[i], and_or<0x01000100u, 0x54005400u>(he)), s1, c1);
            o[16 + 2 * i + 1] = hfma2_bits(and_or<0x00F000F0u>(w[i] >> 8, and_or<0x01000100u, 0x54005400u>(ho >> 1)), s1, c1);
        }
    }
};

// Q2_K / Q3_K: block b = 4 n + pos: bit pair pos of bytes 32 n .. of the codes; a scale per 16 elements, number 2 b + half.
// Q2_K: code q in bits 8-9: the value 4 + q; the operand is sc (2 q - 3), so the row's scale is d / 2 (PLAIN: sc q, d).
template <bool PLAIN> struct Expand<CQ_Q2_K, PLAIN> {
    const uint8_t *p;
    float d, dmin;
    __device__ __forceinline__ void header(const uint8_t *rr, int shift) {
        p = rr + shift;         // a multiple of 4 when the base is, else of 2
        uint32_t dm[1];
        cq_lds_words<1, true>(p + 80, dm);
        d = h16(dm[0]); dmin = h16(dm[0] >> 16);
    }
    __device__ __forceinline__ void scales(float *dst) const {
        if constexpr (PLAIN) {
            uint32_t sc[4];
            cq_lds_words<4, true>(p, sc);
            *dst = d;
#pragma unroll
            for (int j = 0; j < 16; ++j) dst[(1 + 8 * (j & 1) + (j >> 1)) * kRows] = -__fmul_rn(dmin, (float)((sc[j >> 2] >> (8 * (j & 3) + 4)) & 0xFu));
        } else *dst = __fmul_rn(0.5f, d);
    }
    __device__ __forceinline__ void coef(uint8_t *row) const {
        const float d15 = __fmul_rn(1.5f, d);
        uint32_t sc[4];
        cq_lds_words<4, true>(p, sc);
        auto c = [&](int j) {
            const uint32_t by = (sc[j >> 2] >> (8 * (j & 3))) & 0xFFu;
            return __fmaf_rn(-dmin, (float)(by >> 4), __fmul_rn(d15, (float)(by & 0xFu)));
        };
        put_coefs<16>(row, c);
    }
    __device__ __forceinline__ void chunk(int ch, uint32_t (&o)[32]) const {
        uint32_t q[8], sc[1];
        cq_lds_words<8, true>(p + 16 + 32 * (ch >> 1), q);
        cq_lds_words<1, true>(p + 4 * ch, sc);
#pragma unroll
        for (int bb = 0; bb < 2; ++bb) {
            const int pos = 2 * (ch & 1) + bb;
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                const __half2 sv = twice((sc[0] >> (8 * (2 * bb + hf))) & 0xFu), s2 = PLAIN ? sv : __hadd2(sv, sv);
                const __half2 cv = __hmul2(sv, __float2half2_rn(PLAIN ? -4.0f : -11.0f));
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    o[16 * bb + 8 * hf + 2 * i] = hfma2_bits(and_or<0x03000300u, 0x44004400u>(q[4 * hf + i] << (8 - 2 * pos)), s2, cv);
                    o[16 * bb + 8 * hf + 2 * i + 1] = hfma2_bits(and_or<0x03000300u, 0x44004400u>(q[4 * hf + i] >> (2 * pos)), s2, cv);
                }
            }
        }
    }
};
// Q3_K: two bits, plus 4 when the mask bit is set, in bits 7-9: the value 8 + u; the operand is scale * (u - 4).
template <bool PLAIN> struct Expand<CQ_Q3_K, PLAIN> {
    const uint8_t *p;
    uint32_t sc[3];
    __device__ __forceinline__ void header(const uint8_t *rr, int shift) {
        p = rr + shift;         // even
        cq_lds_words<3, true>(p + 96, sc);
    }
    __device__ __forceinline__ void scales(float *dst) const { *dst = __half2float(*reinterpret_cast<const __half *>(p + 108)); }
    __device__ __forceinline__ void coef(uint8_t *) const {}
    __device__ __forceinline__ void chunk(int ch, uint32_t (&o)[32]) const {
        uint32_t q[8], hm[8];
        cq_lds_words<8, true>(p + 32 + 32 * (ch >> 1), q);
        cq_lds_words<8, true>(p, hm);
        // scale number j = 4 ch + 2 bb + half: 4 low bits from bytes 0-7, 2 high bits from bytes 8-11
        const uint32_t scl = (ch & 1 ? sc[1] : sc[0]) >> (ch & 2 ? 4 : 0), sch = sc[2] >> (2 * ch);
#pragma unroll
        for (int bb = 0; bb < 2; ++bb) {
            const int b = 2 * ch + bb, pos = b & 3;
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                const int j = 2 * bb + hf;
                const uint32_t s6 = ((scl >> (8 * j)) & 0xFu) | ((sch >> (8 * j)) & 3u) << 4;
                const __half2 sv = __hsub2(bits_h2(s6 * 0x00010001u | 0x64006400u), __float2half2_rn(1056.0f));
                const __half2 cv = __hmul2(sv, __float2half2_rn(-12.0f));
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t u = q[4 * hf + i], h = hm[4 * hf + i];
                    o[16 * bb + 8 * hf + 2 * i] = hfma2_bits(and_or<0x01800180u>(u << (7 - 2 * pos), and_or<0x02000200u, 0x48004800u>(h << (9 - b))), sv, cv);
                    o[16 * bb + 8 * hf + 2 * i + 1] =
                        hfma2_bits(and_or<0x01800180u>(u >> (1 + 2 * pos), and_or<0x02000200u, 0x48004800u>((h >> 8) << (9 - b))), sv, cv);
                }
            }
        }
    }
};

// bf16 x bf16 from shared memory
template <bool ACC> __device__ __forceinline__ void mma_ss(uint32_t tmem_d, uint32_t desc_a, uint32_t desc_b, uint32_t idesc) {
    if constexpr (ACC)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.eq.b32 p, 0, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                     ::"r"(tmem_d), "l"(desc_of(desc_a)), "l"(desc_of(desc_b)), "r"(idesc) : "memory");
    else
        mma_f16_ss(tmem_d, desc_a, desc_b, idesc);
}
struct Args {
    const uint8_t *w, *act;
    void *out;
    int out_kind, nrows, nch, stride_out, use_map, ntiles;
};

// STORE: see prompt_f16.cuh; N8: tiles of up to 16 N8 tokens, 2 or 4
template <int WTYPE, bool PLAIN, int STORE, int N8>
__global__ void __launch_bounds__(kThreads, 1) prompt32_kernel(const __grid_constant__ CUtensorMap wmap, const Args a, const Tiling tl) {
    using F = Fmt<WTYPE, PLAIN>;
    using S = Smem<WTYPE, PLAIN>;
    constexpr int kCB = chunk_bytes<WTYPE>(), kSums = S::kSums, kMins = F::kMins, kNA = 3;
    constexpr bool kOneCommit = kSums == 0;         // accumulator slots and buffers of operand A go together: bar_acc serves the producers too
    using R = Raw<kCB>;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t *bar_raw = reinterpret_cast<uint64_t *>(smem);        // [3] raw weight bytes landed
    uint64_t *bar_rawfree = bar_raw + 3;                            // [3] read by both producer sets
    uint64_t *bar_fullT = bar_raw + 6;                              // [4] token stage (first half: + scales) landed
    uint64_t *bar_doneT = bar_raw + 10;                             // [4] its MMAs are complete
    uint64_t *bar_fullW = bar_raw + 14;                             // [3] operand A pair stored (a producer set)
    uint64_t *bar_doneW = bar_raw + 17;                             // [3] its MMAs are complete
    uint64_t *bar_acc = bar_raw + 20;                               // [3] the MMAs of two blocks are complete
    uint64_t *bar_free = bar_raw + 23;                              // [3] accumulator slot read (all epilogue warps)
    uint64_t *bar_vis = bar_raw + 26;                               // [2] relay: the scales of this chunk are visible
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + 512);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + 520);
    uint8_t *stT0 = smem + 1024;
    uint8_t *aux0 = stT0 + kStagesT * S::kStageT;       // [4] scales [8][n], then sums: the same, or planes
    uint8_t *ringW = aux0 + 4 * S::kAux;                // [4] d [1 or 8][128 rows], then minima [kMins][8][128 rows]
    uint8_t *coef0 = ringW + 4 * S::kRingW;             // [2] planes of coefficients
    uint8_t *raw0 = coef0 + 2 * S::kCoef;               // 128-byte aligned

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nch = a.nch;
    const uint32_t row_bytes = (uint32_t)nch * kCB;
    const GroupInfo gi{};

    if (tid == 0) {
        for (int i = 0; i < kRawStages; ++i) { cq_mbar_init(&bar_raw[i], a.use_map ? 1 : kRawThreads); cq_mbar_init(&bar_rawfree[i], kProdWarps); }
        for (int i = 0; i < kStagesT; ++i) { cq_mbar_init(&bar_fullT[i], 1); cq_mbar_init(&bar_doneT[i], 1); }
        for (int i = 0; i < 3; ++i) {
            cq_mbar_init(&bar_fullW[i], kProdWarps / 2);
            cq_mbar_init(&bar_doneW[i], 1);
            cq_mbar_init(&bar_acc[i], 1);
            cq_mbar_init(&bar_free[i], kEpiWarps);
        }
        for (int i = 0; i < 2; ++i) cq_mbar_init(&bar_vis[i], 1);
        *abort_flag = 0;
        cq_fence_mbar_init();
    }
    if (warp == 0) {
        tmem_alloc(tmem_slot, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    cq_pdl_wait();

    if (warp >= kMmaWarp) {
    regs_down<kRegsMisc32>();
    if (warp == kLoadWarp) {
        // ===== loader =====
        int it = 0, ti = 0, rs = 0, rs_phase = 1;       // rs_phase: parity of the wait for this stage's previous use
        bool alive = true;
        for (int tile = blockIdx.x; tile < a.ntiles && alive; tile += gridDim.x) {
            TileCtx cx;
            tile_ctx(tile, tl.ntt, tl, gi, cx);
            const int n = cx.n;
            const uint8_t *blob0 = a.act + (size_t)cx.blob_row * nch * tok_bytes(F::kSum);
            for (int c = 0; c < nch && alive; ++c, ++it) {
                if (a.use_map) {
                    if (it >= kRawStages && !wait_warp(&bar_rawfree[rs], rs_phase, abort_flag)) { alive = false; break; }
                    if (lane == 0) {
                        cq_mbar_expect_tx(&bar_raw[rs], R::kBytes);
                        cq_tmap::load_2d(raw0 + rs * R::kBytes, &wmap, (int)(((uint32_t)c * kCB & ~15u) / 2), cx.row0, &bar_raw[rs]);
                    }
                    if (++rs == kRawStages) { rs = 0; rs_phase ^= 1; }
                }
                const uint8_t *blob = blob0 + (size_t)c * n * tok_bytes(F::kSum);
                for (int half = 0; half < 2; ++half, ++ti) {
                    const int s = ti % kStagesT;
                    if (ti >= kStagesT && !wait_warp(&bar_doneT[s], (ti / kStagesT - 1) & 1, abort_flag)) { alive = false; break; }
                    if (lane == 0) {
                        const unsigned bytes = (unsigned)n * 256;
                        if (half == 0) {
                            // a stage of chunk it - 2 (or later) is done: its MMAs had started, so the epilogue has finished it - 4
                            const unsigned aux_bytes = (unsigned)n * (float_bytes(F::kSum) + sum_bytes(F::kSum));
                            cq_mbar_expect_tx(&bar_fullT[s], bytes + aux_bytes);
                            cq_bulk_g2s(aux0 + (it & 3) * S::kAux, blob + (size_t)n * 512, aux_bytes, &bar_fullT[s]);
                        } else {
                            cq_mbar_expect_tx(&bar_fullT[s], bytes);
                        }
                        cq_bulk_g2s(stT0 + s * S::kStageT, blob + (size_t)half * bytes, bytes, &bar_fullT[s]);
                    }
                    __syncwarp();
                }
            }
        }
        // after a give-up the copies already issued must land (or give up themselves) before the shared memory goes away
        if (lane == 0 && (!alive || *abort_flag)) {
            for (int j = it >= kRawStages ? it - kRawStages + 1 : 0; a.use_map && j <= it; ++j)
                (void)cq_mbar_wait_bounded(&bar_raw[j % kRawStages], (j / kRawStages) & 1);
            for (int j = ti > kStagesT ? ti - kStagesT : 0; j < ti; ++j) (void)cq_mbar_wait_bounded(&bar_fullT[j % kStagesT], (j / kStagesT) & 1);
        }
        __syncwarp();
    } else if (warp >= kRawWarp) {
        // ===== raw bytes of rows that are not a multiple of 16 bytes apart =====
        if (!a.use_map) {
            int it = 0;
            bool alive = true;
            for (int tile = blockIdx.x; tile < a.ntiles && alive; tile += gridDim.x) {
                TileCtx cx;
                tile_ctx(tile, tl.ntt, tl, gi, cx);
                const uint8_t *w0 = a.w + cx.wrow0 * row_bytes;
                for (int c = 0; c < nch; ++c, ++it) {
                    const int rs = it % kRawStages;
                    if (it >= kRawStages && !wait_warp(&bar_rawfree[rs], (it / kRawStages - 1) & 1, abort_flag)) { alive = false; break; }
                    R::load_rows(raw0 + rs * R::kBytes, w0 + (uint32_t)c * kCB, min(a.nrows - cx.row0, kRows), row_bytes, tid - kRawWarp * 32, &bar_raw[rs]);
                }
            }
            cq_cp_async_wait<0>();
        }
    } else if (warp == kMmaWarp) {
        // ===== MMA issuer (the warp runs the loop, one elected lane issues): a block = two K = 16 steps into fresh columns =====
        const uint32_t stT = uniform(cq_smem_u32(stT0) >> 4), tm = uniform(tmem_base);
        [[maybe_unused]] const uint32_t coef = uniform(cq_smem_u32(coef0) >> 4), aux = uniform(cq_smem_u32(aux0) >> 4);
        int it = 0, s = 0, s_phase = 0, slot = 0, round = 0;      // token stage; accumulator slot and how often all have been used
        int buf = 0, buf_phase = 0;
        bool alive = true;
        for (int tile = blockIdx.x; tile < a.ntiles && alive; tile += gridDim.x) {
            TileCtx cx;
            tile_ctx(tile, tl.ntt, tl, gi, cx);
            const uint32_t n = uniform((uint32_t)cx.n), idesc = idesc_f16((int)n), bT = stT | (n << 16);
#pragma unroll 1
            for (int c = 0; c < nch && alive; ++c, ++it) {
#pragma unroll
                for (int ch = 0; ch < 4; ++ch) {
                    if (((ch & 1) == 0 && !wait_warp(&bar_fullT[s], s_phase, abort_flag)) ||
                        !wait_warp(&bar_fullW[buf], buf_phase, abort_flag) ||
                        (round > 0 && !wait_warp(&bar_free[slot], (round - 1) & 1, abort_flag))) { alive = false; break; }
                    tc_fence_after();
                    const uint32_t b0 = bT + (uint32_t)s * (S::kStageT >> 4) + (uint32_t)(8 * (ch & 1)) * n, a0 = tm + (uint32_t)(kColA + buf * 32);
                    const uint32_t td = tm + (uint32_t)(slot * 2 * kTok);
                    if (elect_one()) {
                        if (ch == 0) mbar_arrive(&bar_vis[it & 1]);     // what this warp has acquired is visible to the epilogue
                        mma_f16_ts<false>(td, a0, b0, idesc);
                        mma_f16_ts<true>(td, a0 + 8, b0 + 2 * n, idesc);
                        mma_f16_ts<false>(td + kTok, a0 + 16, b0 + 4 * n, idesc);
                        mma_f16_ts<true>(td + kTok, a0 + 24, b0 + 6 * n, idesc);
                        tc_commit(&bar_acc[slot]);
                        if (ch & 1) tc_commit(&bar_doneT[s]);
                        if constexpr (!kOneCommit) tc_commit(&bar_doneW[buf]);
                    }
                    __syncwarp();
                    if (++slot == kSlots) { slot = 0; ++round; }
                    if (++buf == kNA) { buf = 0; buf_phase ^= 1; }
                    if ((ch & 1) && ++s == kStagesT) { s = 0; s_phase ^= 1; }
                }
                if constexpr (kSums > 0) {      // the chunk's sums take a slot like two blocks: the products hi hi, and all others
                    if (!alive || (round > 0 && !wait_warp(&bar_free[slot], (round - 1) & 1, abort_flag))) { alive = false; break; }
                    tc_fence_after();
                    if (elect_one()) {      // A planes lo, hi, mid; B planes: planes_of
                        const uint32_t t1 = tm + (uint32_t)(slot * 2 * kTok), t2 = t1 + kTok, idb = idesc | (1u << 7) | (1u << 10);      // bf16 x bf16
                        const uint32_t ca = (coef + (uint32_t)(it & 1) * (S::kCoef >> 4)) | ((uint32_t)kRows << 16);
                        const uint32_t cb = (aux + (uint32_t)(it & 3) * (S::kAux >> 4) + (float_bytes(F::kSum) / 16) * n) | (n << 16);
                        if constexpr (kSums == 8) {         // a step is two planes of eight
                            mma_ss<false>(t2, ca + kRows, cb, idb);                 // hi lo + mid mid
                            mma_ss<true>(t2, ca, cb + 2 * n, idb);                  // lo hi
                            mma_ss<true>(t2, ca + kRows, cb + n, idb);              // hi mid + mid hi
                            mma_ss<false>(t1, ca, cb + 3 * n, idb);                 // hi hi
                        } else {
                            mma_ss<false>(t2, ca + 2 * kRows, cb, idb);             // hi lo
                            mma_ss<true>(t2, ca + 4 * kRows, cb + 2 * n, idb);      // mid mid
                            mma_ss<true>(t2, ca, cb + 4 * n, idb);                  // lo hi
                            mma_ss<true>(t2, ca + 2 * kRows, cb + 2 * n, idb);      // hi mid
                            mma_ss<true>(t2, ca + 4 * kRows, cb + 4 * n, idb);      // mid hi
                            mma_ss<false>(t1, ca + 2 * kRows, cb + 6 * n, idb);     // hi hi
                        }
                        tc_commit(&bar_acc[slot]);
                    }
                    __syncwarp();
                    if (++slot == kSlots) { slot = 0; ++round; }
                }
            }
        }
    }
    } else if (warp >= kEpiWarps) {
        regs_down<kRegsProd32>();
        // ===== producers: thread = weight row = TMEM lane; set 0 takes the even pairs of blocks, set 1 the odd ones =====
        const int set = (warp - kEpiWarps) >> 2, r = (warp & 3) * 32 + lane;
        const uint32_t ta = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)kColA;
        int it = 0, rs = 0, rs_phase = 0;
        bool alive = true;
        for (int tile = blockIdx.x; tile < a.ntiles && alive; tile += gridDim.x) {
            TileCtx cx;
            tile_ctx(tile, tl.ntt, tl, gi, cx);
            long long wr = cx.wrow0 + r;
            if (wr >= a.nrows) wr = a.nrows - 1;
            const uint32_t row_off = a.use_map ? 0u : (uint32_t)((uintptr_t)(a.w + wr * row_bytes) & 15);
            for (int c = 0; c < nch && alive; ++c, ++it) {
                if (!wait_warp(&bar_raw[rs], rs_phase, abort_flag)) { alive = false; break; }
                Expand<WTYPE, PLAIN> ex;
                ex.header(raw0 + rs * R::kBytes + r * R::kPitch, R::kAligned ? 0 : (int)((row_off + (uint32_t)c * kCB) & 15));
                // Set 0 has waited for the last pair of it - 2 or later, and the epilogue, at most three slots behind the MMAs, has finished it - 4; set 1
                // for the first pair of it - 1, whose completion includes the sums of it - 2.
                if (set == 0) ex.scales(reinterpret_cast<float *>(ringW + (it & 3) * S::kRingW) + r);
                else if constexpr (kSums > 0) {
                    ex.coef(coef0 + (it & 1) * S::kCoef + r * 16);
                    fence_proxy_async_smem();
                }
#pragma unroll 1
                for (int ch = set; ch < 4; ch += 2) {
                    uint32_t o[32];
                    ex.chunk(ch, o);
                    if (ch >= 2) arrive_warp(&bar_rawfree[rs], lane);
                    const int wi = 4 * it + ch, buf = wi % kNA, turn = wi / kNA;
                    if (turn > 0 && !wait_warp(kOneCommit ? &bar_acc[buf] : &bar_doneW[buf], (turn - 1) & 1, abort_flag)) { alive = false; break; }
                    tc_fence_after();
#pragma unroll
                    for (int i = 0; i < 4; ++i) tmem_st8(ta + buf * 32 + 8 * i, o + 8 * i);
                    tmem_st_wait();
                    tc_fence_before();
                    arrive_warp(&bar_fullW[buf], lane);
                }
                if (++rs == kRawStages) { rs = 0; rs_phase ^= 1; }
            }
        }
    } else {
        regs_up<kRegsEpi32>();
        // ===== epilogue: warp = 32 weight rows 32 (warp % 4) .., half of the tokens =====
        // A thread holds rows r0 + 8 i, columns 8 j + csub, + 1 of its half: pair 2 N8 (i / 2) + 2 j + i % 2.
        constexpr bool kComp = F::kQ81;
        const int half = warp >> 2, r0 = (warp & 3) * 32 + (lane >> 2), csub = 2 * (lane & 3);
        const uint64_t minus1 = pack2f(-1.0f, -1.0f), one = pack2f(1.0f, 1.0f);
        int it = 0, slot = 0, round = 0;
        bool alive = true;
        // Every warp works on N8 units of eight columns; those past the tile's tokens are computed and dropped.  (A branch on the size inside the loop, over
        // running sums, made the compiler move every sum, a quarter of the epilogue's instructions.)
        constexpr int kP = 4 * N8;
        for (int tile = blockIdx.x; tile < a.ntiles && alive; tile += gridDim.x) {
            TileCtx cx;
            tile_ctx(tile, tl.ntt, tl, gi, cx);
            const int n = cx.n, col0 = half * (n >> 1);
            const uint32_t tq = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)col0;
            uint64_t acc[kP];                                                 // running sums (or those of this chunk)
            [[maybe_unused]] uint64_t sum[kComp ? kP : 1], low[kComp ? kP : 1];       // compensated sum of the chunks
#pragma unroll
            for (int i = 0; i < kP; ++i) {
                acc[i] = 0ull;
                if constexpr (kComp) { sum[i] = 0ull; low[i] = 0ull; }
            }
            for (int c = 0; c < nch && alive; ++c, ++it) {
                const float *da = reinterpret_cast<const float *>(aux0 + (it & 3) * S::kAux) + col0 + csub;
                const float *rw = reinterpret_cast<const float *>(ringW + (it & 3) * S::kRingW) + r0;
                if (!wait_warp(&bar_vis[it & 1], (it >> 1) & 1, abort_flag)) { alive = false; break; }
                [[maybe_unused]] uint64_t dc[4];
                if constexpr (!F::kBlockScale && PLAIN) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) dc[i] = pack2f(rw[8 * i], rw[8 * i]);
                }
#pragma unroll 1
                for (int ch = 0; ch < 4; ++ch) {
                    if (!wait_warp(&bar_acc[slot], round & 1, abort_flag)) { alive = false; break; }
                    tc_fence_after();
#pragma unroll
                    for (int bb = 0; bb < 2; ++bb) {
                        const int b = 2 * ch + bb;
                        uint32_t p[8 * N8];
                        const uint32_t ts = tq + (uint32_t)((2 * slot + bb) * kTok);
                        tmem_ld_16x256b<N8>(ts, p);
                        tmem_ld_16x256b<N8>(ts + (16u << 16), p + 4 * N8);
                        [[maybe_unused]] uint64_t dw[4] = {}, mw[kMins ? kMins : 1][4], ss[kMins ? kMins : 1][N8];
                        uint64_t dd[N8];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            if constexpr (F::kBlockScale) { const float d = rw[b * kRows + 8 * i]; dw[i] = pack2f(d, d); }
                            else if constexpr (PLAIN) dw[i] = dc[i];
#pragma unroll
                            for (int h = 0; h < kMins; ++h) { const float m = rw[(S::kScales + 8 * h + b) * kRows + 8 * i]; mw[h][i] = pack2f(m, m); }
                        }
#pragma unroll
                        for (int j = 0; j < N8; ++j) {
                            dd[j] = *reinterpret_cast<const uint64_t *>(da + b * n + 8 * j);
#pragma unroll
                            for (int h = 0; h < kMins; ++h) ss[h][j] = *reinterpret_cast<const uint64_t *>(da + (8 + 8 * h + b) * n + 8 * j);
                        }
                        tmem_ld_wait();
                        if (bb == 1) {
                            tc_fence_before();
                            arrive_warp(&bar_free[slot], lane);
                        }
#pragma unroll
                        for (int j = 0; j < N8; ++j) {
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const int x = 2 * N8 * (i >> 1) + 2 * j + (i & 1);
                                const uint64_t pv = pack2(p[2 * x], p[2 * x + 1]);
                                if constexpr (F::kTerm) {       // d_w d_a: two f16, exact
                                    uint64_t v = mul2(mw[0][i], ss[0][j]);
                                    if constexpr (kMins == 2) v = fma2(mw[1][i], ss[1][j], v);
                                    acc[x] = fma2(one, fma2(mul2(dw[i], dd[j]), pv, v), acc[x]);
                                } else if constexpr (PLAIN && !F::kBlockScale) {
                                    acc[x] = fma2(dd[j], mul2(dw[i], pv), acc[x]);
                                    if constexpr (kMins == 1) acc[x] = fma2(mw[0][i], ss[0][j], acc[x]);
                                } else acc[x] = fma2(F::kBlockScale ? mul2(dw[i], dd[j]) : dd[j], pv, acc[x]);       // Q8_0 / Q4_0: the rounding of the int8 kernel
                            }
                        }
                    }
                    if (++slot == kSlots) { slot = 0; ++round; }
                }
                if (!alive) break;
                if constexpr (kComp) {
                    // sum += the chunk, the rounding error of the addition into `low`.  An exact two-sum, but for Q5_K and Q2_K: theirs is the fast one, which
                    // loses up to a rounding of the chunk where the chunk is larger than the sum before it.  It costs the other formats 1 - 9 % of their
                    // error (Q5_0, K = 1024, a few large blocks 5.7e-8 -> 6.1e-8); these two stay far below the sums with a minimum added per block (Q5_K
                    // 6.3e-8 for 8.7e-8, Q2_K 6.0e-8 for 7.2e-8), and three more operations per value are 4 % of the time (Q5_K 254 us -> 267).
                    constexpr bool kExact = F::kBlockScale || kSums == 0;
                    constexpr bool kScaled = !F::kBlockScale && !PLAIN;        // the chunk is d times the blocks' sum
                    [[maybe_unused]] uint64_t dw[4];
                    if constexpr (kScaled) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) dw[i] = pack2f(rw[8 * i], rw[8 * i]);
                    }
                    if constexpr (kSums > 0) {
                        if (!wait_warp(&bar_acc[slot], round & 1, abort_flag)) { alive = false; break; }
                        tc_fence_after();
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        [[maybe_unused]] uint32_t v1[4 * N8], v2[4 * N8];
                        if constexpr (kSums > 0) {
                            tmem_ld_16x256b<N8>(tq + (uint32_t)(2 * slot * kTok) + ((uint32_t)(16 * h) << 16), v1);
                            tmem_ld_16x256b<N8>(tq + (uint32_t)((2 * slot + 1) * kTok) + ((uint32_t)(16 * h) << 16), v2);
                            tmem_ld_wait();
                            if (h == 1) {
                                tc_fence_before();
                                arrive_warp(&bar_free[slot], lane);
                            }
                        }
#pragma unroll
                        for (int i = 0; i < 2 * N8; ++i) {
                            const int x = 2 * N8 * h + i;
                            const uint64_t s0 = sum[x];
                            uint64_t f = one, y = acc[x];            // the chunk is f y
                            if constexpr (kScaled) f = dw[2 * h + (x & 1)];
                            if constexpr (kSums > 0) {
                                y = fma2(f, y, fma2(one, pack2(v2[2 * i], v2[2 * i + 1]), pack2(v1[2 * i], v1[2 * i + 1])));
                                f = one;
                            }
                            const uint64_t s1 = fma2(f, y, s0);
                            if constexpr (kExact) {
                                const uint64_t bb = fma2(minus1, s0, s1), e0 = fma2(minus1, fma2(minus1, bb, s1), s0);
                                const uint64_t e1 = kScaled ? fma2(f, y, bb ^ 0x8000000080000000ull) : fma2(minus1, bb, y);
                                low[x] = fma2(one, fma2(one, e0, e1), low[x]);
                            } else low[x] = fma2(one, fma2(f, y, fma2(minus1, s1, s0)), low[x]);
                            sum[x] = s1;
                            acc[x] = 0ull;
                        }
                    }
                    if constexpr (kSums > 0) {
                        if (++slot == kSlots) { slot = 0; ++round; }
                    }
                }
            }
            if (!alive) break;
            if constexpr (kComp) {
#pragma unroll
                for (int x = 0; x < kP; ++x) {          // an infinite (or NaN) sum has no error term
                    const float s0 = lo2(sum[x]), s1 = hi2(sum[x]);
                    acc[x] = pack2f(fabsf(s0) <= 3.0e38f ? __fadd_rn(s0, lo2(low[x])) : s0, fabsf(s1) <= 3.0e38f ? __fadd_rn(s1, hi2(low[x])) : s1);
                }
            }
            const int left = min(n >> 1, cx.valid - col0);          // columns of this warp that hold tokens
            const int64_t base = ((int64_t)cx.t * tl.tt + col0) * a.stride_out + cx.row0;
#pragma unroll
            for (int j = 0; j < N8; ++j) {
                const uint64_t v[4] = {acc[2 * j], acc[2 * j + 1], acc[2 * N8 + 2 * j], acc[2 * N8 + 2 * j + 1]};       // rows r0 + 8 i
                if constexpr (STORE == kStore16 || STORE == kStore16Any) {
                    const int row = (warp & 3) * 32;
                    uint16_t *dst = (uint16_t *)a.out + base + (int64_t)(8 * j) * a.stride_out + row;
                    if constexpr (STORE == kStore16) store_rows32_wide(v, a.out_kind, dst, a.stride_out, a.nrows - cx.row0 - row, left - 8 * j);
                    else store_rows32_any(v, a.out_kind, dst, a.stride_out, a.nrows - cx.row0 - row, left - 8 * j);
                } else {
                    const int col = 8 * j + csub;
                    float *o = (float *)a.out + base + (int64_t)col * a.stride_out + r0;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const bool in = cx.row0 + r0 + 8 * i < a.nrows;
                        if (in && col < left) o[8 * i] = lo2(v[i]);
                        if (in && col + 1 < left) o[8 * i + a.stride_out] = hi2(v[i]);
                    }
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (tid == 0 && *abort_flag) atomicExch(&g_prompt_b32_timeout_flag, 1);
    if (warp == 0) tmem_dealloc(tmem_base, 512);
}

template <int WTYPE, bool PLAIN, typename T>
void launch_quantize(const void *x, void *scratch, int k, const Tiling &tl, unsigned blocks, cudaStream_t st) {
    using F = Fmt<WTYPE, PLAIN>;
    cq_launch_k(quantize_kernel<T, F::kQ81, F::kSum>, dim3(blocks), dim3(256), 0, st, (const T *)x, (uint8_t *)scratch, k, tl);
}

template <int WTYPE, bool PLAIN, int STORE, int N8> void launch_kernel(int grid, cudaStream_t st, const CUtensorMap &map, const Args &a, const Tiling &tl) {
    static_assert(Smem<WTYPE, PLAIN>::kBytes <= 232448, "shared memory of one CTA");
    static bool attr_done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attr_done[dev]) {
        cudaFuncSetAttribute(prompt32_kernel<WTYPE, PLAIN, STORE, N8>, cudaFuncAttributeMaxDynamicSharedMemorySize, Smem<WTYPE, PLAIN>::kBytes);
        attr_done[dev] = true;
    }
    cq_launch_k(prompt32_kernel<WTYPE, PLAIN, STORE, N8>, dim3(grid), dim3(kThreads), Smem<WTYPE, PLAIN>::kBytes, st, map, a, tl);
}

template <int WTYPE, bool PLAIN = false>
bool launch(const void *w, const void *x, int elem, void *dst, void *scratch, int k, int n, int tokens, int stride_dst, cudaStream_t st) {
    using R = Raw<chunk_bytes<WTYPE>()>;
    const int nch = k / 256, nrt = (n + kRows - 1) / kRows;
    const Tiling tl = plan_tiling(tokens, nrt, sm_count(), kFixedTokens, kTok);
    const long long blocks = (long long)tl.ntt * (tl.tt / 8) * nch;
    if (blocks > INT32_MAX) { cq_set_status(CQ_ERR_UNSUPPORTED, "prompt32: too many tokens for one launch"); return false; }
    const long long row_bytes = (long long)nch * chunk_bytes<WTYPE>();
    CUtensorMap map{};
    const bool use_map = (uintptr_t)w % 16 == 0 && row_bytes % 16 == 0 && row_bytes <= INT32_MAX &&
                         cq_tmap::weight_map(w, (int)row_bytes, n, R::kPitch / 2, kRows, 2, map);
    if (!use_map && R::kAligned && (uintptr_t)w % 16 != 0) {
        cq_set_status(CQ_ERR_BAD_ARG, "prompt32: weights of this format must be 16-byte aligned");
        return false;
    }
    if constexpr (!PLAIN) {
        if (elem == CQ_F32) launch_quantize<WTYPE, false, float>(x, scratch, k, tl, (unsigned)blocks, st);
        if (elem == CQ_F16) launch_quantize<WTYPE, false, __half>(x, scratch, k, tl, (unsigned)blocks, st);
    }
    if (elem == CQ_BF16) launch_quantize<WTYPE, PLAIN, __nv_bfloat16>(x, scratch, k, tl, (unsigned)blocks, st);
    const Args a{(const uint8_t *)w, (const uint8_t *)scratch, dst, elem, n, nch, stride_dst, use_map ? 1 : 0, nrt * tl.ntt};
    const int grid = a.ntiles < sm_count() ? a.ntiles : sm_count();
    if constexpr (!PLAIN) {
        if (elem == CQ_F32) {
            if (tl.tt <= 32) launch_kernel<WTYPE, false, kStoreF32, 2>(grid, st, map, a, tl);
            else launch_kernel<WTYPE, false, kStoreF32, 4>(grid, st, map, a, tl);
            return true;
        }
    }
    if (rows_16_bytes_apart(dst, stride_dst) && n % 8 == 0) {
        if (tl.tt <= 32) launch_kernel<WTYPE, PLAIN, kStore16, 2>(grid, st, map, a, tl);
        else launch_kernel<WTYPE, PLAIN, kStore16, 4>(grid, st, map, a, tl);
    } else {
        if (tl.tt <= 32) launch_kernel<WTYPE, PLAIN, kStore16Any, 2>(grid, st, map, a, tl);
        else launch_kernel<WTYPE, PLAIN, kStore16Any, 4>(grid, st, map, a, tl);
    }
    return true;
}

int sum_of(int wtype, bool plain) {
    switch (wtype) {
    case CQ_Q4_1: case CQ_Q5_1: return kTermSum;
    case CQ_Q5_0: return plain ? kTermSum : kDelta;
    case CQ_Q5_K: return plain ? kPlain32 : kSum32;
    case CQ_Q2_K: return plain ? kPlain16 : kSum16;
    }
    return kNoSum;
}

size_t scratch_bytes(int wtype, int tokens, int k, bool plain) {
    if (tokens <= 0 || k <= 0 || k % 256 != 0) return 0;
    return (size_t)((tokens + 15) / 16 * 16) * (k / 256) * (size_t)tok_bytes(sum_of(wtype, plain)) + 256;
}

bool args_ok(const void *vx, const void *x, const void *dst, const void *scratch, int elem, int ncols_x, int nrows_x, int tokens) {
    if (!vx || !x || !scratch || !dst || ncols_x <= 0 || nrows_x <= 0 || tokens <= 0 || ncols_x % 256 != 0) {
        cq_set_status(CQ_ERR_BAD_ARG, "prompt32 matmul: null pointer, empty shape or K not a multiple of 256");
        return false;
    }
    if ((uintptr_t)scratch % 16 != 0 || (uintptr_t)vx % 2 != 0 || elem < CQ_F32 || elem > CQ_BF16) {
        cq_set_status(CQ_ERR_BAD_ARG, "prompt32 matmul: misaligned scratch or weights, or unknown element type");
        return false;
    }
    return true;
}

}  // namespace

extern "C" size_t cq_prompt32_scratch_bytes(int wtype, int tokens, int k) { return scratch_bytes(wtype, tokens, k, false); }
extern "C" size_t cq_prompt32_bf16_scratch_bytes(int wtype, int tokens, int k) { return scratch_bytes(wtype, tokens, k, true); }

// time of a slice of up to eight rows on the decode kernel; weights: millions of them
static double slice_us(bool super, int rows, int k, double weights) {
    return super ? 5.25 + 0.125e-3 * k + weights * (0.05 + 0.084 * rows) : std::max(5.05, 4.7 + 0.018e-3 * k + weights * (0.21 + 0.02 * rows));
}

// The six Q8_1 formats against slices of eight rows on the decode kernel, which stream the matrix once each.  Models of both sides (9 - 220 tokens,
// 32 - 20000 rows, K to 14336; f32, cold weights): a round of tiles takes a fixed part and one per token and 256 elements of K, measured at 148
// tiles; a slice its two launches, and time per weight that grows with its rows (a fit to 1500 shapes).  Of 240 sampled shapes 10 go to the slower side by
// more than 5 %, all of them to the slices, mostly a matrix of few rows and long K (192 rows of K = 9216, 123 tokens: 77 us here, 113 in slices).
extern "C" int cq_prompt32_pays(int wtype, int tokens, int k, int n) {
    const double sms = cq_sm_count(), weights = 1e-6 * n * (double)k;
    const Tiling tl = plan_tiling(tokens, (n + kRows - 1) / kRows, (int)sms, kFixedTokens, 64);
    const double rounds = std::ceil((double)((n + kRows - 1) / kRows) * tl.ntt / sms);
    const bool super = cq_block_elems(wtype) == 256;
    double fixed = 2.16, per_token = 0.0104;        // Q5_K
    switch (wtype) {
    case CQ_Q4_1: fixed = 2.1; per_token = 0.0215; break;
    case CQ_Q5_0: fixed = 2.58; per_token = 0.0081; break;
    case CQ_Q5_1: fixed = 2.41; per_token = 0.019; break;
    case CQ_Q2_K: fixed = 2.46; per_token = 0.008; break;
    case CQ_Q3_K: fixed = 2.64; per_token = 0.005; break;
    }
    const double idle = (double)((n + kRows - 1) / kRows) * tl.ntt < 0.3 * sms ? 0.85 : 1.0;      // few tiles share the L2
    const double here = 8.5 + rounds * (k / 256) * (fixed + per_token * tl.tt) * idle;
    const int whole = tokens / 8, left = tokens % 8;
    return here < (super ? 1.8 : 2.5) + whole * slice_us(super, 8, k, weights) + (left ? slice_us(super, left, k, weights) : 0.0);
}

// The same with bf16, whose line has not followed the kernel (its constants are those of a kernel that took 468 us where this one takes 325, Q5_K 4096 ->
// 14336, 512 tokens): the two sides add in different orders, so a call that changes sides gets a few in 100 000 of its bf16 results as the neighbouring value.
// Of the same shapes 19 go to the slower side by more than 5 %, all of them to the slices (36 rows of K = 11520, 205 tokens: 95 us here, 197 in slices).
extern "C" int cq_prompt32_bf16_pays(int wtype, int tokens, int k, int n) {
    const double sms = cq_sm_count(), weights = 1e-6 * n * (double)k;
    const Tiling tl = plan_tiling(tokens, (n + kRows - 1) / kRows, (int)sms, 40, 64);
    const double rounds = std::ceil((double)((n + kRows - 1) / kRows) * tl.ntt / sms);
    const bool super = cq_block_elems(wtype) == 256;
    const double fixed = wtype == CQ_Q2_K ? 2.52 : wtype == CQ_Q3_K ? 2.09 : 2.27, per_token = wtype == CQ_Q2_K ? 0.046 : 0.036;
    const double here = 6.7 + rounds * (k / 256) * (fixed + per_token * tl.tt);
    const int whole = tokens / 8, left = tokens % 8;
    return here < (super ? 1.8 : 2.5) + whole * slice_us(super, 8, k, weights) + (left ? slice_us(super, left, k, weights) : 0.0);
}

extern "C" int cq_prompt32_tile_tokens(int tokens, int n) {
    return tokens <= 0 || n <= 0 ? 0 : plan_tiling(tokens, (n + kRows - 1) / kRows, sm_count(), kFixedTokens, kTok).tt;
}

extern "C" void cq_prompt32_matmul(int wtype, const void *vx, const void *x, int elem, void *dst, void *scratch, int ncols_x, int nrows_x,
                                   int tokens, int stride_dst, void *stream) {
    if (!args_ok(vx, x, dst, scratch, elem, ncols_x, nrows_x, tokens)) return;
    cudaStream_t st = (cudaStream_t)stream;
    bool ok = false;
    switch (wtype) {
    case CQ_Q4_0: ok = launch<CQ_Q4_0>(vx, x, elem, dst, scratch, ncols_x, nrows_x, tokens, stride_dst, st); break;
    case CQ_Q8_0: ok = launch<CQ_Q8_0>(vx, x, elem, dst, scratch, ncols_x, nrows_x, tokens, stride_dst, st); break;
    case CQ_Q4_1: ok = launch<CQ_Q4_1>(vx, x, elem, dst, scratch, ncols_x, nrows_x, tokens, stride_dst, st); break;
    case CQ_Q5_0: ok = launch<CQ_Q5_0>(vx, x, elem, dst, scratch, ncols_x, nrows_x, tokens, stride_dst, st); break;
    case CQ_Q5_1: ok = launch<CQ_Q5_1>(vx, x, elem, dst, scratch, ncols_x, nrows_x, tokens, stride_dst, st); break;
    case CQ_Q2_K: ok = launch<CQ_Q2_K>(vx, x, elem, dst, scratch, ncols_x, nrows_x, tokens, stride_dst, st); break;
    case CQ_Q3_K: ok = launch<CQ_Q3_K>(vx, x, elem, dst, scratch, ncols_x, nrows_x, tokens, stride_dst, st); break;
    case CQ_Q5_K: ok = launch<CQ_Q5_K>(vx, x, elem, dst, scratch, ncols_x, nrows_x, tokens, stride_dst, st); break;
    default: cq_set_status(CQ_ERR_UNSUPPORTED, "prompt32 matmul: Q4_K and Q6_K have their own kernel"); return;
    }
    if (ok) cq_check_launch("prompt32 matmul");
}

extern "C" void cq_prompt32_bf16_matmul(int wtype, const void *vx, const void *x, void *dst, void *scratch, int ncols_x, int nrows_x, int tokens,
                                        int stride_dst, void *stream) {
    if (!args_ok(vx, x, dst, scratch, CQ_BF16, ncols_x, nrows_x, tokens)) return;
    cudaStream_t st = (cudaStream_t)stream;
    bool ok = false;
    switch (wtype) {
    case CQ_Q4_1: ok = launch<CQ_Q4_1>(vx, x, CQ_BF16, dst, scratch, ncols_x, nrows_x, tokens, stride_dst, st); break;
    case CQ_Q5_1: ok = launch<CQ_Q5_1>(vx, x, CQ_BF16, dst, scratch, ncols_x, nrows_x, tokens, stride_dst, st); break;
    case CQ_Q5_0: ok = launch<CQ_Q5_0, true>(vx, x, CQ_BF16, dst, scratch, ncols_x, nrows_x, tokens, stride_dst, st); break;
    case CQ_Q2_K: ok = launch<CQ_Q2_K, true>(vx, x, CQ_BF16, dst, scratch, ncols_x, nrows_x, tokens, stride_dst, st); break;
    case CQ_Q3_K: ok = launch<CQ_Q3_K, true>(vx, x, CQ_BF16, dst, scratch, ncols_x, nrows_x, tokens, stride_dst, st); break;
    case CQ_Q5_K: ok = launch<CQ_Q5_K, true>(vx, x, CQ_BF16, dst, scratch, ncols_x, nrows_x, tokens, stride_dst, st); break;
    default: cq_set_status(CQ_ERR_UNSUPPORTED, "prompt32 matmul in bf16: Q4_1, Q5_0, Q5_1, Q2_K, Q3_K, Q5_K"); return;
    }
    if (ok) cq_check_launch("prompt32 matmul");
}

extern "C" int cq_prompt32_timeout_flag(void) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_prompt_b32_timeout_flag, sizeof v) != cudaSuccess) { (void)cudaGetLastError(); return -1; }
    if (v) cq_set_status(CQ_ERR_TIMEOUT, "prompt32 matmul: a bounded wait gave up");
    return v;
}
extern "C" int cq_prompt32_bf16_timeout_flag(void) { return cq_prompt32_timeout_flag(); }
