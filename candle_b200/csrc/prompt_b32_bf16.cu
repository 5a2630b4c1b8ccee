// Prompt-phase GEMM of Q4_1, Q5_0, Q5_1, Q2_K, Q3_K and Q5_K with bf16 inputs and outputs: the summation that prompt_b32.cu replaced for f32 and f16.
//
// Why it is still here: the sums of the two kernels differ by 1e-7 (2-norm; those of prompt_b32.cu are the closer ones to 64 bits), which takes a few in
// 100 000 bf16 results to the neighbouring value, up to 2^-7 away, more than the 6e-3 of a value by which bf16 results may move from one
// version to the next.  f32 and f16 results stay within theirs.  It costs: Q5_K 4096 -> 14336, 512 tokens 490 us where prompt_b32.cu takes 236.
//
// Every 32-element block is two K = 16 steps into a FRESH accumulator slot, exact (sums below 2^24: at most 31 * 63 * 127 * 32); the codes are unsigned and the
// epilogue adds  d_a d_w I + m_w s_a  to f32 running sums, two at a time: the blocks of a 256-element chunk first, the chunks with a compensated
// sum, since the decode kernels, which these formats use otherwise, sum by a balanced tree.
//
// Mapping: tiles of 128 weight rows x up to 64 tokens, warps 0-7 epilogue, 8-11 producers, 12 MMA issuer, 13 loader, 14-15 raw bytes where there is no tensor
// map; tensor memory: three accumulator slots of two blocks (128 columns), 128 columns of operand A.  Bound by the epilogue, 2.5 us per 256
// elements of K.  Every wait is bounded as in prompt_kq.cu.
#include "../../include/candle_q_b200.h"
#include "prompt_f16.cuh"

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace {
using namespace cq_prompt;

constexpr int kEpiWarps = 8, kProdWarps = 4;
constexpr int kMmaWarp = kEpiWarps + kProdWarps, kLoadWarp = kMmaWarp + 1, kRawWarp = kMmaWarp + 2;
constexpr int kThreads = (kEpiWarps + kProdWarps + 4) * 32;      // the last two: raw bytes without a tensor map
constexpr int kColA = 384;
constexpr int kFixedTokens = 40;                // plan_tiling

__device__ int g_prompt_b32_bf16_timeout_flag = 0;

// kMins: terms m_w * s_a per block;  kSum: what s_a is;  kTerm: a block's terms are summed apart from the running sum.  The codes are unsigned,
// so d_a d_w I and m_w s_a are both large and nearly cancel for weights around zero; added to the running sum one after the other they left
// two to four times the decode kernels' error against 64 bits (2-norm, K = 4096, activations of one sign: Q4_1 2.2e-7 for 7.6e-8, Q5_1 2.6e-7
// for 7.7e-8; now 6.7e-8 and 6.9e-8), for 2 - 4 % of the time.  Q5_K stays below the decode kernel's own error without (normal activations
// 1.0e-7 for 1.1e-7, one sign 2.8e-7 for 4.9e-7).
enum { kNoSum, kFloatSum, kIntSum };
template <int WTYPE> struct Fmt;
template <int MINS, int SUM, bool TERM> struct FmtQ81 {
    static constexpr bool kTerm = TERM;
    static constexpr int kMins = MINS, kSum = SUM, kTok = 64, kStagesT = 4;
};
template <> struct Fmt<CQ_Q4_1> : FmtQ81<1, kFloatSum, true> {};
template <> struct Fmt<CQ_Q5_0> : FmtQ81<1, kFloatSum, true> {};
template <> struct Fmt<CQ_Q5_1> : FmtQ81<1, kFloatSum, true> {};
template <> struct Fmt<CQ_Q5_K> : FmtQ81<1, kIntSum, false> {};
template <> struct Fmt<CQ_Q2_K> : FmtQ81<2, kIntSum, true> {};     // one per 16 elements
template <> struct Fmt<CQ_Q3_K> : FmtQ81<0, kNoSum, false> {};

template <int WTYPE> constexpr int chunk_bytes() { return 256 / cq_block_elems(WTYPE) * cq_type_size(WTYPE); }
template <int MINS> constexpr int tok_bytes() { return 512 + 32 + 32 * MINS; }        // f16 values, scales, sums of one chunk
template <int MINS> constexpr int wscale_bytes() { return MINS == 0 ? 4 : MINS == 1 ? 8 : 16; }
template <int WTYPE> struct Smem {
    using F = Fmt<WTYPE>;
    static constexpr int kStageT = 16 * F::kTok * 16, kAux = F::kTok * (32 + 32 * F::kMins), kRingW = 8 * kRows * wscale_bytes<F::kMins>();
    static constexpr int kBytes = 1024 + F::kStagesT * kStageT + 4 * kAux + 4 * kRingW + 2 * Raw<chunk_bytes<WTYPE>()>::kBytes + 16;
};

// ---- activations ---------------------------------------------------------------------------------------------------
// One warp per (token, chunk of 256), 8 tokens of one chunk per block, through shared memory (see prompt_kq.cu).
template <int MINS, int SUM>
__global__ void __launch_bounds__(256) quantize_kernel(const __nv_bfloat16 *__restrict__ x, uint8_t *__restrict__ y, int k, Tiling tl) {
    constexpr int kPitch = 8 * 16 + 16, kVals = 8 * (1 + MINS);
    __shared__ __align__(16) uint8_t sm[32 * kPitch];
    __shared__ float sv[kVals][8];      // [value][token]: block scales, then sums
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
    // mmvq_gguf.cu:811-911
#pragma unroll
    for (int i = 0; i < 8; ++i) q[i] = (amax == 0.0f) ? 0 : (int)(int8_t)roundf(__fdiv_rn(e[i], d));
    const float dh = __half2float(__float2half_rn(d));
    *reinterpret_cast<uint4 *>(sm + lane * kPitch + warp * 16) = pack_q8(q);
    const int b = lane >> 2;
    if ((lane & 3) == 0) sv[b][warp] = dh;
    if constexpr (SUM == kFloatSum) {
        // the f16-rounded sum of the inputs, added in the order of a 32-lane xor butterfly over the block (16, 8, 4, 2, 1)
        float s[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) s[i] = __fadd_rn(e[i], __shfl_xor_sync(0xffffffffu, e[i], 2));
#pragma unroll
        for (int i = 0; i < 8; ++i) s[i] = __fadd_rn(s[i], __shfl_xor_sync(0xffffffffu, s[i], 1));
        const float t0 = __fadd_rn(__fadd_rn(s[0], s[4]), __fadd_rn(s[2], s[6])), t1 = __fadd_rn(__fadd_rn(s[1], s[5]), __fadd_rn(s[3], s[7]));
        if ((lane & 3) == 0) sv[8 + b][warp] = __half2float(__float2half_rn(__fadd_rn(t0, t1)));
    } else if constexpr (SUM == kIntSum) {      // scale times the sum of the int8 values, per block or per 16
        int s = q[0] + q[1] + q[2] + q[3] + q[4] + q[5] + q[6] + q[7];
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        if constexpr (MINS == 1) s += __shfl_xor_sync(0xffffffffu, s, 2);
        if constexpr (MINS == 1) { if ((lane & 3) == 0) sv[8 + b][warp] = __fmul_rn(dh, (float)s); }
        else { if ((lane & 1) == 0) sv[8 + 8 * ((lane >> 1) & 1) + b][warp] = __fmul_rn(dh, (float)s); }
    }
    __syncthreads();
    uint8_t *blob = y + ((size_t)t * tl.tt * nch + (size_t)c * rows) * tok_bytes<MINS>();
    for (int i = threadIdx.x; i < 32 * 8; i += 256)
        *reinterpret_cast<uint4 *>(blob + ((size_t)(i >> 3) * rows + row0 + (i & 7)) * 16) = *reinterpret_cast<const uint4 *>(sm + (i >> 3) * kPitch + (i & 7) * 16);
    for (int i = threadIdx.x; i < kVals * 8; i += 256)
        *reinterpret_cast<float *>(blob + (size_t)rows * 512 + ((size_t)(i >> 3) * rows + row0 + (i & 7)) * 4) = sv[i >> 3][i & 7];
}

// ---- producers: chunk CH = 0..3 covers blocks 2 CH (cells 0-15) and 2 CH + 1 (cells 16-31) -----------------------------
struct WScale { float d, m0, m1; };

// 32-bit word at byte offset OFF (even) of a row chunk held as 16-byte vectors from vector V0 on
template <int OFF, int V0, int NV> __device__ __forceinline__ uint32_t word_at(const uint4 (&v)[NV]) {
    constexpr int w = OFF / 4 - 4 * V0;
    auto get = [&](int i) -> uint32_t { const uint4 &q = v[i >> 2]; return (i & 3) == 0 ? q.x : (i & 3) == 1 ? q.y : (i & 3) == 2 ? q.z : q.w; };
    if constexpr (OFF % 4 == 0) return get(w);
    else return __funnelshift_r(get(w), get(w + 1), 16);
}
__device__ __forceinline__ float h16(uint32_t w) { return __half2float(__ushort_as_half((unsigned short)(w & 0xFFFFu))); }
// pairs (byte 0, byte 2) and (byte 1, byte 3) of a word of small unsigned codes as f16
__device__ __forceinline__ void codes4(uint32_t w, uint32_t &a, uint32_t &b) {
    const __half2 o = __float2half2_rn(1024.0f);
    a = h2_bits(__hsub2(bits_h2((w & 0x00FF00FFu) | 0x64006400u), o));
    b = h2_bits(__hsub2(bits_h2(((w >> 8) & 0x00FF00FFu) | 0x64006400u), o));
}

// 16 consecutive tokens' values of one weight row; values past `valid` are not stored
__device__ __forceinline__ void store16(const uint64_t (&v)[8], __nv_bfloat16 *out, int64_t stride, int valid) {
#pragma unroll
    for (int i = 0; i < 16; ++i)
        if (i < valid) out[i * stride] = __float2bfloat16((i & 1) ? hi2(v[i >> 1]) : lo2(v[i >> 1]));
}

template <int WTYPE> struct Expand;

// the 32-element block formats: their chunk is a whole number of 16-byte vectors
template <int WTYPE> struct ExpandBlock {
    static constexpr int kBlk = cq_type_size(WTYPE);
    static constexpr bool kHasM = WTYPE == CQ_Q4_1 || WTYPE == CQ_Q5_1, kFive = WTYPE == CQ_Q5_0 || WTYPE == CQ_Q5_1;
    const uint8_t *p;
    __device__ __forceinline__ void header(const uint8_t *rr, int) { p = rr; }
    template <int B, int V0, int NV> __device__ __forceinline__ WScale block(const uint4 (&v)[NV], uint32_t *o) const {
        constexpr int off = B * kBlk, qs = off + 2 + (kHasM ? 2 : 0) + (kFive ? 4 : 0);
        WScale s;
        s.d = h16(word_at<off, V0>(v));
        s.m1 = 0.0f;
        s.m0 = kHasM ? h16(word_at<off + 2, V0>(v)) : __fmul_rn(-16.0f, s.d);      // Q5_0: the codes stay unsigned, -16 d s
        {
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
                codes4(lo, o[2 * i], o[2 * i + 1]);
                codes4(hi, o[8 + 2 * i], o[8 + 2 * i + 1]);
            };
            four(std::integral_constant<int, 0>{}); four(std::integral_constant<int, 1>{});
            four(std::integral_constant<int, 2>{}); four(std::integral_constant<int, 3>{});
        }
        return s;
    }
    template <int CH> __device__ __forceinline__ void chunk(uint32_t (&o)[32], WScale (&s)[2]) {
        constexpr int v0 = 2 * CH * kBlk / 16, nv = (2 * (CH + 1) * kBlk + 15) / 16 - v0;
        uint4 v[nv + 1];
#pragma unroll
        for (int i = 0; i < nv; ++i) v[i] = *reinterpret_cast<const uint4 *>(p + 16 * (v0 + i));
        v[nv] = make_uint4(0u, 0u, 0u, 0u);       // word_at may name (not use) the word after the last
        s[0] = block<2 * CH, v0>(v, o);
        s[1] = block<2 * CH + 1, v0>(v, o + 16);
    }
};
template <> struct Expand<CQ_Q4_1> : ExpandBlock<CQ_Q4_1> {};
template <> struct Expand<CQ_Q5_0> : ExpandBlock<CQ_Q5_0> {};
template <> struct Expand<CQ_Q5_1> : ExpandBlock<CQ_Q5_1> {};

// Q5_K: Q4_K with the fifth bits of sub-block g in bit g of 32 bytes; codes times the 6-bit scale, at most 31 * 63 = 1953.
template <> struct Expand<CQ_Q5_K> {
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
    template <int CH> __device__ __forceinline__ void chunk(uint32_t (&o)[32], WScale (&s)[2]) {
        const uint4 a = *reinterpret_cast<const uint4 *>(p + 48 + 32 * CH), b = *reinterpret_cast<const uint4 *>(p + 64 + 32 * CH);
        const uint4 ha = *reinterpret_cast<const uint4 *>(p + 16), hb = *reinterpret_cast<const uint4 *>(p + 32);
        const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}, h[8] = {ha.x, ha.y, ha.z, ha.w, hb.x, hb.y, hb.z, hb.w};
        auto byte_of = [](const uint32_t (&t)[2], int j) { return (t[j >> 2] >> (8 * (j & 3))) & 0xFFu; };
        auto twice = [](uint32_t v) { return __hsub2(bits_h2(v * 0x00010001u | 0x64006400u), bits_h2(0x64006400u)); };
        const __half2 dmh = bits_h2(dm);
        const float d = __low2float(dmh), dmin = __high2float(dmh);
        s[0] = WScale{d, -__fmul_rn(dmin, (float)byte_of(mn, 2 * CH)), 0.0f};
        s[1] = WScale{d, -__fmul_rn(dmin, (float)byte_of(mn, 2 * CH + 1)), 0.0f};
        const __half2 s0 = twice(byte_of(sc, 2 * CH)), s1 = twice(byte_of(sc, 2 * CH + 1));
        const __half2 c0 = __hmul2(s0, __float2half2_rn(-1024.0f));
        const __half2 m1 = __hmul2(s1, __float2half2_rn(0.0625f)), c1 = __hmul2(s1, __float2half2_rn(-64.0f));
#pragma unroll
        for (int i = 0; i < 8; ++i) {
#pragma unroll
            for (int od = 0; od < 2; ++od) {        // bytes 0, 2 | 1, 3
                const uint32_t u = od ? w[i] >> 8 : w[i], v = od ? h[i] >> 8 : h[i];
                const uint32_t lo = (u & 0x000F000Fu) | ((2 * CH >= 4 ? v >> (2 * CH - 4) : v << (4 - 2 * CH)) & 0x00100010u);
                // high nibbles stay in place, so their codes are 16-fold: the fifth bit goes to bit 8
                const uint32_t hi = (u & 0x00F000F0u) | ((v << (7 - 2 * CH)) & 0x01000100u);
                o[2 * i + od] = hfma2_bits(lo | 0x64006400u, s0, c0);
                o[16 + 2 * i + od] = hfma2_bits(hi | 0x64006400u, m1, c1);
            }
        }
    }
};

// Q2_K / Q3_K: block b = 4 n + pos: bit pair pos of bytes 32 n .. of the codes; a scale per 16 elements, number 2 b + half.
template <> struct Expand<CQ_Q2_K> {
    const uint8_t *p;
    uint32_t q[8], sc[4];
    float d, dmin;
    __device__ __forceinline__ void header(const uint8_t *rr, int shift) {
        p = rr + shift;         // a multiple of 4 when the base is, else of 2
        cq_lds_words<4>(p, sc);
        uint32_t dm[1];
        cq_lds_words<1>(p + 80, dm);
        d = h16(dm[0]); dmin = h16(dm[0] >> 16);
    }
    template <int CH> __device__ __forceinline__ void chunk(uint32_t (&o)[32], WScale (&s)[2]) {
        if constexpr ((CH & 1) == 0) cq_lds_words<8>(p + 16 + 16 * CH, q);
#pragma unroll
        for (int bb = 0; bb < 2; ++bb) {
            const int b = 2 * CH + bb, pos = b & 3;
            float m[2];
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                const uint32_t by = (sc[(2 * b + hf) >> 2] >> (8 * ((2 * b + hf) & 3))) & 0xFFu;
                m[hf] = -__fmul_rn(dmin, (float)(by >> 4));
                const __half2 sv = __hsub2(bits_h2((by & 0xFu) * 0x00010001u | 0x64006400u), bits_h2(0x64006400u));
                const __half2 cv = __hmul2(sv, __float2half2_rn(-1024.0f));
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t u = q[4 * hf + i] >> (2 * pos);
                    o[16 * bb + 8 * hf + 2 * i] = hfma2_bits((u & 0x00030003u) | 0x64006400u, sv, cv);
                    o[16 * bb + 8 * hf + 2 * i + 1] = hfma2_bits(((u >> 8) & 0x00030003u) | 0x64006400u, sv, cv);
                }
            }
            s[bb] = WScale{d, m[0], m[1]};
        }
    }
};
template <> struct Expand<CQ_Q3_K> {
    const uint8_t *p;
    uint32_t q[8], hm[8], sc[3];
    float d;
    __device__ __forceinline__ void header(const uint8_t *rr, int shift) {
        p = rr + shift;         // even
        cq_lds_words<3>(p + 96, sc);
        cq_lds_words<8>(p, hm);
        d = __half2float(*reinterpret_cast<const __half *>(p + 108));
    }
    template <int CH> __device__ __forceinline__ void chunk(uint32_t (&o)[32], WScale (&s)[2]) {
        if constexpr ((CH & 1) == 0) cq_lds_words<8>(p + 32 + 16 * CH, q);
#pragma unroll
        for (int bb = 0; bb < 2; ++bb) {
            const int b = 2 * CH + bb, pos = b & 3;
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                const int j = 2 * b + hf;       // scale number: 4 low bits from bytes 0-7, 2 high bits from bytes 8-11
                const uint32_t lo4 = (sc[(j & 7) >> 2] >> (8 * (j & 3) + (j < 8 ? 0 : 4))) & 0xFu, hi2 = (sc[2] >> (8 * (j & 3) + 2 * (j >> 2))) & 3u;
                const __half2 sv = __hsub2(bits_h2((lo4 | hi2 << 4) * 0x00010001u | 0x64006400u), __float2half2_rn(1056.0f));
                const __half2 four = __float2half2_rn(1028.0f);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    // two bits, plus 4 when the mask bit is set, minus 4
                    const uint32_t u = ((q[4 * hf + i] >> (2 * pos)) & 0x03030303u) | (((hm[4 * hf + i] >> b) & 0x01010101u) << 2);
                    o[16 * bb + 8 * hf + 2 * i] = h2_bits(__hmul2(__hsub2(bits_h2((u & 0x00FF00FFu) | 0x64006400u), four), sv));
                    o[16 * bb + 8 * hf + 2 * i + 1] = h2_bits(__hmul2(__hsub2(bits_h2(((u >> 8) & 0x00FF00FFu) | 0x64006400u), four), sv));
                }
            }
            s[bb] = WScale{d, 0.0f, 0.0f};
        }
    }
};

struct Args {
    const uint8_t *w, *act;
    __nv_bfloat16 *out;
    int nrows, nch, stride_out, use_map, ntiles;
};

template <int WTYPE>
__global__ void __launch_bounds__(kThreads, 1) prompt32_bf16_kernel(const __grid_constant__ CUtensorMap wmap, const Args a, const Tiling tl) {
    using F = Fmt<WTYPE>;
    using S = Smem<WTYPE>;
    constexpr int kCB = chunk_bytes<WTYPE>(), kMins = F::kMins, kTok = F::kTok, kStagesT = F::kStagesT, kSlots = 3;
    using R = Raw<kCB>;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t *bar_raw = reinterpret_cast<uint64_t *>(smem);        // [2] raw weight bytes landed
    uint64_t *bar_rawfree = bar_raw + 2;                            // [2] read by all producers
    uint64_t *bar_fullT = bar_raw + 4;                              // [4] token stage (first half: + scales) landed
    uint64_t *bar_doneT = bar_raw + 8;                              // [4] its MMAs are complete
    uint64_t *bar_fullW = bar_raw + 12;                             // [4] operand A chunk stored (all producers)
    uint64_t *bar_doneW = bar_raw + 16;                             // [4] its MMAs are complete
    uint64_t *bar_vis = bar_raw + 20;                               // [4] relay: the scales of this operand chunk are visible
    uint64_t *bar_acc = bar_raw + 24;                               // [3] the MMAs of two blocks are complete
    uint64_t *bar_free = bar_raw + 30;                              // [3] accumulator slot read (all epilogue warps)
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + 512);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + 520);
    uint8_t *stT0 = smem + 1024;
    uint8_t *aux0 = stT0 + kStagesT * S::kStageT;       // [4] scales [8][n], then sums [kMins][8][n]
    uint8_t *ringW = aux0 + 4 * S::kAux;                // [4][8 blocks][128 rows] weight scales (and minima)
    uint8_t *raw0 = ringW + 4 * S::kRingW;              // 128-byte aligned

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nch = a.nch;
    const uint32_t row_bytes = (uint32_t)nch * kCB;
    const GroupInfo gi{};

    if (tid == 0) {
        for (int i = 0; i < 2; ++i) { cq_mbar_init(&bar_raw[i], a.use_map ? 1 : kRawThreads); cq_mbar_init(&bar_rawfree[i], kProdWarps); }
        for (int i = 0; i < 4; ++i) {
            cq_mbar_init(&bar_fullT[i], 1);
            cq_mbar_init(&bar_doneT[i], 1);
            cq_mbar_init(&bar_fullW[i], kProdWarps);
            cq_mbar_init(&bar_doneW[i], 1);
            cq_mbar_init(&bar_vis[i], 1);
        }
        for (int i = 0; i < kSlots; ++i) { cq_mbar_init(&bar_acc[i], 1); cq_mbar_init(&bar_free[i], kEpiWarps); }
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

    if (warp >= kEpiWarps && warp < kMmaWarp) {
        // ===== producers: thread = weight row = TMEM lane =====
        const int r = tid - kEpiWarps * 32;
        const uint32_t ta = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)kColA;
        int it = 0, wi = 0;
        bool alive = true;
        for (int tile = blockIdx.x; tile < a.ntiles && alive; tile += gridDim.x) {
            TileCtx cx;
            tile_ctx(tile, tl.ntt, tl, gi, cx);
            long long wr = cx.wrow0 + r;
            if (wr >= a.nrows) wr = a.nrows - 1;
            const uint32_t row_off = a.use_map ? 0u : (uint32_t)((uintptr_t)(a.w + wr * row_bytes) & 15);
            for (int c = 0; c < nch && alive; ++c, ++it) {
                const int rs = it & 1;
                if (!wait_warp(&bar_raw[rs], (it >> 1) & 1, abort_flag)) { alive = false; break; }
                Expand<WTYPE> ex;
                ex.header(raw0 + rs * R::kBytes + r * R::kPitch, R::kAligned ? 0 : (int)((row_off + (uint32_t)c * kCB) & 15));
                uint8_t *rw = ringW + (it & 3) * S::kRingW + r * wscale_bytes<kMins>();
                auto step = [&](auto chc) {
                    constexpr int CH = decltype(chc)::value;
                    if (!alive) return;
                    uint32_t o[32];
                    WScale s[2];
                    ex.template chunk<CH>(o, s);
                    if constexpr (CH == 3) arrive_warp(&bar_rawfree[rs], lane);
                    const int buf = wi & 3;
                    if (wi >= 4 && !wait_warp(&bar_doneW[buf], ((wi >> 2) - 1) & 1, abort_flag)) { alive = false; return; }
                    tc_fence_after();
                    // the first operand chunk of it - 1 is done, so its MMAs had started and the epilogue, at most three
                    // operand chunks behind them, has finished it - 3: entry it - 4 of the ring is free
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        uint8_t *dst = rw + (2 * CH + b) * kRows * wscale_bytes<kMins>();
                        if constexpr (kMins == 0) *reinterpret_cast<float *>(dst) = s[b].d;
                        else if constexpr (kMins == 1) *reinterpret_cast<float2 *>(dst) = make_float2(s[b].d, s[b].m0);
                        else *reinterpret_cast<float4 *>(dst) = make_float4(s[b].d, s[b].m0, s[b].m1, 0.0f);
                    }
                    tmem_st32(ta + buf * 32, o);
                    tmem_st_wait();
                    tc_fence_before();
                    arrive_warp(&bar_fullW[buf], lane);
                    ++wi;
                };
                step(std::integral_constant<int, 0>{}); step(std::integral_constant<int, 1>{});
                step(std::integral_constant<int, 2>{}); step(std::integral_constant<int, 3>{});
            }
        }
    } else if (warp == kLoadWarp) {
        // ===== loader =====
        int it = 0, ti = 0;
        bool alive = true;
        for (int tile = blockIdx.x; tile < a.ntiles && alive; tile += gridDim.x) {
            TileCtx cx;
            tile_ctx(tile, tl.ntt, tl, gi, cx);
            const int n = cx.n;
            const uint8_t *blob0 = a.act + (size_t)cx.blob_row * nch * tok_bytes<kMins>();
            for (int c = 0; c < nch && alive; ++c, ++it) {
                const int rs = it & 1;
                if (a.use_map) {
                    if (it >= 2 && !wait_warp(&bar_rawfree[rs], ((it >> 1) - 1) & 1, abort_flag)) { alive = false; break; }
                    if (lane == 0) {
                        cq_mbar_expect_tx(&bar_raw[rs], R::kBytes);
                        cq_tmap::load_2d(raw0 + rs * R::kBytes, &wmap, (int)(((uint32_t)c * kCB & ~15u) / 2), cx.row0, &bar_raw[rs]);
                    }
                }
                const uint8_t *blob = blob0 + (size_t)c * n * tok_bytes<kMins>();
                for (int half = 0; half < 2; ++half, ++ti) {
                    const int s = ti % kStagesT;
                    if (ti >= kStagesT && !wait_warp(&bar_doneT[s], (ti / kStagesT - 1) & 1, abort_flag)) { alive = false; break; }
                    if (lane == 0) {
                        const unsigned bytes = (unsigned)n * 256;
                        if (half == 0) {
                            // a stage of chunk it - 2 (or later) is done: its MMAs had started, so the epilogue has finished it - 4
                            const unsigned aux_bytes = (unsigned)n * (32 + 32 * kMins);
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
            for (int j = it >= 2 ? it - 1 : 0; a.use_map && j <= it; ++j) (void)cq_mbar_wait_bounded(&bar_raw[j & 1], (j >> 1) & 1);
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
                    const int rs = it & 1;
                    if (it >= 2 && !wait_warp(&bar_rawfree[rs], ((it >> 1) - 1) & 1, abort_flag)) { alive = false; break; }
                    R::load_rows(raw0 + rs * R::kBytes, w0 + (uint32_t)c * kCB, min(a.nrows - cx.row0, kRows), row_bytes, tid - kRawWarp * 32, &bar_raw[rs]);
                }
            }
            cq_cp_async_wait<0>();
        }
    } else if (warp == kMmaWarp) {
        // ===== MMA issuer (the warp runs the loop, one elected lane issues): a block = two K = 16 steps into fresh columns =====
        const uint32_t stT = uniform(cq_smem_u32(stT0) >> 4), tm = uniform(tmem_base);
        int it = 0, wi = 0, s = 0, s_phase = 0, slot = 0, round = 0;      // token stage; accumulator slot and how often all have been used
        bool alive = true;
        for (int tile = blockIdx.x; tile < a.ntiles && alive; tile += gridDim.x) {
            TileCtx cx;
            tile_ctx(tile, tl.ntt, tl, gi, cx);
            const uint32_t n = uniform((uint32_t)cx.n), idesc = idesc_f16((int)n), bT = stT | (n << 16);
#pragma unroll 1
            for (int c = 0; c < nch && alive; ++c, ++it) {
#pragma unroll
                for (int ch = 0; ch < 4; ++ch, ++wi) {
                    const int buf = wi & 3;
                    if (((ch & 1) == 0 && !wait_warp(&bar_fullT[s], s_phase, abort_flag)) ||
                        !wait_warp(&bar_fullW[buf], (wi >> 2) & 1, abort_flag) ||
                        (round > 0 && !wait_warp(&bar_free[slot], (round - 1) & 1, abort_flag))) { alive = false; break; }
                    tc_fence_after();
                    const uint32_t b0 = bT + (uint32_t)s * (S::kStageT >> 4) + (uint32_t)(8 * (ch & 1)) * n, a0 = tm + (uint32_t)(kColA + buf * 32);
                    const uint32_t td = tm + (uint32_t)(slot * 2 * kTok);
                    if (elect_one()) {
                        mbar_arrive(&bar_vis[buf]);     // what this warp has acquired is visible to the epilogue
                        mma_f16_ts<false>(td, a0, b0, idesc);
                        mma_f16_ts<true>(td, a0 + 8, b0 + 2 * n, idesc);
                        mma_f16_ts<false>(td + kTok, a0 + 16, b0 + 4 * n, idesc);
                        mma_f16_ts<true>(td + kTok, a0 + 24, b0 + 6 * n, idesc);
                        tc_commit(&bar_acc[slot]);
                        if (ch & 1) tc_commit(&bar_doneT[s]);
                        tc_commit(&bar_doneW[buf]);
                    }
                    __syncwarp();
                    if (++slot == kSlots) { slot = 0; ++round; }
                    if ((ch & 1) && ++s == kStagesT) { s = 0; s_phase ^= 1; }
                }
            }
        }
    } else {
        // ===== epilogue: lane = weight row 32 (warp % 4) + lane; 16-token column groups warp / 4, warp / 4 + 2, ... =====
        constexpr int kG = kTok / 32;
        const int quad = warp & 3, ch0 = warp >> 2;
        const int r = quad * 32 + lane;
        const uint32_t tlane = tmem_base + ((uint32_t)(quad * 32) << 16);
        const uint64_t minus1 = pack2f(-1.0f, -1.0f), one = pack2f(1.0f, 1.0f);
        int it = 0, slot = 0, round = 0;
        bool alive = true;
        for (int tile = blockIdx.x; tile < a.ntiles && alive; tile += gridDim.x) {
            TileCtx cx;
            tile_ctx(tile, tl.ntt, tl, gi, cx);
            uint64_t acc[kG][8];                                              // running sums (or those of this chunk)
            uint64_t sum[kG][8], low[kG][8];          // compensated sum of the chunks
#pragma unroll
            for (int g = 0; g < kG; ++g)
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    acc[g][i] = 0ull;
                    sum[g][i] = low[g][i] = 0ull;
                }
            for (int c = 0; c < nch && alive; ++c, ++it) {
                const float *da = reinterpret_cast<const float *>(aux0 + (it & 3) * S::kAux);
                const uint8_t *rw = ringW + (it & 3) * S::kRingW + r * wscale_bytes<kMins>();
#pragma unroll 1
                for (int ch = 0; ch < 4; ++ch) {
                    if (!wait_warp(&bar_vis[ch], it & 1, abort_flag) || !wait_warp(&bar_acc[slot], round & 1, abort_flag)) { alive = false; break; }
                    tc_fence_after();
#pragma unroll
                    for (int bb = 0; bb < 2; ++bb) {
                        const int b = 2 * ch + bb;
                        const uint8_t *wp = rw + b * kRows * wscale_bytes<kMins>();
                        float wd, m0 = 0.0f, m1 = 0.0f;
                        if constexpr (kMins == 0) wd = *reinterpret_cast<const float *>(wp);
                        else if constexpr (kMins == 1) { const float2 v = *reinterpret_cast<const float2 *>(wp); wd = v.x; m0 = v.y; }
                        else { const float4 v = *reinterpret_cast<const float4 *>(wp); wd = v.x; m0 = v.y; m1 = v.z; }
                        const uint64_t dw = pack2f(wd, wd), mm0 = pack2f(m0, m0), mm1 = pack2f(m1, m1);
#pragma unroll
                        for (int g = 0; g < kG; ++g) {
                            const int col = (2 * g + ch0) * 16;
                            if (col < cx.n) {           // warp-uniform
                                uint32_t p[16];
                                tmem_ld16(tlane + (uint32_t)((2 * slot + bb) * kTok + col), p);
                                tmem_ld_wait();
                                const float *dp = da + b * cx.n + col;
#pragma unroll
                                for (int i = 0; i < 8; i += 2) {
                                    const float4 d4 = *reinterpret_cast<const float4 *>(dp + 2 * i);
                                    float4 s4, t4;
                                    if constexpr (kMins >= 1) s4 = *reinterpret_cast<const float4 *>(dp + 8 * cx.n + 2 * i);
                                    if constexpr (kMins >= 2) t4 = *reinterpret_cast<const float4 *>(dp + 16 * cx.n + 2 * i);
#pragma unroll
                                    for (int e = 0; e < 2; ++e) {
                                        const uint64_t dd = e ? pack2f(d4.z, d4.w) : pack2f(d4.x, d4.y);
                                        const uint64_t pv = pack2(p[2 * (i + e)], p[2 * (i + e) + 1]);
                                        uint64_t v;
                                        if constexpr (F::kTerm) {       // the block's two large parts meet before they are added to others
                                            v = mul2(mm0, e ? pack2f(s4.z, s4.w) : pack2f(s4.x, s4.y));
                                            if constexpr (kMins >= 2) v = fma2(mm1, e ? pack2f(t4.z, t4.w) : pack2f(t4.x, t4.y), v);
                                            v = fma2(one, fma2(mul2(dw, dd), pv, v), acc[g][i + e]);      // d_w d_a: two f16, exact
                                        } else {
                                            v = fma2(dd, mul2(dw, pv), acc[g][i + e]);
                                            if constexpr (kMins >= 1) v = fma2(mm0, e ? pack2f(s4.z, s4.w) : pack2f(s4.x, s4.y), v);
                                        }
                                        acc[g][i + e] = v;
                                    }
                                }
                            }
                        }
                    }
                    tc_fence_before();
                    arrive_warp(&bar_free[slot], lane);
                    if (++slot == kSlots) { slot = 0; ++round; }
                }
                {      // sum += acc with the rounding error kept in `low` (two-sum)
#pragma unroll
                    for (int g = 0; g < kG; ++g)
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const uint64_t x = acc[g][i], s0 = sum[g][i], s1 = fma2(one, x, s0), bb = fma2(minus1, s0, s1);
                            const uint64_t e0 = fma2(minus1, fma2(minus1, bb, s1), s0), e1 = fma2(minus1, bb, x);
                            low[g][i] = fma2(one, fma2(one, e0, e1), low[g][i]);
                            sum[g][i] = s1;
                            acc[g][i] = 0ull;
                        }
                }
            }
            if (!alive) break;
            if (cx.row0 + r < a.nrows) {
#pragma unroll
                for (int g = 0; g < kG; ++g) {
                    const int col = (2 * g + ch0) * 16, left = cx.valid - col;
                    if (left <= 0) continue;
                    {
#pragma unroll
                        for (int i = 0; i < 8; ++i) {       // an infinite (or NaN) sum has no error term
                            const float s0 = lo2(sum[g][i]), s1 = hi2(sum[g][i]);
                            acc[g][i] = pack2f(fabsf(s0) <= 3.0e38f ? __fadd_rn(s0, lo2(low[g][i])) : s0,
                                               fabsf(s1) <= 3.0e38f ? __fadd_rn(s1, hi2(low[g][i])) : s1);
                        }
                    }
                    store16(acc[g], a.out + ((int64_t)cx.t * tl.tt + col) * a.stride_out + cx.row0 + r, a.stride_out, left);
                }
            }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (tid == 0 && *abort_flag) atomicExch(&g_prompt_b32_bf16_timeout_flag, 1);
    if (warp == 0) tmem_dealloc(tmem_base, 512);
}

template <int WTYPE>
bool launch(const void *w, const void *x, void *dst, void *scratch, int k, int n, int tokens, int stride_dst, cudaStream_t st) {
    using F = Fmt<WTYPE>;
    using R = Raw<chunk_bytes<WTYPE>()>;
    static_assert(Smem<WTYPE>::kBytes <= 232448, "shared memory of one CTA");
    static bool attr_done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attr_done[dev]) {
        cudaFuncSetAttribute(prompt32_bf16_kernel<WTYPE>, cudaFuncAttributeMaxDynamicSharedMemorySize, Smem<WTYPE>::kBytes);
        attr_done[dev] = true;
    }
    const int nch = k / 256, nrt = (n + kRows - 1) / kRows;
    const Tiling tl = plan_tiling(tokens, nrt, sm_count(), kFixedTokens, F::kTok);
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
    cq_launch_k(quantize_kernel<F::kMins, F::kSum>, dim3((unsigned)blocks), dim3(256), 0, st, (const __nv_bfloat16 *)x, (uint8_t *)scratch, k, tl);
    const Args a{(const uint8_t *)w, (const uint8_t *)scratch, (__nv_bfloat16 *)dst, n, nch, stride_dst, use_map ? 1 : 0, nrt * tl.ntt};
    const int grid = a.ntiles < sm_count() ? a.ntiles : sm_count();
    cq_launch_k(prompt32_bf16_kernel<WTYPE>, dim3(grid), dim3(kThreads), Smem<WTYPE>::kBytes, st, map, a, tl);
    return true;
}

int mins_of(int wtype) {
    return (wtype == CQ_Q4_1 || wtype == CQ_Q5_0 || wtype == CQ_Q5_1 || wtype == CQ_Q5_K) ? 1 : wtype == CQ_Q2_K ? 2 : 0;
}

}  // namespace

extern "C" size_t cq_prompt32_bf16_scratch_bytes(int wtype, int tokens, int k) {
    if (tokens <= 0 || k <= 0 || k % 256 != 0) return 0;
    return (size_t)((tokens + 15) / 16 * 16) * (k / 256) * (size_t)(512 + 32 + 32 * mins_of(wtype)) + 256;
}

// Against slices of eight rows on the decode kernel, which stream the matrix once each (see cq_prompt32_pays): a model of both, fitted to 1500 shapes, of which 21
// go to the slower side by more than 5 %, by 20 % at most where that is this kernel.
extern "C" int cq_prompt32_bf16_pays(int wtype, int tokens, int k, int n) {
    const double sms = cq_sm_count(), weights = 1e-6 * n * (double)k;
    const Tiling tl = plan_tiling(tokens, (n + kRows - 1) / kRows, (int)sms, kFixedTokens, 64);
    const double rounds = std::ceil((double)((n + kRows - 1) / kRows) * tl.ntt / sms);
    const bool super = cq_block_elems(wtype) == 256;
    const double fixed = wtype == CQ_Q2_K ? 2.52 : wtype == CQ_Q3_K ? 2.09 : 2.27, per_token = wtype == CQ_Q2_K ? 0.046 : 0.036;
    const double here = 6.7 + rounds * (k / 256) * (fixed + per_token * tl.tt);
    auto slice = [&](int rows) {
        return super ? 5.25 + 0.125e-3 * k + weights * (0.05 + 0.084 * rows) : std::max(5.05, 4.7 + 0.018e-3 * k + weights * (0.21 + 0.02 * rows));
    };
    const int whole = tokens / 8, left = tokens % 8;
    return here < (super ? 1.8 : 2.5) + whole * slice(8) + (left ? slice(left) : 0.0);
}

extern "C" void cq_prompt32_bf16_matmul(int wtype, const void *vx, const void *x, void *dst, void *scratch, int ncols_x, int nrows_x,
                                   int tokens, int stride_dst, void *stream) {
    if (!vx || !x || !scratch || !dst || ncols_x <= 0 || nrows_x <= 0 || tokens <= 0 || ncols_x % 256 != 0) {
        cq_set_status(CQ_ERR_BAD_ARG, "prompt32 matmul: null pointer, empty shape or K not a multiple of 256");
        return;
    }
    if ((uintptr_t)scratch % 16 != 0 || (uintptr_t)vx % 2 != 0) {
        cq_set_status(CQ_ERR_BAD_ARG, "prompt32 matmul: misaligned scratch or weights");
        return;
    }
    cudaStream_t st = (cudaStream_t)stream;
    bool ok = false;
    switch (wtype) {
    case CQ_Q4_1: ok = launch<CQ_Q4_1>(vx, x, dst, scratch, ncols_x, nrows_x, tokens, stride_dst, st); break;
    case CQ_Q5_0: ok = launch<CQ_Q5_0>(vx, x, dst, scratch, ncols_x, nrows_x, tokens, stride_dst, st); break;
    case CQ_Q5_1: ok = launch<CQ_Q5_1>(vx, x, dst, scratch, ncols_x, nrows_x, tokens, stride_dst, st); break;
    case CQ_Q2_K: ok = launch<CQ_Q2_K>(vx, x, dst, scratch, ncols_x, nrows_x, tokens, stride_dst, st); break;
    case CQ_Q3_K: ok = launch<CQ_Q3_K>(vx, x, dst, scratch, ncols_x, nrows_x, tokens, stride_dst, st); break;
    case CQ_Q5_K: ok = launch<CQ_Q5_K>(vx, x, dst, scratch, ncols_x, nrows_x, tokens, stride_dst, st); break;
    default: cq_set_status(CQ_ERR_UNSUPPORTED, "prompt32 matmul in bf16: Q4_1, Q5_0, Q5_1, Q2_K, Q3_K, Q5_K"); return;
    }
    if (ok) cq_check_launch("prompt32 matmul");
}

extern "C" int cq_prompt32_bf16_timeout_flag(void) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_prompt_b32_bf16_timeout_flag, sizeof v) != cudaSuccess) { (void)cudaGetLastError(); return -1; }
    if (v) cq_set_status(CQ_ERR_TIMEOUT, "prompt32 matmul: a bounded wait gave up");
    return v;
}
