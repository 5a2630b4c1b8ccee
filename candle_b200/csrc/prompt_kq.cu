// Prompt-phase quantized GEMM, out[t, r] = sum_k x[t, k] * W[r, k] for many tokens, Q4_K and Q6_K weights, dense and grouped
// by expert, on tcgen05.mma kind::f16 (see prompt_f16.cuh for the operand scheme).
//
// Replaces candle's MMQ path for these formats (host: candle-core/src/quantized/fast_mmq.rs:253-400; kernels:
// candle-kernels/src/mmq_gguf/mmq_gguf.cuh:3442-3777, mmq_quantize.cu:11-107) and its expert GEMM
// (candle-kernels/src/moe/moe_wmma_gguf.cu:124-300).
//
// Arithmetic: candle's CPU path.  Activations are BlockQ8K (one f32 scale per 256 values, k_quants.rs:2320-2358, bit-identical
// int8); a super-block contributes  d_a * (d_w * P - dmin_w * L)  (k_quants.rs:1460-1540, 2035-2092) with the integers
//      Q4_K:  P = sum (sc_g q) . q8,   |sc_g q| <= 945: one f16 plane;   L = sum_j m_j bsum_j,  |bsum_j| <= 2048, one K = 16 step
//      Q6_K:  P = sum (sc_j (q - 32)) . q8:  a product of up to 4096 = A + B, A the next multiple of 8, |B| <= 4:  two f16 planes
// The accumulators are f32, so every partial sum has to stay within 2^24 to be exact, whatever the data (|q8| <= 127; 128 where an
// activation is infinite or NaN).  P itself reaches 3.1e7 (Q4_K) and 1.3e8 (Q6_K).
//      Q6_K:  an accumulator per plane: multiples of 8 up to 256 * 4096 * 128 = 8 * 2^24, and 256 * 4 * 128; P = Pa + Pb.
//      Q4_K:  945 * sum |q8| bounds the terms.  The quantizer stores sum |q8| per token and super-block; where all tokens of the tile have
//             945 * sum |q8| <= 2^24 (a mean |q8| of 69; normal inputs have 36, uniform ones 64) one accumulator holds P, else the
//             super-block is split into one accumulator per 128 elements, 128 * 945 * 128 = 15.5e6; P = P0 + P1.
// The epilogue joins two accumulators with one f32 operation: P rounded once, as converting an integer sum would.
// L <= 256 * 63 * 128 is exact.
//
// Mapping.  One CTA per SM walks tiles of 128 weight rows x up to 128 tokens.  Warps 0-7 epilogue, 8-15 producers (two sets of
// four, a weight row per thread), 16 MMA issuer, 17 loader, 18-19 raw bytes where there is no tensor map.  K advances in stages of 64 TMEM
// columns of operand A = eight MMAs: 128 elements of Q4_K, 64 of Q6_K (two planes); the sets take turns.  One barrier says that a
// stage's operands are there (its producer set and the copied activations), one commit that its MMAs are complete.  Tensor memory, all
// 512 columns: two accumulators of 128 for P.  Q4_K alternates between them, so that the epilogue of one super-block runs beside the MMAs
// of the next, and takes both for a split one; L in 128 (its single step comes last in a super-block, by which time the epilogue has read
// the previous one); operand A in two stages.  Q6_K takes both for every super-block; operand A in four stages, so that the producers go
// on while the epilogue reads.
//
// Measured (B200, quantizer included, passes back to back; GPUs differ by up to 5 %): Q4_K 4096 -> 14336, 2048 tokens bf16 287 - 293 us (int8 kernel 478),
// Q6_K 14336 -> 4096, 512 tokens f32 139 - 141 (170).  Bound by the hand-offs between the roles: a super-block of 128 tokens takes 1.4 us (Q4_K) and 2.5 us (Q6_K)
// where its MMAs take 0.55 and 1.05.  What follows are shares of the time at that step, both sides on one GPU:
//   * One accumulator for all of P, which rounds past 2^24: 2 % less.  Both halves of all accumulators in two 64-token passes: 9 % (Q4_K) and 6 % (Q6_K) more,
//     twice the MMAs to issue.  Every super-block split: 48 % more (Q4_K).
//   * The epilogue reads the accumulators in the 16x256b shape (four rows x two columns of each eight per thread), 32 columns at a time: an 8-byte shared load
//     of token scales serves eight values, where a row per thread took a 16-byte load, 4.8 clocks of the SM's shared-memory pipe, for four.  A grouped launch
//     fetches a tile's pair numbers and routing weights, a dependent chain of two L2 round trips, while its super-blocks run.  One instantiation per kind of
//     output, since the code between the loops costs instruction fetches.  Expert block of 1024 tokens (below) 26 % less, dense Q4_K 1 - 2 %.
//   * Instructions count wherever a hand-off waits for them: nibbles into mantissas by one LOP3 each (two constants written in C became two), waits without
//     divergence, arrivals by predicate: Q4_K 6 - 7 % less, Q6_K 5 %.
//   * Tried on top: scales and minima written by the idle raw warps (Q4_K the same, Q6_K 3 % more), half a stage expanded at a time in a loop (5 % and 10 %
//     more), row scales stored in pairs (5 % more: 16-byte broadcast reads).
//   * Left out to see its share (Q4_K, 2048 tokens): all of the expansion 7 %, the MMAs 5 %, the copies 1 %.  What is left are the chains of barrier round trips,
//     none of which bounds it alone.
//
// Every wait is bounded (about a second); a give-up raises a CTA-wide abort flag, all roles leave, copies in flight are waited
// for, TMEM is released and a device flag is set for the host.
#include "../../include/candle_q_b200.h"
#include "prompt_f16.cuh"

#include <algorithm>
#include <type_traits>

namespace {
using namespace cq_prompt;

constexpr int kEpiWarps = 8, kProdWarps = 8;     // producers: two sets of four
constexpr int kMmaWarp = kEpiWarps + kProdWarps, kLoadWarp = kMmaWarp + 1, kRawWarp = kMmaWarp + 2;
constexpr int kThreads = (kEpiWarps + kProdWarps + 4) * 32;      // the last two: raw bytes without a tensor map
constexpr int kSlabs = 34;                       // 32 slabs of 8 f16 activations, 2 of f16 run sums (16 bytes per token each)
constexpr int kTokBytes = kSlabs * 16 + 8;       // + the f32 scale and sum |q8|
constexpr int kRingT = 2 * 32 * kTokMax * 16;    // token stages: two super-blocks, 128 KiB
constexpr int kAuxRing = 4;
constexpr int kAux = 2 * kTokMax * 16 + 2 * kTokMax * 4;  // run sums, scales, sums of |q8| of one super-block
constexpr int kColL = 256;
constexpr float kOneAccumulator = (float)((1 << 24) / (63 * 15));      // sum |q8| up to which Q4_K needs one accumulator

__device__ int g_prompt_kq_timeout_flag = 0;

// kSps: stages per super-block; kNA: stages of operand A; kNT: token stages
template <int WTYPE> struct Fmt;
template <> struct Fmt<CQ_Q4_K> { static constexpr int kSps = 2, kNA = 2, kNT = 4, kRawStages = 3, kColA = 384; static constexpr bool kMins = true; };
template <> struct Fmt<CQ_Q6_K> { static constexpr int kSps = 4, kNA = 4, kNT = 8, kRawStages = 2, kColA = 256; static constexpr bool kMins = false; };

template <int WTYPE> constexpr int smem_bytes() {
    return 1024 + kRingT + kAuxRing * kAux + 4 * kRows * 8 + 2 * kRows * 32 + Fmt<WTYPE>::kRawStages * Raw<cq_type_size(WTYPE)>::kBytes + 16;
}

// ---- activations -> f16 operand tiles -------------------------------------------------------------------------
template <typename T> struct LoadRows {            // rows of k elements
    const T *x;
    int64_t k;
    __device__ __forceinline__ void operator()(int64_t row, int col, float (&e)[8]) const { load8(x + row * k + col, ((uintptr_t)x & 15) == 0, e); }
};

__device__ __forceinline__ float round16(float v, int kind) {
    return kind == CQ_F16 ? __half2float(__float2half_rn(v)) : __bfloat162float(__float2bfloat16_rn(v));
}
// f32 rows rounded to the 16-bit type `kind`
struct LoadRounded {
    const float *x;
    int64_t k;
    int kind;
    __device__ __forceinline__ void operator()(int64_t row, int col, float (&e)[8]) const {
        load8(x + row * k + col, ((uintptr_t)x & 15) == 0, e);
#pragma unroll
        for (int i = 0; i < 8; ++i) e[i] = round16(e[i], kind);
    }
};
// up * silu(gate) of two f32 matrices, rounded to the 16-bit type `kind`: the input of an expert block's down projection
struct LoadGateUp {
    const float *gate, *up;
    int64_t k;
    int kind;
    __device__ __forceinline__ void operator()(int64_t row, int col, float (&e)[8]) const {
        float g[8];
        load8(gate + row * k + col, true, g);
        load8(up + row * k + col, true, e);
#pragma unroll
        for (int i = 0; i < 8; ++i) e[i] = round16(__fmul_rn(e[i], __fdiv_rn(g[i], __fadd_rn(1.0f, expf(-g[i])))), kind);
    }
};

// One warp per (token, super-block): BlockQ8K values (the rules of quantize_act.cu).  A block of 8 warps takes 8 consecutive
// tokens of one super-block and goes through shared memory, so that every slab receives 128 contiguous bytes (stored straight
// from the warps it would be 16-byte pieces, half a sector each).
template <typename L>
__global__ void __launch_bounds__(256) quantize_kernel(const L load, uint8_t *__restrict__ y, int nsb, int q6k, Tiling tl, GroupInfo gi) {
    constexpr int kPitch = 8 * 16 + 16;
    __shared__ __align__(16) uint8_t sm[kSlabs * kPitch];
    __shared__ float sd[16];
    cq_pdl_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int sb = blockIdx.x % nsb, g = blockIdx.x / nsb, per_tile = tl.tt / 8;
    const int t = g / per_tile, row0 = (g % per_tile) * 8, row = row0 + warp;
    int64_t src = -1, blob_row = (int64_t)t * tl.tt;      // input row; none: a padding row of zeros
    int rows;
    if (gi.tiles) {
        if (t >= gi.tiles[4 * tl.ntt]) return;
        const int4 ti = *reinterpret_cast<const int4 *>(gi.tiles + 4 * t);
        rows = (ti.z + 15) / 16 * 16;
        blob_row = ti.w;
        if (row < ti.z) {
            const int pair = gi.sorted_token_ids[ti.y + row];
            src = gi.row_per_pair ? pair : pair / gi.topk;
        }
    } else {
        rows = tl.rows(t);
        const int64_t tok = (int64_t)t * tl.tt + row;
        if (row < rows && tok < tl.tokens) src = tok;
    }
    if (row0 >= rows) return;           // block-uniform
    float e[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) e[c] = 0.0f;
    if (src >= 0) load(src, sb * 256 + lane * 8, e);
    // The largest magnitude by one warp reduction over its bits (fmaxf leaves NaN out, as the comparisons of quantize_act.cu do),
    // then the first element that has it: the first lane, the first of its eight.  The values stay in f32, where they and their
    // sums are exact integers: conversions to int and back took a third of this kernel.
    float m = 0.0f;
#pragma unroll
    for (int c = 0; c < 8; ++c) m = fmaxf(m, fabsf(e[c]));
    const unsigned top = __reduce_max_sync(0xffffffffu, __float_as_uint(m));
    float v = 0.0f;
#pragma unroll
    for (int c = 7; c >= 0; --c) v = __float_as_uint(fabsf(e[c])) == top ? e[c] : v;
    const float vmax = __shfl_sync(0xffffffffu, v, __ffs(__ballot_sync(0xffffffffu, __float_as_uint(m) == top)) - 1);
    float q[8];
    float d = 0.0f;
    if (top == 0u) {
#pragma unroll
        for (int c = 0; c < 8; ++c) q[c] = 0.0f;
    } else {
        const float iscale = __fdiv_rn(-127.0f, vmax);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const float r = roundf(__fmul_rn(iscale, e[c]));
            q[c] = __fadd_rn(fminf(fmaxf(r, -128.0f), 127.0f), 0.0f);      // + 0: no negative zero
        }
        d = __fdiv_rn(1.0f, iscale);
    }
    // Slab of this lane's 8 elements.  A Q6_K stage holds the two 32-element groups that share their ql bytes: with lane =
    // 16 h + 4 (p + 2 nib) + j the order is h, p, nib, j.
    const int slab = q6k ? (lane & 0x13) | ((lane & 4) << 1) | ((lane & 8) >> 1) : lane;
    *reinterpret_cast<uint4 *>(sm + slab * kPitch + warp * 16) = pack_q8(q);
    float bs = ((q[0] + q[1]) + (q[2] + q[3])) + ((q[4] + q[5]) + (q[6] + q[7]));
    bs += __shfl_xor_sync(0xffffffffu, bs, 1);
    if ((lane & 1) == 0) {              // sum of run j = lane / 2: slab 32 + j / 8, f16 j % 8
        const int j = lane >> 1;
        *reinterpret_cast<__half *>(sm + (32 + (j >> 3)) * kPitch + warp * 16 + 2 * (j & 7)) = __float2half_rn(bs);
    }
    float mag = 0.0f;                   // at most 1024, a whole number
#pragma unroll
    for (int c = 0; c < 8; ++c) mag += fabsf(q[c]);
    const int sum_mag = __reduce_add_sync(0xffffffffu, (int)mag);
    if (lane == 0) { sd[warp] = d; sd[8 + warp] = (float)sum_mag; }
    __syncthreads();
    uint8_t *blob = y + ((size_t)blob_row * nsb + (size_t)sb * rows) * kTokBytes;
    for (int i = threadIdx.x; i < kSlabs * 8; i += 256)
        *reinterpret_cast<uint4 *>(blob + ((size_t)(i >> 3) * rows + row0 + (i & 7)) * 16) = *reinterpret_cast<const uint4 *>(sm + (i >> 3) * kPitch + (i & 7) * 16);
    if (threadIdx.x < 16)
        *reinterpret_cast<float *>(blob + (size_t)rows * (kSlabs * 16 + (threadIdx.x >> 3) * 4) + (row0 + (threadIdx.x & 7)) * 4) = sd[threadIdx.x];
}

// Grouped launches whose input rows occur topk times: rows quantized once, 16 to a tile (quantize_kernel on a dense tiling), are copied to every pair's place,
// eight pairs and all their super-blocks per block: a block per super-block held three copies per thread behind two dependent loads (28 us at
// 8192 pairs of 2048 values, against the 45 that quantizing each pair took).
__global__ void __launch_bounds__(256) copy_rows_kernel(const uint8_t *__restrict__ src, uint8_t *__restrict__ y, int nsb, Tiling tl, GroupInfo gi) {
    cq_pdl_wait();
    const int per_tile = tl.tt / 8, t = blockIdx.x / per_tile, row0 = (blockIdx.x % per_tile) * 8;
    if (t >= gi.tiles[4 * tl.ntt]) return;
    const int4 ti = *reinterpret_cast<const int4 *>(gi.tiles + 4 * t);
    const int rows = (ti.z + 15) / 16 * 16, rr = threadIdx.x & 7;
    if (row0 >= rows) return;           // block-uniform
    const int tok = row0 + rr < ti.z ? gi.sorted_token_ids[ti.y + row0 + rr] / gi.topk : -1;
    const uint8_t *from = src + (size_t)(max(tok, 0) >> 4) * 16 * nsb * kTokBytes;
    uint8_t *blob = y + (size_t)ti.w * nsb * kTokBytes;
#pragma unroll 4
    for (int i = threadIdx.x >> 3; i < nsb * kSlabs; i += 32) {
        const int sb = i / kSlabs, slab = i - sb * kSlabs;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (tok >= 0) v = *reinterpret_cast<const uint4 *>(from + (size_t)sb * 16 * kTokBytes + (slab * 16 + (tok & 15)) * 16);
        *reinterpret_cast<uint4 *>(blob + (size_t)sb * rows * kTokBytes + ((size_t)slab * rows + row0 + rr) * 16) = v;
    }
    for (int i = threadIdx.x >> 3; i < nsb * 2; i += 32) {          // scales, sums of |q8|
        const int sb = i >> 1, w = i & 1;
        float v = 0.0f;
        if (tok >= 0) v = *reinterpret_cast<const float *>(from + (size_t)sb * 16 * kTokBytes + 16 * (kSlabs * 16 + w * 4) + (tok & 15) * 4);
        *reinterpret_cast<float *>(blob + (size_t)sb * rows * kTokBytes + (size_t)rows * (kSlabs * 16 + w * 4) + (row0 + rr) * 4) = v;
    }
}

// One CTA: the tile table of a grouped launch.  expert_ids ascending (ids outside [0, num_experts) may sit at either end);
// the jobs of one expert are cut into tiles of kTokMax.
__global__ void __launch_bounds__(1024) group_tiles_kernel(const int32_t *__restrict__ expert_ids, int m, int num_experts, int max_tiles,
                                                           int *__restrict__ tiles) {
    __shared__ int start[1025], first_tile[1025], first_row[1024];
    const int tid = threadIdx.x;
    for (int e = tid; e <= num_experts; e += 1024) {       // start[e] = first job whose expert is >= e
        int lo = 0, hi = m;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (expert_ids[mid] < e) lo = mid + 1; else hi = mid;
        }
        start[e] = lo;
    }
    __syncthreads();
    if (tid < 32) {         // tiles and blob rows (a multiple of 16 per expert) before each expert: a warp scan, 32 experts at a time
        int tiles_before = 0, rows_before = 0;
        for (int e0 = 0; e0 < num_experts; e0 += 32) {
            const int e = e0 + tid;
            const int cnt = e < num_experts ? start[e + 1] - start[e] : 0;
            const int my_tiles = (cnt + kTokMax - 1) / kTokMax, my_rows = (cnt + 15) / 16 * 16;
            int v = my_tiles, r = my_rows;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int uv = __shfl_up_sync(0xffffffffu, v, o), ur = __shfl_up_sync(0xffffffffu, r, o);
                if (tid >= o) { v += uv; r += ur; }
            }
            if (e < num_experts) { first_tile[e] = tiles_before + v - my_tiles; first_row[e] = rows_before + r - my_rows; }
            tiles_before += __shfl_sync(0xffffffffu, v, 31);
            rows_before += __shfl_sync(0xffffffffu, r, 31);
        }
        if (tid == 0) first_tile[num_experts] = tiles_before;
    }
    __syncthreads();
    for (int e = tid; e < num_experts; e += 1024) {
        const int cnt = start[e + 1] - start[e];
        for (int j = 0; j * kTokMax < cnt; ++j)
            *reinterpret_cast<int4 *>(tiles + 4 * (first_tile[e] + j)) =
                make_int4(e, start[e] + j * kTokMax, min(kTokMax, cnt - j * kTokMax), first_row[e] + j * kTokMax);
    }
    if (tid == 0) tiles[4 * max_tiles] = first_tile[num_experts];
}

// ---- producers: the GGUF bytes of one row -> stages of 64 TMEM cells ------------------------------------------------
template <int WTYPE, bool MAP> struct Expand;

// Q4_K, a stage is two chunks; chunk ch: elements 64 ch ..: low nibbles of bytes 32 ch .. +31 (sub-block 2 ch), then the high ones (2 ch + 1).
// A nibble in the low mantissa bits of 1024.0 (or 16 times it, for high nibbles left in place) becomes sc * q in one fma.
template <bool MAP> struct Expand<CQ_Q4_K, MAP> {
    const uint8_t *p;
    uint32_t sc[2], mn[2], dm;
    __device__ __forceinline__ void header(const uint8_t *rr, int shift) {
        p = rr + shift;
        const uint4 h = *reinterpret_cast<const uint4 *>(p);
        dm = h.x;           // get_scale_min_k4, candle-core/src/quantized/utils.rs:50-60, four sub-blocks per word
        sc[0] = h.y & 0x3F3F3F3Fu; mn[0] = h.z & 0x3F3F3F3Fu;
        sc[1] = (h.w & 0x0F0F0F0Fu) | ((h.y >> 2) & 0x30303030u);
        mn[1] = ((h.w >> 4) & 0x0F0F0F0Fu) | ((h.z >> 2) & 0x30303030u);
    }
    static __device__ __forceinline__ __half2 byte_h2(uint32_t w, int i) {      // byte i (< 1024) as f16, twice
        return __hsub2(bits_h2(((w >> (8 * i)) & 0xFFu) * 0x00010001u | 0x64006400u), bits_h2(0x64006400u));
    }
    __device__ __forceinline__ float2 scales() const {
        const __half2 h = bits_h2(dm);
        return make_float2(__low2float(h), __high2float(h));
    }
    __device__ __forceinline__ void mins(uint8_t *slab0) const {       // f16 minimum of every 16-element run, two slabs
#pragma unroll
        for (int s = 0; s < 2; ++s)
            *reinterpret_cast<uint4 *>(slab0 + s * kRows * 16) =
                make_uint4(h2_bits(byte_h2(mn[s], 0)), h2_bits(byte_h2(mn[s], 1)), h2_bits(byte_h2(mn[s], 2)), h2_bits(byte_h2(mn[s], 3)));
    }
    // One copy of the code for both stages (and both producer sets): straight-line code of every stage did not fit the
    // instruction caches and ran at five clocks per instruction.
    __device__ __forceinline__ void stage(int st, uint32_t (&o)[2][32]) const {
        const uint32_t scw = st ? sc[1] : sc[0];
        const uint8_t *q = p + 16 + 64 * st;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const uint4 a = *reinterpret_cast<const uint4 *>(q + 32 * c), b = *reinterpret_cast<const uint4 *>(q + 16 + 32 * c);
            const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
            const __half2 s0 = byte_h2(scw, 2 * c), s1 = byte_h2(scw, 2 * c + 1);
            const __half2 c0 = __hmul2(s0, __float2half2_rn(-1024.0f));
            const __half2 m1 = __hmul2(s1, __float2half2_rn(0.0625f)), c1 = __hmul2(s1, __float2half2_rn(-64.0f));
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint32_t u = w[i], v = w[i] >> 8;
                o[c][2 * i] = hfma2_bits(and_or<0x000F000Fu, 0x64006400u>(u), s0, c0);
                o[c][2 * i + 1] = hfma2_bits(and_or<0x000F000Fu, 0x64006400u>(v), s0, c0);
                o[c][16 + 2 * i] = hfma2_bits(and_or<0x00F000F0u, 0x64006400u>(u), m1, c1);
                o[c][16 + 2 * i + 1] = hfma2_bits(and_or<0x00F000F0u, 0x64006400u>(v), m1, c1);
            }
        }
    }
};

// Q6_K stage 2 h + p: the two 32-element groups pos = p (low nibbles) and p + 2 (high ones) of ql[64 h + 32 p ..], bit pairs pos of
// qh[32 h ..]; 16 cells of A, then 16 of B per group.  The 6-bit code q sits in the mantissa of 1024.0; sc * (q - 32) + 12288, where f16 counts
// in eights, rounds to the next multiple of 8 in one fma, and a second one gives the exact rest.
template <bool MAP> struct Expand<CQ_Q6_K, MAP> {
    const uint8_t *p;
    uint32_t sc[4];
    int off;            // distance of p to the 16-byte boundary below it (MAP: the same for all rows)
    __device__ __forceinline__ void header(const uint8_t *rr, int shift) {
        p = rr + shift;
        off = shift;
        cq_lds_words<4, true>(p + 192, sc);
    }
    // 32 bytes from an even address.  Eight words read one by one are four-way bank conflicts, whatever the pitch of the rows, a multiple of 16; three
    // 16-byte reads are none.  Where all rows have the same distance to a 16-byte boundary the words they leave are picked by a uniform branch.
    __device__ __forceinline__ void words32(const uint8_t *a, uint32_t (&o)[8]) const {
        if constexpr (!MAP) cq_lds_words<8, true>(a, o);
        else {
            const uint4 *v = reinterpret_cast<const uint4 *>(a - off);
            const uint4 x = v[0], y = v[1], z = v[2];
            const uint32_t w[12] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w, z.x, z.y, z.z, z.w};
            const unsigned sh = (off & 2) * 8;
            auto pick = [&](auto first) {
                constexpr int f = decltype(first)::value;
#pragma unroll
                for (int i = 0; i < 8; ++i) o[i] = __funnelshift_r(w[f + i], w[f + i + 1 < 12 ? f + i + 1 : 11], sh);
            };
            if (off < 4) pick(std::integral_constant<int, 0>{});
            else if (off < 8) pick(std::integral_constant<int, 1>{});
            else if (off < 12) pick(std::integral_constant<int, 2>{});
            else pick(std::integral_constant<int, 3>{});
        }
    }
    __device__ __forceinline__ float2 scales() const { return make_float2(__half2float(*reinterpret_cast<const __half *>(p + 208)), 0.0f); }
    __device__ __forceinline__ void mins(uint8_t *) const {}
    __device__ __forceinline__ void stage(int st, uint32_t (&o)[2][32]) const {
        const int h = st >> 1, pp = st & 1;
        uint32_t ql[8], qh[8];
        words32(p + 64 * h + 32 * pp, ql);
        words32(p + 128 + 32 * h, qh);
#pragma unroll
        for (int nib = 0; nib < 2; ++nib) {         // pos = pp + 2 nib, scales 8 h + 2 pos + {0, 1}
            const uint32_t scw = (h ? sc[2 + nib] : sc[nib]) >> (16 * pp);
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                const __half2 s2 = __half2half2(__short2half_rn((short)(int8_t)(scw >> (8 * hf))));
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t l = ql[4 * hf + i], b = qh[4 * hf + i] >> (2 * pp);
                    const uint32_t c = and_or<0x0F0F0F0Fu>(nib ? l >> 4 : l, (nib ? b : b << 4) & 0x30303030u);
#pragma unroll
                    for (int od = 0; od < 2; ++od) {        // bytes 0, 2 | 1, 3
                        const __half2 y = __hsub2(bits_h2(and_or<0x00FF00FFu, 0x64006400u>(od ? c >> 8 : c)), __float2half2_rn(1056.0f));
                        const __half2 a = __hsub2(__hfma2(s2, y, __float2half2_rn(12288.0f)), __float2half2_rn(12288.0f));
                        o[nib][8 * hf + 2 * i + od] = h2_bits(a);
                        o[nib][16 + 8 * hf + 2 * i + od] = h2_bits(__hfma2(s2, y, __hneg2(a)));
                    }
                }
            }
        }
    }
};

struct Args {
    const uint8_t *w, *w2, *act;        // w2: null, or a second matrix of the same shape for the same activations
    void *out, *out2;
    long long total_rows;               // weight rows in memory (all experts)
    int out_kind, nrows, nsb, stride_out, nrt;
};

// STORE: see prompt_f16.cuh; Q: tiles of up to 64 Q tokens, 0: of any size (grouped launches, where each tile has its own); MAP: rows lie a multiple of 16 bytes
// apart and come by tiled copies, so that a chunk starts at the same distance to a 16-byte boundary in all of them
template <int WTYPE, int STORE, int Q, bool MAP>
__global__ void __launch_bounds__(kThreads, 1)
prompt_kernel(const __grid_constant__ CUtensorMap wmap, const __grid_constant__ CUtensorMap wmap2, const Args a, const Tiling tl, const GroupInfo gi) {
    using F = Fmt<WTYPE>;
    using R = Raw<cq_type_size(WTYPE)>;
    constexpr int kCB = cq_type_size(WTYPE), kStageT = kRingT / F::kNT;
    extern __shared__ __align__(1024) uint8_t smem[];
    uint64_t *bar_raw = reinterpret_cast<uint64_t *>(smem);        // [3] raw weight bytes landed
    uint64_t *bar_rawfree = bar_raw + 3;                            // [3] read by both producer sets
    uint64_t *bar_full = bar_raw + 6;                               // [kNT] stage: operand A stored (four warps), activations landed
    uint64_t *bar_done = bar_raw + 14;                              // [kNT] its MMAs are complete
    uint64_t *bar_free = bar_raw + 22;                              // [2] accumulators of an even / odd super-block drained (all epilogue warps)
    uint64_t *bar_vis = bar_raw + 24;                               // [2] relay: the scale rings of this super-block are visible
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + 256);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + 264);
    int *split_of = reinterpret_cast<int *>(smem + 272);           // [2] the super-block takes both accumulators (Q4_K)
    uint8_t *stT0 = smem + 1024;
    uint8_t *aux0 = stT0 + kRingT;
    uint8_t *ringW = aux0 + kAuxRing * kAux;            // (d, dmin) of the rows: [4][128] float2
    uint8_t *mins0 = ringW + 4 * kRows * 8;             // operand A of the sums step: [2][2 slabs][128][16]
    uint8_t *raw0 = mins0 + 2 * kRows * 32;             // 128-byte aligned

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nsb = a.nsb;
    const uint32_t row_bytes = (uint32_t)nsb * kCB;

    if (tid == 0) {
        for (int i = 0; i < 3; ++i) { cq_mbar_init(&bar_raw[i], MAP ? 1 : kRawThreads); cq_mbar_init(&bar_rawfree[i], kProdWarps); }
        for (int i = 0; i < F::kNT; ++i) { cq_mbar_init(&bar_full[i], 4 + 1); cq_mbar_init(&bar_done[i], 1); }
        for (int i = 0; i < 2; ++i) { cq_mbar_init(&bar_free[i], kEpiWarps); cq_mbar_init(&bar_vis[i], 1); }
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
    cq_pdl_wait();              // activations and the tile table come from the preceding launches
    // grouped: the table says how many of its tiles are in use.  With a second matrix its tiles follow those of the first.
    const int ntt = gi.tiles ? gi.tiles[4 * tl.ntt] : tl.ntt;
    const int per_matrix = a.nrt * ntt, ntiles = a.w2 ? 2 * per_matrix : per_matrix;

    if (warp >= kMmaWarp) {
    regs_down<kRegsMisc>();
    if (warp == kLoadWarp) {
        // ===== loader: raw weights and activations of up to three / two super-blocks ahead =====
        int it = 0, h = 0;
        bool alive = true;
        for (int tile = blockIdx.x; tile < ntiles && alive; tile += gridDim.x) {
            TileCtx cx;
            const bool second = tile >= per_matrix;
            tile_ctx(second ? tile - per_matrix : tile, ntt, tl, gi, cx);
            const int n = cx.n;
            const uint8_t *blob0 = a.act + (size_t)cx.blob_row * nsb * kTokBytes;
            for (int sb = 0; sb < nsb && alive; ++sb, ++it) {
                const int rs = it % F::kRawStages;
                if constexpr (MAP) {
                    if (it >= F::kRawStages && !wait_warp(&bar_rawfree[rs], (it / F::kRawStages - 1) & 1, abort_flag)) { alive = false; break; }
                    if (lane == 0) {
                        cq_mbar_expect_tx(&bar_raw[rs], R::kBytes);
                        cq_tmap::load_2d(raw0 + rs * R::kBytes, second ? &wmap2 : &wmap, (int)(((uint32_t)sb * kCB & ~15u) / 2), (int)cx.wrow0, &bar_raw[rs]);
                    }
                }
                const uint8_t *blob = blob0 + (size_t)sb * n * kTokBytes;
                for (int st = 0; st < F::kSps; ++st, ++h) {
                    const int s = h % F::kNT;
                    if (h >= F::kNT && !wait_warp(&bar_done[s], (h / F::kNT - 1) & 1, abort_flag)) { alive = false; break; }
                    if (lane == 0) {
                        const unsigned bytes = (unsigned)n * (512 / F::kSps);
                        if (st == 0) {
                            // done with the first stage of it - 2: its MMAs started after the epilogue of it - 4
                            uint8_t *ax = aux0 + (it & 3) * kAux;
                            const unsigned aux_bytes = (unsigned)n * (F::kMins ? 40 : 4);
                            cq_mbar_expect_tx(&bar_full[s], bytes + aux_bytes);
                            cq_bulk_g2s(ax + (F::kMins ? 0 : n * 32), blob + (size_t)n * (F::kMins ? 512 : 544), aux_bytes, &bar_full[s]);
                        } else {
                            cq_mbar_expect_tx(&bar_full[s], bytes);
                        }
                        cq_bulk_g2s(stT0 + s * kStageT, blob + (size_t)st * bytes, bytes, &bar_full[s]);
                    }
                    __syncwarp();
                }
            }
        }
        // after a give-up the copies of raw bytes must land (or give up themselves) before the shared memory goes away, and those
        // of activations have a second to (their barrier also waits for producers that may have left)
        if (lane == 0 && (!alive || *abort_flag)) {
            for (int j = it >= F::kRawStages ? it - F::kRawStages + 1 : 0; MAP && j <= it; ++j)
                (void)cq_mbar_wait_bounded(&bar_raw[j % F::kRawStages], (j / F::kRawStages) & 1);
            for (int j = h > F::kNT ? h - F::kNT : 0; j < h; ++j) {
                if (cq_mbar_wait_bounded(&bar_full[j % F::kNT], (j / F::kNT) & 1)) continue;
                break;
            }
        }
        __syncwarp();
    } else if (warp >= kRawWarp) {
        // ===== raw bytes of rows that are not a multiple of 16 bytes apart =====
        if constexpr (!MAP) {
            int it = 0;
            bool alive = true;
            for (int tile = blockIdx.x; tile < ntiles && alive; tile += gridDim.x) {
                TileCtx cx;
                const bool second = tile >= per_matrix;
                tile_ctx(second ? tile - per_matrix : tile, ntt, tl, gi, cx);
                const uint8_t *w0 = (second ? a.w2 : a.w) + cx.wrow0 * row_bytes;
                const int rows_left = (int)min(a.total_rows - cx.wrow0, (long long)kRows);
                for (int sb = 0; sb < nsb; ++sb, ++it) {
                    const int rs = it % F::kRawStages;
                    if (it >= F::kRawStages && !wait_warp(&bar_rawfree[rs], (it / F::kRawStages - 1) & 1, abort_flag)) { alive = false; break; }
                    R::load_rows(raw0 + rs * R::kBytes, w0 + (uint32_t)sb * kCB, rows_left, row_bytes, tid - kRawWarp * 32, &bar_raw[rs]);
                }
            }
            cq_cp_async_wait<0>();
        }
    } else if (warp == kMmaWarp) {
        // ===== MMA issuer: the warp runs the loop, one elected lane issues =====
        const uint32_t stT = uniform(cq_smem_u32(stT0) >> 4), mins = uniform(cq_smem_u32(mins0) >> 4), aux = uniform(cq_smem_u32(aux0) >> 4);
        const uint32_t tm = uniform(tmem_base);
        int it = 0;
        bool alive = true;
        // ---- Q4_K: the super-blocks alternate between the accumulators of P, a split one takes both ----
        bool split = false;                         // the last super-block whose first stage has been issued
        auto epilogue_done = [&](int j) { return j < 0 || wait_warp(&bar_free[j & 1], (j >> 1) & 1, abort_flag); };
        auto super_block4 = [&](uint32_t n, uint32_t idesc, uint32_t bT) {
            const int c = it & 1;
            const uint32_t tp = tm + (uint32_t)(c * kTokMax), tp2 = tm + (uint32_t)((c ^ 1) * kTokMax);
            // The epilogue has read P of it - 2: known from the wait for L of it - 1, unless that took this accumulator too.
            if (split && !epilogue_done(it - 1)) return false;
#pragma unroll
            for (int st = 0; st < 2; ++st) {
                const int h = it * 2 + st, s = h % F::kNT;
                if (st == 1) {
                    // Where this super-block's second stage goes.  Looked up behind the first stage's MMAs: in front of them it cost 170 clocks.
                    const float4 m = *reinterpret_cast<const float4 *>(aux0 + (it & 3) * kAux + n * 36 + min(16u * lane, 4u * n - 16u));
                    split = __any_sync(0xffffffffu, fmaxf(fmaxf(m.x, m.y), fmaxf(m.z, m.w)) > kOneAccumulator);
                    if (split && !epilogue_done(it - 1)) return false;
                }
                if (!wait_warp(&bar_full[s], (h / F::kNT) & 1, abort_flag)) return false;
                tc_fence_after();
                const uint32_t b0 = bT + (uint32_t)s * (kStageT >> 4), a0 = tm + (uint32_t)(F::kColA + (h % F::kNA) * 64);
                if (elect_one()) {
                    if (st == 1) {
                        split_of[c] = split;
                        mbar_arrive(&bar_vis[c]);       // relay: what this warp has acquired is visible to the epilogue
                    }
                    if (st == 1 && split) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            if (j == 0) mma_f16_ts<false>(tp2, a0, b0, idesc);
                            else mma_f16_ts<true>(tp2, a0 + 8 * j, b0 + 2 * j * n, idesc);
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            if (st == 0 && j == 0) mma_f16_ts<false>(tp, a0, b0, idesc);
                            else mma_f16_ts<true>(tp, a0 + 8 * j, b0 + 2 * j * n, idesc);
                        }
                    }
                }
                if (st == 1) {
                    // L has one buffer: the epilogue of the previous super-block must have read it
                    if (!epilogue_done(it - 1)) return false;
                    tc_fence_after();
                    if (elect_one())
                        mma_f16_ss(tm + (uint32_t)kColL, (mins + (uint32_t)c * (kRows * 32 >> 4)) | ((uint32_t)kRows << 16),
                                   (aux + (uint32_t)(it & 3) * (kAux >> 4)) | (n << 16), idesc);
                }
                __syncwarp();
                if (elect_one()) tc_commit(&bar_done[s]);
            }
            return true;
        };
        // ---- Q6_K: an accumulator per plane ----
        auto super_block6 = [&](uint32_t n, uint32_t idesc, uint32_t bT) {
            if (!epilogue_done(it - 1)) return false;
#pragma unroll
            for (int st = 0; st < F::kSps; ++st) {
                const int h = it * F::kSps + st, s = h % F::kNT;
                if (!wait_warp(&bar_full[s], (h / F::kNT) & 1, abort_flag)) return false;
                tc_fence_after();
                const uint32_t b0 = bT + (uint32_t)s * (kStageT >> 4), a0 = tm + (uint32_t)(F::kColA + (h % F::kNA) * 64);
                if (elect_one()) {
                    if (st == 0) mbar_arrive(&bar_vis[it & 1]);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {           // a group's two planes (two steps each) meet the same 32 activations
                        const uint32_t dst = tm + (uint32_t)((j >> 1 & 1) * kTokMax), b1 = b0 + (uint32_t)(4 * (j >> 2) + 2 * (j & 1)) * n;
                        if (st == 0 && (j & ~2) == 0) mma_f16_ts<false>(dst, a0 + 8 * j, b1, idesc);
                        else mma_f16_ts<true>(dst, a0 + 8 * j, b1, idesc);
                    }
                    tc_commit(&bar_done[s]);
                }
                __syncwarp();
            }
            return true;
        };
        for (int tile = blockIdx.x; tile < ntiles && alive; tile += gridDim.x) {
            TileCtx cx;
            const bool second = tile >= per_matrix;
            tile_ctx(second ? tile - per_matrix : tile, ntt, tl, gi, cx);
            const uint32_t n = uniform((uint32_t)cx.n), idesc = idesc_f16((int)n), bT = stT | (n << 16);
#pragma unroll 1
            for (int sb = 0; sb < nsb && alive; ++sb, ++it) {
                if constexpr (F::kMins) alive = super_block4(n, idesc, bT);
                else alive = super_block6(n, idesc, bT);
            }
        }
    }
    } else if (warp >= kEpiWarps) {
        regs_down<kRegsProd>();
        // ===== producers: thread = weight row = TMEM lane; set 0 takes the even stages, set 1 the odd ones =====
        const int set = (warp - kEpiWarps) >> 2, r = (warp & 3) * 32 + lane;
        const uint32_t ta = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)F::kColA;
        int it = 0, rs = 0, rs_phase = 0;
        bool alive = true;
        for (int tile = blockIdx.x; tile < ntiles && alive; tile += gridDim.x) {
            TileCtx cx;
            const bool second = tile >= per_matrix;
            tile_ctx(second ? tile - per_matrix : tile, ntt, tl, gi, cx);
            long long wr = cx.wrow0 + r;
            if (wr >= a.total_rows) wr = a.total_rows - 1;
            // without the tensor map every row has its own distance to the 16-byte boundary below it
            const uint32_t row_off = MAP ? 0u : (uint32_t)((uintptr_t)((second ? a.w2 : a.w) + wr * row_bytes) & 15);
            for (int sb = 0; sb < nsb && alive; ++sb, ++it) {
                if (!wait_warp(&bar_raw[rs], rs_phase, abort_flag)) { alive = false; break; }
                Expand<WTYPE, MAP> ex;
                ex.header(raw0 + rs * R::kBytes + r * R::kPitch, R::kAligned ? 0 : (int)((row_off + (uint32_t)sb * kCB) & 15));
                // This set's wait in super-block it - 1 was for a stage of it - 2: its MMAs had started, so the epilogue had finished it - 4
                // (the ring entry written here), and set 1's was for the last one, with the sums step that read this copy of the minima.
                if (set == 0) *reinterpret_cast<float2 *>(ringW + (it & 3) * kRows * 8 + r * 8) = ex.scales();
                else if (F::kMins) {
                    ex.mins(mins0 + (it & 1) * kRows * 32 + r * 16);
                    fence_proxy_async_smem();
                }
#pragma unroll 1
                for (int st = set; st < F::kSps; st += 2) {
                    uint32_t o[2][32];
                    ex.stage(st, o);
                    if (st >= F::kSps - 2) arrive_warp(&bar_rawfree[rs], lane);
                    const int h = it * F::kSps + st, before = h - F::kNA;       // the stage whose columns are taken over
                    if (before >= 0 && !wait_warp(&bar_done[before % F::kNT], (before / F::kNT) & 1, abort_flag)) { alive = false; break; }
                    tc_fence_after();
                    const uint32_t dst = ta + (uint32_t)((h % F::kNA) * 64);
#pragma unroll
                    for (int i = 0; i < 8; ++i) tmem_st8(dst + 8 * i, &o[i >> 2][8 * (i & 3)]);
                    tmem_st_wait();
                    tc_fence_before();
                    arrive_warp(&bar_full[h % F::kNT], lane);
                }
                if (++rs == F::kRawStages) { rs = 0; rs_phase ^= 1; }
            }
        }
    } else {
        regs_up<kRegsEpi>();
        // ===== epilogue: warp = 32 weight rows 32 (warp % 4) .., half of the tile's tokens =====
        // A thread holds rows r0 + 8 i, columns 8 j + csub, + 1 of each 32 of its half: pair 8 (i / 2) + 2 j + i % 2 (prompt_f16.cuh, 16x256b).
        const int half = warp >> 2, r0 = (warp & 3) * 32 + (lane >> 2), csub = 2 * (lane & 3);
        const uint32_t tlane = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
        [[maybe_unused]] const uint64_t one = pack2f(1.0f, 1.0f);
        int it = 0;
        bool alive = true;
        // A tile whose warps have up to 32 kQ columns; those past its tokens are computed and dropped (a branch on the number of tokens inside, over
        // running sums, makes the compiler move them).
        auto run_tile = [&](const TileCtx &cx, bool second, auto quarters) {
            constexpr int kQ = decltype(quarters)::value;
            const int n = cx.n, col0 = half * (n >> 1);
            const uint32_t tcol = tlane + (uint32_t)col0;
            uint64_t acc[kQ][16];
#pragma unroll
            for (int q = 0; q < kQ; ++q)
#pragma unroll
                for (int i = 0; i < 16; ++i) acc[q][i] = 0ull;
            // grouped: the pairs of this warp's columns, a lane per column of each 32; their loads have the whole tile to arrive
            int pair[kQ];
            float pw[kQ];
#pragma unroll
            for (int q = 0; q < kQ; ++q) {
                pair[q] = 0;
                pw[q] = 1.0f;
                if (STORE == kStorePairs && col0 + 32 * q + lane < cx.valid) pair[q] = gi.sorted_token_ids[cx.job0 + col0 + 32 * q + lane];
            }
            for (int sb = 0; sb < nsb; ++sb, ++it) {
                const int c = it & 1;
                // the last stage of the super-block is done; its barrier cannot come round again before this epilogue is through
                const int h = it * F::kSps + F::kSps - 1;
                if (!wait_warp(&bar_vis[c], (it >> 1) & 1, abort_flag) || !wait_warp(&bar_done[h % F::kNT], (h / F::kNT) & 1, abort_flag)) return false;
                tc_fence_after();
                const float2 *rw = reinterpret_cast<const float2 *>(ringW + (it & 3) * kRows * 8) + r0;
                const float *da = reinterpret_cast<const float *>(aux0 + (it & 3) * kAux + n * 32) + col0 + csub;
                const uint32_t tp = tcol + (uint32_t)(F::kMins ? c * kTokMax : 0);
                if (F::kMins && split_of[c]) {      // rare: P0 + P1 into the place of P
#pragma unroll 1
                    for (int col = 0; col < n >> 1; col += 8) {
                        uint32_t p[8], p1[8];
                        tmem_ld8(tp + (uint32_t)col, p);
                        tmem_ld8(tcol + (uint32_t)((c ^ 1) * kTokMax + col), p1);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 8; ++i) p[i] = __float_as_uint(__fadd_rn(__uint_as_float(p[i]), __uint_as_float(p1[i])));
                        tmem_st8(tp + (uint32_t)col, p);
                    }
                    tmem_st_wait();
                }
#pragma unroll
                for (int q = 0; q < kQ; ++q) {
                    uint64_t dd[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) dd[j] = *reinterpret_cast<const uint64_t *>(da + 32 * q + 8 * j);
#pragma unroll
                    for (int hf = 0; hf < 2; ++hf) {
                        uint32_t p[16], l[16];      // l: L, or the sum of the second plane
                        tmem_ld_16x256b<4>(tp + (uint32_t)(32 * q) + ((uint32_t)(16 * hf) << 16), p);
                        tmem_ld_16x256b<4>(tcol + (uint32_t)((F::kMins ? kColL : kTokMax) + 32 * q) + ((uint32_t)(16 * hf) << 16), l);
                        const float2 w0 = rw[16 * hf], w1 = rw[16 * hf + 8];
                        const uint64_t dw[2] = {pack2f(w0.x, w0.x), pack2f(w1.x, w1.x)}, ndm[2] = {pack2f(-w0.y, -w0.y), pack2f(-w1.y, -w1.y)};
                        tmem_ld_wait();
                        if (q == kQ - 1 && hf == 1) {
                            tc_fence_before();
                            arrive_warp(&bar_free[c], lane);       // (the scales are in registers by now)
                        }
#pragma unroll
                        for (int j = 0; j < 4; ++j)
#pragma unroll
                            for (int s = 0; s < 2; ++s) {
                                const int x = 2 * j + s;
                                const uint64_t pv = pack2(p[2 * x], p[2 * x + 1]), lv = pack2(l[2 * x], l[2 * x + 1]);
                                uint64_t tv;
                                if constexpr (F::kMins) tv = fma2(dw[s], pv, mul2(ndm[s], lv));
                                else tv = mul2(dw[s], fma2(one, pv, lv));
                                acc[q][8 * hf + x] = fma2(dd[j], tv, acc[q][8 * hf + x]);
                            }
                    }
                }
                if (STORE == kStorePairs && sb == 0 && gi.topk_weights) {
#pragma unroll
                    for (int q = 0; q < kQ; ++q)
                        if (col0 + 32 * q + lane < cx.valid) pw[q] = gi.topk_weights[pair[q]];
                }
            }
            const int left = min(n >> 1, cx.valid - col0);          // columns of this warp that hold tokens
            void *out = second ? a.out2 : a.out;
            const int64_t base = ((int64_t)cx.t * tl.tt + col0) * a.stride_out + cx.row0;
#pragma unroll
            for (int q = 0; q < kQ; ++q)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint64_t v[4] = {acc[q][2 * j], acc[q][2 * j + 1], acc[q][8 + 2 * j], acc[q][9 + 2 * j]};       // rows r0 + 8 i
                    if constexpr (STORE == kStore16 || STORE == kStore16Any) {
                        const int col = 32 * q + 8 * j, row = (warp & 3) * 32;
                        uint16_t *dst = (uint16_t *)out + base + (int64_t)col * a.stride_out + row;
                        if constexpr (STORE == kStore16) store_rows32_wide(v, a.out_kind, dst, a.stride_out, a.nrows - cx.row0 - row, left - col);
                        else store_rows32_any(v, a.out_kind, dst, a.stride_out, a.nrows - cx.row0 - row, left - col);
                    } else {
                        const int col = 32 * q + 8 * j + csub;
                        float *o0 = (float *)out + base + (int64_t)col * a.stride_out + r0, *o1 = o0 + a.stride_out;
                        float w0 = 1.0f, w1 = 1.0f;
                        if constexpr (STORE == kStorePairs) {       // output row = the pair of this job, scaled by its routing weight
                            const int p0 = __shfl_sync(0xffffffffu, pair[q], col & 31), p1 = __shfl_sync(0xffffffffu, pair[q], (col & 31) + 1);
                            w0 = __shfl_sync(0xffffffffu, pw[q], col & 31);
                            w1 = __shfl_sync(0xffffffffu, pw[q], (col & 31) + 1);
                            o0 = (float *)out + (int64_t)p0 * a.stride_out + cx.row0 + r0;
                            o1 = (float *)out + (int64_t)p1 * a.stride_out + cx.row0 + r0;
                        }
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const bool in = cx.row0 + r0 + 8 * i < a.nrows;
                            if (in && col < left) o0[8 * i] = STORE == kStorePairs ? __fmul_rn(lo2(v[i]), w0) : lo2(v[i]);
                            if (in && col + 1 < left) o1[8 * i] = STORE == kStorePairs ? __fmul_rn(hi2(v[i]), w1) : hi2(v[i]);
                        }
                    }
                }
            return true;
        };
        for (int tile = blockIdx.x; tile < ntiles && alive; tile += gridDim.x) {
            TileCtx cx;
            const bool second = tile >= per_matrix;
            tile_ctx(second ? tile - per_matrix : tile, ntt, tl, gi, cx);
            if constexpr (Q == 0) alive = cx.n > 64 ? run_tile(cx, second, std::integral_constant<int, 2>{}) : run_tile(cx, second, std::integral_constant<int, 1>{});
            else alive = run_tile(cx, second, std::integral_constant<int, Q>{});
        }
    }

    tc_fence_before();
    __syncthreads();
    if (tid == 0 && *abort_flag) atomicExch(&g_prompt_kq_timeout_flag, 1);
    if (warp == 0) tmem_dealloc(tmem_base, 512);
}

// the fixed part of a tile's time per super-block in tokens (plan_tiling); Q6_K is bound by its producers, 2 us at any token count
template <int WTYPE> constexpr int fixed_tokens() { return WTYPE == CQ_Q4_K ? 150 : 400; }

template <int WTYPE, int STORE, int Q, bool MAP> void launch_kernel(int grid, cudaStream_t st, const CUtensorMap &map, const CUtensorMap &map2, const Args &a, const Tiling &tl, const GroupInfo &gi) {
    static_assert(smem_bytes<WTYPE>() <= 232448, "shared memory of one CTA");
    static bool attr_done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attr_done[dev]) {
        cudaFuncSetAttribute(prompt_kernel<WTYPE, STORE, Q, MAP>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes<WTYPE>());
        attr_done[dev] = true;
    }
    cq_launch_k(prompt_kernel<WTYPE, STORE, Q, MAP>, dim3(grid), dim3(kThreads), smem_bytes<WTYPE>(), st, map, map2, a, tl, gi);
}

template <int WTYPE>
bool launch_gemm(const void *w, const void *act, void *out, int out_elem, int k, int n, long long total_rows, int stride_out, const Tiling &tl,
                 const GroupInfo &gi, cudaStream_t st, const void *w2 = nullptr, void *out2 = nullptr) {
    using R = Raw<cq_type_size(WTYPE)>;
    const long long row_bytes = (long long)(k / 256) * cq_type_size(WTYPE);
    CUtensorMap map{}, map2{};
    const uintptr_t both = (uintptr_t)w | (uintptr_t)w2;
    const bool use_map = both % 16 == 0 && row_bytes % 16 == 0 && row_bytes <= INT32_MAX && total_rows <= INT32_MAX &&
                         cq_tmap::weight_map(w, (int)row_bytes, (int)total_rows, R::kPitch / 2, kRows, 2, map) &&
                         (!w2 || cq_tmap::weight_map(w2, (int)row_bytes, (int)total_rows, R::kPitch / 2, kRows, 2, map2));
    if (!use_map && R::kAligned && both % 16 != 0) {
        cq_set_status(CQ_ERR_BAD_ARG, "prompt gemm: Q4_K weights must be 16-byte aligned");
        return false;
    }
    const Args a{(const uint8_t *)w, (const uint8_t *)w2, (const uint8_t *)act, out, out2, total_rows, out_elem, n, k / 256, stride_out, (n + kRows - 1) / kRows};
    const long long ntiles = (long long)a.nrt * tl.ntt * (w2 ? 2 : 1);
    const int grid = ntiles < sm_count() ? (int)ntiles : sm_count();
    auto run = [&](auto map_) {
        constexpr bool M = decltype(map_)::value;
        if (gi.tiles) launch_kernel<WTYPE, kStorePairs, 0, M>(grid, st, map, map2, a, tl, gi);
        else if (out_elem == CQ_F32 && tl.tt <= 64) launch_kernel<WTYPE, kStoreF32, 1, M>(grid, st, map, map2, a, tl, gi);
        else if (out_elem == CQ_F32) launch_kernel<WTYPE, kStoreF32, 2, M>(grid, st, map, map2, a, tl, gi);
        else if (rows_16_bytes_apart(out, stride_out) && n % 8 == 0) {
            if (tl.tt <= 64) launch_kernel<WTYPE, kStore16, 1, M>(grid, st, map, map2, a, tl, gi);
            else launch_kernel<WTYPE, kStore16, 2, M>(grid, st, map, map2, a, tl, gi);
        } else if (tl.tt <= 64) launch_kernel<WTYPE, kStore16Any, 1, M>(grid, st, map, map2, a, tl, gi);
        else launch_kernel<WTYPE, kStore16Any, 2, M>(grid, st, map, map2, a, tl, gi);
    };
    if (use_map) run(std::true_type{});
    else run(std::false_type{});
    return true;
}

template <typename L> bool launch_quantize(int wtype, const L &load, void *scratch, int k, const Tiling &tl, const GroupInfo &gi, cudaStream_t st) {
    const long long blocks = (long long)tl.ntt * (tl.tt / 8) * (k / 256);
    if (blocks > INT32_MAX) { cq_set_status(CQ_ERR_UNSUPPORTED, "prompt quantize: too many tokens for one launch"); return false; }
    cq_launch_k(quantize_kernel<L>, dim3((unsigned)blocks), dim3(256), 0, st, load, (uint8_t *)scratch, k / 256, wtype == CQ_Q6_K ? 1 : 0, tl, gi);
    return true;
}
bool launch_quantize_rows(int wtype, const void *x, int x_elem, void *scratch, int k, const Tiling &tl, const GroupInfo &gi, cudaStream_t st) {
    if (x_elem == CQ_F32) return launch_quantize(wtype, LoadRows<float>{(const float *)x, k}, scratch, k, tl, gi, st);
    if (x_elem == CQ_F16) return launch_quantize(wtype, LoadRows<__half>{(const __half *)x, k}, scratch, k, tl, gi, st);
    if (x_elem == CQ_BF16) return launch_quantize(wtype, LoadRows<__nv_bfloat16>{(const __nv_bfloat16 *)x, k}, scratch, k, tl, gi, st);
    cq_set_status(CQ_ERR_BAD_ARG, "prompt quantize: unknown element type");
    return false;
}

Tiling dense_tiling(int wtype, int tokens, int n) {
    return plan_tiling(tokens, (n + kRows - 1) / kRows, sm_count(), wtype == CQ_Q4_K ? fixed_tokens<CQ_Q4_K>() : fixed_tokens<CQ_Q6_K>());
}
int group_max_tiles(int size_m, int num_experts) { return (size_m + kTokMax - 1) / kTokMax + num_experts; }
size_t table_bytes(int max_tiles) { return ((size_t)(max_tiles + 1) * 16 + 255) / 256 * 256; }
// every expert pads its rows to a multiple of 16
size_t group_blob_bytes(int size_m, int num_experts, int k) { return ((size_t)size_m + 15 * (size_t)num_experts) * kTokBytes * (k / 256); }

}  // namespace

// prefill_tcgen05.cu
size_t cq_prefill_grouped_blob_bytes(int max_tiles, int k);
bool cq_prefill_grouped_q6k(const void *input, int in_elem, const void *weights, const int *tiles, int max_tiles, const int32_t *sorted_token_ids,
                            const float *topk_weights, float *out, uint8_t *blobs, int topk, int n, int k, cudaStream_t st);

extern "C" size_t cq_prompt_scratch_bytes(int tokens, int k) {
    if (tokens <= 0 || k <= 0 || k % 256 != 0) return 0;
    // whatever the tile size, only the last tile is padded, to a multiple of 16 rows
    return (size_t)((tokens + 15) / 16 * 16) * (k / 256) * kTokBytes + 256;
}

// Q6_K against the int8 kernel behind cq_prefill_gemm (the same bits): a round of tiles of 128 rows takes 2.3 us per super-block here (2.45 where
// rows are not a multiple of 16 bytes apart and have no tiled copy), 1.6 us for its tiles of 64 rows x 128 tokens.  So a launch that leaves SMs
// idle either way is faster with the smaller tiles (8192 -> 2368, 86 tokens: 73 against 63 us; 10240 -> 3587, 393 tokens: 99 against
// 133; K = 9728, 9856 rows, 51 tokens: 97 against 118).  Of 90 shapes measured the rule takes the slower one five times, by 10 % at most.
extern "C" int cq_prompt_pays(int wtype, int tokens, int k, int n) {
    if (wtype != CQ_Q6_K) return 1;
    const long long sms = cq_sm_count(), tt = (tokens + kTokMax - 1) / kTokMax;
    const long long rounds64 = ((n + 63) / 64 * tt + sms - 1) / sms, rounds128 = ((n + kRows - 1) / kRows * tt + sms - 1) / sms;
    return rounds64 * 1.6 >= rounds128 * (k % 2048 == 0 ? 2.3 : 2.45);
}

extern "C" int cq_prompt_tile_tokens(int wtype, int tokens, int n) { return tokens <= 0 || n <= 0 ? 0 : dense_tiling(wtype, tokens, n).tt; }

extern "C" void cq_prompt_matmul(int wtype, const void *vx, const void *x, int elem, void *dst, void *scratch, int ncols_x, int nrows_x,
                                 int tokens, int stride_dst, void *stream) {
    if (!vx || !x || !scratch || !dst || ncols_x <= 0 || nrows_x <= 0 || tokens <= 0 || ncols_x % 256 != 0) {
        cq_set_status(CQ_ERR_BAD_ARG, "prompt matmul: null pointer, empty shape or K not a multiple of 256");
        return;
    }
    if (wtype != CQ_Q4_K && wtype != CQ_Q6_K) {
        cq_set_status(CQ_ERR_UNSUPPORTED, "prompt matmul: covers Q4_K and Q6_K");
        return;
    }
    if ((uintptr_t)vx % (wtype == CQ_Q4_K ? 16 : 4) != 0 || (uintptr_t)scratch % 16 != 0) {
        cq_set_status(CQ_ERR_BAD_ARG, "prompt matmul: misaligned weights (16 bytes for Q4_K, 4 for Q6_K) or scratch (16)");
        return;
    }
    cudaStream_t st = (cudaStream_t)stream;
    const Tiling tl = dense_tiling(wtype, tokens, nrows_x);
    if (!launch_quantize_rows(wtype, x, elem, scratch, ncols_x, tl, GroupInfo{}, st)) return;
    const bool ok = wtype == CQ_Q4_K
                        ? launch_gemm<CQ_Q4_K>(vx, scratch, dst, elem, ncols_x, nrows_x, nrows_x, stride_dst, tl, GroupInfo{}, st)
                        : launch_gemm<CQ_Q6_K>(vx, scratch, dst, elem, ncols_x, nrows_x, nrows_x, stride_dst, tl, GroupInfo{}, st);
    if (ok) cq_check_launch("prompt matmul");
}

// ---- grouped entry point (quantized mixture-of-experts, many tokens) ----
extern "C" size_t cq_moe_prefill_scratch_bytes(int size_m, int num_experts, int k) {
    if (size_m <= 0 || num_experts <= 0 || num_experts > 1024 || k <= 0 || k % 256 != 0) return 0;
    const int mt = group_max_tiles(size_m, num_experts);
    return table_bytes(mt) + std::max(group_blob_bytes(size_m, num_experts, k), cq_prefill_grouped_blob_bytes(mt, k)) + 256;
}

// Q6_K experts against the int8 kernel's grouped form (the same bits), by the rule of cq_prompt_pays on an expected number of token tiles:
// half way between evenly spread pairs and a tile of each expert besides the full ones.  The int8 kernel is the faster as long as its tiles
// of 64 rows find an SM each: 8 experts, 320 pairs, K = 2816 -> 768: 46 us against 34; 16 experts, 432 pairs, K = 4096 -> 512, which do
// not: 52 against 73.  Of 12222 launches measured (1 - 64 experts, 128 - 3584 rows) 712 take the side that is slower by more than 3 %; by
// this kernel alone 5070 would.
extern "C" int cq_moe_prompt_pays(int wtype, int size_m, int num_experts, int n) {
    if (wtype != CQ_Q6_K) return 1;
    const int experts = size_m < num_experts ? size_m : num_experts;
    const int even = experts * ((size_m + 128 * num_experts - 1) / (128 * num_experts)), uneven = experts + size_m / 128;
    return (n + 63) / 64 * (long long)(even + uneven) / 2 > cq_sm_count() * 3 / 4;
}

// out[pair, :] = W[expert of the pair] . x[input row of the pair] (times topk_weights[pair]) for all size_m sorted pairs
// (candle-nn/src/moe.rs:286-337): jobs sorted by expert; job m: pair = sorted_token_ids[m], expert = expert_ids[m]; input row =
// pair when routing weights are given, else pair / topk.  The host never sees the routing: a table of tiles is built on the
// device, over-sized to ceil(M / 128) + experts entries.  Rows of pairs whose expert id is outside [0, num_experts) are not
// written.
extern "C" void cq_moe_prefill_gemm(int wtype, const void *input, int in_elem, const void *weights, const int32_t *sorted_token_ids,
                                    const int32_t *expert_ids, const float *topk_weights, float *out, void *scratch, int num_experts,
                                    int topk, int size_m, int size_n, int size_k, void *stream) {
    if (!input || !weights || !sorted_token_ids || !expert_ids || !out || !scratch || num_experts <= 0 || num_experts > 1024 ||
        topk <= 0 || size_m <= 0 || size_n <= 0 || size_k <= 0 || size_k % 256 != 0) {
        cq_set_status(CQ_ERR_BAD_ARG, "moe prefill: null pointer, empty shape, more than 1024 experts or K not a multiple of 256");
        return;
    }
    if (wtype != CQ_Q4_K && wtype != CQ_Q6_K) {
        cq_set_status(CQ_ERR_UNSUPPORTED, "moe prefill: the tensor-core kernel covers Q4_K and Q6_K");
        return;
    }
    const long long expert_stride = (long long)size_n * (size_k / 256) * cq_type_size(wtype);
    if ((uintptr_t)weights % 16 != 0 || (uintptr_t)scratch % 256 != 0 || (wtype == CQ_Q4_K ? expert_stride % 16 : expert_stride % 4) != 0) {
        cq_set_status(CQ_ERR_BAD_ARG, "moe prefill: misaligned weights or scratch");
        return;
    }
    cudaStream_t st = (cudaStream_t)stream;
    const int mt = group_max_tiles(size_m, num_experts);
    int *tiles = (int *)scratch;
    uint8_t *blobs = (uint8_t *)scratch + table_bytes(mt);
    group_tiles_kernel<<<1, 1024, 0, st>>>(expert_ids, size_m, num_experts, mt, tiles);
    if (!cq_moe_prompt_pays(wtype, size_m, num_experts, size_n)) {
        (void)cq_prefill_grouped_q6k(input, in_elem, weights, tiles, mt, sorted_token_ids, topk_weights, out, blobs, topk, size_n, size_k, st);
        return;
    }
    const GroupInfo gi{tiles, sorted_token_ids, topk_weights, size_n, topk, topk_weights ? 1 : 0};
    const Tiling tl{mt * kTokMax, kTokMax, mt};
    if (!launch_quantize_rows(wtype, input, in_elem, blobs, size_k, tl, gi, st)) return;
    const long long total = (long long)size_n * num_experts;
    const bool ok = wtype == CQ_Q4_K ? launch_gemm<CQ_Q4_K>(weights, blobs, out, CQ_F32, size_k, size_n, total, size_n, tl, gi, st)
                                     : launch_gemm<CQ_Q6_K>(weights, blobs, out, CQ_F32, size_k, size_n, total, size_n, tl, gi, st);
    if (ok) cq_check_launch("moe prefill gemm");
}

// ---- the expert matmuls of a mixture-of-experts block, many tokens (candle-transformers/src/fused_moe.rs:262-295) ----
// The three products with what lies between them: x is rounded to `kind` (the reference casts before its prompt kernel) and
// quantized ONCE for gate and up, which run as one launch; up * silu(gate), rounded to `kind`, is computed while the down
// projection's operand is quantized.  As three calls of cq_moe_prefill_gemm the same block built the tile table three times and
// quantized x twice, and moved gate, up and their product through memory four times more.
extern "C" size_t cq_moe_block_prompt_scratch_bytes(int size_m, int num_experts, int hidden, int ffn) {
    if (size_m <= 0 || num_experts <= 0 || num_experts > 1024 || hidden <= 0 || ffn <= 0 || hidden % 256 != 0 || ffn % 256 != 0) return 0;
    return table_bytes(group_max_tiles(size_m, num_experts)) + group_blob_bytes(size_m, num_experts, hidden > ffn ? hidden : ffn) + 256 +
           (size_t)size_m * ffn * 8;
}

extern "C" void cq_moe_block_prompt(int wtype, int wtype_down, const float *x, int kind, const void *gate, const void *up, const void *down,
                                    const int32_t *sorted_token_ids, const int32_t *expert_ids, const float *topk_weights, float *out,
                                    void *scratch, int num_experts, int topk, int size_m, int hidden, int ffn, void *stream) {
    if (!x || !gate || !up || !down || !sorted_token_ids || !expert_ids || !topk_weights || !out || !scratch || topk <= 0 ||
        cq_moe_block_prompt_scratch_bytes(size_m, num_experts, hidden, ffn) == 0 || (kind != CQ_F16 && kind != CQ_BF16)) {
        cq_set_status(CQ_ERR_BAD_ARG, "moe block: null pointer, empty or odd shape, more than 1024 experts, or a rounding type that is not 16-bit");
        return;
    }
    if ((wtype != CQ_Q4_K && wtype != CQ_Q6_K) || (wtype_down != CQ_Q4_K && wtype_down != CQ_Q6_K)) {
        cq_set_status(CQ_ERR_UNSUPPORTED, "moe block: the tensor-core kernel covers Q4_K and Q6_K");
        return;
    }
    if ((((uintptr_t)gate | (uintptr_t)up | (uintptr_t)down) % 16) != 0 || (uintptr_t)scratch % 256 != 0) {
        cq_set_status(CQ_ERR_BAD_ARG, "moe block: misaligned weights or scratch");
        return;
    }
    cudaStream_t st = (cudaStream_t)stream;
    const int mt = group_max_tiles(size_m, num_experts);
    int *tiles = (int *)scratch;
    uint8_t *blobs = (uint8_t *)scratch + table_bytes(mt);
    float *g = (float *)(blobs + (group_blob_bytes(size_m, num_experts, hidden > ffn ? hidden : ffn) + 255) / 256 * 256), *u = g + (size_t)size_m * ffn;
    const Tiling tl{mt * kTokMax, kTokMax, mt};
    group_tiles_kernel<<<1, 1024, 0, st>>>(expert_ids, size_m, num_experts, mt, tiles);
    const GroupInfo gu{tiles, sorted_token_ids, nullptr, ffn, topk, 0};
    const int tokens = (size_m + topk - 1) / topk, nsb = hidden / 256;
    if (topk > 1 && (size_t)(tokens + 15) / 16 * 16 * nsb * kTokBytes <= (size_t)size_m * ffn * 8) {       // each row once, into the space of gate and up
        const Tiling rows{tokens, 16, (tokens + 15) / 16};
        if (!launch_quantize(wtype, LoadRounded{x, hidden, kind}, g, hidden, rows, GroupInfo{}, st)) return;
        cq_launch_k(copy_rows_kernel, dim3(tl.ntt * (tl.tt / 8)), dim3(256), 0, st, (const uint8_t *)g, blobs, nsb, tl, gu);
    } else if (!launch_quantize(wtype, LoadRounded{x, hidden, kind}, blobs, hidden, tl, gu, st)) return;
    const long long rows_gu = (long long)ffn * num_experts, rows_d = (long long)hidden * num_experts;
    bool ok = wtype == CQ_Q4_K ? launch_gemm<CQ_Q4_K>(gate, blobs, g, CQ_F32, hidden, ffn, rows_gu, ffn, tl, gu, st, up, u)
                               : launch_gemm<CQ_Q6_K>(gate, blobs, g, CQ_F32, hidden, ffn, rows_gu, ffn, tl, gu, st, up, u);
    const GroupInfo gd{tiles, sorted_token_ids, topk_weights, hidden, topk, 1};
    if (!ok || !launch_quantize(wtype_down, LoadGateUp{g, u, ffn, kind}, blobs, ffn, tl, gd, st)) return;
    ok = wtype_down == CQ_Q4_K ? launch_gemm<CQ_Q4_K>(down, blobs, out, CQ_F32, ffn, hidden, rows_d, hidden, tl, gd, st)
                               : launch_gemm<CQ_Q6_K>(down, blobs, out, CQ_F32, ffn, hidden, rows_d, hidden, tl, gd, st);
    if (ok) cq_check_launch("moe block");
}

extern "C" int cq_prompt_timeout_flag(void) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_prompt_kq_timeout_flag, sizeof v) != cudaSuccess) { (void)cudaGetLastError(); return -1; }
    if (v) cq_set_status(CQ_ERR_TIMEOUT, "prompt matmul: a bounded wait gave up");
    return v;
}
