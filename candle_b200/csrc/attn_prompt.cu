// Causal attention of a prompt over an f32 KV cache: many queries per sequence, the results of attention_f32_kernel (attn.cu) bit
// for bit.
//
// That kernel gives every query a CTA of its own, which reads the whole context from L2: 512 queries x 32 heads x 2 sequences
// move 8.6 GB per layer, 1.2 ms.  Here one CTA takes 32 queries of one head, so a key or value is read once per 32 queries, and
// the work is bound by f32 arithmetic and the shared-memory reads that feed it.  Every sum is added in the other kernel's order:
//   scores : eight chains of 16 dims {4 (g + 8 i) .. + 3}, then the tree ((0+4)+(2+6)) + ((1+5)+(3+7)) of its lane butterfly;
//   softmax: the maximum; exp(score - max); blocks of 32 keys added as its warp butterfly does (16, 8, 4, 2, 1 apart; keys 1024
//            apart first), blocks in ascending order;
//   output : keys w, w + 32, ... in ascending order for each w, the 32 partial sums in ascending order, then the division.
// That needs all scores of a query at once, so they stay in shared memory: 128 bytes per key of the cache, which limits the
// kernel to caches of kMaxKeys positions (longer ones keep the other kernel, and so do grids that would leave SMs idle).
#include "../../include/candle_q_b200.h"
#include "common.cuh"

namespace {

constexpr int kD = 128, kQ = 32, kKeys = 128, kThreads = 256;
constexpr int kPitchK = kD + 4;                     // floats: 33 16-byte units, so eight keys of one column do not conflict
constexpr int kTileBytes = kKeys * kPitchK * 4;     // the key tile; later two value tiles of 64 rows
constexpr int kValRows = 64;
constexpr int kFixedBytes = kQ * kD * 4 + kTileBytes;
constexpr int kMaxKeys = (232448 - kFixedBytes) / (kQ * 4);      // 1160

// address of (key, query) in the scores: 32 floats per key, groups of four queries permuted by the key so that eight keys of
// one group lie in different banks
__device__ __forceinline__ int sidx(int key, int q) { return key * kQ + ((((q >> 2) ^ (key & 7)) << 2) | (q & 3)); }

__global__ void __launch_bounds__(kThreads, 1)
attention_prompt_kernel(const float *__restrict__ q, const float *__restrict__ kc, const float *__restrict__ vc, float *__restrict__ out,
                        const int *__restrict__ pos, int tq, int hq, int hkv, int tmax, float scale, int q_stride) {
    extern __shared__ __align__(16) float sm[];
    float *sq = sm, *tile = sq + kQ * kD, *sc = tile + kTileBytes / 4;
    cq_pdl_launch_dependents();
    cq_pdl_wait();
    // the last queries have the longest context: they start first
    const int t0 = ((int)gridDim.x - 1 - (int)blockIdx.x) * kQ, h = blockIdx.y, b = blockIdx.z;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int kvh = h / (hq / hkv), pos0 = pos[0];
    const float *qp = q + (size_t)b * tq * q_stride + (size_t)h * kD;
    const float *kp = kc + ((size_t)b * hkv + kvh) * (size_t)tmax * kD;
    const float *vp = vc + ((size_t)b * hkv + kvh) * (size_t)tmax * kD;
    // query t sees keys 0 .. min(pos0 + t, tmax - 1)
    const int n_keys = min(pos0 + min(t0 + kQ, tq), tmax);
    auto last_of = [&](int qi) { return min(pos0 + t0 + qi, tmax - 1); };

    for (int i = tid; i < kQ * (kD / 4); i += kThreads)
        cq_cp_async16(sq + i * 4, qp + (int64_t)min(t0 + (i >> 5), tq - 1) * q_stride + (i & 31) * 4);

    // ---- scores: warp = 8 queries x 64 keys of the tile, a lane holds keys lane and lane + 32 of them ----
    {
        const int q0 = (warp & 3) * 8, k0 = (warp >> 2) * 64 + lane;
        for (int j0 = 0; j0 < n_keys; j0 += kKeys) {
            __syncthreads();                // the previous tile has been read
            for (int i = tid; i < kKeys * (kD / 4); i += kThreads)
                cq_cp_async16(tile + (i >> 5) * kPitchK + (i & 31) * 4, kp + (int64_t)min(j0 + (i >> 5), n_keys - 1) * kD + (i & 31) * 4);
            cq_cp_async_commit();
            cq_cp_async_wait<0>();
            __syncthreads();
            float a[8][2], c[8][2];
#pragma unroll 1
            for (int pair = 0; pair < 4; ++pair) {              // lane groups (0, 4), (2, 6), (1, 5), (3, 7)
                float s[8][2];
#pragma unroll 1
                for (int second = 0; second < 2; ++second) {
                    const int g = ((pair & 1) << 1 | pair >> 1) + 4 * second;
                    float t[8][2];
#pragma unroll
                    for (int x = 0; x < 8; ++x) t[x][0] = t[x][1] = 0.0f;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int d = 4 * (g + 8 * i);
                        const float4 ka = *reinterpret_cast<const float4 *>(tile + k0 * kPitchK + d);
                        const float4 kb = *reinterpret_cast<const float4 *>(tile + (k0 + 32) * kPitchK + d);
#pragma unroll
                        for (int x = 0; x < 8; ++x) {
                            const float4 qv = *reinterpret_cast<const float4 *>(sq + (q0 + x) * kD + d);
                            t[x][0] = __fmaf_rn(qv.x, ka.x, t[x][0]); t[x][0] = __fmaf_rn(qv.y, ka.y, t[x][0]);
                            t[x][0] = __fmaf_rn(qv.z, ka.z, t[x][0]); t[x][0] = __fmaf_rn(qv.w, ka.w, t[x][0]);
                            t[x][1] = __fmaf_rn(qv.x, kb.x, t[x][1]); t[x][1] = __fmaf_rn(qv.y, kb.y, t[x][1]);
                            t[x][1] = __fmaf_rn(qv.z, kb.z, t[x][1]); t[x][1] = __fmaf_rn(qv.w, kb.w, t[x][1]);
                        }
                    }
#pragma unroll
                    for (int x = 0; x < 8; ++x) {
                        s[x][0] = second ? __fadd_rn(s[x][0], t[x][0]) : t[x][0];
                        s[x][1] = second ? __fadd_rn(s[x][1], t[x][1]) : t[x][1];
                    }
                }
#pragma unroll
                for (int x = 0; x < 8; ++x)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        if (pair == 0) a[x][e] = s[x][e];
                        else if (pair == 1) a[x][e] = __fadd_rn(a[x][e], s[x][e]);
                        else if (pair == 2) c[x][e] = s[x][e];
                        else a[x][e] = __fmul_rn(__fadd_rn(a[x][e], __fadd_rn(c[x][e], s[x][e])), scale);
                    }
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int key = j0 + k0 + 32 * e;
                if (key < n_keys) {
                    *reinterpret_cast<float4 *>(sc + sidx(key, q0)) = make_float4(a[0][e], a[1][e], a[2][e], a[3][e]);
                    *reinterpret_cast<float4 *>(sc + sidx(key, q0 + 4)) = make_float4(a[4][e], a[5][e], a[6][e], a[7][e]);
                }
            }
        }
    }
    __syncthreads();

    // ---- softmax: lane = query, warp = every eighth block of 32 keys; the key tile holds the partial results ----
    float *redmax = tile, *redsum = tile + 8 * kQ;          // [8][32], [32 blocks][32]
    // at least one block: a context without keys (a position before the cache) divides 0 by 0, as in the other kernel
    const int my_last = last_of(lane), nblk = min(max((n_keys + 31) / 32, 1), 32);
    float mx = -INFINITY;
    for (int j0 = warp * 32; j0 < n_keys; j0 += 256)
        for (int j = j0; j < min(j0 + 32, n_keys); ++j)
            if (j <= my_last) mx = fmaxf(mx, sc[sidx(j, lane)]);
    redmax[warp * kQ + lane] = mx;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 8; ++w) mx = fmaxf(mx, redmax[w * kQ + lane]);
    for (int w = warp; w < nblk; w += 8) {
        float p[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            p[i] = 0.0f;
            const int j = 32 * w + i;
            if (j <= my_last && j < n_keys) { p[i] = expf(sc[sidx(j, lane)] - mx); sc[sidx(j, lane)] = p[i]; }
        }
        for (int j1 = 32 * w + 1024; j1 < n_keys; j1 += 1024)
#pragma unroll
            for (int i = 0; i < 32; ++i)
                if (j1 + i <= my_last && j1 + i < n_keys) {
                    const float e = expf(sc[sidx(j1 + i, lane)] - mx);
                    sc[sidx(j1 + i, lane)] = e;
                    p[i] += e;
                }
#pragma unroll
        for (int m = 16; m > 0; m >>= 1)
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if (i < m) p[i] = __fadd_rn(p[i], p[i + m]);
        redsum[w * kQ + lane] = p[0];
    }
    __syncthreads();
    // ---- output: warp = 8 queries x 64 dims, a lane holds two of them ----
    const int q0 = (warp & 3) * 8, d0 = (warp >> 2) * 64 + 2 * lane;
    float den[8];
#pragma unroll
    for (int x = 0; x < 8; ++x) {
        den[x] = redsum[q0 + x];
        for (int w = 1; w < nblk; ++w) den[x] = __fadd_rn(den[x], redsum[w * kQ + q0 + x]);
    }
    __syncthreads();                        // the partial results have been read; the tile takes values now
    const int rpw = max((n_keys + 31) / 32, 1), wg = kValRows / rpw;        // keys per w; w's per value tile (at least one: n_keys <= kMaxKeys)
    const int ngrp = (32 + wg - 1) / wg, all_see = last_of(0);      // keys up to all_see are in every query's context
    auto load_values = [&](int grp) {
        float *dst = tile + (grp & 1) * kValRows * kD;
        for (int i = tid; i < wg * rpw * 32; i += kThreads) {
            const int row = i >> 5, key = grp * wg + row / rpw + 32 * (row % rpw);
            if (grp * wg + row / rpw < 32 && key < n_keys) cq_cp_async16(dst + row * kD + (i & 31) * 4, vp + (int64_t)key * kD + (i & 31) * 4);
        }
        cq_cp_async_commit();
    };
    float o[8][2];
#pragma unroll
    for (int x = 0; x < 8; ++x) o[x][0] = o[x][1] = 0.0f;
    load_values(0);
    for (int grp = 0; grp < ngrp; ++grp) {
        if (grp + 1 < ngrp) load_values(grp + 1);
        else cq_cp_async_commit();          // an empty group keeps the count
        cq_cp_async_wait<1>();
        __syncthreads();
        const float *val = tile + (grp & 1) * kValRows * kD + d0;
        for (int wl = 0; wl < wg && grp * wg + wl < 32; ++wl) {
            const int w = grp * wg + wl;
            float t[8][2];
#pragma unroll
            for (int x = 0; x < 8; ++x) t[x][0] = t[x][1] = 0.0f;
            const float *row = val + wl * rpw * kD;
#pragma unroll 2
            for (int j = w; j < n_keys; j += 32, row += kD) {
                const float2 v = *reinterpret_cast<const float2 *>(row);
                const float4 pa = *reinterpret_cast<const float4 *>(sc + sidx(j, q0)), pb = *reinterpret_cast<const float4 *>(sc + sidx(j, q0 + 4));
                const float p[8] = {pa.x, pa.y, pa.z, pa.w, pb.x, pb.y, pb.z, pb.w};
#pragma unroll
                for (int x = 0; x < 8; ++x)
                    if (j <= all_see || j <= last_of(q0 + x)) {     // warp-uniform; a key past the context is left out, not added as zero
                        t[x][0] = __fmaf_rn(p[x], v.x, t[x][0]);
                        t[x][1] = __fmaf_rn(p[x], v.y, t[x][1]);
                    }
            }
#pragma unroll
            for (int x = 0; x < 8; ++x) {
                o[x][0] = w == 0 ? t[x][0] : __fadd_rn(o[x][0], t[x][0]);
                o[x][1] = w == 0 ? t[x][1] : __fadd_rn(o[x][1], t[x][1]);
            }
        }
        __syncthreads();                    // this tile is filled again two groups later
    }
#pragma unroll
    for (int x = 0; x < 8; ++x) {
        const int t = t0 + q0 + x;
        if (t < tq)
            *reinterpret_cast<float2 *>(out + (((size_t)b * tq + t) * hq + h) * kD + d0) = make_float2(__fdiv_rn(o[x][0], den[x]), __fdiv_rn(o[x][1], den[x]));
    }
}

}  // namespace

// Which kernel cq_attention_f32 runs: 1 the one that reads the context once per 32 queries (attn_prompt.cu, the same bits), 0 a CTA
// per query.  The first has 32 times fewer CTAs, one per SM, and each walks its whole context alone, so it needs enough of them:
// 21 queries of 4 heads behind 954 keys take 13 us per query and 129 us by 32, 512 queries of 32 heads and 2 sequences 1180 and 343.
// Fitted to 260 shapes (1 - 64 heads, 1 - 8 sequences, 17 - 1020 queries, caches to 1152; within 12 % on average): a CTA of the
// first takes 17 us + 0.12 per key, a round of two CTAs per SM of the other 7 us + 0.016 per key.  The position is on the device,
// so the first is taken only if it is the faster both at position 0 and at the end of the cache.
extern "C" int cq_attention_reads_by_32(int batch, int tq, int hq, int tmax) {
    if (tq < 17 || tmax > kMaxKeys || hq > 65535) return 0;
    const double sms = cq_sm_count(), heads = (double)batch * hq;
    const double rounds32 = heads * ((tq + 31) / 32) / sms, rounds1 = heads * tq / (2 * sms);
    for (int last : {tq < tmax ? tq : tmax, tmax}) {            // keys of the last query
        const double mean = last - 0.5 * (tq < last ? tq : last);
        const double by32 = rounds32 > 1 ? rounds32 * (17 + 0.12 * mean) : 17 + 0.12 * last;
        const double by1 = rounds1 > 1 ? rounds1 * (7 + 0.016 * mean) : 7 + 0.016 * last;
        if (by32 >= by1) return 0;
    }
    return 1;
}

// Called by cq_attention_f32 for the shapes above, arguments checked there.
void cq_attention_prompt_launch(const float *q, const float *k_cache, const float *v_cache, float *out, const int *pos, int batch, int tq,
                                int hq, int hkv, int tmax, float scale, int q_stride, cudaStream_t st) {
    static bool attr_done[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && !attr_done[dev]) {
        cudaFuncSetAttribute(attention_prompt_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448);
        attr_done[dev] = true;
    }
    cq_launch_k(attention_prompt_kernel, dim3((tq + kQ - 1) / kQ, hq, batch), dim3(kThreads), (size_t)kFixedBytes + (size_t)tmax * kQ * 4, st, q,
                k_cache, v_cache, out, pos, tq, hq, hkv, tmax, scale, q_stride);
}
