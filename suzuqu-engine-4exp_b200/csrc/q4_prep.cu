/*
 * Q / K preparation ahead of the append and the attention: per-head RMSNorm (optional weight),
 * interleaved-pair RoPE on the first n_rot dims, and for Q the split of the packed [q | gate]
 * projection.  Restates qsa_q_prep_k / qsa_k_prep_k (src/q4_rocm.cu:6229-6294) and their launchers
 * (:6296-6343); position = pos0 + t or the device position word + t.
 *
 * Head sizes 64, 128 and 256: a block takes the heads of one token, one warp per head.  The rotation of a pair depends
 * on the token alone, so its power, sine and cosine are taken once per token (one block per (head, token) took them
 * n_head times: 72 us for 2048 tokens x 24 heads of 256, which read and write 200 MB).  Every sum keeps the order of
 * that form, so the cache bytes quantised from the rows stay the same.  Other head sizes: one block per (head, token).
 */
#include <string.h>

#include "q4_internal.h"

namespace {

__device__ __forceinline__ float block_sum_128(float v, float *sh) {
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    return sh[0] + sh[1] + sh[2] + sh[3];
}

/* src == dst is allowed (K is prepared in place). */
__device__ __forceinline__ void norm_rope(const float *src, float *dst, const float *wn, uint32_t hd,
                                          uint32_t n_rot, int32_t pos, float base, float eps, float *sh) {
    float ss = 0.f;
    for (uint32_t i = threadIdx.x; i < hd; i += blockDim.x) ss += src[i] * src[i];
    ss = block_sum_128(ss, sh);
    const float scale = 1.0f / sqrtf(ss / (float)hd + eps);
    const uint32_t np = n_rot / 2;
    /* each thread normalises and rotates whole pairs, so in-place operation needs no barrier */
    for (uint32_t p = threadIdx.x; p < hd / 2; p += blockDim.x) {
        float x0 = src[2 * p] * scale * (wn ? wn[2 * p] : 1.f);
        float x1 = src[2 * p + 1] * scale * (wn ? wn[2 * p + 1] : 1.f);
        if (p < np) {
            const float freq = powf(base, -(float)p / (float)np);
            const float ang = (float)pos * freq;
            const float c = cosf(ang), si = sinf(ang);
            const float y0 = x0 * c - x1 * si, y1 = x0 * si + x1 * c;
            x0 = y0;
            x1 = y1;
        }
        dst[2 * p] = x0;
        dst[2 * p + 1] = x1;
    }
}

__global__ void q4_q_prep_k(const float *qg, const float *wn, float *q, float *g, uint32_t hd, uint32_t n_rot,
                            int32_t pos0, float base, float eps, uint32_t n_head, const int32_t *pp) {
    __shared__ float sh[4];
    const uint32_t h = blockIdx.x, t = blockIdx.y;
    const int32_t pos = (pp ? *pp : pos0) + (int32_t)t;
    const float *src = qg + ((size_t)t * n_head + h) * hd * 2;
    float *qd = q + ((size_t)t * n_head + h) * hd, *gd = g + ((size_t)t * n_head + h) * hd;
    for (uint32_t i = threadIdx.x; i < hd; i += blockDim.x) gd[i] = src[hd + i];
    norm_rope(src, qd, wn, hd, n_rot, pos, base, eps, sh);
}
__global__ void q4_k_prep_k(float *k, const float *wn, uint32_t hd, uint32_t n_rot, int32_t pos0, float base,
                            float eps, uint32_t n_kvh, const int32_t *pp) {
    __shared__ float sh[4];
    const uint32_t h = blockIdx.x, t = blockIdx.y;
    const int32_t pos = (pp ? *pp : pos0) + (int32_t)t;
    float *kh = k + ((size_t)t * n_kvh + h) * hd;
    norm_rope(kh, kh, wn, hd, n_rot, pos, base, eps, sh);
}


/* ---- one warp per head */
constexpr uint32_t PREP_WARPS = 8;
/* cos and sin of a token's rotation of pair p, by thread p of `threads`; np <= 128 */
__device__ __forceinline__ void rope_table(float2 *cs, uint32_t np, int32_t pos, float base, uint32_t p, uint32_t threads) {
    for (; p < np; p += threads) {
        const float freq = powf(base, -(float)p / (float)np);
        const float ang = (float)pos * freq;
        cs[p] = make_float2(cosf(ang), sinf(ang));
    }
}
/* a row as the warp holds it: register k of lane l = elements 64 k + 2 l, + 1 */
template <int HD>
__device__ __forceinline__ void row_load(const float *src, float2 (&v)[HD / 64]) {
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
    for (int k = 0; k < HD / 64; k++) v[k] = __ldcg(reinterpret_cast<const float2 *>(src) + 32 * k + lane);
}
/* the weights of those elements; l2: the launch before last may have written them (q4d_apart_begin).  A launch of few rows asks
 * for them beside the row: behind its sums they came a trip to L2 later. */
template <int HD>
__device__ __forceinline__ void row_weights(const float *wn, float2 (&w)[HD / 64], bool l2) {
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
    for (int k = 0; k < HD / 64; k++) {
        const float *p = wn + 64 * k + 2 * lane;
        w[k] = !wn ? make_float2(1.f, 1.f) : l2 ? make_float2(__ldcg(p), __ldcg(p + 1)) : make_float2(p[0], p[1]);
    }
}
/* RMSNorm and rotation in place.  Sum of squares as 128 threads of a block would take it: thread i adds elements i and
 * i + 128, a butterfly over each 32 threads, then the four totals in order (element 2 l + e of a register is thread
 * 2 l + e: the butterfly's last step is the addition inside the lane). */
template <int HD>
__device__ __forceinline__ void row_norm_rope(float2 (&v)[HD / 64], const float2 (&w)[HD / 64], const float2 *cs, uint32_t np, float eps) {
    const uint32_t lane = threadIdx.x & 31u;
    float tot[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < (HD / 64 < 2 ? HD / 64 : 2); k++) {
        float a = __fmul_rn(v[k].x, v[k].x), b = __fmul_rn(v[k].y, v[k].y);
        if (HD == 256) { a = __fmaf_rn(v[k + HD / 128].x, v[k + HD / 128].x, a); b = __fmaf_rn(v[k + HD / 128].y, v[k + HD / 128].y, b); }
#pragma unroll
        for (int o = 8; o; o >>= 1) {
            a = __fadd_rn(a, __shfl_xor_sync(0xffffffffu, a, o));
            b = __fadd_rn(b, __shfl_xor_sync(0xffffffffu, b, o));
        }
        a = __fadd_rn(a, b);
        tot[2 * k] = __shfl_sync(0xffffffffu, a, 0);
        tot[2 * k + 1] = __shfl_sync(0xffffffffu, a, 16);
    }
    const float ss = __fadd_rn(__fadd_rn(__fadd_rn(tot[0], tot[1]), tot[2]), tot[3]);
    const float scale = 1.0f / sqrtf(ss / (float)HD + eps);
#pragma unroll
    for (int k = 0; k < HD / 64; k++) {
        const uint32_t p = 32u * k + lane;
        float x0 = v[k].x * scale * w[k].x, x1 = v[k].y * scale * w[k].y;
        if (p < np) {
            const float c = cs[p].x, si = cs[p].y;
            const float y0 = x0 * c - x1 * si, y1 = x0 * si + x1 * c;
            x0 = y0;
            x1 = y1;
        }
        v[k] = make_float2(x0, x1);
    }
}
template <int HD>
__device__ __forceinline__ void row_store(float *dst, const float2 (&v)[HD / 64]) {
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
    for (int k = 0; k < HD / 64; k++) reinterpret_cast<float2 *>(dst)[32 * k + lane] = v[k];
}
/* SPLIT: rows are [q | gate] pairs, q goes to `q` and the gate to `g`; else rows of `q` in place.  blockIdx.x: a group of
 * `per` heads, blockIdx.y: TOK tokens (several where a token has few heads: a block with 2 rows for its 8 warps is mostly
 * the wait for its rotation table). */
template <int HD, bool SPLIT, uint32_t TOK>
__global__ void __launch_bounds__(PREP_WARPS * 32) q4_prep_rows_k(const float *src, const float *wn, float *q, float *g, uint32_t n_rot,
                                                                  int32_t pos0, float base, float eps, uint32_t n_head, uint32_t per,
                                                                  uint32_t n_tok, const int32_t *pp, bool early, bool apart) {
    __shared__ float2 cs[TOK][128];
    constexpr uint32_t W = PREP_WARPS / TOK;   /* warps of a token */
    const uint32_t warp = threadIdx.x >> 5, sub = warp / W, t = blockIdx.y * TOK + sub, h0 = blockIdx.x * per, h1 = min(h0 + per, n_head);
    if (apart) q4d_apart_begin();
    else if (!early) q4d_pdl_wait();
    rope_table(cs[sub], n_rot / 2u, (pp ? __ldcg(pp) : pos0) + (int32_t)t, base, threadIdx.x % (W * 32u), W * 32u);   /* a settled position's under the previous kernel's tail */
    if (early && !apart) q4d_pdl_wait();
    __syncthreads();
    for (uint32_t h = h0 + warp % W; h < h1 && t < n_tok; h += W) {
        const size_t row = (size_t)t * n_head + h;
        float2 v[HD / 64], wt[HD / 64];
        row_weights<HD>(wn, wt, apart);
        row_load<HD>(SPLIT ? src + row * 2u * HD : q + row * HD, v);
        if (SPLIT) {
            float2 w[HD / 64];
            row_load<HD>(src + row * 2u * HD + HD, w);
            row_store<HD>(g + row * HD, w);
        }
        row_norm_rope<HD>(v, wt, cs[sub], n_rot / 2u, eps);
        row_store<HD>(q + row * HD, v);
    }
    if (apart) q4d_apart_end();
}

/* false in `done` where the head size or an address is not the warp form's */
template <bool SPLIT>
bool prep_rows(const float *src, const float *wn, float *q, float *g, uint32_t n_head, uint32_t hd, uint32_t n_rot, int32_t pos0, float base,
               float eps, uint32_t n_tok, const int32_t *pp, bool &done) {
    done = (hd == 64 || hd == 128 || hd == 256) && (((uintptr_t)src | (uintptr_t)q | (uintptr_t)g) & 7u) == 0;
    if (!done) return false;
    /* few tokens: a token's heads over several SMs, eight to a block; many: one block each, or four where heads are few */
    const bool four = n_tok >= 2u * (uint32_t)g_q4.sm_count && n_head <= 4u;
    const uint32_t per = n_tok < (uint32_t)g_q4.sm_count ? PREP_WARPS : n_head;
    const dim3 grid((n_head + per - 1u) / per, four ? (n_tok + 3u) / 4u : n_tok);
    const bool early = !pp || q4i_settled(g_q4.pos_written);
    Q4Touch touch = {};
    const uint64_t rows = (uint64_t)n_tok * n_head * hd * 4u;
    touch.reads(src, 2u * rows);
    touch.reads(wn, hd * 4u);
    touch.reads(pp, 4);
    touch.writes(q, rows);
    touch.writes(g, rows);
    const bool apart = early && q4i_apart(touch);
    auto start = [&](auto kernel) {
        return q4i_launched(q4i_launch_dep("prep launch", kernel, grid, PREP_WARPS * 32u, 0, src, wn, q, g, n_rot, pos0, base, eps, n_head, per, n_tok, pp,
                                           early, apart), &touch, apart);
    };
    if (hd == 64) return four ? start(q4_prep_rows_k<64, SPLIT, 4>) : start(q4_prep_rows_k<64, SPLIT, 1>);
    if (hd == 128) return four ? start(q4_prep_rows_k<128, SPLIT, 4>) : start(q4_prep_rows_k<128, SPLIT, 1>);
    return four ? start(q4_prep_rows_k<256, SPLIT, 4>) : start(q4_prep_rows_k<256, SPLIT, 1>);
}
bool q_prep(const float *qg, const float *wn, float *q, float *g, uint32_t n_head, uint32_t hd, uint32_t n_rot, int32_t pos0, float base,
            float eps, uint32_t n_tok, const int32_t *pp) {
    bool done;
    const bool ok = prep_rows<true>(qg, wn, q, g, n_head, hd, n_rot, pos0, base, eps, n_tok, pp, done);
    if (done) return ok;
    q4_q_prep_k<<<dim3(n_head, n_tok), 128, 0, g_q4.stream>>>(qg, wn, q, g, hd, n_rot, pos0, base, eps, n_head, pp);
    return q4i_check(cudaGetLastError(), "q_prep launch");
}
bool k_prep(float *k, const float *wn, uint32_t n_kvh, uint32_t hd, uint32_t n_rot, int32_t pos0, float base, float eps, uint32_t n_tok,
            const int32_t *pp) {
    bool done;
    const bool ok = prep_rows<false>(nullptr, wn, k, nullptr, n_kvh, hd, n_rot, pos0, base, eps, n_tok, pp, done);
    if (done) return ok;
    q4_k_prep_k<<<dim3(n_kvh, n_tok), 128, 0, g_q4.stream>>>(k, wn, hd, n_rot, pos0, base, eps, n_kvh, pp);
    return q4i_check(cudaGetLastError(), "k_prep launch");
}

}  // namespace

extern "C" bool q4_hip_qsa_q_prep_n(const float *d_qg, const float *d_wn, float *d_q, float *d_g, uint32_t n_head,
                                    uint32_t hd, uint32_t n_rot, int32_t pos0, float base, float eps,
                                    uint32_t n_tok) {
    if (!g_q4.ok || !d_qg || !d_q || !d_g || n_head == 0 || n_tok == 0 || hd == 0 || (hd & 1) || n_rot > hd)
        return false;
    return q_prep(d_qg, d_wn, d_q, d_g, n_head, hd, n_rot, pos0, base, eps, n_tok, nullptr);
}
extern "C" bool q4_hip_qsa_q_prep_d(const float *qg, const float *wn, float *q, float *g, uint32_t n_head,
                                    uint32_t hd, uint32_t n_rot, float base, float eps) {
    if (!g_q4.ok || !g_q4.pos_d || !qg || !q || !g || n_head == 0 || hd == 0 || (hd & 1) || n_rot > hd)
        return false;
    return q_prep(qg, wn, q, g, n_head, hd, n_rot, 0, base, eps, 1, g_q4.pos_d);
}
extern "C" bool q4_hip_qsa_q_prep(const float *d_qg, const float *d_wn, float *d_q, float *d_g, uint32_t n_head,
                                  uint32_t hd, uint32_t n_rot, int32_t pos, float base, float eps) {
    return q4_hip_qsa_q_prep_n(d_qg, d_wn, d_q, d_g, n_head, hd, n_rot, pos, base, eps, 1);
}
extern "C" bool q4_hip_qsa_k_prep_n(float *d_k, const float *d_wn, uint32_t n_kvh, uint32_t hd, uint32_t n_rot,
                                    int32_t pos0, float base, float eps, uint32_t n_tok) {
    if (!g_q4.ok || !d_k || n_kvh == 0 || n_tok == 0 || hd == 0 || (hd & 1) || n_rot > hd) return false;
    return k_prep(d_k, d_wn, n_kvh, hd, n_rot, pos0, base, eps, n_tok, nullptr);
}
extern "C" bool q4_hip_qsa_k_prep_d(float *k, const float *wn, uint32_t n_kvh, uint32_t hd, uint32_t n_rot,
                                    float base, float eps) {
    if (!g_q4.ok || !g_q4.pos_d || !k || n_kvh == 0 || hd == 0 || (hd & 1) || n_rot > hd) return false;
    return k_prep(k, wn, n_kvh, hd, n_rot, 0, base, eps, 1, g_q4.pos_d);
}
extern "C" bool q4_hip_qsa_k_prep(float *d_k, const float *d_wn, uint32_t n_kvh, uint32_t hd, uint32_t n_rot,
                                  int32_t pos, float base, float eps) {
    return q4_hip_qsa_k_prep_n(d_k, d_wn, n_kvh, hd, n_rot, pos, base, eps, 1);
}

/* ---- K prep fused into the append: RMSNorm + RoPE of the new K rows, q8_0 quantisation (or fp16 /
 * fp32 conversion) of K and V, and the scatter into the store, in one launch -- replaces
 * q4_hip_qsa_k_prep_d + q4_hip_kv_append_d (src/q4_fwd.c:884,891) and the prefill pair
 * q4_hip_qsa_k_prep_n + 2 x kv_write (:1734,1738-1741).  The normalised, rotated K row is built in
 * shared memory with exactly the arithmetic of q4_k_prep_k, then quantised with the append kernel's
 * arithmetic, so the cache bytes equal those of the two-launch sequence. */
namespace {

struct PrepAppendParams {
    Q4Cache C;
    int layout;
    uint32_t layer, n_kvh, hd, n_rot, n_tok;
    const float *k, *v, *wn;
    const int32_t *pos;      /* device position word or null */
    int32_t pos0;
    float base, eps;
    uint32_t *err;
    uint32_t early;          /* the position is settled */
};

/* head sizes 32 and 64: a block per (row, K or V) */
__global__ void q4_prep_append_k(const PrepAppendParams P) {
    __shared__ float sh[4];
    __shared__ __align__(16) float row_s[256];
    const uint32_t kh = blockIdx.x, t = blockIdx.y;
    const bool which = blockIdx.z != 0;
    const int32_t pos = (P.pos ? *P.pos : P.pos0) + (int32_t)t;
    const float *src = (which ? P.v : P.k) + ((size_t)t * P.n_kvh + kh) * P.hd;
    if (!which) norm_rope(src, row_s, P.wn, P.hd, P.n_rot, pos, P.base, P.eps, sh);
    else for (uint32_t i = threadIdx.x; i < P.hd; i += blockDim.x) row_s[i] = src[i];
    __syncthreads();
    if (pos < 0 || (uint32_t)pos >= P.C.max_kv) {
        if (threadIdx.x == 0) atomicOr(P.err, (uint32_t)Q4E_RANGE);
        return;
    }
    /* 8 lanes per 32-value block, as the append kernel: hd / 4 lanes are busy */
    const uint32_t nb = P.hd / 32u, sub = threadIdx.x & 7u, b = threadIdx.x >> 3;
    const bool live = b < nb;
    const float4 x = live ? *reinterpret_cast<const float4 *>(row_s + b * 32 + sub * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    float d, id;
    q4d_block_scale(x, d, id);
    if (!live) return;
    uint8_t *row = const_cast<uint8_t *>(which ? P.C.v : P.C.k) + (uint64_t)P.layer * P.C.layer_stride +
                   (uint64_t)kh * P.C.kvh_stride + (uint64_t)pos * P.C.tok_stride;
    if (P.layout == LAY_Q8P) {
        *reinterpret_cast<uint32_t *>(row + b * 32 + sub * 4) = q4d_quant4(x, id);
        if (sub == 0) {
            uint8_t *srow = const_cast<uint8_t *>(P.C.s) + (uint64_t)P.layer * P.C.s_layer_stride +
                            (uint64_t)kh * P.C.s_kvh_stride + (uint64_t)pos * P.C.s_tok_stride;
            reinterpret_cast<__half *>(srow)[(which ? nb : 0u) + b] = __float2half_rn(d);
        }
    } else if (P.layout == LAY_F16) {
        __half2 *o = reinterpret_cast<__half2 *>(row + (b * 32 + sub * 4) * 2);
        o[0] = __floats2half2_rn(x.x, x.y);
        o[1] = __floats2half2_rn(x.z, x.w);
    } else {
        *reinterpret_cast<float4 *>(row + (b * 32 + sub * 4) * 4) = x;
    }
}

/* Head sizes 128 and 256: a block per TOK tokens, a warp per row (K heads, then V heads), the rotation once per token.  The row
 * passes through the warp's part of shared memory to be quantised eight lanes per 32 values, as everywhere. */
template <int HD, uint32_t TOK>
__global__ void __launch_bounds__(PREP_WARPS * 32) q4_prep_append_rows_k(const PrepAppendParams P) {
    __shared__ float2 cs[TOK][128];
    constexpr uint32_t W = PREP_WARPS / TOK;   /* warps of a token */
    __shared__ __align__(16) float row_s[PREP_WARPS][HD];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, sub = warp / W, t = blockIdx.x * TOK + sub;
    if (!P.early) q4d_pdl_wait();
    const int32_t pos = (P.pos ? *P.pos : P.pos0) + (int32_t)t;
    rope_table(cs[sub], P.n_rot / 2u, pos, P.base, threadIdx.x % (W * 32u), W * 32u);
    if (P.early) q4d_pdl_wait();
    __syncthreads();
    if (t >= P.n_tok) return;
    if (pos < 0 || (uint32_t)pos >= P.C.max_kv) {
        if (lane == 0) atomicOr(P.err, (uint32_t)Q4E_RANGE);
        return;
    }
    for (uint32_t r = warp % W; r < 2u * P.n_kvh; r += W) {
        const bool which = r >= P.n_kvh;
        const uint32_t kh = which ? r - P.n_kvh : r;
        float2 v[HD / 64];
        row_load<HD>((which ? P.v : P.k) + ((size_t)t * P.n_kvh + kh) * HD, v);
        if (!which) {
            float2 wt[HD / 64];
            row_weights<HD>(P.wn, wt, false);
            row_norm_rope<HD>(v, wt, cs[sub], P.n_rot / 2u, P.eps);
        }
        __syncwarp();
        row_store<HD>(row_s[warp], v);
        __syncwarp();
        uint8_t *row = const_cast<uint8_t *>(which ? P.C.v : P.C.k) + (uint64_t)P.layer * P.C.layer_stride +
                       (uint64_t)kh * P.C.kvh_stride + (uint64_t)pos * P.C.tok_stride;
#pragma unroll
        for (uint32_t i = lane; i < HD / 4u; i += 32u) {
            const float4 x = *reinterpret_cast<const float4 *>(row_s[warp] + i * 4u);
            float d, id;
            if (P.layout == LAY_Q8P) {
                q4d_block_scale(x, d, id);
                *reinterpret_cast<uint32_t *>(row + i * 4u) = q4d_quant4(x, id);
                if ((i & 7u) == 0) {
                    uint8_t *srow = const_cast<uint8_t *>(P.C.s) + (uint64_t)P.layer * P.C.s_layer_stride +
                                    (uint64_t)kh * P.C.s_kvh_stride + (uint64_t)pos * P.C.s_tok_stride;
                    reinterpret_cast<__half *>(srow)[(which ? HD / 32u : 0u) + (i >> 3)] = __float2half_rn(d);
                }
            } else if (P.layout == LAY_F16) {
                const __half2 a = __floats2half2_rn(x.x, x.y), b = __floats2half2_rn(x.z, x.w);
                *reinterpret_cast<uint2 *>(row + i * 8u) = make_uint2(*reinterpret_cast<const uint32_t *>(&a), *reinterpret_cast<const uint32_t *>(&b));
            } else {
                *reinterpret_cast<float4 *>(row + i * 16u) = x;
            }
        }
    }
}

bool prep_append_launch(q4_gpu_kv *kv, uint32_t layer, const float *k, const float *v, const float *wn, uint32_t n_rot,
                 float base, float eps, const int32_t *pos_dev, int32_t pos0, uint32_t n_tok) {
    if (!g_q4.ok) return q4i_fail(Q4E_INIT, "kv_prep_append: library not initialised");
    Q4_REQUIRE(kv && k && v && n_tok && layer < kv->n_layers && n_rot <= kv->hd && !(n_rot & 1), "kv_prep_append: bad argument");
    Q4_REQUIRE(pos_dev || (pos0 >= 0 && (uint64_t)pos0 + n_tok <= kv->max_kv), "kv_prep_append: rows beyond max_kv");
    PrepAppendParams p;
    p.C = kv->view;
    p.layout = kv->kind == Q4K_Q8 ? LAY_Q8P : kv->kind == Q4K_F16 ? LAY_F16 : LAY_F32;
    p.layer = layer; p.n_kvh = kv->n_kvh; p.hd = kv->hd; p.n_rot = n_rot; p.n_tok = n_tok;
    p.k = k; p.v = v; p.wn = wn; p.pos = pos_dev; p.pos0 = pos0; p.base = base; p.eps = eps; p.err = g_q4.err_d;
    p.early = !pos_dev || q4i_settled(g_q4.pos_written);
    if ((kv->hd == 128 || kv->hd == 256) && (((uintptr_t)k | (uintptr_t)v) & 7u) == 0)
    {
        const bool two = n_tok >= 2u * (uint32_t)g_q4.sm_count && kv->n_kvh <= 2u;   /* 4 rows a token: two tokens for 8 warps */
        const dim3 grid(two ? (n_tok + 1u) / 2u : n_tok);
        auto start = [&](auto kernel) { return q4i_launch_pdl("kv_prep_append launch", kernel, grid, PREP_WARPS * 32u, 0, p); };
        if (kv->hd == 128) return two ? start(q4_prep_append_rows_k<128, 2>) : start(q4_prep_append_rows_k<128, 1>);
        return two ? start(q4_prep_append_rows_k<256, 2>) : start(q4_prep_append_rows_k<256, 1>);
    }
    q4_prep_append_k<<<dim3(kv->n_kvh, n_tok, 2), 128, 0, g_q4.stream>>>(p);
    return q4i_check(cudaGetLastError(), "kv_prep_append launch");
}

bool prep_append(q4_gpu_kv *kv, uint32_t layer, const float *k, const float *v, const float *wn, uint32_t n_rot,
                 float base, float eps, const int32_t *pos_dev, int32_t pos0, uint32_t n_tok) {
    const bool ok = prep_append_launch(kv, layer, k, v, wn, n_rot, base, eps, pos_dev, pos0, n_tok);
    if (kv && layer < kv->n_layers) q4i_kv_written(kv, layer);
    return ok;
}

}  // namespace

extern "C" bool q4_gpu_kv_prep_append(q4_gpu_kv *kv, uint32_t layer, const float *k_raw, const float *v, const float *k_norm_w,
                                      uint32_t n_rot, float rope_base, float eps, uint32_t pos0, uint32_t n_tok) {
    return prep_append(kv, layer, k_raw, v, k_norm_w, n_rot, rope_base, eps, nullptr, (int32_t)pos0, n_tok);
}
extern "C" bool q4_gpu_kv_prep_append_d(q4_gpu_kv *kv, uint32_t layer, const float *k_raw, const float *v,
                                        const float *k_norm_w, uint32_t n_rot, float rope_base, float eps) {
    if (!g_q4.ok || !g_q4.pos_d) return q4i_fail(Q4E_INIT, "kv_prep_append_d: library not initialised");
    return prep_append(kv, layer, k_raw, v, k_norm_w, n_rot, rope_base, eps, g_q4.pos_d, 0, 1);
}
