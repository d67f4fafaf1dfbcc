/*
 * QSA indexer: the step that produces the 2051-wide selection lists the sparse decode consumes.
 *
 *   pool   qsa_pool_k / qsa_pool_dk (src/q4_rocm.cu:7366-7402, 7880-7933): block b of `ratio` tokens =
 *          mean of their raw fp16 keys, RMSNorm, RoPE at the block's first position, fp32 [block][128]
 *   score  qsa_score_k / qsa_score_dk (:7405-7436, 7469-7502): score[b] = sum_h relu(q_h . pool[b])
 *          over the blocks the token can see -- at ctx 262 144 a 33.5 MB scan per layer, 30x the
 *          bytes of the sparse attention it feeds, so this is the HBM-bound part
 *   top-k  qsa_topk_k / the qsa_tk_* family (:7506-7666, 7722-7846): exact top-512 blocks by (score
 *          descending, index ascending), expanded to positions plus the newest partial block
 *
 * Results are defined by the reference down to the order of the list, so the arithmetic keeps its
 * association: the sum of squares is the same pairwise tree, a dot product is one fused multiply-add
 * per dim in dim order (four heads = four independent chains per thread), and the selection is an
 * exact radix select followed by an index-ordered compaction.  What changes is the mapping: a warp
 * per pooled block with the tree in shuffles, a thread per pooled block for the scan with each warp's
 * 32 rows staged in shared memory by coalesced asynchronous copies (many tokens: a tiled product with the
 * same chains), and ONE launch for the whole selection instead of the reference's 12 per token, in one of
 * three forms: a cluster of 1, 2, 4 or 8 blocks per token with the keys in registers, a pivot from the
 * threads' maxima summed through distributed shared memory and the keys that reach it pushed to every
 * block; many tokens at once, a block each that streams its row twice into an index-ordered bitmap; rows
 * longer than 65 536 blocks, one block that re-reads the row, 16 independent loads at a time.
 */
#include <math_constants.h>
#include <string.h>

#include <type_traits>

#include "q4_internal.h"

namespace {

constexpr uint32_t IX_HD = 128;
constexpr uint32_t IX_TK_THREADS = 1024, IX_MAX_KBLK = 512;

/* ---- pool: one warp per block, lane l holds dims l, l+32, l+64, l+96 */
__global__ void __launch_bounds__(128) q4_ix_pool_k(const __half *raw, float *pool, const float *wn, uint32_t ratio,
                                                    uint32_t b0, uint32_t b1, uint32_t n_rot, float base, float eps,
                                                    const int32_t *pp, bool early, bool apart) {
    const uint32_t lane = threadIdx.x & 31u, w = blockIdx.x * 4u + (threadIdx.x >> 5);
    if (apart) q4d_apart_begin();
    else if (!early) q4d_pdl_wait();
    if (pp) {   /* device position: the block this token completes, if any */
        const uint32_t pos = (uint32_t)__ldcg(pp);
        b0 = pos / ratio;
        b1 = (pos + 1u) / ratio;
    }
    const uint32_t b = b0 + w;
    /* the rotation depends on the block alone: a settled position's is taken under the previous kernel's tail */
    float cs[4], sn[4];
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const uint32_t d = lane + 32u * c;
        cs[c] = 1.f;
        sn[c] = 0.f;
        if (b < b1 && (d & ~1u) < n_rot) {
            const uint32_t p = d >> 1;
            const float freq = powf(base, -(float)p / (float)(n_rot / 2u));
            const float ang = (float)(b * ratio) * freq;
            cs[c] = cosf(ang);
            sn[c] = sinf(ang);
        }
    }
    if (early && !apart) q4d_pdl_wait();
    if (b >= b1) {
        if (apart) q4d_apart_end();
        return;
    }
    const __half *src = raw + (size_t)b * ratio * IX_HD;
    float v[4], r[4], g[4] = {1.f, 1.f, 1.f, 1.f};
    if (wn) {
#pragma unroll
        for (int c = 0; c < 4; c++) g[c] = __ldcg(wn + lane + 32u * c);
    }
#pragma unroll
    for (int c = 0; c < 4; c++) {
        float s = 0.f;
        for (uint32_t j = 0; j < ratio; j++) s += __half2float(__ldcg(src + (size_t)j * IX_HD + lane + 32u * c));
        v[c] = __fdiv_rn(s, (float)ratio);
        r[c] = __fmul_rn(v[c], v[c]);
    }
    /* red[d] += red[d + st] for st = 64, 32 is local to the lane; 16 .. 1 are shuffles */
    float a = __fadd_rn(__fadd_rn(r[0], r[2]), __fadd_rn(r[1], r[3]));
#pragma unroll
    for (int st = 16; st > 0; st >>= 1) a = __fadd_rn(a, __shfl_down_sync(0xffffffffu, a, st));
    const float tot = __shfl_sync(0xffffffffu, a, 0);
    const float inv = rsqrtf(__fadd_rn(__fdiv_rn(tot, (float)IX_HD), eps));
#pragma unroll
    for (int c = 0; c < 4; c++) v[c] = __fmul_rn(__fmul_rn(v[c], inv), g[c]);
#pragma unroll
    for (int c = 0; c < 4; c++) {
        const uint32_t d = lane + 32u * c;
        const float other = __shfl_xor_sync(0xffffffffu, v[c], 1);
        /* even dim: x0 * c - x1 * s; odd dim: x0 * s + x1 * c, with (x0, x1) the pair */
        if ((d & ~1u) < n_rot)
            v[c] = (d & 1u) ? __fadd_rn(__fmul_rn(other, sn[c]), __fmul_rn(v[c], cs[c]))
                            : __fsub_rn(__fmul_rn(v[c], cs[c]), __fmul_rn(other, sn[c]));
        pool[(size_t)b * IX_HD + d] = v[c];
    }
    if (apart) q4d_apart_end();
}

/* ---- score: one thread per pooled block, 4 heads = 4 fused-multiply-add chains in dim order.
 * Persistent warps: a warp takes every n-th tile of 32 rows (512 B each), brings the next tile into
 * the other of its two shared-memory buffers with one 16-byte asynchronous copy per lane and row --
 * fully coalesced, 16 KB in flight per warp while the previous tile is being scored -- and every lane
 * walks its own row there.  Rows are 132 floats apart: 16-byte reads of eight consecutive rows fall
 * into eight different bank groups, so the walk is conflict free; the query is read as a broadcast. */
/* Q4_IX_PDL=0 switches it off for the score and selection launches */
bool ix_pdl() {
    static int on = -1;
    if (on < 0) { const char *e = getenv("Q4_IX_PDL"); on = e ? atoi(e) : 1; }
    return on != 0;
}
template <typename K, typename... A>
bool ix_start(const char *what, K kernel, dim3 grid, uint32_t threads, size_t smem, uint32_t cluster, A... args) {
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = g_q4.stream;
    cudaLaunchAttribute at[2];
    unsigned n = 0;
    if (cluster > 1) {
        at[n].id = cudaLaunchAttributeClusterDimension;
        at[n].val.clusterDim.x = cluster;
        at[n].val.clusterDim.y = 1;
        at[n].val.clusterDim.z = 1;
        n++;
    }
    if (ix_pdl()) {
        at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[n].val.programmaticStreamSerializationAllowed = 1;
        n++;
    }
    cfg.attrs = at;
    cfg.numAttrs = n;
    return q4i_launched(q4i_check(cudaLaunchKernelEx(&cfg, kernel, args...), what));
}
constexpr uint32_t SC_ROW_FLOATS = IX_HD + 4, SC_WARPS = 2;
constexpr uint32_t SC_TILE_BYTES = 32u * SC_ROW_FLOATS * sizeof(float);
constexpr uint32_t SC_SMEM = SC_WARPS * 2u * SC_TILE_BYTES + IX_HD * sizeof(float4);
/* SC_EACH: sessions with a pool and a position of their own, while there is room for a block per two tiles of every session; more
 * rows share the blocks (q4_ix_score_batch_k), which costs some counting (score + select, shared out / so: 2 sessions of 512 blocks
 * 6.2 / 4.2 us, of 14 000, almost all the room, 11.7 / 10.7; 8 of 3500 10.5 / 9.6). */
enum { SC_ONE, SC_EACH };
template <int FORM>
__global__ void __launch_bounds__(SC_WARPS * 32) q4_ix_score_k(const float *q, const float *pool, float *score,
                                                               uint32_t n_blocks, uint32_t stride, uint32_t n_head,
                                                               uint32_t pos0, uint32_t ratio, const int32_t *pp,
                                                               const float *const *pools, const int32_t *pos_arr, uint32_t n_sess, bool early) {
    extern __shared__ __align__(16) uint8_t sc_smem[];
    float4 *qs = reinterpret_cast<float4 *>(sc_smem);   /* [dim] = the 4 heads' values (0 for heads that do not exist) */
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t buf0 = (uint32_t)__cvta_generic_to_shared(sc_smem + IX_HD * sizeof(float4)) + warp * 2u * SC_TILE_BYTES;
    /* rows [0, lim) of token t's pool, tiles of 32: first, first + step, .. below n_tiles */
    auto scan = [&](uint32_t t, const float *pool, uint32_t lim, uint32_t first, uint32_t n_tiles, uint32_t step) {
    auto fetch = [&](uint32_t tile, uint32_t which) {
        if (tile < n_tiles) {
            const uint32_t r0 = tile * 32u, rows = min(32u, lim - r0);
            const uint32_t dst = buf0 + which * SC_TILE_BYTES + lane * 16u;
            const float *src = pool + (size_t)r0 * IX_HD + lane * 4u;
            for (uint32_t r = 0; r < rows; r++)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + r * SC_ROW_FLOATS * 4u),
                             "l"(src + (size_t)r * IX_HD) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");   /* one group per call keeps the wait count uniform */
    };
    fetch(first, 0);
    /* the query is staged while the first tile is in flight */
    for (uint32_t d = threadIdx.x; d < IX_HD; d += SC_WARPS * 32u) {
        const float *qt = q + (size_t)t * n_head * IX_HD + d;
        qs[d] = make_float4(qt[0], n_head > 1 ? qt[IX_HD] : 0.f, n_head > 2 ? qt[2 * IX_HD] : 0.f,
                            n_head > 3 ? qt[3 * IX_HD] : 0.f);
    }
    __syncthreads();
    uint32_t which = 0;
    for (uint32_t tile = first; tile < n_tiles; tile += step, which ^= 1u) {
        fetch(tile + step, which ^ 1u);
        asm volatile("cp.async.wait_group 1;" ::: "memory");   /* this tile has landed, the next may be in flight */
        __syncwarp();
        const uint32_t b = tile * 32u + lane;
        if (b < lim) {
            const uint32_t row = buf0 + which * SC_TILE_BYTES + lane * SC_ROW_FLOATS * 4u;
            float d0 = 0.f, d1 = 0.f, d2 = 0.f, d3 = 0.f;
            /* the row is read two steps ahead of the multiply-adds that use it */
            float4 kq[3];
            asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(kq[0].x), "=f"(kq[0].y), "=f"(kq[0].z), "=f"(kq[0].w) : "r"(row));
            asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(kq[1].x), "=f"(kq[1].y), "=f"(kq[1].z), "=f"(kq[1].w) : "r"(row + 16u));
#pragma unroll
            for (uint32_t i = 0; i < IX_HD / 4; i++) {
                if (i + 2 < IX_HD / 4)
                    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];"
                                 : "=f"(kq[(i + 2) % 3].x), "=f"(kq[(i + 2) % 3].y), "=f"(kq[(i + 2) % 3].z), "=f"(kq[(i + 2) % 3].w)
                                 : "r"(row + 16u * (i + 2)));
                const float4 k = kq[i % 3];
                const float4 q0 = qs[4 * i], q1 = qs[4 * i + 1], q2 = qs[4 * i + 2], q3 = qs[4 * i + 3];
                d0 = __fmaf_rn(q0.x, k.x, d0); d1 = __fmaf_rn(q0.y, k.x, d1); d2 = __fmaf_rn(q0.z, k.x, d2); d3 = __fmaf_rn(q0.w, k.x, d3);
                d0 = __fmaf_rn(q1.x, k.y, d0); d1 = __fmaf_rn(q1.y, k.y, d1); d2 = __fmaf_rn(q1.z, k.y, d2); d3 = __fmaf_rn(q1.w, k.y, d3);
                d0 = __fmaf_rn(q2.x, k.z, d0); d1 = __fmaf_rn(q2.y, k.z, d1); d2 = __fmaf_rn(q2.z, k.z, d2); d3 = __fmaf_rn(q2.w, k.z, d3);
                d0 = __fmaf_rn(q3.x, k.w, d0); d1 = __fmaf_rn(q3.y, k.w, d1); d2 = __fmaf_rn(q3.z, k.w, d2); d3 = __fmaf_rn(q3.w, k.w, d3);
            }
            float sc = __fadd_rn(0.f, fmaxf(d0, 0.f));          /* s = 0; s += relu(dot_h) in head order */
            if (n_head > 1) sc = __fadd_rn(sc, fmaxf(d1, 0.f));
            if (n_head > 2) sc = __fadd_rn(sc, fmaxf(d2, 0.f));
            if (n_head > 3) sc = __fadd_rn(sc, fmaxf(d3, 0.f));
            score[(size_t)t * stride + b] = sc;
        }
        __syncwarp();   /* every lane is done with this buffer before the fetch after next refills it */
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    };
    const uint32_t t = blockIdx.y;
    if (!early) q4d_pdl_wait();
    const uint32_t pos = FORM == SC_EACH ? (uint32_t)pos_arr[t] : (pp ? (uint32_t)*pp : pos0) + t;
    const uint32_t n_vis = ratio ? (pos + 1u) / ratio : 0u;
    if (early) q4d_pdl_wait();
    if (FORM == SC_EACH) pool = pools[t];
    if (FORM == SC_EACH || pp) n_blocks = min(n_vis, stride);      /* device position: the bound is derived here */
    const uint32_t lim = min(n_blocks, n_vis);  /* rows to score */
    scan(t, pool, lim, blockIdx.x * SC_WARPS + warp, (lim + 31u) / 32u, gridDim.x * SC_WARPS);
    /* blocks the token cannot see (host-position form only): -1e30 */
    for (uint32_t b = n_vis + blockIdx.x * (SC_WARPS * 32u) + threadIdx.x; b < n_blocks; b += gridDim.x * SC_WARPS * 32u)
        score[(size_t)t * stride + b] = -1.0e30f;
}
/* ---- score of one token over as many rows as one block per SM holds at once (66 304 on 148 SMs: every context of the
 * engine's).  The form above has two parts per warp and three blocks per SM, so of 65 536 rows the last third waits for
 * parts to be walked (1.2 us), and reading shared memory takes longer than HBM: a 16-byte read costs four cycles of what it
 * returns to a warp, the query's broadcasts too, 5 of them per 4 dims of 32 rows.  Here every warp requests all it will need
 * at once, and where a block has more than SC1_SHORT rows a lane walks two (6 reads per 4 dims of 64 rows).  Chunk c of row r
 * lies at c ^ (r & 7): 16-byte reads of eight consecutive rows fall into eight different bank groups, without the padding
 * that would not fit.  Eight steps in line, not 32: the kernel's image is fetched anew by every launch.
 * us, the form above / here: 64 rows 2.57 / 2.4, 4096 2.66 / 2.14, 16 384 4.28 / 4.1, 32 768 6.66 / 5.2, 65 536 9.3 / 8.5.
 * ahead: all blocks but the newest are requested before the wait (q4i_blocks_ahead), under whatever this launch's pooling still
 * waits for: a 262144-token select step 298.5 -> 255 to 272 us from one card to another, the reference host's token 361 -> 340 to 350. */
constexpr uint32_t SC1_WARPS = 7, SC1_ROWS = SC1_WARPS * 64, SC1_SHORT = 128, SC1_SMEM = IX_HD * (uint32_t)sizeof(float4) + SC1_ROWS * IX_HD * (uint32_t)sizeof(float);
/* rows at .. at + 32 R - 1, below r1, by one warp */
template <int R>
__device__ __forceinline__ void sc1_fetch(uint32_t buf, const float *pool, uint32_t at, uint32_t r1) {
    const uint32_t lane = threadIdx.x & 31u, rows = at < r1 ? min(32u * R, r1 - at) : 0u;
    const float *src = pool + (size_t)at * IX_HD + lane * 4u;
    for (uint32_t r = 0; r < rows; r++)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(buf + r * (IX_HD * 4u) + ((lane ^ (r & 7u)) << 4)), "l"(src + (size_t)r * IX_HD) : "memory");
}
template <int R>
__device__ __forceinline__ void sc1_walk(uint32_t buf, const float4 *qs, float *score, uint32_t at, uint32_t r1, uint32_t n_head) {
    const uint32_t lane = threadIdx.x & 31u, row = buf + lane * (IX_HD * 4u), x = lane & 7u;
    auto chunk = [&](uint32_t i, float4 (&k)[R]) {   /* rows lane, lane + 32; stale bytes behind r1 are walked and not stored */
#pragma unroll
        for (int u = 0; u < R; u++)
            asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(k[u].x), "=f"(k[u].y), "=f"(k[u].z), "=f"(k[u].w)
                         : "r"(row + ((i ^ x) << 4) + u * (32u * IX_HD * 4u)) : "memory");
    };
    float d[R][4];
#pragma unroll
    for (int u = 0; u < R; u++) d[u][0] = d[u][1] = d[u][2] = d[u][3] = 0.f;
    float4 k[4][R];   /* a row is read two steps ahead of the multiply-adds that use it */
    chunk(0, k[0]);
    chunk(1, k[1]);
#pragma unroll 8
    for (uint32_t i = 0; i < IX_HD / 4; i++) {
        if (i < IX_HD / 4 - 2) chunk(i + 2u, k[(i + 2u) & 3u]);
        const float4 q0 = qs[4 * i], q1 = qs[4 * i + 1], q2 = qs[4 * i + 2], q3 = qs[4 * i + 3];
        auto step = [&](const float4 qd, float kd, float (&a)[4]) {
            a[0] = __fmaf_rn(qd.x, kd, a[0]); a[1] = __fmaf_rn(qd.y, kd, a[1]); a[2] = __fmaf_rn(qd.z, kd, a[2]); a[3] = __fmaf_rn(qd.w, kd, a[3]);
        };
#pragma unroll
        for (int u = 0; u < R; u++) step(q0, k[i & 3u][u].x, d[u]);
#pragma unroll
        for (int u = 0; u < R; u++) step(q1, k[i & 3u][u].y, d[u]);
#pragma unroll
        for (int u = 0; u < R; u++) step(q2, k[i & 3u][u].z, d[u]);
#pragma unroll
        for (int u = 0; u < R; u++) step(q3, k[i & 3u][u].w, d[u]);
    }
#pragma unroll
    for (int u = 0; u < R; u++) {
        float sc = __fadd_rn(0.f, fmaxf(d[u][0], 0.f));          /* s = 0; s += relu(dot_h) in head order */
        if (n_head > 1) sc = __fadd_rn(sc, fmaxf(d[u][1], 0.f));
        if (n_head > 2) sc = __fadd_rn(sc, fmaxf(d[u][2], 0.f));
        if (n_head > 3) sc = __fadd_rn(sc, fmaxf(d[u][3], 0.f));
        if (at + lane + 32u * u < r1) score[at + lane + 32u * u] = sc;
    }
}
__global__ void __launch_bounds__(SC1_WARPS * 32) q4_ix_score1_k(const float *q, const float *pool, float *score, uint32_t n_blocks, uint32_t stride,
                                                                 uint32_t n_head, uint32_t pos0, uint32_t ratio, const int32_t *pp, bool early, bool ahead) {
    extern __shared__ __align__(16) uint8_t sc_smem[];
    float4 *qs = reinterpret_cast<float4 *>(sc_smem);   /* [dim] = the 4 heads' values (0 for heads that do not exist) */
    const uint32_t warp = threadIdx.x >> 5;
    if (!early) q4d_pdl_wait();
    const uint32_t pos = pp ? (uint32_t)*pp : pos0, n_vis = ratio ? (pos + 1u) / ratio : 0u;
    if (pp) n_blocks = min(n_vis, stride);      /* device position: the bound is derived here */
    const uint32_t lim = min(n_blocks, n_vis), per = (lim + gridDim.x - 1u) / gridDim.x;   /* at most SC1_ROWS */
    const uint32_t r0 = min(blockIdx.x * per, lim), r1 = min(r0 + per, lim);
    const bool two = per > SC1_SHORT;
    const uint32_t at = r0 + warp * (two ? 64u : 32u);
    const uint32_t buf = (uint32_t)__cvta_generic_to_shared(sc_smem + IX_HD * sizeof(float4)) + warp * (64u * IX_HD * 4u);
    if (early && !ahead) q4d_pdl_wait();
    const uint32_t newest = n_vis ? n_vis - 1u : 0u, old = ahead ? min(r1, newest) : r1;
    if (two) sc1_fetch<2>(buf, pool, at, old);
    else sc1_fetch<1>(buf, pool, at, old);
    if (ahead) {
        q4d_pdl_wait();
        if (newest >= at && newest < min(r1, at + (two ? 64u : 32u))) {
            const uint32_t r = newest - at, lane = threadIdx.x & 31u;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(buf + r * (IX_HD * 4u) + ((lane ^ (r & 7u)) << 4)), "l"(pool + (size_t)newest * IX_HD + lane * 4u) : "memory");
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    /* the query is staged while the rows are in flight */
    if (threadIdx.x < IX_HD) {
        const float *qt = q + threadIdx.x;
        qs[threadIdx.x] = make_float4(qt[0], n_head > 1 ? qt[IX_HD] : 0.f, n_head > 2 ? qt[2 * IX_HD] : 0.f, n_head > 3 ? qt[3 * IX_HD] : 0.f);
    }
    __syncthreads();
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    if (at < r1) {
        if (two) sc1_walk<2>(buf, qs, score, at, r1, n_head);
        else sc1_walk<1>(buf, qs, score, at, r1, n_head);
    }
    /* blocks the token cannot see (host-position form only): -1e30 */
    for (uint32_t b = n_vis + blockIdx.x * blockDim.x + threadIdx.x; b < n_blocks; b += gridDim.x * blockDim.x) score[b] = -1.0e30f;
}
/* ---- scores of many sessions, one token and one pool each.  The sessions' rows are counted through and every warp takes an equal
 * share of the whole, which may end in one session and begin in the next.  Bound by HBM as long as shared memory keeps up: a
 * 16-byte read costs four cycles of what it returns to a warp, so a lane walks two rows (six reads per 4 dims of 64 rows; with one
 * row per lane ten), but one where a tile has no more than 32.  A stage is 64 rows x 32 dims, 128 bytes of each row, two in flight
 * per warp behind the one that is read; chunk c of row r lies at c ^ (r & 7).  A few sessions are two to five tiles a warp, and
 * with fewer warps and deeper rings the last, partial one came late.  us from HBM, this kernel alone, six warps of 32-row tiles in
 * two buffers / four warps of six stages / so: 8 sessions up to 131 072 (74 MB) 19.4 / 20.5 / 18.4, of 131 072 27.8 / 27.0 / 26.3,
 * 64 up to 131 072 98.5 / 93.1 / 89.9, of 8000 18.4 / 19.7 / 17.4, 33 up to 30 000 18.5 / 19.7 / 18.6, 12 up to 60 000 15.9 / 16.4 /
 * 16.1, 2 up to 131 072 (16 MB) 9.6 / 10.8 / 10.0. */
constexpr uint32_t SB_WARPS = 8, SB_STAGES = 3, SB_ROWS = 64, SB_CD = 32, SB_STAGE = SB_ROWS * SB_CD * 4u;
constexpr uint32_t SB_SMEM = SB_WARPS * (SB_STAGES * SB_STAGE + IX_HD * (uint32_t)sizeof(float4));
struct SbAt { uint32_t t, row, end, left; const float *pool; };   /* session, rows [row, end) of it, rows of later sessions */
__global__ void __launch_bounds__(SB_WARPS * 32, 1) q4_ix_score_batch_k(const float *q, float *score, uint32_t stride, uint32_t n_head, uint32_t ratio,
                                                                        const float *const *pools, const int32_t *pos_arr, uint32_t n_sess) {
    extern __shared__ __align__(16) uint8_t sc_smem[];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t buf = (uint32_t)__cvta_generic_to_shared(sc_smem) + warp * (SB_STAGES * SB_STAGE);
    float4 *qs = reinterpret_cast<float4 *>(sc_smem + SB_WARPS * SB_STAGES * SB_STAGE) + warp * IX_HD;   /* [dim] = the 4 heads' values */
    q4d_pdl_wait();
    auto rows_of = [&](uint32_t t) -> uint32_t { return min(((uint32_t)pos_arr[t] + 1u) / ratio, stride); };
    /* the first 32 sessions' rows and pools are kept for the search below */
    uint32_t rows = lane < n_sess ? rows_of(lane) : 0u;
    const float *pool = lane < n_sess ? pools[lane] : nullptr;
    uint64_t total = __reduce_add_sync(0xffffffffu, rows);
    for (uint32_t t0 = 32u; t0 < n_sess; t0 += 32u) total += __reduce_add_sync(0xffffffffu, t0 + lane < n_sess ? rows_of(t0 + lane) : 0u);
    const uint32_t w = blockIdx.x * SB_WARPS + warp, n_w = gridDim.x * SB_WARPS;
    const uint64_t share0 = total * w / n_w, share1 = total * (w + 1u) / n_w;
    if (share0 == share1) return;
    /* the session that the share begins in */
    SbAt at = {0u, 0u, 0u, 0u, nullptr};
    uint64_t before = 0;
    for (uint32_t t0 = 0;; t0 += 32u) {
        if (t0) {
            rows = t0 + lane < n_sess ? rows_of(t0 + lane) : 0u;
            pool = t0 + lane < n_sess ? pools[t0 + lane] : nullptr;
        }
        uint32_t incl = rows;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += y;
        }
        const uint32_t here = __ballot_sync(0xffffffffu, before + incl > share0);
        if (here) {
            const int l = __ffs(here) - 1;
            at.t = t0 + (uint32_t)l;
            at.row = (uint32_t)(share0 - before) - __shfl_sync(0xffffffffu, incl - rows, l);
            at.end = min(__shfl_sync(0xffffffffu, rows, l), at.row + (uint32_t)(share1 - share0));
            at.left = (uint32_t)(share1 - share0) - (at.end - at.row);
            at.pool = reinterpret_cast<const float *>(__shfl_sync(0xffffffffu, (unsigned long long)pool, l));
            break;
        }
        before += __shfl_sync(0xffffffffu, incl, 31);
    }
    auto next = [&](SbAt &a) {   /* the tile after; row == end: none */
        a.row = min(a.row + SB_ROWS, a.end);
        while (a.row == a.end && a.left) {
            a.t++;
            a.row = 0;
            a.end = min(rows_of(a.t), a.left);
            a.left -= a.end;
            a.pool = pools[a.t];
        }
    };
    SbAt ahead = at;
    uint32_t chunk = 0, fill = 0;
    auto fetch = [&]() {
        const uint32_t rows = min(SB_ROWS, ahead.end - ahead.row), r0 = lane >> 3, c = lane & 7u;
        const float *src = ahead.pool + (size_t)(ahead.row + r0) * IX_HD + chunk * SB_CD + c * 4u;
        const uint32_t dst = buf + fill * SB_STAGE + r0 * (SB_CD * 4u);
#pragma unroll
        for (uint32_t j = 0; j < SB_ROWS / 4u; j++)
            if (4u * j + r0 < rows)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + j * (SB_CD * 16u) + ((c ^ ((4u * j + r0) & 7u)) << 4)), "l"(src + (size_t)j * (4u * IX_HD)) : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");   /* one group per call keeps the wait count uniform */
        if (++fill == SB_STAGES) fill = 0;
        if (++chunk == IX_HD / SB_CD) {
            chunk = 0;
            next(ahead);
        }
    };
#pragma unroll 1
    for (uint32_t i = 0; i < SB_STAGES - 1u; i++) fetch();
    uint32_t stage = 0, of = 0xffffffffu;
    while (at.row < at.end) {
        if (at.t != of) {   /* another query */
            of = at.t;
            __syncwarp();
            const float *qt = q + (size_t)of * n_head * IX_HD;
            for (uint32_t d = lane; d < IX_HD; d += 32u)
                qs[d] = make_float4(qt[d], n_head > 1 ? qt[IX_HD + d] : 0.f, n_head > 2 ? qt[2 * IX_HD + d] : 0.f, n_head > 3 ? qt[3 * IX_HD + d] : 0.f);
        }
        auto walk = [&](auto r) {
            constexpr int R = decltype(r)::value;   /* rows per lane */
            float d[R][4];
#pragma unroll
            for (int u = 0; u < R; u++) d[u][0] = d[u][1] = d[u][2] = d[u][3] = 0.f;
#pragma unroll 1
            for (uint32_t c = 0; c < IX_HD / SB_CD; c++) {
                asm volatile("cp.async.wait_group %0;" ::"n"(SB_STAGES - 2u) : "memory");
                __syncwarp();   /* this stage has landed, and every lane is done with the one before, which is filled again */
                fetch();
                const uint32_t row = buf + stage * SB_STAGE + lane * (SB_CD * 4u), x = lane & 7u;
                if (++stage == SB_STAGES) stage = 0;
                auto read = [&](uint32_t i, float4 (&k)[R]) {   /* rows lane, lane + 32; stale bytes behind the end are walked and not stored */
#pragma unroll
                    for (int u = 0; u < R; u++)
                        asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(k[u].x), "=f"(k[u].y), "=f"(k[u].z), "=f"(k[u].w)
                                     : "r"(row + ((i ^ x) << 4) + u * (32u * SB_CD * 4u)));   /* no clobber: the query's reads may go ahead */
                };
                float4 k[3][R];
                read(0, k[0]);
                read(1, k[1]);
                const float4 *qc = qs + c * SB_CD;
#pragma unroll
                for (uint32_t i = 0; i < SB_CD / 4u; i++) {
                    if (i + 2u < SB_CD / 4u) read(i + 2u, k[(i + 2u) % 3u]);
                    const float4 q0 = qc[4 * i], q1 = qc[4 * i + 1], q2 = qc[4 * i + 2], q3 = qc[4 * i + 3];
                    auto step = [&](const float4 qd, float kd, float (&a)[4]) {
                        a[0] = __fmaf_rn(qd.x, kd, a[0]); a[1] = __fmaf_rn(qd.y, kd, a[1]); a[2] = __fmaf_rn(qd.z, kd, a[2]); a[3] = __fmaf_rn(qd.w, kd, a[3]);
                    };
#pragma unroll
                    for (int u = 0; u < R; u++) step(q0, k[i % 3u][u].x, d[u]);
#pragma unroll
                    for (int u = 0; u < R; u++) step(q1, k[i % 3u][u].y, d[u]);
#pragma unroll
                    for (int u = 0; u < R; u++) step(q2, k[i % 3u][u].z, d[u]);
#pragma unroll
                    for (int u = 0; u < R; u++) step(q3, k[i % 3u][u].w, d[u]);
                }
            }
#pragma unroll
            for (int u = 0; u < R; u++) {
                float sc = __fadd_rn(0.f, fmaxf(d[u][0], 0.f));          /* s = 0; s += relu(dot_h) in head order */
                if (n_head > 1) sc = __fadd_rn(sc, fmaxf(d[u][1], 0.f));
                if (n_head > 2) sc = __fadd_rn(sc, fmaxf(d[u][2], 0.f));
                if (n_head > 3) sc = __fadd_rn(sc, fmaxf(d[u][3], 0.f));
                const uint32_t b = at.row + lane + 32u * u;
                if (b < at.end) score[(size_t)at.t * stride + b] = sc;
            }
        };
        if (at.end - at.row > 32u) walk(std::integral_constant<int, 2>());
        else walk(std::integral_constant<int, 1>());
        next(at);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}
/* ---- score for many tokens over one pool (a prompt's slice).  The scan above reads the pool once per token, 17 GB
 * through L2 for 512 tokens x 32 768 blocks (1.67 ms).  This form is a tiled fp32 product on the FMA pipe (the
 * result is defined as one fused multiply-add per dim in dim order, which rules the tensor cores out): 32 tokens x 4
 * heads against 64 M pooled blocks per tile, 8 x 4 M chains per thread -- two tokens' four heads, so the relu sum over
 * heads stays in the thread.  Both operands lie dim by dim in shared memory (a chunk of 32 dims is transposed on its way
 * in, through registers; the columns of dim group c are stored at column ^ 4 (c & 7), so that neither the four-byte stores
 * nor the 16-byte reads meet in a bank), two neighbouring blocks' chains share an instruction (fma.rn.f32x2, one rounding
 * per chain), and the fragments of the next dim are requested under the products of this one, all 32 dims in line.
 * 512 tokens x 32 768 blocks, us, all with the same bits:
 *   one chain per instruction, rows of 4 dims from both operands, cp.async            370  (the FMA pipe 66 % busy: 0.44
 *                                              warps per issue held up in dispatch, by the register file's ports)
 *   two chains per instruction, dim by dim, requested in the order of the rows        347  (16 bytes of 32 rows per request)
 *   requested in whole 128-byte pieces of four rows                                   331
 *   every dim in line (4 dims in line 324, 8 321), half a chunk in registers at once  294
 * The FMA pipe alone takes 268 (64.1 TFLOP/s of such products out of registers).  Reading the queries as pairs ready in shared
 * memory instead of doubling them by moves: 407, bound by what shared memory returns.  Two blocks of 128 threads: 314. */
constexpr uint32_t SM_TOK = 32, SM_ROWS = SM_TOK * 4, SM_THREADS = 256, SM_CD = 32, SM_CHUNKS = IX_HD / SM_CD;
template <uint32_t M>
constexpr uint32_t sm_smem() { return ((IX_HD + 1u) * SM_ROWS + 2u * (SM_CD + 1u) * 64u * M) * (uint32_t)sizeof(float); }   /* a row more each: read ahead, not used */
__device__ __forceinline__ uint64_t ix_pair(float a, float b) {
    uint64_t v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
    return v;
}
__device__ __forceinline__ float2 ix_unpair(uint64_t v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}
__device__ __forceinline__ uint64_t ix_fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
template <uint32_t M>
__global__ void __launch_bounds__(SM_THREADS, 1) q4_ix_score_mt_k(const float *q, const float *pool, float *score, uint32_t n_tok,
                                                                 uint32_t n_blocks, uint32_t stride, uint32_t n_head,
                                                                 uint32_t pos0, uint32_t ratio) {
    constexpr uint32_t COLS = 64u * M, BUF = (SM_CD + 1u) * COLS;
    extern __shared__ __align__(16) float sm_tiles[];   /* queries [dim][row] | pool, two chunks [dim][column ^ 4 (dim / 4 % 8)] */
    float *sk = sm_tiles + (IX_HD + 1u) * SM_ROWS;
    const uint32_t tid = threadIdx.x;
    const uint32_t ty = tid >> 4, tc = tid & 15u;       /* tokens 2 ty, 2 ty + 1; pooled blocks 4 tc + 64 m .. + 3 */
    const uint32_t lr = tid >> 3, lc = tid & 7u;        /* staging: rows lr + 32 k, dims 4 lc .. + 3 of a chunk */
    const uint32_t col_tiles = (n_blocks + COLS - 1u) / COLS, tok_tiles = (n_tok + SM_TOK - 1u) / SM_TOK;
    const uint64_t total = (uint64_t)col_tiles * tok_tiles;
    const uint32_t first = (uint32_t)(total * blockIdx.x / gridDim.x), last = (uint32_t)(total * (blockIdx.x + 1u) / gridDim.x);
    const bool vec = ((uintptr_t)score & 15u) == 0u && (stride & 3u) == 0u;
    auto visible = [&](uint32_t tok) { return (pos0 + tok + 1u) / ratio; };
    float4 stage[M];
    /* rows of a tile that no token of the group can see are not read: they need not exist yet */
    auto request = [&](uint32_t it, uint32_t half) {
        const uint32_t tile = first + it / SM_CHUNKS;
        uint32_t lim = 0, c0 = 0;
        if (tile < last) {
            c0 = (tile % col_tiles) * COLS + half * (COLS / 2u);
            lim = min(visible(min((tile / col_tiles + 1u) * SM_TOK, n_tok) - 1u), n_blocks);
        }
        const float *src = pool + (size_t)(c0 + lr) * IX_HD + (it % SM_CHUNKS) * SM_CD + 4u * lc;
#pragma unroll
        for (uint32_t k = 0; k < M; k++) {
            stage[k] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (c0 + lr + 32u * k < lim) stage[k] = *reinterpret_cast<const float4 *>(src + (size_t)(32u * k) * IX_HD);
        }
    };
    auto put = [&](uint32_t it, uint32_t half) {
        float *dst = sk + (it & 1u) * BUF + 4u * lc * COLS + half * (COLS / 2u) + (lr ^ (4u * lc));
#pragma unroll
        for (uint32_t k = 0; k < M; k++) {
            dst[32u * k] = stage[k].x;
            dst[COLS + 32u * k] = stage[k].y;
            dst[2u * COLS + 32u * k] = stage[k].z;
            dst[3u * COLS + 32u * k] = stage[k].w;
        }
    };
    q4d_pdl_wait();
    uint32_t have = 0xffffffffu, it = 0;
    request(0, 0);
    put(0, 0);
    request(0, 1);
    put(0, 1);
    for (uint32_t tile = first; tile < last; tile++) {
        const uint32_t group = tile / col_tiles, c0 = (tile % col_tiles) * COLS;
        if (group != have) {
            __syncthreads();   /* everyone is done with the queries of the group before */
            for (uint32_t i = tid; i < SM_ROWS * 32u; i += SM_THREADS) {
                const uint32_t r = i % SM_ROWS, c = i / SM_ROWS, tok = group * SM_TOK + (r >> 2), h = r & 3u;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (tok < n_tok && h < n_head) v = *reinterpret_cast<const float4 *>(q + ((size_t)tok * n_head + h) * IX_HD + c * 4u);
                float *dst = sm_tiles + 4u * c * SM_ROWS + r;
                dst[0] = v.x; dst[SM_ROWS] = v.y; dst[2u * SM_ROWS] = v.z; dst[3u * SM_ROWS] = v.w;
            }
            have = group;
        }
        uint64_t acc[8][2 * M];
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
            for (uint32_t j = 0; j < 2 * M; j++) acc[i][j] = 0ull;
#pragma unroll 1
        for (uint32_t ch = 0; ch < SM_CHUNKS; ch++, it++) {
            __syncthreads();   /* chunk `it` is in; everyone is done with the buffer that chunk it + 1 goes to */
            request(it + 1u, 0);
            const float *qa = sm_tiles + ch * SM_CD * SM_ROWS + ty * 8u, *kb = sk + (it & 1u) * BUF;
            float4 an[2], bn[M];
            an[0] = *reinterpret_cast<const float4 *>(qa);
            an[1] = *reinterpret_cast<const float4 *>(qa + 4);
#pragma unroll
            for (uint32_t m = 0; m < M; m++) bn[m] = *reinterpret_cast<const float4 *>(kb + 64u * m + 4u * tc);
#pragma unroll
            for (uint32_t d = 0; d < SM_CD; d++) {
                const float a[8] = {an[0].x, an[0].y, an[0].z, an[0].w, an[1].x, an[1].y, an[1].z, an[1].w};
                uint64_t b[2 * M];
#pragma unroll
                for (uint32_t m = 0; m < M; m++) {
                    b[2 * m] = ix_pair(bn[m].x, bn[m].y);
                    b[2 * m + 1] = ix_pair(bn[m].z, bn[m].w);
                }
                an[0] = *reinterpret_cast<const float4 *>(qa + (d + 1u) * SM_ROWS);
                an[1] = *reinterpret_cast<const float4 *>(qa + (d + 1u) * SM_ROWS + 4);
#pragma unroll
                for (uint32_t m = 0; m < M; m++)
                    bn[m] = *reinterpret_cast<const float4 *>(kb + (d + 1u) * COLS + 64u * m + ((4u * tc) ^ ((d + 1u) & 28u)));
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const uint64_t x = ix_pair(a[i], a[i]);
#pragma unroll
                    for (uint32_t j = 0; j < 2 * M; j++) acc[i][j] = ix_fma2(x, b[j], acc[i][j]);
                }
                if (d == SM_CD / 2u) {
                    put(it + 1u, 0);
                    request(it + 1u, 1);
                }
            }
            put(it + 1u, 1);
        }
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const uint32_t tok = group * SM_TOK + 2u * ty + u;
            if (tok >= n_tok) continue;
            const uint32_t n_vis = visible(tok);
            float *row = score + (size_t)tok * stride;
#pragma unroll
            for (uint32_t m = 0; m < M; m++) {
                const uint32_t c = c0 + 4u * tc + 64u * m;
                float sc[4];
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    /* heads that do not exist have zero queries: their relu adds exactly nothing */
                    float v = 0.f;
#pragma unroll
                    for (int h = 0; h < 4; h++) {
                        const float2 f = ix_unpair(acc[4 * u + h][2 * m + (e >> 1)]);
                        v = __fadd_rn(v, fmaxf(e & 1 ? f.y : f.x, 0.f));
                    }
                    sc[e] = c + e < n_vis ? v : -1.0e30f;
                }
                if (vec && c + 3u < n_blocks) {
                    *reinterpret_cast<float4 *>(row + c) = make_float4(sc[0], sc[1], sc[2], sc[3]);
                } else {
#pragma unroll
                    for (int e = 0; e < 4; e++)
                        if (c + e < n_blocks) row[c + e] = sc[e];
                }
            }
        }
    }
}
/* Estimated ns of the product with tiles of 64 M blocks, and of the scan; fitted to 2 .. 512 tokens over 64 .. 65 536 blocks,
 * within 10 % where the forms are close.  Product: a tile takes a time of its own however few of its 32 tokens exist (us,
 * narrow / wide tiles: 32 tokens over 8192 blocks 16.6 / 25.6, 33 over 16 384 28.5 / 26.3, 512 over 65 536 667 / 602; with
 * tiles of the earlier form 18.7, 31.0 and 726). */
uint64_t score_mt_ns(uint32_t n_tok, uint32_t n_blocks, uint32_t m) {
    const uint64_t tiles = (uint64_t)((n_blocks + 64u * m - 1u) / (64u * m)) * ((n_tok + SM_TOK - 1u) / SM_TOK);
    return (m == 4u ? 4300u : 5000u) + (tiles + (uint64_t)g_q4.sm_count - 1u) / (uint64_t)g_q4.sm_count * (m == 4u ? 21000u : 11750u);
}
/* Scan: tiles of 32 blocks a warp takes one after the other, and again (with the card nearly to itself) where the tokens'
 * grids do not fit at once: 4 tokens over 65 536 blocks 25.0 us, 5 (445 blocks of 444) 40.3, 8 62.7, 12 62.5. */
uint64_t score_scan_ns(uint32_t n_tok, uint32_t n_blocks) {
    const uint32_t all = (uint32_t)g_q4.sm_count * 3u, need = (n_blocks + SC_WARPS * 32u - 1u) / (SC_WARPS * 32u);
    uint32_t gx = (all + n_tok - 1u) / n_tok;
    if (gx > need) gx = need;
    const uint64_t per_warp = ((n_blocks + 31u) / 32u + gx * SC_WARPS - 1u) / (gx * SC_WARPS), waves = ((uint64_t)gx * n_tok + all - 1u) / all;
    return 3000u + per_warp * (2150u + (waves - 1u) * 1250u);
}
template <uint32_t M>
bool score_mt_launch(const float *q, const float *pool, float *score, uint32_t n_tok, uint32_t n_blocks, uint32_t stride, uint32_t n_head,
                     uint32_t pos0, uint32_t ratio) {
    static bool done = false;
    if (!done && !q4i_check(cudaFuncSetAttribute(q4_ix_score_mt_k<M>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_smem<M>()),
                            "qsa_score smem attribute"))
        return false;
    done = true;
    const uint64_t tiles = (uint64_t)((n_blocks + 64u * M - 1u) / (64u * M)) * ((n_tok + SM_TOK - 1u) / SM_TOK);
    const uint32_t grid = (uint32_t)(tiles < (uint64_t)g_q4.sm_count ? tiles : (uint64_t)g_q4.sm_count);
    return ix_start("qsa_score launch", q4_ix_score_mt_k<M>, dim3(grid), SM_THREADS, sm_smem<M>(), 1u, q, pool, score, n_tok, n_blocks, stride,
                    n_head, pos0, ratio);
}
template <int FORM>
bool score_start(dim3 grid, const float *q, const float *pool, float *score, uint32_t n_tok, uint32_t n_blocks, uint32_t stride,
                 uint32_t n_head, uint32_t pos0, uint32_t ratio, const int32_t *pp, const float *const *pools, const int32_t *pos_arr) {
    static bool done = false;
    if (!done) {
        if (!q4i_check(cudaFuncSetAttribute(q4_ix_score_k<FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SC_SMEM),
                       "qsa_score smem attribute"))
            return false;
        done = true;
    }
    return ix_start("qsa_score launch", q4_ix_score_k<FORM>, grid, SC_WARPS * 32u, SC_SMEM, 1u, q, pool, score, n_blocks, stride, n_head, pos0, ratio, pp,
                    pools, pos_arr, n_tok, FORM == SC_ONE && ix_pdl() && (!pp || q4i_settled(g_q4.pos_written)));
}
/* persistent grid: 3 blocks of 2 warps per SM share 227 KB; fewer when the rows are short */
bool score_launch(const float *q, const float *pool, float *score, uint32_t n_tok, uint32_t n_blocks, uint32_t stride,
                  uint32_t n_head, uint32_t pos0, uint32_t ratio, const int32_t *pp, const float *const *pools, const int32_t *pos_arr) {
    const uint32_t all = (uint32_t)g_q4.sm_count * 3u, need = ((pp || pools ? stride : n_blocks) + SC_WARPS * 32u - 1u) / (SC_WARPS * 32u);
    if (pools && (uint64_t)need * n_tok > all) {
        static bool done = false;
        if (!done && !q4i_check(cudaFuncSetAttribute(q4_ix_score_batch_k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SB_SMEM), "qsa_score smem attribute")) return false;
        done = true;
        return ix_start("qsa_score launch", q4_ix_score_batch_k, dim3((unsigned)g_q4.sm_count), SB_WARPS * 32u, SB_SMEM, 1u, q, score, stride, n_head, ratio, pools, pos_arr, n_tok);
    }
    if (pools) return score_start<SC_EACH>(dim3(need, n_tok), q, pool, score, n_tok, n_blocks, stride, n_head, pos0, ratio, pp, pools, pos_arr);
    const uint32_t rows = pp ? stride : n_blocks;
    if (n_tok == 1 && rows <= (uint32_t)g_q4.sm_count * SC1_ROWS) {
        static bool done = false;
        if (!done && !q4i_check(cudaFuncSetAttribute(q4_ix_score1_k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SC1_SMEM), "qsa_score smem attribute"))
            return false;
        done = true;
        const bool early = ix_pdl() && (!pp || q4i_settled(g_q4.pos_written));
        const uint32_t fill = (rows + 31u) / 32u, grid = fill < (uint32_t)g_q4.sm_count ? (fill ? fill : 1u) : (uint32_t)g_q4.sm_count;
        /* a position of the host's need not be the word's: what pooling writes there may be any of the blocks */
        const bool ahead = early && q4i_blocks_ahead(pool, (uint64_t)rows * IX_HD * 4u, pp ? ratio : 0u);
        g_q4.n_ahead += ahead;
        return ix_start("qsa_score launch", q4_ix_score1_k, dim3(grid), SC1_WARPS * 32u, SC1_SMEM, 1u, q, pool, score, n_blocks, stride, n_head, pos0, ratio,
                        pp, early, ahead);
    }
    uint32_t gx = n_tok > 1 ? (all + n_tok - 1u) / n_tok : all;
    if (gx > need) gx = need;
    if (gx < 1) gx = 1;
    return score_start<SC_ONE>(dim3(gx, n_tok), q, pool, score, n_tok, n_blocks, stride, n_head, pos0, ratio, pp, nullptr, nullptr);
}

/* ---- selection: one block per token */
__device__ __forceinline__ uint32_t ix_key(float f) {   /* order-preserving uint of a float (:7464-7467) */
    uint32_t u;
    /* bits out of the compiler's sight: it turned a conversion's  u | sign  into -|f|, which leaves a NaN its sign */
    asm("mov.b32 %0, %1;" : "=r"(u) : "f"(f));
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
/* exclusive prefix sum of one value per thread over the block; returns the block total */
__device__ uint32_t block_excl_scan(uint32_t v, uint32_t &excl, uint32_t *warp_tot /* [33] shared */) {
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    __syncthreads();   /* warp_tot may still be read from the previous scan */
    if (lane == 31) warp_tot[w] = x;
    __syncthreads();
    if (w == 0) {
        uint32_t t = lane < IX_TK_THREADS / 32 ? warp_tot[lane] : 0u, s = t;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= (uint32_t)o) s += y;
        }
        warp_tot[lane] = s - t;
        if (lane == 31) warp_tot[32] = s;
    }
    __syncthreads();
    excl = warp_tot[w] + x - v;
    return warp_tot[32];
}

/* A warp walks its contiguous share of the row in batches of IX_BATCH x 32 keys: the IX_BATCH loads of
 * a batch are independent (one memory round trip per batch instead of one per key), lane l of load k
 * holds index base + 32 k + l, so (batch, k, lane) is ascending index order inside the warp. */
constexpr uint32_t IX_BATCH = 16;
template <typename F>
__device__ __forceinline__ void ix_walk(const float *row, uint32_t n_vis, uint32_t per_warp, F f) {
    const uint32_t lane = threadIdx.x & 31u, w0 = (threadIdx.x >> 5) * per_warp;
    const uint32_t w1 = min(w0 + per_warp, n_vis);
    for (uint32_t base = w0; base < w1; base += 32u * IX_BATCH) {
        uint32_t key[IX_BATCH];
#pragma unroll
        for (uint32_t k = 0; k < IX_BATCH; k++) {
            const uint32_t b = base + 32u * k + lane;
            key[k] = b < w1 ? ix_key(__ldcg(row + b)) : 0u;
        }
#pragma unroll
        for (uint32_t k = 0; k < IX_BATCH; k++) {
            const uint32_t b = base + 32u * k + lane;
            f(b, key[k], b < w1);
        }
    }
}

__global__ void __launch_bounds__(IX_TK_THREADS) q4_ix_topk1_k(const float *score, int32_t *sel, uint32_t stride,
                                                              uint32_t k_blk, uint32_t ratio, uint32_t pos0,
                                                              uint32_t width, const int32_t *pp, const int32_t *pos_arr) {
    __shared__ uint32_t hist[256], warp_tot[33], st_prefix, st_hi;
    __shared__ int32_t chosen[IX_MAX_KBLK];
    const uint32_t t = blockIdx.x, tx = threadIdx.x, lane = tx & 31u;
    const uint32_t pos = pos_arr ? (uint32_t)pos_arr[t] : (pp ? (uint32_t)*pp : pos0) + t;
    const uint32_t n_vis = ratio ? (pos + 1u) / ratio : 0u;
    const uint32_t need = n_vis < k_blk ? n_vis : k_blk;
    const float *row = score + (size_t)t * stride;
    int32_t *out = sel + (size_t)t * width;
    if (need == n_vis) {   /* every complete block fits: the dense prefix */
        for (uint32_t w = tx; w < width; w += IX_TK_THREADS) out[w] = w <= pos ? (int32_t)w : -1;
        return;
    }
    /* contiguous share of each of the 32 warps, a whole number of batches */
    const uint32_t per_warp = ((n_vis + 31u) / 32u + 32u * IX_BATCH - 1u) / (32u * IX_BATCH) * (32u * IX_BATCH);

    /* exact need-th largest key: 4 passes over the 8-bit digits, most significant first */
    if (tx == 0) { st_prefix = 0u; st_hi = 0u; }
    for (int p = 0; p < 4; p++) {
        if (tx < 256) hist[tx] = 0u;
        __syncthreads();
        const uint32_t sh = 24u - 8u * p, pre = st_prefix;
        ix_walk(row, n_vis, per_warp, [&](uint32_t, uint32_t u, bool live) {
            const bool in = live && (p == 0 || (u >> (sh + 8u)) == pre);
            const uint32_t bin = (u >> sh) & 255u;
            /* Keys often share a digit (the leading digits of non-negative scores, relu zeros, padding):
             * when every participating lane has the same bin one lane adds the count; otherwise the bins
             * are spread and each lane adds for itself. */
            const uint32_t m = __ballot_sync(0xffffffffu, in);
            if (m) {
                const uint32_t first = __shfl_sync(0xffffffffu, bin, __ffs(m) - 1);
                if (__all_sync(0xffffffffu, !in || bin == first)) {
                    if (lane == (uint32_t)(__ffs(m) - 1)) atomicAdd(&hist[first], (uint32_t)__popc(m));
                } else if (in) {
                    atomicAdd(&hist[bin], 1u);
                }
            }
        });
        __syncthreads();
        if (tx < 32) {
            /* digit = the highest bin whose count, added to those above it, reaches the target: lane l owns
             * bins 255 - 8 l .. 248 - 8 l, a warp scan gives the count above each lane's bins */
            const uint32_t target = need - st_hi;
            uint32_t c[8], tot = 0;
#pragma unroll
            for (int j = 0; j < 8; j++) { c[j] = hist[255 - 8 * (int)lane - j]; tot += c[j]; }
            uint32_t incl = tot;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= (uint32_t)o) incl += y;
            }
            uint32_t above = incl - tot;
            if (above < target && incl >= target) {   /* exactly one lane */
                uint32_t dg = 0;
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    if (above + c[j] >= target) { dg = 255u - 8u * lane - (uint32_t)j; break; }
                    above += c[j];
                }
                st_hi += above;
                st_prefix = (pre << 8) | dg;
            }
        }
        __syncthreads();
    }
    const uint32_t thr = st_prefix, n_gt = st_hi;   /* keys above the threshold: n_gt < need <= n_gt + ties */

    /* ordered compaction: blocks above the threshold in ascending index order, then threshold ties in
     * ascending index order until `need` is full.  Per-warp counts, a scan over the warps, then ranks
     * by ballots. */
    uint32_t ng = 0, ne = 0;
    ix_walk(row, n_vis, per_warp, [&](uint32_t, uint32_t u, bool live) {
        ng += __popc(__ballot_sync(0xffffffffu, live && u > thr));
        ne += __popc(__ballot_sync(0xffffffffu, live && u == thr));
    });
    uint32_t og, oe;
    (void)block_excl_scan(lane == 0 ? ng : 0u, og, warp_tot);
    (void)block_excl_scan(lane == 0 ? ne : 0u, oe, warp_tot);
    og = __shfl_sync(0xffffffffu, og, 0);
    oe = __shfl_sync(0xffffffffu, oe, 0);
    const uint32_t lt = (1u << lane) - 1u;
    ix_walk(row, n_vis, per_warp, [&](uint32_t b, uint32_t u, bool live) {
        const bool gt = live && u > thr, eq = live && u == thr;
        const uint32_t mg = __ballot_sync(0xffffffffu, gt), me = __ballot_sync(0xffffffffu, eq);
        if (gt) {
            const uint32_t at = og + __popc(mg & lt);
            if (at < IX_MAX_KBLK) chosen[at] = (int32_t)b;
        } else if (eq) {
            const uint32_t at = n_gt + oe + __popc(me & lt);
            if (at < need) chosen[at] = (int32_t)b;
        }
        og += __popc(mg);
        oe += __popc(me);
    });
    __syncthreads();
    const uint32_t ncs = need * ratio;
    for (uint32_t w = tx; w < width; w += IX_TK_THREADS) {
        int32_t v;
        if (w < ncs) {
            const uint32_t i = w / ratio, j = w - i * ratio;
            v = (int32_t)((uint32_t)chosen[i] * ratio + j);
        } else {
            const uint32_t tail = n_vis * ratio + (w - ncs);
            v = tail <= pos ? (int32_t)tail : -1;
        }
        out[w] = v;
    }
}

/* ---- selection with the keys in registers (rows of up to 65 536 pooled blocks = ctx 262 144): a cluster of
 * NB = 1, 2, 4 or 8 blocks (8192 keys each), 8 keys per thread; block r, step i, thread t holds index 8192 r + 1024 i + t.
 * Bound by latency and by issue: 32 warps share an SM's four schedulers, so every instruction per key is paid for eight times,
 * and what keeps the chain short is that all keys are looked at twice only.
 *   pivot    the digit (12 bits: sign, exponent, 3 mantissa bits) of the need-th largest among the threads' own maxima: at least
 *            `need` keys reach it, and not many more than that do (8192 normal scores: 820 for 512).  A thread's keys are 1024
 *            apart, so that a run of high scores is many threads' maxima.  One count per thread instead of eight.  In a cluster
 *            every block adds its occupied bins to EVERY block's sum: no read-back after the meeting.
 *   collect  the keys that reach it into shared memory; in a cluster to every block, which then finishes alone.
 *   finish   one count of the collected keys by the next 12 bits (bins of 2^12 from the pivot's edge on), and the few in the
 *            threshold's bin against one another.  Two cluster meetings after the launch wait (one block: none).
 *   emit     every chosen key finds its place in the list from a bitmap of the block's keys.
 * With the first digit counted over all keys, the threshold bin's keys collected by ballots, and two more passes of ballots
 * over all keys for the list, a selection took 6.7 us of one block (8192 normal keys, a chain of such launches) and 9.4 of eight
 * (65 536); now 5.3 and 6.7.
 *   wide     where the pivot's digit is many keys': those above it are collected, and the blocks tell one another in the same
 *            meeting how many are at it, the least and the largest of them and their next digits.  So rows of ties need no more
 *            meetings (all zeros 8.1 and 10.8 us with every digit counted, now 5.3 and 6.9; a row whose 560 keys above zero are
 *            enough 7.95 / 7.3; with the pivot and then every digit 15.9).  Keys that differ behind their first 12 bits are
 *            collected by their first 24 (1000 +- 0.5: 6.8 / 7.6, 10.8 / 10.4), and only where 1500 share 24 are the last 8
 *            counted (7.3 / 8.7, 11.3 / 11.4).
 * What a row of the usual kind does not need stands behind the end of its list: 0.1 to 0.2 us of 6 are instruction fetches. */
constexpr uint32_t TKC_KPT = 8, TKC_KEYS = IX_TK_THREADS * TKC_KPT, TKC_MAX_ROW = 8 * TKC_KEYS;
constexpr uint32_t TK_BINS = 4096, TK_B1 = 20, TK_B2 = 8;   /* digits: bits 31..20, 19..8, 7..0 */
constexpr uint32_t TK_B2F = 12;   /* bits of a bin of collected keys */
constexpr uint32_t TKC_ROUNDS = 6;                         /* of telling, at most: twice by the pivot and by the threshold's digit, once by its next one and behind its last */
constexpr uint32_t TKC_NEAR = 32;                          /* keys of the threshold's bin that are compared with one another */
__device__ __forceinline__ uint32_t tkc_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
template <uint32_t NB>
__device__ __forceinline__ void tkc_sync() {
    if (NB == 1) __syncthreads();
    else asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t tkc_remote(const void *p, uint32_t rank) {
    uint32_t a = (uint32_t)__cvta_generic_to_shared(p), r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void tkc_st(uint32_t ra, uint32_t v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(ra), "r"(v) : "memory");
}
__device__ __forceinline__ void tkc_red_add(uint32_t ra, uint32_t v) {
    asm volatile("red.relaxed.cluster.shared::cluster.add.u32 [%0], %1;" ::"r"(ra), "r"(v) : "memory");
}
struct TkPick { uint32_t digit, above, cnt; };   /* the digit that holds the target-th key from the top, keys above it, keys in it */
/* from TK_BINS counts, by the whole block (two block barriers); `tot` and `st` are scratch of the block */
template <uint32_t NT>
__device__ __forceinline__ TkPick tk_pick(const uint32_t *hist, uint32_t target, uint32_t *tot /* [32] */, TkPick *st) {
    constexpr uint32_t PER = TK_BINS / NT;
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5, top = TK_BINS - 1u - PER * threadIdx.x;
    static_assert(PER % 4 == 0, "whole 16-byte words of counts per thread: a count at a time they met in PER-way bank conflicts");
    uint32_t c[PER], sum = 0;
#pragma unroll
    for (uint32_t j = 0; j < PER; j += 4) {
        const uint4 x = *reinterpret_cast<const uint4 *>(hist + top - j - 3u);
        c[j] = x.w; c[j + 1] = x.z; c[j + 2] = x.y; c[j + 3] = x.x;
        sum += (x.x + x.y) + (x.z + x.w);
    }
    const uint32_t of_warp = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0) tot[w] = of_warp;
    __syncthreads();
    const uint32_t mine = lane < NT / 32 ? tot[lane] : 0u;
    uint32_t above = __reduce_add_sync(0xffffffffu, lane < w ? mine : 0u);
    if (above < target && above + of_warp >= target) {   /* one warp, which alone works out where in its bins */
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += y;
        }
        above += incl - sum;
        if (above < target && above + sum >= target) {   /* one thread */
#pragma unroll
            for (uint32_t j = 0; j < PER; j++) {
                if (above + c[j] >= target) { st->digit = top - j; st->above = above; st->cnt = c[j]; break; }
                above += c[j];
            }
        }
    }
    __syncthreads();
    return *st;
}
/* the same over 256 counts; every warp works it out for itself, no barrier */
__device__ __forceinline__ TkPick tk_pick256(const uint32_t *hist, uint32_t target) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t c[8], sum = 0;
#pragma unroll
    for (int j = 0; j < 8; j++) { c[j] = hist[255 - 8 * (int)lane - j]; sum += c[j]; }
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= (uint32_t)o) incl += y;
    }
    uint32_t above = incl - sum, digit = 0, cnt = 0;
    const bool here = above < target && incl >= target;
    if (here) {
#pragma unroll
        for (int j = 0; j < 8; j++) {
            if (above + c[j] >= target) { digit = 255u - 8u * lane - (uint32_t)j; cnt = c[j]; break; }
            above += c[j];
        }
    }
    const int src = __ffs(__ballot_sync(0xffffffffu, here)) - 1;
    return {__shfl_sync(0xffffffffu, digit, src), __shfl_sync(0xffffffffu, above, src), __shfl_sync(0xffffffffu, cnt, src)};
}
/* exclusive prefix sum of one value per warp over the block's warps (all lanes hold the warp's value); one block barrier */
__device__ __forceinline__ uint32_t tk_warp_prefix(uint32_t v, uint32_t *tot /* [32] */) {
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    if (lane == 0) tot[w] = v;
    __syncthreads();
    const uint32_t mine = lane < (blockDim.x >> 5) ? tot[lane] : 0u;
    return __reduce_add_sync(0xffffffffu, lane < w ? mine : 0u);
}

template <uint32_t NB>
struct TkcShared {
    static constexpr uint32_t CAP = NB > 1 ? IX_TK_THREADS : 2u * IX_TK_THREADS;   /* collected keys of a block, at most */
    __align__(16) uint32_t ha[TK_BINS];   /* this block's counts of the first digit; cluster: the collected keys' */
    __align__(16) uint32_t hb[NB > 1 ? TK_BINS : 4];   /* the cluster's counts of the first digit */
    __align__(16) uint32_t h2[TK_BINS];   /* one block: the collected keys' counts; cluster: its counts of the pivot's next digit */
    __align__(16) uint32_t h3[256];       /* counts of the last digit */
    uint32_t bg[TKC_KEYS / 32], be[TKC_KEYS / 32], before[TKC_KEYS / 32];   /* this block's keys above / at the threshold, a bit each; those of earlier words */
    uint32_t tot[4][32];
    uint32_t cand[NB][CAP], idx[CAP];     /* the keys that each block has collected; this block's indices */
    struct { uint32_t n[NB], lo[NB], hi[NB], next[NB]; } told[2];   /* of every block in this round: keys that it has to collect, those at the pivot << 16, the least and largest of them, the least above them */
    struct { uint32_t n, lo, hi, next; } own[TKC_ROUNDS];   /* this block's, as they are counted */
    uint32_t n_near, low;                 /* low: keys above (low half-word) and at the threshold, of earlier blocks */
    uint32_t near[TKC_NEAR], thr, n_gt;
    TkPick st[3];
};
template <uint32_t NB>
__global__ void __launch_bounds__(IX_TK_THREADS) q4_ix_topkc_k(const float *score, int32_t *sel, uint32_t stride,
                                                               uint32_t k_blk, uint32_t ratio, uint32_t pos0,
                                                               uint32_t width, const int32_t *pp, const int32_t *pos_arr, uint32_t last_read, bool early) {
    extern __shared__ __align__(16) uint8_t tkc_smem[];
    TkcShared<NB> &S = *reinterpret_cast<TkcShared<NB> *>(tkc_smem);
    const uint32_t t = blockIdx.y, tx = threadIdx.x, lane = tx & 31u, warp = tx >> 5, rank = NB > 1 ? tkc_rank() : 0u;
    /* A position that comes with the launch or is settled in its word tells before anything is prepared whether every complete
     * block fits, the list of a short context (one token, 512 blocks: 2.9 -> 2.4 us; costs the others 0.3 of 7.5). */
    uint32_t pos = pos0 + t, n_read = t + 1u < gridDim.y ? stride : last_read, n_vis = 0u;
    if (early) {
        if (pp) pos = (uint32_t)*pp;
        if (pos + 1u < (k_blk + 1u) * ratio) {   /* the same decision in all blocks */
            q4d_pdl_wait();
            for (uint32_t w = rank * IX_TK_THREADS + tx; w < width; w += NB * IX_TK_THREADS) sel[(size_t)t * width + w] = w <= pos ? (int32_t)w : -1;
            return;
        }
        n_vis = (pos + 1u) / ratio;
        if (pp) n_read = min(stride, n_vis);
    }
    /* The block's own shared memory is prepared before the launch waits for the previous kernel: with programmatic dependent
     * launch this part runs under that kernel's tail. */
    constexpr uint32_t BPT = TK_BINS / IX_TK_THREADS;   /* bins per thread */
    static_assert(BPT == 4, "one 16-byte word of counts per thread");
    uint32_t *hist = NB > 1 ? S.ha : S.h2;
    reinterpret_cast<uint4 *>(S.ha)[tx] = make_uint4(0u, 0u, 0u, 0u);
    reinterpret_cast<uint4 *>(S.h2)[tx] = make_uint4(0u, 0u, 0u, 0u);
    if (NB > 1) reinterpret_cast<uint4 *>(S.hb)[tx] = make_uint4(0u, 0u, 0u, 0u);
    if (tx < 256) S.h3[tx] = S.bg[tx] = S.be[tx] = 0u;
    if (tx < TKC_ROUNDS) {
        S.own[tx].n = S.own[tx].hi = 0u;
        S.own[tx].lo = S.own[tx].next = 0xffffffffu;
    }
    if (tx == 0) S.n_near = S.low = 0u;
    /* the sums are zero before anyone adds to them; a cluster meets while the keys are on their way (8
     * sessions' step, met before the wait 416 us, so 411.5: its blocks find room late) */
    if (NB == 1) __syncthreads();
    else asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    q4d_pdl_wait();
    /* The keys are requested before a position that has yet to be read arrives.  Only visible ones of the last row: a host's
     * need not reach to `stride` (those of a batch do by its interface, and there the last row has stride too). */
    if (!early && pp) {
        pos = (uint32_t)*pp;
        n_read = min(stride, (pos + 1u) / ratio);
    }
    const float *row = score + (size_t)t * stride;
    const uint32_t base = rank * TKC_KEYS + tx;
    uint32_t key[TKC_KPT];
#pragma unroll
    for (uint32_t i = 0; i < TKC_KPT; i++) key[i] = base + IX_TK_THREADS * i < n_read ? __float_as_uint(__ldcg(row + base + IX_TK_THREADS * i)) : 0u;
    if (!early) {
        if (pos_arr) pos = (uint32_t)pos_arr[t];
        n_vis = ratio ? (pos + 1u) / ratio : 0u;
    }
    if (NB > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    const uint32_t need = n_vis < k_blk ? n_vis : k_blk;
    int32_t *out = sel + (size_t)t * width;
    const uint32_t w_per = (width + NB - 1u) / NB;
    const uint32_t w0 = min(rank * w_per, width), w1 = min(w0 + w_per, width);   /* this block's slice of the list */
    if (need == n_vis) {   /* every complete block fits: the dense prefix (same decision in all blocks) */
        for (uint32_t w = w0 + tx; w < w1; w += IX_TK_THREADS) out[w] = w <= pos ? (int32_t)w : -1;
        return;
    }
    /* ---- pivot: at least min(n_vis, 1024) threads have a key, which is `need` or more */
    auto live = [&](uint32_t i) { return base + IX_TK_THREADS * i < n_vis; };
    uint32_t most = 0u;
#pragma unroll
    for (uint32_t i = 0; i < TKC_KPT; i++) {
        key[i] = live(i) ? ix_key(__uint_as_float(key[i])) : 0u;
        most = max(most, key[i]);
    }
    if (live(0)) atomicAdd(&S.ha[most >> TK_B1], 1u);
    /* the tail of the list (positions behind the last complete block) does not depend on the selection */
    const uint32_t ncs = need * ratio;
    for (uint32_t w = max(w0, ncs) + tx; w < w1; w += IX_TK_THREADS) {
        const uint32_t tail = n_vis * ratio + (w - ncs);
        out[w] = tail <= pos ? (int32_t)tail : -1;
    }
    __syncthreads();
    /* this block's counts into every block's sum; the local array is left at zero for the next digit */
    auto spread = [&](uint32_t *sum, uint32_t bins) {
#pragma unroll
        for (uint32_t j = 0; j < BPT; j++) {   /* occupied bins are neighbours: one per thread */
            const uint32_t at = tx + j * IX_TK_THREADS, c = at < bins ? S.ha[at] : 0u;
            if (c) {
#pragma unroll
                for (uint32_t r = 0; r < NB; r++) tkc_red_add(tkc_remote(&sum[at], r), c);
                S.ha[at] = 0u;
            }
        }
        tkc_sync<NB>();
    };
    if (NB > 1) spread(S.hb, TK_BINS);
    const TkPick p1 = tk_pick<IX_TK_THREADS>(NB > 1 ? S.hb : S.ha, need, S.tot[0], &S.st[0]);
    /* The keys that are above the threshold or at it are found among those that reach a pivot, the digits `at` << shift.  Where a
     * block has no room for them, or so many threads' maxima reach the pivot that it will have none (of 8 keys per thread an eighth,
     * of one block a quarter, are some among 11, 15, threads of 16), many keys share its digits: then only those above it are
     * collected, and the blocks tell one another what lies at it (wide).  Those above may be enough; or the keys at it are equal, as
     * in rows of ties, and that is the threshold; or its next digit is counted. */
    uint32_t at = p1.digit, shift = TK_B1, n_round = 0, n_own, above, edge;   /* above: keys that have been collected */
    uint32_t thr = 0, n_gt = 0, low = 0;   /* the need-th largest key, keys above it: n_gt < need <= n_gt + ties; of earlier blocks, and their ties << 16 */
    bool clean = NB > 1;   /* the sums of the pivot's next digit are zero */
    /* Collects in any order, one add per warp.  Whether every block had room for its keys and they are enough: like all that
     * follows, the same in all blocks. */
    auto collect = [&](auto is_wide) -> bool {
        constexpr bool wide = decltype(is_wide)::value;
        edge = (wide ? at + 1u : at) << shift;
        if (wide) {
            if (!clean) {
                reinterpret_cast<uint4 *>(NB > 1 ? S.h2 : S.ha)[tx] = make_uint4(0u, 0u, 0u, 0u);
                tkc_sync<NB>();
            }
            clean = false;
        }
        uint32_t n = 0;
        if (!wide) {
#pragma unroll
            for (uint32_t i = 0; i < TKC_KPT; i++) n += key[i] >= edge;
        } else {
            uint32_t lo = 0xffffffffu, hi = 0u, next = 0xffffffffu;
#pragma unroll
            for (uint32_t i = 0; i < TKC_KPT; i++) {
                const uint32_t d = key[i] >> TK_B1;
                if (d > at) {
                    n++;
                    next = min(next, key[i]);
                }
                if (live(i) && d == at) {
                    n += 1u << 16;
                    lo = min(lo, key[i]);
                    hi = max(hi, key[i]);
                }
            }
            lo = __reduce_min_sync(0xffffffffu, lo);
            hi = __reduce_max_sync(0xffffffffu, hi);
            next = __reduce_min_sync(0xffffffffu, next);
            if (lane == 0) {
                atomicMin(&S.own[n_round].lo, lo);
                atomicMax(&S.own[n_round].hi, hi);
                atomicMin(&S.own[n_round].next, next);
            }
        }
        uint32_t slot = n;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, slot, o);
            if (lane >= (uint32_t)o) slot += y;
        }
        uint32_t first = 0;
        if (lane == 31 && slot) first = atomicAdd(&S.own[n_round].n, slot);
        slot += __shfl_sync(0xffffffffu, first, 31) - n;
        if (wide) slot &= 0xffffu;
        static_assert(TKC_KEYS < 65536, "two counts share a word");
        if (!wide || (n & 0xffffu)) {
#pragma unroll
            for (uint32_t i = 0; i < TKC_KPT; i++)
                if (key[i] >= edge) {
                    if (slot < S.CAP) {
                        S.cand[rank][slot] = key[i];
                        S.idx[slot] = IX_TK_THREADS * i + tx;
                    }
                    slot++;
                }
        }
        __syncthreads();
        const uint32_t mine = S.own[n_round].n;
        auto &told = S.told[n_round & 1u];
        n_own = wide ? mine & 0xffffu : mine;
        if (wide) {   /* the keys at the pivot by their next digit: one bin's where they are equal */
            const uint32_t lo = S.own[n_round].lo;
            if (lo < S.own[n_round].hi) {
#pragma unroll
                for (uint32_t i = 0; i < TKC_KPT; i++)
                    if (live(i) && key[i] >> TK_B1 == at) atomicAdd(&S.ha[(key[i] >> TK_B2) & (TK_BINS - 1u)], 1u);
            } else if (tx == 0 && mine >> 16) {
                S.ha[(lo >> TK_B2) & (TK_BINS - 1u)] = mine >> 16;
            }
            __syncthreads();
        }
        if (NB > 1) {
            if (tx < n_own && n_own <= S.CAP) {
                const uint32_t k = S.cand[rank][tx];
#pragma unroll
                for (uint32_t r = 0; r < NB; r++)
                    if (r != rank) tkc_st(tkc_remote(&S.cand[rank][tx], r), k);
            }
            if (tx < NB) {
                tkc_st(tkc_remote(&told.n[rank], tx), mine);
                if (wide) {
                    tkc_st(tkc_remote(&told.lo[rank], tx), S.own[n_round].lo);
                    tkc_st(tkc_remote(&told.hi[rank], tx), S.own[n_round].hi);
                    tkc_st(tkc_remote(&told.next[rank], tx), S.own[n_round].next);
                }
            }
            /* the last access to another block's shared memory, unless there is another round */
            if (wide) spread(S.h2, TK_BINS);
            else tkc_sync<NB>();
        }
        n_round++;
        if (NB == 1) {
            above = n_own;
            return n_own <= S.CAP && above >= need;
        }
        bool fits = true;
        above = 0;
#pragma unroll
        for (uint32_t r = 0; r < NB; r++) {
            const uint32_t c = wide ? told.n[r] & 0xffffu : told.n[r];
            fits = fits && c <= S.CAP;
            if (wide) above += c;
        }
        return fits && (!wide || above >= need);   /* a pivot is chosen so that enough keys reach it */
    };
    /* The threshold and this block's share of the list, from all collected keys, a warp's lanes at one block's; every block's begin
     * at other warps, for they are a hundred or two each.  Not where it lies beyond the bins, four times `edge` or more. */
    constexpr uint32_t CPT = NB > 1 ? NB : 2u;
    auto place = [&](uint32_t j) { return NB > 1 ? (tx - 128u * j) % IX_TK_THREADS : tx + j * IX_TK_THREADS; };
    auto finish = [&]() -> bool {
        const uint32_t *n = S.told[(n_round - 1u) & 1u].n;
        uint32_t ck[CPT];   /* 0: none */
#pragma unroll
        for (uint32_t j = 0; j < CPT; j++) {
            const uint32_t c = place(j);
            ck[j] = c < (NB > 1 ? n[j % NB] & 0xffffu : n_own) ? S.cand[j % NB][c] : 0u;
            if (ck[j]) atomicAdd(&hist[min((ck[j] - edge) >> TK_B2F, TK_BINS - 1u)], 1u);
        }
        __syncthreads();
        const TkPick p2 = tk_pick<IX_TK_THREADS>(hist, need, S.tot[1], &S.st[1]);
        if (p2.digit == TK_BINS - 1u) return false;
        const uint32_t left = need - p2.above;
        if (p2.cnt <= TKC_NEAR) {   /* mostly one to three */
#pragma unroll
            for (uint32_t j = 0; j < CPT; j++)
                if (ck[j] && (ck[j] - edge) >> TK_B2F == p2.digit) S.near[atomicAdd(&S.n_near, 1u)] = ck[j];
            __syncthreads();
            if (tx < p2.cnt) {
                const uint32_t k = S.near[tx];
                uint32_t more = 0, same = 0;
                for (uint32_t j = 0; j < p2.cnt; j++) {
                    more += S.near[j] > k;
                    same += S.near[j] == k;
                }
                if (more < left && left <= more + same) {
                    S.thr = k;
                    S.n_gt = p2.above + more;
                }
            }
        } else {   /* many keys share 24 bits */
            uint32_t *h = NB > 1 ? S.hb : S.ha;
            reinterpret_cast<uint4 *>(h)[tx] = make_uint4(0u, 0u, 0u, 0u);
            __syncthreads();
#pragma unroll
            for (uint32_t j = 0; j < CPT; j++)
                if (ck[j] && (ck[j] - edge) >> TK_B2F == p2.digit) atomicAdd(&h[(ck[j] - edge) & (TK_BINS - 1u)], 1u);
            __syncthreads();
            const TkPick p3 = tk_pick<IX_TK_THREADS>(h, left, S.tot[2], &S.st[2]);
            if (tx == 0) {
                S.thr = edge + (p2.digit << TK_B2F) + p3.digit;
                S.n_gt = p2.above + p3.above;
            }
        }
        __syncthreads();
        thr = S.thr;
        n_gt = S.n_gt;
#pragma unroll
        for (uint32_t j = 0; j < CPT; j++)
            if (ck[j] >= thr) {
                if (NB > 1 && j != rank) {
                    if (j < rank) atomicAdd(&S.low, ck[j] > thr ? 1u : 1u << 16);
                } else {
                    const uint32_t i = S.idx[place(j)];
                    atomicOr(ck[j] > thr ? &S.bg[i >> 5] : &S.be[i >> 5], 1u << (i & 31u));
                }
            }
        __syncthreads();
        low = S.low;
        return true;
    };
    /* ---- ordered emit: above the threshold in index order, then ties until `need` is full.  The bits' counts before every word: */
    auto count_words = [&]() {
        if (tx < TKC_KEYS / 32u) {
            const uint32_t v = __popc(S.bg[tx]) | __popc(S.be[tx]) << 16;
            uint32_t sum = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= (uint32_t)o) sum += y;
            }
            if (lane == 31) S.tot[3][warp] = sum;
            asm volatile("bar.sync 1, %0;" ::"n"(TKC_KEYS / 32u) : "memory");
            S.before[tx] = sum - v + __reduce_add_sync(0xffffffffu, lane < warp ? S.tot[3][lane] : 0u);
        }
        __syncthreads();
    };
    auto put = [&](uint32_t w, uint32_t i) {   /* the w-th of the list: key i of the block's */
        const uint32_t b = rank * TKC_KEYS + i;
        for (uint32_t j = 0; j < ratio && w * ratio + j < width; j++) out[w * ratio + j] = (int32_t)(b * ratio + j);
    };
    auto emit = [&]() {
        count_words();
#pragma unroll
        for (uint32_t j = 0; j < S.CAP / IX_TK_THREADS; j++) {
            const uint32_t c = tx + j * IX_TK_THREADS;
            if (c < n_own && S.cand[rank][c] >= thr) {
                const bool gt = S.cand[rank][c] > thr;
                const uint32_t i = S.idx[c], all = S.before[i >> 5] + low;
                uint32_t w = gt ? all & 0xffffu : n_gt + (all >> 16);
                if (w < need) {
                    w += __popc((gt ? S.bg[i >> 5] : S.be[i >> 5]) & ((1u << (i & 31u)) - 1u));
                    if (w < need) put(w, i);
                }
            }
        }
    };
    constexpr uint32_t ROOM = NB * S.CAP / 4u * 3u;   /* of all blocks, where their shares differ a little */
    bool wide = at == 0u || (n_vis > S.CAP && (p1.above + p1.cnt) * 16u >= (n_vis / TKC_KEYS * IX_TK_THREADS + min(n_vis % TKC_KEYS, IX_TK_THREADS)) * (NB > 1 ? 11u : 15u));
    bool over = false;   /* the threshold is above the pivot */
    if (!wide) {
        if (collect(std::false_type())) {
            if (finish()) {
                emit();
                return;
            }
            over = true;
        }
        wide = true;
    }
    bool known = true;   /* `low` is */
#pragma unroll 1
    while (true) {
        if (!over) {
            if (wide ? collect(std::true_type()) : collect(std::false_type())) {
                if (wide) {   /* they may begin far above the pivot */
                    uint32_t next = S.own[n_round - 1u].next;
                    for (uint32_t r = 0; NB > 1 && r < NB; r++) next = min(next, S.told[(n_round - 1u) & 1u].next[r]);
                    edge = next >> TK_B1 << TK_B1;
                }
                if (finish()) {
                    emit();
                    return;
                }
                over = true;
            } else if (wide) {
                over = above >= need;
            } else if (shift == TK_B1) {
                wide = true;
                continue;
            }
        }
        uint32_t *sums = NB > 1 ? S.h2 : S.ha;
        if (over) {   /* the first digit, of all keys */
            reinterpret_cast<uint4 *>(hist)[tx] = make_uint4(0u, 0u, 0u, 0u);   /* may have been counted into */
            reinterpret_cast<uint4 *>(sums)[tx] = make_uint4(0u, 0u, 0u, 0u);
            clean = false;
            tkc_sync<NB>();
#pragma unroll
            for (uint32_t i = 0; i < TKC_KPT; i++)
                if (live(i)) atomicAdd(&S.ha[key[i] >> TK_B1], 1u);
            __syncthreads();
            if (NB > 1) spread(sums, TK_BINS);
            const TkPick p = tk_pick<IX_TK_THREADS>(sums, need, S.tot[2], &S.st[2]);
            at = p.digit;
            over = false;
            wide = at == 0u || p.above + p.cnt > ROOM;
            continue;
        }
        if (shift == TK_B1) {
            const auto &told = S.told[(n_round - 1u) & 1u];
            uint32_t lo = S.own[n_round - 1u].lo, hi = S.own[n_round - 1u].hi;
            for (uint32_t r = 0; NB > 1 && r < NB; r++) {
                lo = min(lo, told.lo[r]);
                hi = max(hi, told.hi[r]);
            }
            n_gt = above;
            if (lo == hi) {   /* as in rows of ties: the threshold */
                thr = lo;
                for (uint32_t r = 0; NB > 1 && r < rank; r++) low += told.n[r];
                break;
            }
            const TkPick p = tk_pick<IX_TK_THREADS>(sums, need - n_gt, S.tot[2], &S.st[2]);
            at = at << (TK_B1 - TK_B2) | p.digit;
            shift = TK_B2;
            n_gt += p.above;
            wide = false;
            if (at && n_gt + p.cnt <= ROOM) continue;
        }
        /* the last digit */
#pragma unroll
        for (uint32_t i = 0; i < TKC_KPT; i++)
            if (live(i) && key[i] >> TK_B2 == at) atomicAdd(&(NB > 1 ? S.ha : S.h3)[key[i] & 255u], 1u);
        __syncthreads();
        if (NB > 1) spread(S.h3, 256u);
        const TkPick p = tk_pick256(S.h3, need - n_gt);
        thr = at << TK_B2 | p.digit;
        n_gt += p.above;
        known = NB == 1;
        break;
    }
    /* the list of all keys that reach the threshold; a key that is not there is 0 */
    uint32_t mg[TKC_KPT], me[TKC_KPT], all[TKC_KPT];
#pragma unroll
    for (uint32_t i = 0; i < TKC_KPT; i++) {
        mg[i] = __ballot_sync(0xffffffffu, key[i] > thr);
        me[i] = __ballot_sync(0xffffffffu, live(i) && key[i] == thr);
        if (lane == 0) { S.bg[32u * i + warp] = mg[i]; S.be[32u * i + warp] = me[i]; }
    }
    if (!known) {   /* the blocks tell one another what they hold */
        uint32_t n = 0;
#pragma unroll
        for (uint32_t i = 0; i < TKC_KPT; i++) n += __popc(mg[i]) | __popc(me[i]) << 16;
        if (lane == 0 && n) atomicAdd(&S.own[n_round].n, n);
        __syncthreads();
        if (tx < NB) tkc_st(tkc_remote(&S.told[n_round & 1u].n[rank], tx), S.own[n_round].n);
        tkc_sync<NB>();
        for (uint32_t r = 0; NB > 1 && r < rank; r++) low += S.told[n_round & 1u].n[r];
    }
    __syncthreads();
    count_words();
#pragma unroll
    for (uint32_t i = 0; i < TKC_KPT; i++) all[i] = S.before[32u * i + warp] + low;
#pragma unroll
    for (uint32_t i = 0; i < TKC_KPT; i++) {
        const bool gt = (mg[i] >> lane) & 1u;
        const uint32_t m = gt ? mg[i] : me[i], w = (gt ? all[i] & 0xffffu : n_gt + (all[i] >> 16)) + __popc(m & ((1u << lane) - 1u));
        if (((m >> lane) & 1u) && w < need) put(w, IX_TK_THREADS * i + tx);
    }
}

/* ---- selection for many tokens at once (a prompt's slice): one block of 512 threads per token, four blocks per
 * SM.  The cluster form above holds 16 SMs' worth of threads per token for a dozen block barriers (409 us for 512
 * tokens x 32 768 keys); here a token's row is read twice from L2, once to count the first digits and once to collect the
 * keys of the threshold bin, and the exact finish works on those.  Chosen keys are marked in a bitmap in index order; the
 * ordered emit is a prefix sum of its population counts.
 * Counting every key's digit in shared memory costs more than reading it, because most keys of a row share few leading
 * digits.  So the first pass over a long row is a sample of 2048 keys: it gives a pivot, 24 bits of a key, which `need` keys of the
 * row fall short of by five standard deviations.  The second collects the keys above the pivot's bin and counts, by their last 8
 * bits, those in it: where the first are too few (rows of ties, whose pivot is the threshold itself) the threshold is known by
 * then, and a third pass marks the row.  Where the sample misled the row is counted in full.  Only with more than one block per
 * SM: a block that has an SM to itself waits for the sample longer than it saves.
 * us, counted / sampled: 512 tokens x 65 536 keys 86.7 / 73.7, 32 768 44.2 / 35.4, 24 576 35.5 / 30.3; 200 tokens x 32 768 24.4 /
 * 22.3, 24 576 20.0 / 19.3, rounded keys 20.5 / 21.9; 100 x 32 768 17.3 / 19.5; 512 x 32 768 zeros 68.6 / 65.2 (111 where all keys
 * that reach the pivot are collected, until the room ends). */
constexpr uint32_t TKM_THREADS = 512, TKM_CAND = 2048, TKM_BATCH = 8, TKM_SAMPLE = 2048, TKM_SAMPLED_FROM = 24576;   /* keys */
struct TkmShared {
    __align__(16) uint32_t hist[TK_BINS], h3[256], tot[4][32];
    uint32_t ckey[TKM_CAND];
    uint32_t cidx[TKM_CAND];
    uint32_t chosen[IX_MAX_KBLK];
    uint32_t n_cand;
    TkPick st[2];
};
/* keys above the pivot's bin of 256, in any order (the count goes on where the room ends), and how many lie where in the bin */
__device__ __forceinline__ void tkm_collect(TkmShared &S, const float *row, uint32_t n, uint32_t pivot) {
    const float pf = __uint_as_float(pivot & 0x80000000u ? pivot & 0x7fffffffu : ~pivot);   /* ix_key's inverse */
    auto one = [&](uint32_t b, float x) {
        if (!(x < pf)) {   /* and NaN, which ix_key orders by its sign */
            const uint32_t u = ix_key(x);
            if (u > (pivot | 255u)) {
                const uint32_t slot = atomicAdd(&S.n_cand, 1u);
                if (slot < TKM_CAND) {
                    S.ckey[slot] = u;
                    S.cidx[slot] = b;
                }
            } else if (u >= pivot) {
                atomicAdd(&S.h3[u & 255u], 1u);
            }
        }
    };
    const uint32_t head = min(n, (4u - (uint32_t)((uintptr_t)row >> 2)) & 3u), quads = (n - head) / 4u, done = head + 4u * quads;
    if (threadIdx.x < head) one(threadIdx.x, __ldcg(row + threadIdx.x));
    if (threadIdx.x < n - done) one(done + threadIdx.x, __ldcg(row + done + threadIdx.x));
    const float4 *body = reinterpret_cast<const float4 *>(row + head);
    /* Eight keys at a time into a mask, then one by one what is in it: with one key of 30 above the pivot a warp goes round
     * once or twice. */
    for (uint32_t i0 = threadIdx.x; i0 < quads; i0 += TKM_THREADS * 2u) {
        const uint32_t i1 = i0 + TKM_THREADS;
        const float4 x = __ldcg(body + i0), y = __ldcg(body + min(i1, quads - 1u));
        uint32_t m = (uint32_t)!(x.x < pf) | (uint32_t)!(x.y < pf) << 1 | (uint32_t)!(x.z < pf) << 2 | (uint32_t)!(x.w < pf) << 3;
        if (i1 < quads) m |= (uint32_t)!(y.x < pf) << 4 | (uint32_t)!(y.y < pf) << 5 | (uint32_t)!(y.z < pf) << 6 | (uint32_t)!(y.w < pf) << 7;
        for (; m; m &= m - 1u) {
            const uint32_t k = (uint32_t)__ffs(m) - 1u;
            const float4 z = k & 4u ? y : x;
            const float2 w = k & 2u ? make_float2(z.z, z.w) : make_float2(z.x, z.y);
            one(head + 4u * (k & 4u ? i1 : i0) + (k & 3u), k & 1u ? w.y : w.x);
        }
    }
}
/* all keys of a row in steps of the block's width: f(index, key, live) with the lanes of a warp on 32 consecutive indices */
template <typename F>
__device__ __forceinline__ void tkm_walk(const float *row, uint32_t n, F f) {
    for (uint32_t b0 = threadIdx.x; b0 - threadIdx.x < n; b0 += TKM_THREADS * TKM_BATCH) {
        float x[TKM_BATCH];
#pragma unroll
        for (uint32_t k = 0; k < TKM_BATCH; k++) {
            const uint32_t b = b0 + k * TKM_THREADS;
            x[k] = b < n ? __ldcg(row + b) : 0.f;
        }
#pragma unroll
        for (uint32_t k = 0; k < TKM_BATCH; k++) {
            const uint32_t b = b0 + k * TKM_THREADS;
            f(b, ix_key(x[k]), b < n);
        }
    }
}
template <bool SAMPLED>
__global__ void __launch_bounds__(TKM_THREADS, 4) q4_ix_topkm_k(const float *score, int32_t *sel, uint32_t stride, uint32_t k_blk,
                                                               uint32_t ratio, uint32_t pos0, uint32_t width, uint32_t words,
                                                               const int32_t *pp, const int32_t *pos_arr) {
    extern __shared__ __align__(16) uint8_t tkm_smem[];
    TkmShared &S = *reinterpret_cast<TkmShared *>(tkm_smem);
    uint32_t *bg = reinterpret_cast<uint32_t *>(tkm_smem + sizeof(TkmShared)), *be = bg + words;   /* above / at the threshold */
    const uint32_t t = blockIdx.x, tx = threadIdx.x, lane = tx & 31u;
    q4d_pdl_wait();
    const uint32_t pos = pos_arr ? (uint32_t)pos_arr[t] : (pp ? (uint32_t)*pp : pos0) + t;
    const uint32_t n_vis = ratio ? (pos + 1u) / ratio : 0u;
    const uint32_t need = n_vis < k_blk ? n_vis : k_blk;
    const float *row = score + (size_t)t * stride;
    int32_t *out = sel + (size_t)t * width;
    if (need == n_vis) {   /* every complete block fits: the dense prefix */
        for (uint32_t w = tx; w < width; w += TKM_THREADS) out[w] = w <= pos ? (int32_t)w : -1;
        return;
    }
    const uint32_t n = min(n_vis, words * 32u);   /* the launcher sizes the bitmaps for the row */
    auto clear = [&]() {
        for (uint32_t i = tx; i < TK_BINS / 4; i += TKM_THREADS) reinterpret_cast<uint4 *>(S.hist)[i] = make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();
    };
    if (tx < 256) S.h3[tx] = 0u;
    if (tx == 0) S.n_cand = 0u;
    for (uint32_t i = tx; i < words; i += TKM_THREADS) { bg[i] = 0u; be[i] = 0u; }
    clear();
    uint32_t n_cand = 0, thr = 0, n_gt = 0;
    bool sampled = false, known = false, mark = false;   /* candidates from the sampled pivot; threshold known already; the row is marked by walking it */
    if (SAMPLED && n > TKM_SAMPLED_FROM) {
        /* the pivot: 24 bits of a key */
        constexpr uint32_t PER = TKM_SAMPLE * 9u / 8u / TKM_THREADS + 1u;
        const uint32_t step = n / TKM_SAMPLE, n_s = (n + step - 1u) / step;
        uint32_t ks[PER];
#pragma unroll
        for (uint32_t j = 0; j < PER; j++) {
            const uint32_t i = tx + j * TKM_THREADS, at = min(i * step + (i * 0x9E3779B1u >> 16) % step, n - 1u);
            ks[j] = i < n_s ? ix_key(__ldcg(row + at)) : 0u;
        }
#pragma unroll
        for (uint32_t j = 0; j < PER; j++)
            if (tx + j * TKM_THREADS < n_s) atomicAdd(&S.hist[ks[j] >> TK_B1], 1u);
        __syncthreads();
        const float mean = (float)need / (float)step;
        const uint32_t target = (uint32_t)(mean + 5.f * sqrtf(mean)) + 4u;   /* at most 64 + 40 + 4 of 2048 */
        const TkPick s1 = tk_pick<TKM_THREADS>(S.hist, target, S.tot[0], &S.st[0]);
        clear();
#pragma unroll
        for (uint32_t j = 0; j < PER; j++)
            if (tx + j * TKM_THREADS < n_s && (ks[j] >> TK_B1) == s1.digit) atomicAdd(&S.hist[(ks[j] >> TK_B2) & (TK_BINS - 1u)], 1u);
        __syncthreads();
        const TkPick s2 = tk_pick<TKM_THREADS>(S.hist, target - s1.above, S.tot[1], &S.st[1]);
        clear();
        const uint32_t pivot = (s1.digit << TK_B1) | (s2.digit << TK_B2);
        tkm_collect(S, row, n, pivot);
        __syncthreads();
        n_cand = S.n_cand;
        sampled = n_cand >= need && n_cand <= TKM_CAND;
        if (n_cand < need) {   /* the threshold lies in the pivot's bin, if that has enough keys */
            const TkPick p3 = tk_pick256(S.h3, need - n_cand);
            thr = pivot | p3.digit;
            n_gt = n_cand + p3.above;
            known = mark = p3.cnt != 0u;
        }
        __syncthreads();
        if (tx < 256) S.h3[tx] = 0u;
    }
    if (!known) {
        if (sampled) {
            for (uint32_t i = tx; i < n_cand; i += TKM_THREADS) atomicAdd(&S.hist[S.ckey[i] >> TK_B1], 1u);
        } else {
            tkm_walk(row, n, [&](uint32_t, uint32_t u, bool live) { if (live) atomicAdd(&S.hist[u >> TK_B1], 1u); });
        }
        __syncthreads();
        const TkPick p1 = tk_pick<TKM_THREADS>(S.hist, need, S.tot[0], &S.st[0]);
        if (tx == 0) S.n_cand = 0u;   /* everyone has read it */
        clear();
        if (sampled || p1.cnt <= TKM_CAND) {
            if (sampled) {
                for (uint32_t i = tx; i < n_cand; i += TKM_THREADS)
                    if ((S.ckey[i] >> TK_B1) == p1.digit) atomicAdd(&S.hist[(S.ckey[i] >> TK_B2) & (TK_BINS - 1u)], 1u);
            } else {
                n_cand = p1.cnt;
                tkm_walk(row, n, [&](uint32_t b, uint32_t u, bool live) {
                    const uint32_t m = __ballot_sync(0xffffffffu, live && (u >> TK_B1) > p1.digit);
                    if (lane == 0 && m) bg[b >> 5] = m;
                    if (live && (u >> TK_B1) == p1.digit) {
                        const uint32_t slot = atomicAdd(&S.n_cand, 1u);
                        S.ckey[slot] = u;
                        S.cidx[slot] = b;
                        atomicAdd(&S.hist[(u >> TK_B2) & (TK_BINS - 1u)], 1u);
                    }
                });
            }
            __syncthreads();
            const TkPick p2 = tk_pick<TKM_THREADS>(S.hist, need - p1.above, S.tot[1], &S.st[1]);
            const uint32_t pre = (p1.digit << 12) | p2.digit;
            for (uint32_t i = tx; i < n_cand; i += TKM_THREADS)
                if ((S.ckey[i] >> TK_B2) == pre) atomicAdd(&S.h3[S.ckey[i] & 255u], 1u);
            __syncthreads();
            const TkPick p3 = tk_pick256(S.h3, need - p1.above - p2.above);
            thr = (pre << 8) | p3.digit;
            n_gt = p1.above + p2.above + p3.above;
            for (uint32_t i = tx; i < n_cand; i += TKM_THREADS) {
                const uint32_t u = S.ckey[i], b = S.cidx[i];
                if (u > thr) atomicOr(&bg[b >> 5], 1u << (b & 31u));
                else if (u == thr) atomicOr(&be[b >> 5], 1u << (b & 31u));
            }
        } else {   /* rows of ties: the second and third digit are counted over the row too */
            tkm_walk(row, n, [&](uint32_t, uint32_t u, bool live) {
                if (live && (u >> TK_B1) == p1.digit) atomicAdd(&S.hist[(u >> TK_B2) & (TK_BINS - 1u)], 1u);
            });
            __syncthreads();
            const TkPick p2 = tk_pick<TKM_THREADS>(S.hist, need - p1.above, S.tot[1], &S.st[1]);
            const uint32_t pre = (p1.digit << 12) | p2.digit;
            tkm_walk(row, n, [&](uint32_t, uint32_t u, bool live) {
                if (live && (u >> TK_B2) == pre) atomicAdd(&S.h3[u & 255u], 1u);
            });
            __syncthreads();
            const TkPick p3 = tk_pick256(S.h3, need - p1.above - p2.above);
            thr = (pre << 8) | p3.digit;
            n_gt = p1.above + p2.above + p3.above;
            mark = true;
        }
    }
    if (mark)
        tkm_walk(row, n, [&](uint32_t b, uint32_t u, bool live) {
            const uint32_t mg = __ballot_sync(0xffffffffu, live && u > thr), me = __ballot_sync(0xffffffffu, live && u == thr);
            if (lane == 0 && mg) bg[b >> 5] = mg;
            if (lane == 0 && me) be[b >> 5] = me;
        });
    __syncthreads();
    /* ranks: every thread owns consecutive words of the bitmaps */
    const uint32_t wpt = (words + TKM_THREADS - 1u) / TKM_THREADS, wa = min(tx * wpt, words), wb = min(wa + wpt, words);
    uint32_t ng = 0, ne = 0;
    for (uint32_t i = wa; i < wb; i++) { ng += __popc(bg[i]); ne += __popc(be[i]); }
    uint32_t ig = ng, ie = ne;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t yg = __shfl_up_sync(0xffffffffu, ig, o), ye = __shfl_up_sync(0xffffffffu, ie, o);
        if (lane >= (uint32_t)o) { ig += yg; ie += ye; }
    }
    uint32_t og = tk_warp_prefix(__shfl_sync(0xffffffffu, ig, 31), S.tot[2]) + ig - ng;
    uint32_t oe = n_gt + tk_warp_prefix(__shfl_sync(0xffffffffu, ie, 31), S.tot[3]) + ie - ne;
    for (uint32_t i = wa; i < wb; i++) {
        for (uint32_t m = bg[i]; m; m &= m - 1u, og++)
            if (og < need) S.chosen[og] = 32u * i + (uint32_t)__ffs(m) - 1u;
        for (uint32_t m = be[i]; m && oe < need; m &= m - 1u, oe++) S.chosen[oe] = 32u * i + (uint32_t)__ffs(m) - 1u;
    }
    __syncthreads();
    const uint32_t ncs = need * ratio;
    for (uint32_t w = tx; w < width; w += TKM_THREADS) {
        int32_t v;
        if (w < ncs) {
            const uint32_t i = w / ratio;
            v = (int32_t)(S.chosen[i] * ratio + (w - i * ratio));
        } else {
            const uint32_t tail = n_vis * ratio + (w - ncs);
            v = tail <= pos ? (int32_t)tail : -1;
        }
        out[w] = v;
    }
}

template <uint32_t NB>
bool topkc_start(const float *score, int32_t *sel, uint32_t n_tok, uint32_t stride, uint32_t k_blk, uint32_t ratio, uint32_t pos0,
                 uint32_t width, const int32_t *pp, const int32_t *pos_arr) {
    static bool done = false;
    if (!done && !q4i_check(cudaFuncSetAttribute(q4_ix_topkc_k<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TkcShared<NB>)),
                            "qsa_topk smem attribute"))
        return false;
    done = true;
    const uint32_t vis = ratio ? (pos0 + n_tok) / ratio : 0u;   /* of the last token, where the host gives the position */
    return ix_start("qsa_topk launch", q4_ix_topkc_k<NB>, dim3(NB, n_tok), IX_TK_THREADS, sizeof(TkcShared<NB>), NB, score, sel, stride, k_blk, ratio, pos0,
                      width, pp, pos_arr, pos_arr || vis > stride ? stride : vis, ix_pdl() && ratio && !pos_arr && (!pp || q4i_settled(g_q4.pos_written)));
}
template <bool SAMPLED>
bool topkm_start(const float *score, int32_t *sel, uint32_t n_tok, uint32_t stride, uint32_t k_blk, uint32_t ratio, uint32_t pos0,
                 uint32_t width, const int32_t *pp, const int32_t *pos_arr) {
    static bool done = false;
    if (!done && !q4i_check(cudaFuncSetAttribute(q4_ix_topkm_k<SAMPLED>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)(sizeof(TkmShared) + 2 * TKC_MAX_ROW / 8)), "qsa_topk smem attribute"))
        return false;
    done = true;
    const uint32_t words = (stride + 31u) / 32u;
    return ix_start("qsa_topk launch", q4_ix_topkm_k<SAMPLED>, dim3(n_tok), TKM_THREADS, sizeof(TkmShared) + 2u * words * 4u, 1u, score, sel, stride, k_blk,
                    ratio, pos0, width, words, pp, pos_arr);
}
/* Which form: rows of up to 8192 keys need one block either way, which keeps them in registers.  Longer rows take the
 * cluster form up to two blocks per SM, which are two or three waves, for a block of 1024 threads fills an SM's registers (us, the
 * last so / the next one streamed: 37 / 38 tokens of 65 536 keys 21.7 / 27.6, 74 / 75 of 32 768 18.9 / 17.4, 148 / 149 of 16 384 13.1 /
 * 14.5), the streaming form beyond (512 tokens x 32 768 keys), and the single block that re-reads the row behind 65 536 keys. */
bool launch_topk(const float *score, int32_t *sel, uint32_t n_tok, uint32_t stride, uint32_t k_blk, uint32_t ratio,
                 uint32_t pos0, uint32_t width, const int32_t *pp, const int32_t *pos_arr = nullptr) {
    if (stride > TKC_MAX_ROW) {
        q4_ix_topk1_k<<<n_tok, IX_TK_THREADS, 0, g_q4.stream>>>(score, sel, stride, k_blk, ratio, pos0, width, pp, pos_arr);
        return q4i_launched(q4i_check(cudaGetLastError(), "qsa_topk launch"));
    }
    if (stride <= TKC_KEYS) return topkc_start<1>(score, sel, n_tok, stride, k_blk, ratio, pos0, width, pp, pos_arr);
    const uint32_t nb = stride <= 2 * TKC_KEYS ? 2u : stride <= 4 * TKC_KEYS ? 4u : 8u;
    if ((uint64_t)n_tok * nb > 2ull * (uint64_t)g_q4.sm_count) {
        const uint32_t rows = pp || pos_arr || !ratio ? stride : (pos0 + n_tok) / ratio;   /* the last token's, at most */
        return n_tok > (uint32_t)g_q4.sm_count && rows > TKM_SAMPLED_FROM ? topkm_start<true>(score, sel, n_tok, stride, k_blk, ratio, pos0, width, pp, pos_arr)
                                                                          : topkm_start<false>(score, sel, n_tok, stride, k_blk, ratio, pos0, width, pp, pos_arr);
    }
    if (nb == 2) return topkc_start<2>(score, sel, n_tok, stride, k_blk, ratio, pos0, width, pp, pos_arr);
    if (nb == 4) return topkc_start<4>(score, sel, n_tok, stride, k_blk, ratio, pos0, width, pp, pos_arr);
    return topkc_start<8>(score, sel, n_tok, stride, k_blk, ratio, pos0, width, pp, pos_arr);
}

bool pool_start(const char *what, uint32_t grid, const void *raw, float *pool, const float *wn, uint32_t ratio, uint32_t b0, uint32_t b1, uint32_t n_rot,
                float base, float eps, const int32_t *pp) {
    Q4Touch t = {};
    const uint64_t row = (uint64_t)IX_HD * 2u * ratio;
    if (pp) {
        t.reads(raw, 0);
        t.writes(pool, 0);
        t.r[t.n - 1u].newest = ratio;
    } else {
        t.reads((const __half *)raw + (size_t)b0 * ratio * IX_HD, (b1 - b0) * row);
        t.writes(pool + (size_t)b0 * IX_HD, (uint64_t)(b1 - b0) * IX_HD * 4u);
    }
    t.reads(wn, IX_HD * 4u);
    t.reads(pp, 4);
    const bool early = !pp || q4i_settled(g_q4.pos_written), apart = early && q4i_apart(t);
    return q4i_launched(q4i_launch_dep(what, q4_ix_pool_k, dim3(grid), 128u, 0, (const __half *)raw, pool, wn, ratio, b0, b1, n_rot, base, eps, pp, early,
                                       apart), &t, apart);
}

}  // namespace

/* ======================================================================= reference ABI ===== */
extern "C" bool q4_hip_qsa_pool(const void *raw_f16, float *pool, const float *wn, uint32_t hd, uint32_t ratio,
                                uint32_t b0, uint32_t b1, uint32_t n_rot, float rope_base, float eps) {
    if (!g_q4.ok || !raw_f16 || !pool || b1 <= b0 || hd != IX_HD || ratio == 0) return false;
    return pool_start("qsa_pool launch", (b1 - b0 + 3u) / 4u, raw_f16, pool, wn, ratio, b0, b1, n_rot, rope_base, eps, nullptr);
}
extern "C" bool q4_hip_qsa_pool_d(const void *raw, float *pool, const float *wn, uint32_t hd, uint32_t ratio,
                                  uint32_t n_rot, float rope_base, float eps) {
    if (!g_q4.ok || !g_q4.pos_d || !raw || !pool || hd != IX_HD || ratio == 0) return false;
    return pool_start("qsa_pool_d launch", 1u, raw, pool, wn, ratio, 0u, 0u, n_rot, rope_base, eps, g_q4.pos_d);
}
extern "C" bool q4_hip_qsa_score(const float *q, const float *pool, float *score, uint32_t n_tok, uint32_t n_blocks,
                                 uint32_t stride, uint32_t n_head, uint32_t hd, uint32_t pos0, uint32_t ratio) {
    if (!g_q4.ok || !q || !pool || !score || n_tok == 0 || hd != IX_HD || n_head == 0 || n_head > 4) return false;
    if (n_blocks == 0) return true;
    if (ratio && n_tok > 1 && (((uintptr_t)q | (uintptr_t)pool) & 15u) == 0) {
        const uint64_t wide = score_mt_ns(n_tok, n_blocks, 4), narrow = score_mt_ns(n_tok, n_blocks, 2), scan = score_scan_ns(n_tok, n_blocks);
        const uint64_t below = scan - scan / 16u;   /* of 8 tokens over 24 576 blocks: 23.2 us where 26.8 are estimated, the product takes 24.3 */
        if (wide <= narrow && wide < below) return score_mt_launch<4>(q, pool, score, n_tok, n_blocks, stride, n_head, pos0, ratio);
        if (narrow < below) return score_mt_launch<2>(q, pool, score, n_tok, n_blocks, stride, n_head, pos0, ratio);
    }
    return score_launch(q, pool, score, n_tok, n_blocks, stride, n_head, pos0, ratio, nullptr, nullptr, nullptr);
}
/* Device position (graph-captured decode): the grid covers `stride` blocks, the bound comes from the
 * position word inside the kernel. */
extern "C" bool q4_hip_qsa_score_d(const float *q, const float *pool, float *score, uint32_t stride, uint32_t n_head,
                                   uint32_t hd, uint32_t ratio) {
    if (!g_q4.ok || !g_q4.pos_d || !q || !pool || !score || hd != IX_HD || n_head == 0 || n_head > 4 || stride == 0)
        return false;
    return score_launch(q, pool, score, 1, 0, stride, n_head, 0, ratio, g_q4.pos_d, nullptr, nullptr);
}
extern "C" bool q4_hip_qsa_topk(const float *score, int32_t *sel, uint32_t n_tok, uint32_t n_blocks, uint32_t stride,
                                uint32_t k_blk, uint32_t ratio, uint32_t pos0, uint32_t width) {
    (void)n_blocks;
    if (!g_q4.ok || !score || !sel || n_tok == 0 || k_blk == 0 || k_blk > IX_MAX_KBLK || width == 0) return false;
    return launch_topk(score, sel, n_tok, stride, k_blk, ratio, pos0, width, nullptr);
}
extern "C" bool q4_hip_qsa_topk_d(const float *score, int32_t *sel, uint32_t stride, uint32_t k_blk, uint32_t ratio,
                                  uint32_t width) {
    if (!g_q4.ok || !g_q4.pos_d || !score || !sel || k_blk == 0 || k_blk > IX_MAX_KBLK || width == 0) return false;
    return launch_topk(score, sel, 1, stride, k_blk, ratio, 0, width, g_q4.pos_d);
}

/* Batched form for concurrent sessions (additive): row t of q / score / sel belongs to session t, which
 * has its own pool (pools[t], device array of device pointers) and its own position (pos[t], device
 * array); scoring and selection of all sessions in two launches.  Every session must have at most
 * `stride` visible blocks.  Same arithmetic and the same lists as one q4_hip_qsa_score_d +
 * q4_hip_qsa_topk_d pair per session. */
extern "C" bool q4_gpu_qsa_select_batch(const float *const *pools, const int32_t *pos, const float *q, float *score,
                                        int32_t *sel, uint32_t n_sess, uint32_t stride, uint32_t n_head, uint32_t hd,
                                        uint32_t k_blk, uint32_t ratio, uint32_t width) {
    if (!g_q4.ok) return q4i_fail(Q4E_INIT, "qsa_select_batch: library not initialised");
    Q4_REQUIRE(pools && pos && q && score && sel && n_sess && stride && ratio && width, "qsa_select_batch: bad argument");
    Q4_REQUIRE(hd == IX_HD && n_head >= 1 && n_head <= 4 && k_blk >= 1 && k_blk <= IX_MAX_KBLK,
               "qsa_select_batch: unsupported shape");
    return score_launch(q, nullptr, score, n_sess, 0, stride, n_head, 0, ratio, nullptr, pools, pos) &&
           launch_topk(score, sel, n_sess, stride, k_blk, ratio, 0, width, nullptr, pos);
}
