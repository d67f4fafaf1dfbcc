/*
 * Dense causal attention of a chunk of query tokens on the 5th-generation tensor cores (tcgen05.mma, accumulators
 * in tensor memory, operands brought in by bulk copies).  Query t of the chunk attends rows
 * [0, min(kv_base + t + 1, max_kv)) -- the semantics of gqa_prefill_k (src/q4_rocm.cu:7019-7206) as launched by
 * q4_hip_qsa_decode_n with n_tok > 1 (:7263,7286-7298); the reference computes it with scalar FMAs and
 * re-dequantises every K/V tile for every query token.
 *
 * Launches per call:
 *
 *  1. q4_pf_stage_k turns the rows the chunk can see, once, into fp16 operand tiles: 32 KB images of 128 K rows x 128
 *     dims and of V^T, already in the 128-byte-swizzled K-major layout that the tensor core reads, so that a tile
 *     comes in with one plain bulk copy (no tensor maps).  The q8_0 caches of the reference ABI get two images of both,
 *     fp16(code * scale) and the rest, which together are exact: that entry point always multiplied exact codes.  (A code
 *     times its scale is a multiple of 2^-24, like the scale: the rest is one too and has 8 bits at most.)  With one image
 *     of V the outputs' error against 64 bits was 13 to 24 % above that of the decode form, six times on a token that
 *     attends one row; the second costs the 2048-token prompt of the reference's host 2340 -> 2755 us.
 *  2. q4_prefill_k: one block = one kv head x NQ groups of query tokens whose (token, head) pairs fill the 128 rows
 *     of the MMA each (NQ = 2: 32 tokens x 8 heads at the benchmark shape), against 128-position tiles.
 *
 *       producer warp (one thread): bulk copies into a ring of five 32 KB slots
 *       issuer warp (one elected lane): a sequence of units.  O += P . V of unit i as soon as the softmax warps have
 *                     published its P (64 positions at a time), then S = Q . K^T of the unit that takes over the score
 *                     buffer just freed (products of one thread run in order)
 *       softmax warps: thread r owns row r (NQ = 1: two threads, half of the unit's positions each): its scores out of
 *                     tensor memory, causal mask, running max with lazy rescale, P = exp2(..) as fp16 back into the
 *                     first half of the columns it came from.
 *
 *     A score buffer holds S and then P of one unit, and every group of softmax warps has two, so that the scores of
 *     its next unit are computed under its present exponentials.  NQ = 2 (hd 128): units are (64 positions, group),
 *     four buffers of 64 columns; both groups share every K/V tile.  NQ = 1: units are tiles of 128 positions, two
 *     buffers of 128 columns; two warps per 32 rows instead of one take the 2048-token prefill of the reference's host
 *     (24 / 2 heads of 256) from 2591 to 2340 us.  Tensor memory: 256 columns of scores, NQ x hd of O.
 *     PAIR: behind a prefix two blocks on neighbouring SMs form one product of 256 rows (cta_group::2): each has queries,
 *     scores, weights and outputs of its own and half of every K and V image, which the tensor cores read from both.  The first
 *     block issues; the second tells it what has landed.  Half the images' traffic from L2, and Q . K^T at the tensor core's
 *     pace: 128 positions of hd 256 with both images 4650 -> 4130 cycles (4096 of products), of two groups at hd 128 3370 -> 3170.
 *     What orders the two blocks.  Weights, scores and outputs lie in tensor memory: tcgen05 fences before an arrival and behind a
 *     wait, both relaxed at cluster scope.  Images: a warp of the second block waits for its halves (acquire), and
 *     arrives behind a release that is restricted to shared memory, which the first block's wait acquires.  A full release takes
 *     1000 cycles: one for each image, slower than one block; one for all that has landed meanwhile, 0.8 us per block (512 tokens
 *     over 640 rows of 24 / 2 heads of 256 38.9 -> 39.9 us); restricted it is not to be seen.  A copy by tensor map can count
 *     its bytes on the other block's barrier, but fetching the map cost the reference host's 2048-token chunk 2674 -> 2751 us.
 *  3. Where the last wave of blocks leaves much of the SMs idle, the positions of its blocks, or of all, are split over
 *     several; those write (O, m, l) and q4_pf_merge_k combines them.
 *
 * Measured rates of tcgen05.mma with both operands in shared memory: 64 cycles per 128 x 128 x 16, 48 per 128 x 64 x 16
 * (4 KB of Q and 2 KB of K at 128 B/clk).  Single score buffers of 128 columns per group (all 512 columns in use as
 * well) make the products cheaper but leave a serial chain S -> softmax -> P . V -> Q . K^T per group: 3270 cycles per
 * 128 positions of both groups at 8192 tokens over 16 384, the tensor core 63 % busy.
 *
 * Every mbarrier wait is bounded: on expiry the thread raises a block-wide abort flag that every other wait polls, the
 * block records Q4E_CUDA in the status word, and still frees its tensor memory.
 */
#include <cuda_bf16.h>
#include <math_constants.h>
#include <string.h>
#include <type_traits>

#include "q4_internal.h"

namespace {

constexpr uint32_t PF_ROWS = 128, PF_BN = 128;              /* rows of a query group, positions of a tile */
constexpr uint32_t PF_CHUNK = 32768, PF_RING = 5;           /* operand image bytes, ring slots */
constexpr uint32_t PF_Q_BYTES = 65536;                      /* NQ x 128 rows x hd fp16, in every configuration at most this */
constexpr uint32_t PF_BAR_BYTES = 288 + 1024;               /* barriers and words; one float per softmax thread */
constexpr uint32_t PF_THREADS = 320;                        /* 8 softmax warps, the issuer, the producer */
constexpr uint32_t PF_SMEM = PF_Q_BYTES + PF_RING * PF_CHUNK + PF_BAR_BYTES + 1024;
constexpr uint32_t PF_SPIN_LIMIT = 1u << 22;
constexpr unsigned long long PF_LIMIT_NS = 2000000000ull;   /* a block that has not finished by then gives up */
constexpr float PF_RESCALE_TAU = 8.f;

struct __align__(16) PfMark { float k, v; uint32_t bad_rows, pad; };   /* factors of 32 staged rows, V rows that are not finite */

struct PrefillParams {
    uint32_t n_head, n_kvh, gqa, tpc /* tokens per query group */;
    const void *q;           /* [n_tok][n_head][hd] */
    const float *gate;
    void *out;               /* [n_tok][n_head][hd] */
    int q_bf16, out_bf16;
    uint32_t n_tok, kv_base, max_kv;
    float scale_log2e;
    const uint8_t *kimg, *vimg;   /* operand images [kv head][tile][chunk][32 KB] */
    uint32_t img_tiles;           /* tiles per kv head in the images */
    uint32_t n_split;             /* position ranges of equal tile count of the items that are split; > 1: partial results */
    float *part;                  /* [split][token][head][hd] unnormalised O */
    float2 *part_ml;              /* [split][token][head] running max (log2 units), sum */
    const PfMark *marks;          /* [kv head][32 positions], of caches that are not the library's */
    const uint32_t *flags;        /* [kv head][64 positions]: bytes that are not zero where K or V of 32 of them is marked */
    uint32_t *err;
};
struct PrefillTail : PrefillParams {
    uint32_t n_groups;            /* items, of a block's or a pair's query groups, per kv head; work items: kv head by kv head, last tokens first */
    uint32_t n_whole, n_late;     /* items that are one block each; later ones, n_split blocks each */
    uint32_t part_tok;            /* tokens below this may have parts */
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ float ex2f(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
/* two fp32 in one 64-bit register pair */
__device__ __forceinline__ uint64_t pack2(float a, float b) {
    uint64_t v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b));
    return v;
}
__device__ __forceinline__ float2 unpack2(uint64_t v) {
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
/* x * sigmoid(g); a gate below -126 / log2(e) gives 0 (1 / (1 + inf)) */
__device__ __forceinline__ float gated(float x, float g) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.f + ex2f(g * -1.4426950408889634f)));
    return x * r;
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ uint32_t h2u(__half2 h) { return *reinterpret_cast<uint32_t *>(&h); }

__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr) {
    /* K-major operand tile, 128-byte rows, 16-byte chunks XOR-swizzled by (row & 7) inside 8-row groups:
     * start >> 4 | LBO (unused with swizzle) = 1 | SBO = 1024 B >> 4 | version 1 | SWIZZLE_128B (2) */
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
/* The issuing warp runs converged and one elected lane's predicate guards the instruction: the descriptors then stay in
 * uniform registers.  Issued from a branch that only one lane takes, each product costs about 107 cycles of moves
 * instead of the 64 that the tensor core needs for 128 x 128 x 16. */
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(p));
    return p;
}
template <bool PAIR>
__device__ __forceinline__ void umma_f16(uint32_t el, uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
    if constexpr (PAIR)
        asm volatile(
            "{\n\t.reg .pred p, e;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 e, %5, 0;\n\t"
            "@e tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(el) : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p, e;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 e, %5, 0;\n\t"
            "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(el) : "memory");
}
/* same product with the A operand in tensor memory (lane = row, one 32-bit column = two consecutive k) */
template <bool PAIR>
__device__ __forceinline__ void umma_f16_ta(uint32_t el, uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate) {
    if constexpr (PAIR)
        asm volatile(
            "{\n\t.reg .pred p, e;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 e, %5, 0;\n\t"
            "@e tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
            ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(el) : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p, e;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 e, %5, 0;\n\t"
            "@e tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
            ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(el) : "memory");
}
/* of a pair: on the barrier at that place in both blocks */
template <bool PAIR>
__device__ __forceinline__ void umma_commit(uint32_t el, uint32_t bar) {
    if constexpr (PAIR)
        asm volatile(
            "{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %1, 0;\n\t"
            "@e tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %2;\n\t}"
            ::"r"(bar), "r"(el), "h"((uint16_t)3) : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred e;\n\tsetp.ne.b32 e, %1, 0;\n\t"
            "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
            ::"r"(bar), "r"(el) : "memory");
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
/* One probe of a phase; the callers bound the number of probes.  What the arrivals order: OWN, what the block itself does; of either
 * block of a pair PAIR_TENSOR, accesses of tensor memory, between tcgen05 fences, and PAIR_BYTES, what lies in shared memory */
enum { OWN, PAIR_TENSOR, PAIR_BYTES };
template <int WHAT>
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t done;
    if constexpr (WHAT == PAIR_TENSOR)
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.relaxed.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    else if constexpr (WHAT == PAIR_BYTES)
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    return done != 0u;
}
/* a probe that returns at once */
__device__ __forceinline__ bool mbar_peek(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done) : "r"(bar), "r"(parity) : "memory");
    return done != 0u;
}
/* on the barrier at that place in the first block of the pair; what comes before it is ordered by a fence, of tcgen05 or release_shared */
__device__ __forceinline__ void mbar_arrive_first(uint32_t bar) {
    asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %0, 0;\n\tmbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [a];\n\t}"
                 ::"r"(bar) : "memory");
}
__device__ __forceinline__ void release_shared() { asm volatile("fence.release.sync_restrict::shared::cta.cluster;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t *r = reinterpret_cast<uint32_t *>(v);
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const float (&v)[32]) {
    const uint32_t *r = reinterpret_cast<const uint32_t *>(v);
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};"
        ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
          "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
          "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
          "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31]),
          "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }


/* ---- staging: rows [0, n) of (layer, kv head) -> operand images.  Per tile of 128 positions: NP * HD / 128 images of
 * K (128 rows x 128 dims: two blocks of 64 dims, rows of 128 bytes) and as many images' worth of V^T (two blocks of
 * 64 positions x HD dims).  Rows behind n are zero.  Block = 32 positions of one kv head, K or V (blockIdx.z); V goes
 * through shared memory to come out position-contiguous.  Short and bound by latency, hence the small blocks: 64
 * positions of K and V per block took 12.8 us for 2048 rows of hd 256, 2 kv heads. */
/* dims d .. d + 7 of a row as fp32 (exact for every kind) */
template <int LAY>
__device__ __forceinline__ void load8(const uint8_t *row, const uint8_t *srow, uint32_t d, float (&x)[8]) {
    if constexpr (LAY == LAY_F32) {
        const float4 a = *reinterpret_cast<const float4 *>(row + d * 4u), b = *reinterpret_cast<const float4 *>(row + d * 4u + 16u);
        x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
    } else if constexpr (LAY == LAY_F16) {
        const uint4 w = *reinterpret_cast<const uint4 *>(row + d * 2u);
        const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&u[i]));
            x[2 * i] = f.x; x[2 * i + 1] = f.y;
        }
    } else {
        uint32_t u[2];
        float s;
        if constexpr (LAY == LAY_Q8P) {
            const uint2 w = *reinterpret_cast<const uint2 *>(row + d);
            u[0] = w.x; u[1] = w.y;
            s = __half2float(reinterpret_cast<const __half *>(srow)[d >> 5]);
        } else {   /* 34-byte blocks {fp16 scale, 32 codes}, 2-byte aligned */
            const uint16_t *b = reinterpret_cast<const uint16_t *>(row + (d >> 5) * 34u);
            const uint16_t *c = b + 1 + ((d & 31u) >> 1);
            u[0] = (uint32_t)c[0] | ((uint32_t)c[1] << 16);
            u[1] = (uint32_t)c[2] | ((uint32_t)c[3] << 16);
            s = __half2float(__ushort_as_half(b[0]));
        }
#pragma unroll
        for (int i = 0; i < 8; i++) x[i] = (float)(int8_t)(u[i >> 2] >> (8 * (i & 3))) * s;   /* 8 + 11 bits: exact */
    }
}
/* A caller's cache may hold what fp16 does not: a code times its scale reaches 8.3e6, and rows may hold infinities or NaN.  A
 * group of 32 rows with a value beyond fp16 is staged by 2^-7, and its mark says so (K: scores are multiplied by it, V:
 * weights; both exact).  A V row with a value that is still not finite has that value staged as 0, or a token that does not
 * attend the row would get 0 x infinity, and its bit set: tokens that do attend it get NaN. */
constexpr float PF_HALF_END = 65520.f, PF_DOWN = 1.f / 128.f;   /* the least magnitude that rounds to an fp16 infinity */
template <int LAY, int HD, int NP>
__global__ void __launch_bounds__(256) q4_pf_stage_k(const Q4Cache C, uint32_t layer, uint32_t n, uint32_t tiles, uint32_t unit, uint8_t *kimg, uint8_t *vimg, PfMark *marks,
                                                     uint8_t *flags) {
    constexpr bool MARKS = LAY != LAY_Q8P;
    constexpr uint32_t PITCH = 34;   /* halves per dim row of the transposition tile (odd word count) */
    constexpr uint32_t CK = NP * HD / 128, CV = NP * HD / 128, PER = HD * 32u / 8u / 256u;   /* groups of 8 dims per thread */
    __shared__ __half tile[NP][HD * PITCH];
    __shared__ uint32_t bad_rows;
    const uint32_t kh = blockIdx.y, p0 = blockIdx.x * 32u, tid = threadIdx.x;
    q4d_pdl_wait();
    const uint8_t *sc = LAY == LAY_Q8P ? C.s + (uint64_t)layer * C.s_layer_stride + (uint64_t)kh * C.s_kvh_stride : nullptr;
    const uint64_t base = (uint64_t)layer * C.layer_stride + (uint64_t)kh * C.kvh_stride;
    float x[PER][8];
    auto fit = [&]() -> float {   /* the group's factor; all threads */
        bool over = false;
#pragma unroll
        for (uint32_t it = 0; it < PER; it++)
#pragma unroll
            for (int j = 0; j < 8; j++) over = over || (fabsf(x[it][j]) >= PF_HALF_END && fabsf(x[it][j]) < PF_HALF_END / PF_DOWN);
        if (!__syncthreads_or(over)) return 1.f;
#pragma unroll
        for (uint32_t it = 0; it < PER; it++)
#pragma unroll
            for (int j = 0; j < 8; j++) x[it][j] *= PF_DOWN;
        return 1.f / PF_DOWN;
    };
    const size_t group = (size_t)kh * tiles * (PF_BN / 32u) + blockIdx.x;
    PfMark *mark = marks + group;
    if (blockIdx.z == 0) {
        const uint8_t *kq = C.k + base;
        uint8_t *kt = kimg + ((size_t)kh * tiles + p0 / PF_BN) * CK * PF_CHUNK;
        /* of a pair each block holds half of every unit's rows */
        const uint32_t in = p0 % PF_BN, second = unit ? in >> (unit - 1u) & 1u : 0u, dims64 = unit ? 8192u : 16384u;   /* unit: log2 of its positions */
        const uint32_t row0 = unit ? (in >> unit << (unit - 1u)) + (in & ((1u << (unit - 1u)) - 1u)) : in;
        kt += second * (PF_CHUNK / 2u);
#pragma unroll
        for (uint32_t it = 0; it < PER; it++) {
            const uint32_t i = tid + 256u * it, p = p0 + i / (HD / 8u), c = i % (HD / 8u);
#pragma unroll
            for (int j = 0; j < 8; j++) x[it][j] = 0.f;
            if (p < n) load8<LAY>(kq + (uint64_t)p * C.tok_stride, sc + (uint64_t)p * C.s_tok_stride, c * 8u, x[it]);
        }
        if (MARKS) {
            const float f = fit();
            if (tid == 0) {
                mark->k = f;
                flags[group * 2u] = f != 1.f;
            }
        }
#pragma unroll
        for (uint32_t it = 0; it < PER; it++) {
            const uint32_t i = tid + 256u * it, R = row0 + i / (HD / 8u), c = i % (HD / 8u);
            uint8_t *dst = kt + (c >> 4) * PF_CHUNK + ((c >> 3) & 1u) * dims64 + R * 128u + (((c & 7u) ^ (R & 7u)) << 4);
            __half2 hi[4], lo[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                hi[j] = __floats2half2_rn(x[it][2 * j], x[it][2 * j + 1]);
                const float2 f = __half22float2(hi[j]);
                lo[j] = __floats2half2_rn(x[it][2 * j] - f.x, x[it][2 * j + 1] - f.y);
            }
            *reinterpret_cast<uint4 *>(dst) = make_uint4(h2u(hi[0]), h2u(hi[1]), h2u(hi[2]), h2u(hi[3]));
            if (NP == 2) *reinterpret_cast<uint4 *>(dst + (HD / 128) * PF_CHUNK) = make_uint4(h2u(lo[0]), h2u(lo[1]), h2u(lo[2]), h2u(lo[3]));
        }
        return;
    }
    const uint8_t *vq = C.v + base;
    /* a tile's images in the order of their use: hd 256 {value, rest} of its first 64 positions, then of the others; hd 128
     * value, rest, both halves in each */
    const uint32_t half = (p0 / 64u) & 1u;
    uint8_t *vt = vimg + ((size_t)kh * tiles + p0 / PF_BN) * CV * PF_CHUNK + (HD == 256 ? half * NP * PF_CHUNK : half * (unit ? HD * 64u : HD * 128u));
    if (MARKS && tid == 0) bad_rows = 0u;
#pragma unroll
    for (uint32_t it = 0; it < PER; it++) {   /* lanes on consecutive rows: the 2-byte stores below do not conflict */
        const uint32_t i = tid + 256u * it, p = p0 + (i & 31u), c = i >> 5;
#pragma unroll
        for (int j = 0; j < 8; j++) x[it][j] = 0.f;
        if (p < n) load8<LAY>(vq + (uint64_t)p * C.tok_stride, sc + (uint64_t)p * C.s_tok_stride + 2u * (HD / 32u), c * 8u, x[it]);
    }
    float f = 1.f;
    if (MARKS) f = fit();
    uint32_t bad = 0;
#pragma unroll
    for (uint32_t it = 0; it < PER; it++) {
        const uint32_t i = tid + 256u * it;
        bool finite = true;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            if (MARKS && !(fabsf(x[it][j]) < PF_HALF_END)) {
                finite = false;
                x[it][j] = 0.f;
            }
            const __half h = __float2half_rn(x[it][j]);
            tile[0][((i >> 5) * 8u + j) * PITCH + (i & 31u)] = h;
            if (NP == 2) tile[NP - 1][((i >> 5) * 8u + j) * PITCH + (i & 31u)] = __float2half_rn(x[it][j] - __half2float(h));
        }
        if (MARKS) bad |= __ballot_sync(0xffffffffu, !finite);
    }
    if (MARKS && bad && (tid & 31u) == 0u) atomicOr(&bad_rows, bad);
    __syncthreads();
    if (MARKS && tid == 0) {
        mark->v = f;
        mark->bad_rows = bad_rows;
        flags[group * 2u + 1u] = f != 1.f || bad_rows;
    }
#pragma unroll
    for (int im = 0; im < NP; im++)
#pragma unroll
        for (uint32_t it = 0; it < PER; it++) {
            const uint32_t i = tid + 256u * it, d = i >> 2, c = (p0 & 63u) / 8u + (i & 3u), second = unit && HD == 128 ? d >> 6 : 0u;   /* hd 256: halves lie behind one another anyway */
            const uint32_t *w = reinterpret_cast<const uint32_t *>(tile[im] + d * PITCH + (i & 3u) * 8u);
            *reinterpret_cast<uint4 *>(vt + im * PF_CHUNK + second * 8192u + d * 128u + ((c ^ (d & 7u)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
        }
}

/* the rest of a wait whose first test found the phase incomplete: at most two seconds from the block's start, and no
 * longer than every other thread of the block; out of line, so that the loops around it stay short */
template <int WHAT>
__device__ __noinline__ bool pf_wait(uint32_t bar, uint32_t parity, uint32_t s_abort, unsigned long long t_start) {
    for (uint32_t i = 0; i < PF_SPIN_LIMIT; i++) {
        if (mbar_test<WHAT>(bar, parity)) return true;
        if ((i & 63u) == 63u) {
            uint32_t a;
            asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(a) : "r"(s_abort) : "memory");
            if (a) return false;
            if (global_ns() - t_start > PF_LIMIT_NS) break;
        }
    }
    asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(s_abort), "r"(1u) : "memory");
    return false;
}
/* HD: head size; NQ: query groups per block; NP: images per 128 dims of K and V (2: value and remainder); MARKS: rows may
 * have been scaled or not be finite; PAIR: two blocks per item; TAIL: the grid is a list of items, the last ones in ranges, else (groups, kv heads, ranges):
 * where a block learns only when it runs whether it writes parts, one group's epilogue takes 0.6 us more (333 tokens 10.6 -> 11.2
 * us), two groups' no more.  Only the list's launches carry its numbers: with 16 bytes more of parameters the other forms were
 * compiled to 1 to 6 % slower code (24 / 2 heads of 256, fp16, 1500 tokens 62.5 -> 65.4 us). */
template <int HD, int NQ, int NP, bool MARKS, bool TAIL, bool PAIR>
__global__ void __launch_bounds__(PF_THREADS, 1) q4_prefill_k(const std::conditional_t<TAIL, PrefillTail, PrefillParams> P) {
    constexpr uint32_t CK = NP * HD / 128, CV = NP * HD / 128;   /* ring slots a K / V tile takes */
    static_assert(NQ == 1 || NP == 1, "two groups hold a tile's V and the next one's K at once: both images of them leave the ring no slack");
    constexpr uint32_t SW = 8;                                 /* softmax warps; then the issuer, then the producer */
    constexpr uint32_t O_COL = 256, TMEM_COLS = 512;           /* scores in the first 256 columns, O of group g at 256 + 128 g */
    constexpr uint32_t UN = NQ == 2 ? 64 : 128, SB = 2 * NQ;   /* positions of a unit, score buffers */
    constexpr uint32_t TU = 64;                                /* of them, those of one softmax thread */
    constexpr uint32_t QG_BYTES = PF_ROWS * HD * 2;            /* one group's queries */
    constexpr uint32_t CTAS = PAIR ? 2 : 1, SLOTS = PF_RING * CTAS, PIECE = PF_CHUNK / CTAS;   /* a pair's blocks hold half of each image */
    static_assert(NQ * QG_BYTES <= PF_Q_BYTES && O_COL + NQ * HD <= TMEM_COLS, "shared / tensor memory");
    extern __shared__ uint8_t smem_dyn[];
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    /* later token groups see more rows: launch them first so the tail of the grid is made of short blocks */
    const uint32_t rank = PAIR ? blockIdx.x & 1u : 0u, work = blockIdx.x / CTAS;
    uint32_t kh = blockIdx.y, t0 = (gridDim.x / CTAS - 1u - work) * (P.tpc * NQ * CTAS), range = 0, ranges = 1;
    if constexpr (TAIL) {
        const Q4PfItem it = q4i_pf_item(work, P.n_groups, P.n_whole, P.n_late, P.n_split);
        kh = it.kh;
        t0 = (P.n_groups - 1u - it.group) * (P.tpc * NQ * CTAS);
        range = it.range;
        ranges = it.ranges;
    }
    const uint32_t t_last = min(t0 + P.tpc * NQ * CTAS, P.n_tok) - 1u;
    t0 += rank * (P.tpc * NQ);   /* a pair's second block may have no tokens left: rows of zeros, none stored */

    /* 1024-byte aligned operand tiles (the swizzle pattern is anchored to the address) */
    const uint32_t sQ = (smem_u32(smem_dyn) + 1023u) & ~1023u, sR = sQ + PF_Q_BYTES, bars = sR + PF_RING * PF_CHUNK;
    const uint32_t full = bars, empty = bars + 80, bar_s = bars + 160, bar_p = bars + 192, bar_o = bars + 224,
                   s_tmem = bars + 240, s_abort = bars + 244, s_item = bars + 256, s_xch = bars + 288;

    const uint32_t inv_gqa = 65536u / P.gqa + 1u;   /* row / gqa = row * inv_gqa >> 16 for rows below 128, gqa up to 16 */
    const uint32_t cta_nkv = min(P.kv_base + t_last + 1u, P.max_kv);
    const uint32_t all_tiles = (cta_nkv + PF_BN - 1u) / PF_BN;
    /* this block's range of tiles */
    const uint32_t j0 = TAIL ? all_tiles * range / ranges : (uint32_t)((uint64_t)all_tiles * blockIdx.z / P.n_split);   /* at most 2^25 tiles, 16 ranges */
    const uint32_t j1 = TAIL ? all_tiles * (range + 1u) / ranges : (uint32_t)((uint64_t)all_tiles * (blockIdx.z + 1u) / P.n_split);
    const uint32_t n_tiles = j1 - j0;
    /* units per group: the last tile may be needed in half only */
    const uint32_t n_seq = NQ == 2 ? min(n_tiles * 2u, (cta_nkv - j0 * PF_BN + 63u) / 64u) : n_tiles;

    if (warp == SW) {
        if (lane == 0) {
#pragma unroll
            for (uint32_t s = 0; s < SLOTS; s++) {
                mbar_init(full + 8 * s, PAIR && rank == 0u ? 2 : 1);   /* the other block's half counts too */
                mbar_init(empty + 8 * s, 1);
            }
#pragma unroll
            for (uint32_t s = 0; s < 4; s++) {
                mbar_init(bar_s + 8 * s, 1);
                mbar_init(bar_p + 8 * s, PAIR ? 2u * SW / NQ : SW * 32u / NQ);
            }
            mbar_init(bar_o, 1);
            mbar_init(bar_o + 8, 1);
            asm volatile("st.shared.u32 [%0], %1;" ::"r"(s_abort), "r"(0u) : "memory");
            if (TAIL) asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(s_item), "r"(t0), "r"(kh), "r"(range), "r"((uint32_t)(ranges > 1u)) : "memory");
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncwarp();
        if constexpr (PAIR) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_tmem), "r"(TMEM_COLS) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(s_tmem), "r"(TMEM_COLS) : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
    }
    /* Queries and gates are older than the staging launch before this one, and that lets this grid start only after it has
     * waited for everything older: they need no wait.  The images do. */
    if (warp >= SW) q4d_pdl_wait();
    if (warp < SW) {
        /* ---- queries as fp16 (exact for normal bf16 values), K-major swizzled, blocks of 64 dims: 8 dims per thread
         * and step, whole rows per warp step */
        constexpr uint32_t PER = HD / 8u, STEPS = NQ * PF_ROWS * PER / (SW * 32u), BATCH = 8u;   /* loads in flight before the first store */
#pragma unroll 1
        for (uint32_t k0 = 0; k0 < STEPS; k0 += BATCH) {
            uint4 w[BATCH][2];
#pragma unroll
            for (uint32_t k = 0; k < BATCH; k++) {
                const uint32_t i = tid + (k0 + k) * SW * 32u, row = i / PER, c = i % PER, g = row / PF_ROWS, r = row % PF_ROWS;
                const uint32_t tl = r * inv_gqa >> 16, tok = t0 + g * P.tpc + tl;
                w[k][0] = w[k][1] = make_uint4(0u, 0u, 0u, 0u);
                if (tl < P.tpc && tok < P.n_tok) {
                    const size_t off = ((size_t)tok * P.n_head + (size_t)kh * P.gqa + (r - tl * P.gqa)) * HD + c * 8u;
                    if (P.q_bf16) {
                        w[k][0] = *reinterpret_cast<const uint4 *>(reinterpret_cast<const __nv_bfloat16 *>(P.q) + off);
                    } else {
                        w[k][0] = *reinterpret_cast<const uint4 *>(reinterpret_cast<const float *>(P.q) + off);
                        w[k][1] = *reinterpret_cast<const uint4 *>(reinterpret_cast<const float *>(P.q) + off + 4);
                    }
                }
            }
#pragma unroll
            for (uint32_t k = 0; k < BATCH; k++) {
                const uint32_t i = tid + (k0 + k) * SW * 32u, row = i / PER, c = i % PER, g = row / PF_ROWS, r = row % PF_ROWS;
                const uint32_t in[8] = {w[k][0].x, w[k][0].y, w[k][0].z, w[k][0].w, w[k][1].x, w[k][1].y, w[k][1].z, w[k][1].w};
                uint32_t o[4];
#pragma unroll
                for (int e = 0; e < 4; e++)
                    o[e] = P.q_bf16 ? h2u(__floats2half2_rn(__uint_as_float(in[e] << 16), __uint_as_float(in[e] & 0xffff0000u)))
                                    : h2u(__floats2half2_rn(__uint_as_float(in[2 * e]), __uint_as_float(in[2 * e + 1])));
                const uint32_t a = sQ + g * QG_BYTES + (c >> 3) * (PF_ROWS * 128u) + r * 128u + (((c & 7u) ^ (r & 7u)) << 4);
                asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(a), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]) : "memory");
            }
        }
        fence_async_smem();
        q4d_pdl_wait();
    }
    tc_fence_before();
    if (PAIR) {               /* barriers initialised, queries in place, tensor memory allocated */
        cluster_arrive();
        cluster_wait();
    } else {
        __syncthreads();
    }
    tc_fence_after();
    uint32_t tmem;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(s_tmem));

    constexpr uint32_t IDESC_QK = (1u << 4) | ((uint32_t)(UN >> 3) << 17) | ((uint32_t)(PF_ROWS * CTAS >> 4) << 24);
    constexpr uint32_t IDESC_PV = (1u << 4) | ((uint32_t)(HD >> 3) << 17) | ((uint32_t)(PF_ROWS * CTAS >> 4) << 24);
    const unsigned long long t_start = global_ns();
    constexpr int BYTES = PAIR ? PAIR_BYTES : OWN, TENSOR = PAIR ? PAIR_TENSOR : OWN;
    auto wait = [&](uint32_t bar, uint32_t parity) -> bool { return mbar_test<TENSOR>(bar, parity) || pf_wait<TENSOR>(bar, parity, s_abort, t_start); };
    /* by a whole warp, which goes on as one; the test that succeeds at once stays in line */
    auto all_wait = [&](uint32_t bar, uint32_t parity) -> bool {
        if (__builtin_expect(__all_sync(0xffffffffu, mbar_test<TENSOR>(bar, parity)), 1)) return true;
        return __all_sync(0xffffffffu, pf_wait<TENSOR>(bar, parity, s_abort, t_start));
    };
    auto all_landed = [&](uint32_t bar, uint32_t parity) -> bool {
        if (__builtin_expect(__all_sync(0xffffffffu, mbar_test<BYTES>(bar, parity)), 1)) return true;
        return __all_sync(0xffffffffu, pf_wait<BYTES>(bar, parity, s_abort, t_start));
    };
    /* order of the images in the ring, that of their first use: K0 V0 K1 V1 .. where two groups share a tile, K0 K1 V0 K2
     * V1 .. V(n-1) where units are tiles (the scores run a tile and two tiles ahead of P . V) */
    bool ok = true;

    if (warp == SW + 1) {
        /* ================= producer: one thread keeps the ring full ================= */
        if (lane == 0 && n_tiles > 0) {
            uint32_t at = 0;
            auto load = [&](const uint8_t *src, uint32_t chunks) {
                for (uint32_t c = 0; c < chunks && ok; c++, at++) {
                    const uint32_t s = at % SLOTS, use = at / SLOTS;
                    if (use > 0) ok = mbar_test<BYTES>(empty + 8 * s, (use - 1u) & 1u) || pf_wait<BYTES>(empty + 8 * s, (use - 1u) & 1u, s_abort, t_start);
                    if (ok) {
                        mbar_expect_tx(full + 8 * s, PIECE);
                        bulk_load(sR + s * PIECE, src + (size_t)c * PF_CHUNK + rank * PIECE, PIECE, full + 8 * s);
                    } else {
                        return;
                    }
                }
            };
            const uint8_t *ks = P.kimg + ((size_t)kh * P.img_tiles + j0) * CK * PF_CHUNK, *vs = P.vimg + ((size_t)kh * P.img_tiles + j0) * CV * PF_CHUNK;
            load(ks, CK);
            if (NQ == 1 && n_tiles > 1) load(ks + (size_t)CK * PF_CHUNK, CK);
            for (uint32_t j = 0; j < n_tiles && ok; j++) {
                load(vs + (size_t)j * CV * PF_CHUNK, CV);
                if (j + (3u - NQ) < n_tiles) load(ks + (size_t)(j + (3u - NQ)) * CK * PF_CHUNK, CK);
            }
            /* A pair: the last images' slots have been told free before either block leaves, or that would reach shared memory that is
             * another block's by then.  (Of two groups the last tile's V is not, where only its first half is needed.) */
            if (PAIR && ok)
                for (uint32_t t = at > SLOTS ? at - SLOTS : 0, end = at - (NQ == 2 ? n_seq & 1u : 0u); t < end && ok; t++)
                    ok = mbar_test<BYTES>(empty + 8 * (t % SLOTS), (t / SLOTS) & 1u) || pf_wait<BYTES>(empty + 8 * (t % SLOTS), (t / SLOTS) & 1u, s_abort, t_start);
            /* Gave up somewhere: copies still in flight must land before the block's shared memory is released
             * (bounded again; these probes ignore the abort flag; phases that completed long ago answer at once). */
            if (!ok)
                for (uint32_t t = at > SLOTS ? at - SLOTS : 0; t < at; t++)
                    for (uint32_t i = 0; i < 4096u && !mbar_test<BYTES>(full + 8 * (t % SLOTS), (t / SLOTS) & 1u); i++) {}
        }
    } else if (PAIR && warp == SW && rank != 0u) {
        /* ================= second block of a pair: the products are issued in the first, which learns here what has landed ====== */
        /* All that has landed at once (one by one the reference host's chunk takes 2683 us, so 2671).  A slot's next image is not
         * requested before this one has been told and used: the phases that are looked at are the present ones. */
        for (uint32_t at = 0, n = n_tiles * (CK + CV); at < n;) {
            const uint32_t i = at + lane;
            const uint32_t here = __ballot_sync(0xffffffffu, lane < SLOTS && i < n && mbar_peek(full + 8 * (i % SLOTS), (i / SLOTS) & 1u));
            const uint32_t k = (uint32_t)__ffs((int)~here) - 1u;
            if (k == 0u) {
                ok = all_landed(full + 8 * (at % SLOTS), (at / SLOTS) & 1u);
                if (!ok) break;
                continue;
            }
            release_shared();
            if (lane < k) mbar_arrive_first(full + 8 * (i % SLOTS));
            at += k;
        }
    } else if (warp == SW) {
        /* ================= tensor-core issuer: a converged warp, one elected lane ================= */
        if (n_tiles > 0) {
            const uint32_t el = elect_one();
            /* the ring is consumed in order: (slot, phase) of the next image */
            uint32_t slot = 0, phase = 0;
            auto take = [&]() -> uint32_t {
                const uint32_t s = slot;
                ok = ok && all_landed(full + 8 * s, phase);
                if (++slot == SLOTS) { slot = 0; phase ^= 1u; }
                return s;
            };
            const uint64_t q_desc = umma_desc(sQ), r_desc = umma_desc(sR);   /* byte offsets / 16 are added to these */
            auto qk_chunk = [&](uint32_t s_col, uint32_t g, uint32_t c, uint32_t s, uint32_t row0) {
                const uint64_t qd = q_desc + ((g * QG_BYTES + (c % (HD / 128)) * (2u * PF_ROWS * 128u)) >> 4), kd = r_desc + ((s * PIECE + row0 * 128u / CTAS) >> 4);
#pragma unroll
                for (uint32_t kk = 0; kk < 8; kk++)
                    umma_f16<PAIR>(el, tmem + s_col, qd + (((kk >> 2) * (PF_ROWS * 128u) + (kk & 3) * 32u) >> 4),
                                   kd + (((kk >> 2) * (PF_BN / CTAS * 128u) + (kk & 3) * 32u) >> 4), IDESC_QK, (c | kk) > 0);
            };
            auto pv_half = [&](uint32_t s_col, uint32_t g, uint32_t s, uint32_t half_off, bool first) {
                const uint64_t vd = r_desc + ((s * PIECE + half_off / CTAS) >> 4);
#pragma unroll
                for (uint32_t kk = 0; kk < 4; kk++)
                    umma_f16_ta<PAIR>(el, tmem + O_COL + g * 128u, tmem + s_col + kk * 8u, vd + kk * 2u, IDESC_PV, (first && kk == 0) ? 0u : 1u);
            };
            if (NQ == 2) {
                /* per tile: its P . V for both groups and both halves, each followed by the scores that take over the buffer */
                uint32_t ks[CK];
#pragma unroll
                for (uint32_t c = 0; c < CK; c++) ks[c] = take();
                tc_fence_after();
                if (ok) {
#pragma unroll
                    for (uint32_t e = 0; e < 4; e++)
                        if ((e >> 1) < n_seq) {
#pragma unroll
                            for (uint32_t c = 0; c < CK; c++) qk_chunk((e & 1u) * 128u + (e >> 1) * 64u, e & 1u, c, ks[c], (e >> 1) * 64u);
                            umma_commit<PAIR>(el, bar_s + 8 * e);
                        }
#pragma unroll
                    for (uint32_t c = 0; c < CK; c++) umma_commit<PAIR>(el, empty + 8 * ks[c]);
                }
                for (uint32_t j = 0; j < n_tiles && ok; j++) {
                    const uint32_t sv = take();
                    const bool more = j + 1u < n_tiles;
                    if (more) {
#pragma unroll
                        for (uint32_t c = 0; c < CK; c++) ks[c] = take();
                    }
#pragma unroll
                    for (uint32_t e = 0; e < 4; e++) {   /* buffer e: half e >> 1, group e & 1 */
                        if (2u * j + (e >> 1) >= n_seq) continue;
                        ok = ok && all_wait(bar_p + 8 * e, j & 1u);
                        tc_fence_after();
                        if (!ok) break;
                        pv_half((e & 1u) * 128u + (e >> 1) * 64u, e & 1u, sv, (e >> 1) * (HD * 128u), j == 0 && e < 2);
                        umma_commit<PAIR>(el, bar_o + 8 * (e & 1u));
                        if (e == 3) umma_commit<PAIR>(el, empty + 8 * sv);
                        if (2u * (j + 1u) + (e >> 1) < n_seq) {
#pragma unroll
                            for (uint32_t c = 0; c < CK; c++) qk_chunk((e & 1u) * 128u + (e >> 1) * 64u, e & 1u, c, ks[c], (e >> 1) * 64u);
                            umma_commit<PAIR>(el, bar_s + 8 * e);
                        }
                    }
                    if (more && ok) {
#pragma unroll
                        for (uint32_t c = 0; c < CK; c++) umma_commit<PAIR>(el, empty + 8 * ks[c]);
                    }
                }
            } else {
                auto issue_qk = [&](uint32_t j) {
                    for (uint32_t c = 0; c < CK && ok; c++) {
                        const uint32_t s = take();
                        tc_fence_after();
                        if (!ok) return;
                        qk_chunk((j & 1u) * 128u, 0u, c, s, 0u);
                        umma_commit<PAIR>(el, empty + 8 * s);
                    }
                    umma_commit<PAIR>(el, bar_s + 8 * (j & 1u));
                };
                issue_qk(0);
                if (ok && n_tiles > 1) issue_qk(1);
                for (uint32_t j = 0; j < n_tiles && ok; j++) {
                    uint32_t sv[NP];
#pragma unroll
                    for (uint32_t h = 0; h < 2; h++) {   /* 64 positions each; the operands land while the softmax runs */
                        if (HD == 256 || h == 0) {
#pragma unroll
                            for (int im = 0; im < NP; im++) sv[im] = take();
                        }
                        if (h == 0) ok = ok && all_wait(bar_p + 8 * (j & 1u), (j >> 1) & 1u);
                        tc_fence_after();
                        if (!ok) break;
#pragma unroll
                        for (int im = 0; im < NP; im++) pv_half((j & 1u) * 128u + h * 64u, 0u, sv[im], HD == 256 ? 0u : h * (HD * 128u), j == 0 && h == 0 && im == 0);
                        if (HD == 256 || h == 1) {
#pragma unroll
                            for (int im = 0; im < NP; im++) umma_commit<PAIR>(el, empty + 8 * sv[im]);
                        }
                    }
                    if (ok) {
                        umma_commit<PAIR>(el, bar_o);
                        if (j + 2u < n_tiles) issue_qk(j + 2u);
                    }
                }
            }
        }
    } else {
        /* ================= softmax: thread r of group g owns row r of that group's queries; with one group, thread r of
         * half h owns 64 of a unit's positions of row r ================= */
        const uint32_t g = NQ == 2 ? warp >> 2 : 0u, h = NQ == 2 ? 0u : warp >> 2, r = tid & 127u, t_lane = tmem + (((warp & 3u) * 32u) << 16);
        const uint32_t tl = r * inv_gqa >> 16, tok = t0 + g * P.tpc + tl, head = kh * P.gqa + r - tl * P.gqa;   /* rows past tpc * gqa or past n_tok are padding */
        const bool row_live = tl < P.tpc && tok < P.n_tok;
        /* this row attends positions [0, row_nkv); padding rows (queries of zeros, never stored) need no mask */
        const uint32_t row_nkv = row_live ? min(P.kv_base + tok + 1u, P.max_kv) : 0xffffffffu;
        const uint32_t warp_min = __reduce_min_sync(0xffffffffu, row_nkv);
        /* the two warps of the same 32 rows (one group): all meetings are unconditional, so that they also end where one
         * of the two has given up */
        auto pair_sync = [&]() {
            __syncwarp();
            asm volatile("bar.sync %0, 64;" ::"r"(1u + (warp & 3u)) : "memory");
        };
        auto pair_any = [&](bool x) -> bool {
            uint32_t any;
            __syncwarp();
            asm volatile("{ .reg .pred p, q; setp.ne.u32 q, %1, 0; bar.red.or.pred p, %2, 64, q; selp.u32 %0, 1, 0, p; }"
                         : "=r"(any) : "r"((uint32_t)x), "r"(1u + (warp & 3u)) : "memory");
            return any != 0u;
        };
        auto partner = [&](float x) -> float {   /* the other half's value of this row; a meeting lies between two calls */
            asm volatile("st.shared.f32 [%0], %1;" ::"r"(s_xch + 4u * tid), "f"(x) : "memory");
            pair_sync();
            asm volatile("ld.shared.f32 %0, [%1];" : "=f"(x) : "r"(s_xch + 4u * (tid ^ 128u)) : "memory");
            return x;
        };
        float m_ref = -CUDART_INF_F, l_run = 0.f;
        /* of unit u, this thread's 64 positions; units of one group per block are 128 positions */
        const uint32_t *flag_at = P.flags + (size_t)kh * P.img_tiles * 2u + j0 * 2u + h;
        constexpr uint32_t FLAG_STEP = UN / 64u;
        uint32_t flag = MARKS && n_seq > 0 ? flag_at[0] : 0u;
        for (uint32_t u = 0; u < n_seq && (NQ == 1 || ok); u++) {
            const uint32_t i = u * NQ + g, b = i % SB, use = (i / SB) & 1u, p0 = j0 * PF_BN + u * UN + h * TU;
            const uint32_t t_s = t_lane + (NQ == 2 ? g * 128u + (u & 1u) * 64u : b * 128u + h * TU);
            bool marked = false;   /* the same in all lanes; requested a unit ahead (with the marks themselves, and none ahead, 157 -> 187 us for 512 tokens over 32768 fp16 rows) */
            if (MARKS) {
                marked = flag != 0u;
                if (u + 1u < n_seq) flag = flag_at[(u + 1u) * FLAG_STEP];
            }
            ok = ok && all_wait(bar_s + 8 * b, use);   /* a warp goes on as one */
            if (NQ == 1 && !ok) {
                if (u == 0 || pair_any(false)) partner(0.f);
                continue;
            }
            tc_fence_after();
            float s[TU];
#pragma unroll
            for (int c = 0; c < (int)TU / 32; c++) tmem_ld32(t_s + 32 * c, *reinterpret_cast<float(*)[32]>(&s[32 * c]));
            tmem_wait_ld();
            if (MARKS && __builtin_expect(marked, 0)) {
#pragma unroll
                for (int i2 = 0; i2 < 2; i2++) {
                    const PfMark mk = P.marks[(size_t)kh * P.img_tiles * (PF_BN / 32u) + p0 / 32u + i2];
#pragma unroll
                    for (int k = 0; k < 32; k++) s[32 * i2 + k] = (mk.bad_rows >> k) & 1u ? CUDART_NAN_F : s[32 * i2 + k] * mk.k;
                }
            }
            if (__builtin_expect(p0 + TU > warp_min, 0)) {
#pragma unroll
                for (int k = 0; k < (int)TU; k++)
                    if (p0 + k >= row_nkv) s[k] = -CUDART_INF_F;
            }
            /* P against the reference maximum, as fp16 pairs; sums into ls */
            uint32_t pk[TU / 2];
            uint64_t ls[2];
            auto exps = [&]() {
                const float mneg = m_ref == -CUDART_INF_F ? 0.f : -m_ref;
                const uint64_t sc2 = pack2(P.scale_log2e, P.scale_log2e), mn2 = pack2(mneg, mneg);
                ls[0] = ls[1] = 0ull;
#pragma unroll
                for (int k = 0; k < (int)TU / 2; k++) {
                    const float2 x = unpack2(fma2(pack2(s[2 * k], s[2 * k + 1]), sc2, mn2));
                    const float e0 = ex2f(x.x), e1 = ex2f(x.y);
                    ls[k & 1] = add2(ls[k & 1], pack2(e0, e1));
                    pk[k] = h2u(__floats2half2_rn(e0, e1));
                }
            };
            /* The exponentials start against the maximum of the units before, while this unit's own is still being
             * formed: the reference only has to be within 2^8 of it.  Where it is not (the first unit, a large new
             * score) the reference moves and they are taken again. */
            if (NQ == 2 || u > 0) exps();   /* of a short chunk the first unit is a good part */
            float mx[4] = {-CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F, -CUDART_INF_F};
#pragma unroll
            for (int k = 0; k < (int)TU; k += 8) {
                mx[0] = fmaxf(fmaxf(mx[0], s[k]), s[k + 1]); mx[1] = fmaxf(fmaxf(mx[1], s[k + 2]), s[k + 3]);
                mx[2] = fmaxf(fmaxf(mx[2], s[k + 4]), s[k + 5]); mx[3] = fmaxf(fmaxf(mx[3], s[k + 6]), s[k + 7]);
            }
            float m_new = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * P.scale_log2e;   /* scale > 0 */
            bool grow = m_new > m_ref + PF_RESCALE_TAU;   /* also true on the first live unit (m_ref = -inf) */
            const bool any = NQ == 2 ? __any_sync(0xffffffffu, grow) : u == 0 || pair_any(grow);
            if (__builtin_expect(any, 0)) {
                if (NQ == 1) {   /* both halves of a row keep one reference: they share its O */
                    m_new = fmaxf(m_new, partner(m_new));
                    grow = m_new > m_ref + PF_RESCALE_TAU;
                }
                float alpha = 1.f;
                if (grow) {
                    alpha = ex2f(m_ref - m_new);             /* 0 on the first live unit */
                    m_ref = m_new;
                    l_run *= alpha;
                }
                exps();
                /* O is rescaled only here (one group: half of its columns by each half); the group's previous P . V must
                 * have drained first */
                if (u > 0) {
                    ok = all_wait(bar_o + 8 * g, (u - 1u) & 1u) && ok;
                    tc_fence_after();
#pragma unroll 1
                    for (uint32_t c = h * (HD / 64); c < (NQ == 2 ? HD / 32 : (h + 1u) * (HD / 64)); c++) {
                        float o[32];
                        tmem_ld32(t_lane + O_COL + g * 128u + 32 * c, o);
                        tmem_wait_ld();
#pragma unroll
                        for (int k = 0; k < 32; k++) o[k] *= alpha;
                        tmem_st32(t_lane + O_COL + g * 128u + 32 * c, o);
                    }
                }
            }
            if (MARKS && __builtin_expect(marked, 0)) {   /* up to 2^8 x 2^7 */
#pragma unroll
                for (int i2 = 0; i2 < 2; i2++) {
                    const __half2 f = __float2half2_rn(P.marks[(size_t)kh * P.img_tiles * (PF_BN / 32u) + p0 / 32u + i2].v);
#pragma unroll
                    for (int k = 0; k < 16; k++) pk[16 * i2 + k] = h2u(__hmul2(*reinterpret_cast<const __half2 *>(&pk[16 * i2 + k]), f));
                }
            }
            /* P goes into the first half of the columns this thread has just read (two fp16 per column) */
            tmem_st32(t_s, *reinterpret_cast<const float(*)[32]>(&pk[0]));
            tmem_wait_st();
            /* A parity wait can tell the current phase from the one before it, no further, and bar_o's phases are not
             * followed unit by unit.  So the phase before the last is waited for here, while the last cannot
             * complete without this thread (that of unit n - 3 has: the scores of unit n - 1 were committed behind it). */
            if (u > 0 && u + 1u == n_seq) ok = all_wait(bar_o + 8 * g, (u - 1u) & 1u) && ok;
            tc_fence_before();
            if (PAIR) {
                __syncwarp();
                if (lane == 0) mbar_arrive_first(bar_p + 8 * b);
            } else {
                mbar_arrive(bar_p + 8 * b);
            }
            const float2 l0 = unpack2(ls[0]), l1 = unpack2(ls[1]);
            l_run += (l0.x + l0.y) + (l1.x + l1.y);
        }
        if (NQ == 1) {
            pair_sync();
            l_run += partner(l_run);
        }
        /* ---- epilogue: O / l * sigmoid(gate), or the unnormalised part of a split range.  32 columns at a time go
         * through the warp's share of the query tiles (read by no product any more), so that rows leave in whole lines.
         * Step q of a column block: 4 rows of 32 columns, 8 lanes each.  The gates are requested a whole column block
         * ahead, the first ones under the last product (requested behind their use a block took 2600 cycles, most of it
         * their latency).  One group: each half takes half of the columns (a warp alone is held up in turn by its
         * special-function steps, 700 cycles a block, and its stores, 450). */
        /* two groups: which item this is was left in shared memory (kept in registers through the loop above it cost the softmax 4
         * to 8 %; one group has registers to spare) */
        uint32_t e_t0 = t0, e_kh = kh, e_range = TAIL ? range : blockIdx.z, e_split = ranges > 1u;
        if (NQ == 2)
            asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(e_t0), "=r"(e_kh), "=r"(e_range), "=r"(e_split) : "r"(s_item) : "memory");
        const bool parts = TAIL ? e_split != 0u : P.n_split > 1u, gates = P.gate && !parts;
        const uint32_t w_row0 = (warp & 3u) * 32u;
        uint32_t off[8], live = 0;   /* in 16-byte units from the chunk's first token */
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const uint32_t row = w_row0 + 4u * q + (lane >> 3), ti = row * inv_gqa >> 16;
            if (ti < P.tpc && e_t0 + g * P.tpc + ti < P.n_tok) live |= 1u << q;
            off[q] = ((g * P.tpc + ti) * P.n_head + e_kh * P.gqa + (row - ti * P.gqa)) * (HD / 4u) + (lane & 7u);
        }
        const size_t first = (size_t)e_t0 * P.n_head * (HD / 4u);
        auto fetch_gates = [&](int c, float4 (&to)[8]) {
#pragma unroll
            for (int q = 0; q < 8; q++)
                if (gates && ((live >> q) & 1u)) to[q] = reinterpret_cast<const float4 *>(P.gate)[first + off[q] + 8u * c];
        };
        constexpr int NC = NQ == 2 ? HD / 32 : HD / 64;   /* column blocks of this warp */
        const int c0 = h * NC;
        float4 gt0[8], gt1[8];
        fetch_gates(c0, gt0);
        if (ok && n_seq > 0) ok = wait(bar_o + 8 * g, (n_seq - 1u) & 1u);
        ok = __all_sync(0xffffffffu, ok);
        tc_fence_after();

        if (ok) {
            const float inv = parts ? 1.f : l_run > 0.f ? 1.f / l_run : 0.f;
            float *buf = reinterpret_cast<float *>(smem_dyn + (sQ - smem_u32(smem_dyn)) + warp * (PF_Q_BYTES / SW));   /* [32][36] */
            uint32_t part_tok = P.n_tok;
            if constexpr (TAIL) part_tok = P.part_tok;
            const uint32_t etl = TAIL ? r * inv_gqa >> 16 : tl, etok = TAIL ? e_t0 + g * P.tpc + etl : tok, ehead = TAIL ? e_kh * P.gqa + (r - etl * P.gqa) : head;
            if (parts && (TAIL ? etl < P.tpc && etok < P.n_tok : row_live) && h == 0)
                P.part_ml[((size_t)e_range * part_tok + etok) * P.n_head + ehead] = make_float2(m_ref, l_run);
            auto columns = [&](int c, float4 (&gs)[8]) {
                float o[32];
                if (n_tiles > 0) {
                    tmem_ld32(t_lane + O_COL + g * 128u + 32 * c, o);
                    tmem_wait_ld();
                } else {
#pragma unroll
                    for (int k = 0; k < 32; k++) o[k] = 0.f;
                }
                __syncwarp();
#pragma unroll
                for (int k = 0; k < 32; k += 4)
                    *reinterpret_cast<float4 *>(buf + lane * 36u + k) = make_float4(o[k] * inv, o[k + 1] * inv, o[k + 2] * inv, o[k + 3] * inv);
                __syncwarp();
                float4 x[8];   /* all eight at once: a step after the other is 300 cycles of latency each */
#pragma unroll
                for (int q = 0; q < 8; q++) x[q] = *reinterpret_cast<const float4 *>(buf + (4u * q + (lane >> 3)) * 36u + 4u * (lane & 7u));
                if (gates) {
#pragma unroll
                    for (int q = 0; q < 8; q++) {
                        x[q].x = gated(x[q].x, gs[q].x); x[q].y = gated(x[q].y, gs[q].y);
                        x[q].z = gated(x[q].z, gs[q].z); x[q].w = gated(x[q].w, gs[q].w);
                    }
                }
                if (parts) {
#pragma unroll
                    for (int q = 0; q < 8; q++)
                        if ((live >> q) & 1u) reinterpret_cast<float4 *>(P.part)[(size_t)e_range * part_tok * P.n_head * (HD / 4u) + first + off[q] + 8u * c] = x[q];
                } else if (P.out_bf16) {
#pragma unroll
                    for (int q = 0; q < 8; q++) {
                        const __nv_bfloat162 b0 = __floats2bfloat162_rn(x[q].x, x[q].y), b1 = __floats2bfloat162_rn(x[q].z, x[q].w);
                        if ((live >> q) & 1u)
                            reinterpret_cast<uint2 *>(P.out)[first + off[q] + 8u * c] = make_uint2(*reinterpret_cast<const uint32_t *>(&b0), *reinterpret_cast<const uint32_t *>(&b1));
                    }
                } else {
#pragma unroll
                    for (int q = 0; q < 8; q++)
                        if ((live >> q) & 1u) reinterpret_cast<float4 *>(P.out)[first + off[q] + 8u * c] = x[q];
                }
            };
#pragma unroll 1
            for (int c = c0; c < c0 + NC; c += 2) {
                fetch_gates(c + 1, gt1);
                columns(c, gt0);
                if (c + 2 < c0 + NC) fetch_gates(c + 2, gt0);
                columns(c + 1, gt1);
            }
        }
    }
    if (!ok && lane == 0) atomicOr(P.err, (uint32_t)Q4E_CUDA);
    tc_fence_before();
    if (PAIR) {   /* neither block leaves while products read its memory or the other arrives on its barriers */
        __syncwarp();
        cluster_arrive();
        cluster_wait();
    } else {
        __syncthreads();
    }
    if (warp == SW) {
        if constexpr (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
    }
}

/* ---- the parts of split position ranges -> out: thread = 4 dims of one (token, head); TAIL: only some items have parts */
template <bool TAIL>
__global__ void __launch_bounds__(256) q4_pf_merge_k(const std::conditional_t<TAIL, PrefillTail, PrefillParams> P, uint32_t hd, uint64_t total4, uint32_t tok_per_group) {
    const uint64_t i = (uint64_t)blockIdx.x * 256u + threadIdx.x;
    q4d_pdl_wait();
    if (i >= total4) return;
    const uint64_t row = i / (hd / 4u);
    uint64_t rows = (uint64_t)P.n_tok * P.n_head;
    if constexpr (TAIL) {   /* at most a block's rows per SM; where all items have parts these divisions took 0.5 us */
        const uint32_t tok = (uint32_t)row / P.n_head, head = (uint32_t)row % P.n_head;
        if (head / P.gqa * P.n_groups + (P.n_groups - 1u - tok / tok_per_group) < P.n_whole) return;   /* one block's, finished */
        rows = (uint64_t)P.part_tok * P.n_head;
    }
    float M = -CUDART_INF_F;
    for (uint32_t s = 0; s < P.n_split; s++) M = fmaxf(M, P.part_ml[s * rows + row].x);
    const float Mu = M == -CUDART_INF_F ? 0.f : M;
    float L = 0.f;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t s = 0; s < P.n_split; s++) {
        const float2 ml = P.part_ml[s * rows + row];
        const float w = ml.y > 0.f ? ex2f(ml.x - Mu) : 0.f;
        const float4 a = reinterpret_cast<const float4 *>(P.part)[s * total4 + i];
        L = fmaf(w, ml.y, L);
        x.x = fmaf(w, a.x, x.x); x.y = fmaf(w, a.y, x.y); x.z = fmaf(w, a.z, x.z); x.w = fmaf(w, a.w, x.w);
    }
    const float inv = L > 0.f ? 1.f / L : 0.f;
    x.x *= inv; x.y *= inv; x.z *= inv; x.w *= inv;
    if (P.gate) {
        const float4 gt = reinterpret_cast<const float4 *>(P.gate)[i];
        x.x = gated(x.x, gt.x); x.y = gated(x.y, gt.y);
        x.z = gated(x.z, gt.z); x.w = gated(x.w, gt.w);
    }
    if (P.out_bf16) {
        const __nv_bfloat162 b0 = __floats2bfloat162_rn(x.x, x.y), b1 = __floats2bfloat162_rn(x.z, x.w);
        reinterpret_cast<uint2 *>(P.out)[i] = make_uint2(*reinterpret_cast<const uint32_t *>(&b0), *reinterpret_cast<const uint32_t *>(&b1));
    } else {
        reinterpret_cast<float4 *>(P.out)[i] = x;
    }
}

/* ---- host side: workspace, launches */
/* operand images of the rows a chunk can see, and the parts of split ranges; grows on demand, never inside a capture */
uint8_t *g_stage = nullptr;
size_t g_stage_bytes = 0;
uint32_t g_layout[3] = {};   /* of the last chunk: whole items, split ones, their ranges */
/* 1 = there, 0 = an error, -1 = not to be had: inside a capture, or no memory is left for it */
int stage_reserve(size_t bytes) {
    if (bytes <= g_stage_bytes) {
        g_q4.stage_captured = g_q4.stage_captured || g_q4.capturing;
        return 1;
    }
    if (g_q4.capturing) return -1;
    if (!q4i_check(cudaStreamSynchronize(g_q4.stream), "prefill staging sync")) return 0;
    q4i_give_back(g_stage, g_q4.stage_captured);
    g_stage = nullptr;
    g_stage_bytes = 0;
    g_q4.stage_captured = false;
    const size_t wants[2] = {bytes + bytes / 4, bytes};   /* with room to grow, if that can be had */
    for (size_t want : wants) {
        const cudaError_t e = cudaMalloc(&g_stage, want);
        if (e == cudaSuccess) {
            g_stage_bytes = want;
            return 1;
        }
        g_stage = nullptr;
        if (e != cudaErrorMemoryAllocation) return q4i_check(e, "prefill staging alloc");
        (void)cudaGetLastError();
    }
    return -1;
}

template <int HD, int NQ, int NP, bool MARKS, bool TAIL, bool PAIR>
bool attend(const PrefillTail &p, dim3 grid) {
    static bool attr = false;
    const auto kernel = q4_prefill_k<HD, NQ, NP, MARKS, TAIL, PAIR>;
    if (!attr && !q4i_check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PF_SMEM), "prefill smem attribute")) return false;
    attr = true;
    grid.x *= PAIR ? 2u : 1u;
    return q4i_launched(q4i_launch_dep_in<PAIR ? 2u : 1u>("prefill launch", kernel, grid, PF_THREADS, PF_SMEM, static_cast<const std::conditional_t<TAIL, PrefillTail, PrefillParams> &>(p)));
}
template <int HD, int NQ, int NP, bool MARKS, bool TAIL>
bool attend(const PrefillTail &p, dim3 grid, bool pair) {
    if constexpr (NP == 2 || HD == 256 || (NQ == 2 && !MARKS))
        if (pair) return attend<HD, NQ, NP, MARKS, TAIL, true>(p, grid);
    return attend<HD, NQ, NP, MARKS, TAIL, false>(p, grid);
}
template <int HD, int NP, bool MARKS>
bool attend_one(const PrefillTail &p, uint32_t n_kvh, bool pair) {
    if (p.n_whole && p.n_late) return attend<HD, 1, NP, MARKS, true>(p, dim3(p.n_whole + p.n_late * p.n_split), pair);
    return attend<HD, 1, NP, MARKS, false>(p, dim3(p.n_groups, n_kvh, p.n_split), pair);
}
template <int LAY, int HD, int NP>
bool stage(const Q4PrefillArgs &a, uint32_t n, uint32_t tiles, uint32_t unit, uint8_t *kimg, uint8_t *vimg, PfMark *marks, uint8_t *flags) {
    return q4i_launch_pdl("prefill launch", q4_pf_stage_k<LAY, HD, NP>, dim3(tiles * (PF_BN / 32u), a.n_kvh, 2), 256u, 0, a.cache, a.layer, n, tiles, unit, kimg, vimg, marks, flags);
}

/* Which blocks' (pairs') positions are split, and into how many ranges: the choice with the least estimated time, waves x (tiles of a
 * range + what a block takes besides) + the merge with its traffic.  In ns, one group per block, from chunks of 33 to 1500
 * tokens over 0 to 16 384: a tile 1.0 us at hd 128, 2.2 at 256 with both images; a block 4 and 6 us besides; the merge
 * 1.2 us, 0.2 per range, and 7 KB per ns.  600 tokens over 16 384 (76 blocks): 146 us in one range, 112 in three.
 * Two groups per block: a tile 1.8 us, a block 5.  There, and with more blocks than SMs, only those of the last wave are split,
 * the shortest of the chunk: 8192 tokens over 16 384 are 512 blocks, 444 and 68 x 2. */
struct PfSplit { uint32_t whole, ranges; uint64_t ns; };   /* ns: the estimate, to compare single blocks and pairs by */
PfSplit best_split(uint32_t groups, uint32_t n_kvh, uint32_t sms, uint32_t kv_base, uint32_t tok_per_group, uint32_t tiles, uint64_t rows, uint32_t rows_per_group, uint32_t hd,
                   uint32_t np, uint32_t nq, bool pair) {
    const uint32_t blocks = groups * n_kvh, waves = blocks / sms, rest = blocks % sms;
    uint64_t tile = nq == 2 ? 1800u : 640u + 190u * (hd / 128u) * 2u * np, block = nq == 2 ? 5000u : 2000u + 2000u * (hd / 128u);
    auto merge = [&](uint64_t n, uint32_t s) -> uint64_t { return 1200u + 200u * s + n * hd * s * 8u / 7000u; };
    /* The last wave's blocks are the last kv head's first tokens. */
    const uint32_t seen = (kv_base + (rest < groups ? rest : groups) * tok_per_group + PF_BN - 1u) / PF_BN, n = seen < tiles ? seen : tiles;
    auto all_in = [&](uint32_t s) -> uint64_t { return ((uint64_t)blocks * s + sms - 1u) / sms * ((tiles + s - 1u) / s * tile + block) + (s > 1u ? merge(rows, s) : 0u); };
    auto rest_in = [&](uint32_t s) -> uint64_t { return waves * (tiles * tile + block) + (n + s - 1u) / s * tile + block + merge((uint64_t)rest * rows_per_group, s); };
    PfSplit r = {blocks, 1u, 0u};
    const uint64_t whole = all_in(1u);
    uint64_t best = whole - whole / 16u;   /* whole blocks need no merge: left for a clear gain only (causal chunks have less work) */
    for (uint32_t s = 2; s <= 16u && s <= tiles; s++) {
        if (nq == 1) {
            const uint64_t t = all_in(s);
            if (t < best) {
                best = t;
                r = {0u, s, 0u};
            }
        }
        /* Where they are much shorter than the chunk's last tokens', as without a prefix, the blocks before them end so far apart that
         * they fill the gaps (8192 tokens over none 240 us, split 255). */
        if (waves && rest && rest * s <= sms && n >= 2u * (tiles - kv_base / PF_BN)) {
            const uint64_t t = rest_in(s), now = waves * (tiles * tile + block) + n * tile + block;
            if (t < best && t < now) {
                best = t;
                r = {blocks - rest, s, 0u};
            }
        }
    }
    /* Pairs: their products are the tensor core's 64 cycles per 128 x 128 x 16 where one block's wait for shared memory, and meeting
     * costs a microsecond. */
    if (pair) {
        tile = tile * (np == 2 ? 89u : nq == 2 ? 97u : 93u) / 100u;
        block += 1000u;
    }
    r.ns = r.ranges == 1u ? all_in(1u) : r.whole ? rest_in(r.ranges) : all_in(r.ranges);
    if (r.ranges == 1u) r.ns -= r.ns / 32u;
    return r;
}

}  // namespace

void q4i_prefill_release() {
    if (g_stage) cudaFree(g_stage);
    g_stage = nullptr;
    g_stage_bytes = 0;
}

extern "C" void q4_gpu_prefill_layout(uint32_t *whole, uint32_t *split, uint32_t *ranges) {
    if (whole) *whole = g_layout[0];
    if (split) *split = g_layout[1];
    if (ranges) *ranges = g_layout[2];
}

int q4i_prefill(const Q4PrefillArgs &a) {
    const uint32_t gqa = a.n_head / a.n_kvh, hd = a.hd;
    const uint64_t n64 = (uint64_t)a.kv_base + a.n_tok;
    const uint32_t n = (uint32_t)(n64 < a.cache.max_kv ? n64 : a.cache.max_kv), tiles = (n + PF_BN - 1u) / PF_BN;
    /* a code times its scale has 19 bits: the reference ABI's q8_0 caches keep what the first image leaves over */
    const uint32_t np = a.layout == LAY_Q8R ? 2u : 1u;
    const uint32_t tpc = PF_ROWS / gqa, groups = (a.n_tok + tpc - 1u) / tpc, sms = (uint32_t)g_q4.sm_count;
    /* Two groups per block share every K/V tile and hide one another's softmax; one group per block while that takes few
     * waves: 1000 tokens over 4000 (126 blocks) 52 against 83 us, 2500 over 16 384 (314) 450 against 505, 3600 (450) 643
     * against 591; between 300 and 400 it depends on the depth. */
    const uint32_t nq = hd == 128 && np == 1u && groups * a.n_kvh * 2u > sms * 5u ? 2u : 1u;
    const uint32_t prefix = a.kv_base / PF_BN;
    /* Pairs of blocks behind a prefix, where they are estimated to take 1.5 % less.  How many pairs fill the places of a wave, and how
     * many ranges fit, moves a chunk by up to 20 % either way: 24 / 2 heads of 256 over 2048 rows of fp16, 350 tokens 1 % more in
     * pairs, 380 2 % less; one kv head with 8 heads of 256 over 2048 rows of q8_0, 850 tokens 4 % less, but 770, 25 pairs in two ranges
     * instead of 49 blocks in three, 10 % more; 32 / 2 heads, 290 tokens 35 % more.  us, one block / pairs.  Both images: 512 tokens over
     * 512 at hd 256 39.5 / 37.8, 2048 over 4000 392 / 361, at hd 128 144 / 128, 512 over 512 21.4 / 22.4, over 1536 27.7 / 27.5 (2048
     * over none at hd 256 120 / 121).  One image at hd 256: 512 over 512 24.8 / 25.4, 2048 over 4000 227 / 212.  Two groups per block:
     * 8192 over 5000 515 / 514, 16 384 1159 / 1130, 40 000 2463 / 2389 (as long up to 12 000 rows, 1 % less over 14 336 and 20 000);
     * with marks 8192 over 8000 758 / 760; one group at hd 128 600 over 16 384 115 / 121.  And not for a few blocks in ranges (100 over
     * 4000 39.6 / 40.2). */
    const size_t k_bytes = (size_t)a.n_kvh * tiles * np * (hd / 128u) * PF_CHUNK, v_bytes = k_bytes, m_bytes = (size_t)a.n_kvh * tiles * (PF_BN / 32u) * (sizeof(PfMark) + 4u);   /* marks, flags (two bytes used per mark) */
    auto layout = [&](uint32_t ctas) -> PfSplit {
        const uint32_t per = tpc * nq * ctas;
        return best_split((groups + nq * ctas - 1u) / (nq * ctas), a.n_kvh, sms / ctas, a.kv_base, per, tiles, (uint64_t)a.n_tok * a.n_head, per * gqa, hd, np, nq, ctas == 2u);
    };
    PfSplit sp = layout(1u);
    bool pair = groups * a.n_kvh >= 48u && (np == 2u ? prefix >= (hd == 256u ? 4u : 12u) : hd == 256u ? prefix >= 16u : nq == 2u && a.layout == LAY_Q8P && prefix >= 112u);
    if (pair) {
        const PfSplit two = layout(2u);
        pair = two.ns * 1000u < sp.ns * 985u;
        if (pair) sp = two;
    }
    const uint32_t ctas = pair ? 2u : 1u, unit = pair ? (nq == 2u ? 6u : 7u) : 0u;
    const uint32_t n_groups = (groups + nq * ctas - 1u) / (nq * ctas), tok_per_group = tpc * nq * ctas, blocks = n_groups * a.n_kvh;
    uint32_t part_tok;
    size_t rows, part_bytes;
    int room;
    for (;; sp = {blocks, 1u, 0u}) {
        /* tokens that parts are kept for: those of the groups at the end of the order */
        const uint32_t late = blocks - sp.whole;
        const uint64_t late_tok = (uint64_t)(late < n_groups ? late : n_groups) * tok_per_group;
        part_tok = (uint32_t)(late_tok < a.n_tok ? late_tok : a.n_tok);
        rows = (size_t)part_tok * a.n_head;
        part_bytes = sp.ranges * rows * hd * sizeof(float);
        room = stage_reserve(k_bytes + v_bytes + m_bytes + part_bytes + sp.ranges * rows * sizeof(float2));
        if (room != -1 || sp.ranges == 1u) break;   /* no room for parts: whole blocks need none */
    }
    if (room != 1) return room;
    const uint32_t split = sp.ranges;
    g_layout[0] = sp.whole * ctas; g_layout[1] = (blocks - sp.whole) * ctas; g_layout[2] = split;

    PrefillTail p;
    memset(&p, 0, sizeof(p));
    p.n_head = a.n_head; p.n_kvh = a.n_kvh; p.gqa = gqa; p.tpc = tpc;
    p.q = a.q; p.q_bf16 = a.q_bf16; p.gate = a.gate; p.out = a.out; p.out_bf16 = a.out_bf16;
    p.n_tok = a.n_tok; p.kv_base = a.kv_base; p.max_kv = a.cache.max_kv;
    p.scale_log2e = a.scale * 1.4426950408889634f;
    uint8_t *kimg = g_stage, *vimg = g_stage + k_bytes;
    p.kimg = kimg; p.vimg = vimg; p.img_tiles = tiles;
    p.n_groups = n_groups; p.n_whole = sp.whole; p.n_late = blocks - sp.whole; p.n_split = split; p.part_tok = part_tok;
    PfMark *marks = reinterpret_cast<PfMark *>(g_stage + k_bytes + v_bytes);
    uint8_t *flags = reinterpret_cast<uint8_t *>(marks + (size_t)a.n_kvh * tiles * (PF_BN / 32u));
    p.marks = marks;
    p.flags = reinterpret_cast<const uint32_t *>(flags);
    p.part = reinterpret_cast<float *>(g_stage + k_bytes + v_bytes + m_bytes);
    p.part_ml = reinterpret_cast<float2 *>(g_stage + k_bytes + v_bytes + m_bytes + part_bytes);
    p.err = g_q4.err_d;

    bool ok;
    if (a.layout == LAY_Q8P) ok = stage<LAY_Q8P, 128, 1>(a, n, tiles, unit, kimg, vimg, marks, flags);
    else if (a.layout == LAY_Q8R) ok = hd == 128 ? stage<LAY_Q8R, 128, 2>(a, n, tiles, unit, kimg, vimg, marks, flags) : stage<LAY_Q8R, 256, 2>(a, n, tiles, unit, kimg, vimg, marks, flags);
    else if (a.layout == LAY_F16) ok = hd == 128 ? stage<LAY_F16, 128, 1>(a, n, tiles, unit, kimg, vimg, marks, flags) : stage<LAY_F16, 256, 1>(a, n, tiles, unit, kimg, vimg, marks, flags);
    else ok = hd == 128 ? stage<LAY_F32, 128, 1>(a, n, tiles, unit, kimg, vimg, marks, flags) : stage<LAY_F32, 256, 1>(a, n, tiles, unit, kimg, vimg, marks, flags);
    if (!ok) return 0;
    const bool own = a.layout == LAY_Q8P;
    if (nq == 2) {
        const dim3 grid(p.n_whole + p.n_late * split);
        ok = own ? attend<128, 2, 1, false, true>(p, grid, pair) : attend<128, 2, 1, true, true>(p, grid, pair);
    } else if (hd == 256) {
        ok = np == 2 ? attend_one<256, 2, true>(p, a.n_kvh, pair) : attend_one<256, 1, true>(p, a.n_kvh, pair);
    } else {
        ok = np == 2 ? attend_one<128, 2, true>(p, a.n_kvh, pair) : own ? attend_one<128, 1, false>(p, a.n_kvh, pair) : attend_one<128, 1, true>(p, a.n_kvh, pair);
    }
    if (ok && split > 1) {
        const uint64_t total4 = (uint64_t)rows * hd / 4u;
        const dim3 grid((unsigned)((total4 + 255u) / 256u));
        ok = sp.whole ? q4i_launch_pdl("prefill launch", q4_pf_merge_k<true>, grid, 256u, 0, p, hd, total4, tok_per_group)
                      : q4i_launch_pdl("prefill launch", q4_pf_merge_k<false>, grid, 256u, 0, static_cast<const PrefillParams &>(p), hd, total4, tok_per_group);
    }
    return ok ? 1 : 0;
}

extern "C" bool q4_gpu_kv_prefill(const q4_gpu_kv *kv, uint32_t layer, const void *q_bf16, const float *gate,
                                  void *out_bf16, uint32_t n_head, uint32_t n_tok, uint32_t kv_base, float scale) {
    if (!g_q4.ok) return q4i_fail(Q4E_INIT, "kv_prefill: library not initialised");
    Q4_REQUIRE(kv && q_bf16 && out_bf16 && n_head && n_tok && layer < kv->n_layers, "kv_prefill: bad argument");
    Q4_REQUIRE(kv->kind == Q4K_Q8 && kv->hd == 128, "kv_prefill: tensor-core path needs a q8_0 store with hd 128");
    Q4_REQUIRE(n_head % kv->n_kvh == 0 && n_head / kv->n_kvh <= 16, "kv_prefill: n_head/n_kvh must be 1..16");
    Q4_REQUIRE(scale > 0.f, "kv_prefill: scale must be positive");
    Q4_REQUIRE((uint64_t)kv_base + 1 <= kv->max_kv, "kv_prefill: kv_base beyond max_kv");
    Q4PrefillArgs a;
    memset(&a, 0, sizeof(a));
    a.cache = kv->view;
    a.layout = LAY_Q8P;
    a.layer = layer;
    a.n_head = n_head; a.n_kvh = kv->n_kvh; a.hd = kv->hd;
    a.q = q_bf16; a.q_bf16 = 1; a.gate = gate; a.out = out_bf16; a.out_bf16 = 1;
    a.n_tok = n_tok; a.kv_base = kv_base; a.scale = scale;
    const int r = q4i_prefill(a);
    if (r < 0)
        return g_q4.capturing ? q4i_fail(Q4E_SCRATCH, "kv_prefill: staging buffer too small inside a capture")
                              : q4i_fail(Q4E_CUDA, "kv_prefill: no device memory for the staging buffer");
    return r == 1;
}
