/* Internal declarations shared by the libq4gpu translation units (not installed). */
#ifndef Q4_INTERNAL_H
#define Q4_INTERNAL_H

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "../../include/q4_gpu.h"

/* KV kinds of the public ABI, plus the two q8_0 layouts the kernels distinguish. */
enum { Q4K_F32 = 0, Q4K_F16 = 1, Q4K_Q8 = 2 };
enum { LAY_F32 = 0, LAY_F16 = 1, LAY_Q8P = 2 /* native store: 16-byte aligned records */, LAY_Q8R = 3 /* reference 34-byte blocks */ };

enum {
    Q4E_ARG = 1, Q4E_CUDA = 2, Q4E_RANGE = 4, Q4E_SCRATCH = 8, Q4E_INIT = 16,
    Q4E_PEER = 32,   /* a peer's record did not arrive within the time limit */
};

/* One cache as the kernels see it.  Row (layer, kv head kh, token p) of the K plane lives at
 * k + layer*layer_stride + kh*kvh_stride + p*tok_stride (same for v); for the native q8_0 store the
 * scale row is at s + layer*s_layer_stride + kh*s_kvh_stride + p*s_tok_stride and holds the K block
 * scales followed by the V block scales (fp16).  The native q8_0 layout is always the record
 * {K codes hd | V codes hd | scales}: v = k + hd, s = k + 2*hd, equal strides (kernels rely on it). */
struct Q4Cache {
    const uint8_t *k, *v, *s;
    uint64_t layer_stride, kvh_stride, s_layer_stride, s_kvh_stride;
    uint32_t tok_stride, s_tok_stride;
    uint32_t max_kv, pad;
};

/* Per layer of a store: g_q4.launches when its rows were last written.  Shared by the store and the batches it is bound to:
 * a batch may outlive a store of a session that has ended. */
struct Q4Writes { uint32_t refs; uint64_t *at; };

struct q4_gpu_kv {
    uint32_t n_layers, n_kvh, hd, max_kv;
    int kind;
    uint8_t *k, *v, *s;          /* device planes (s only for q8_0) */
    uint64_t plane_bytes, s_bytes;
    uint32_t rec_bytes;          /* bytes per (kv head, position): q8_0 record, or fp16 / fp32 row */
    Q4Cache view;                /* host copy of the kernel view */
    Q4Cache *d_view;             /* same, in device memory (for batched launches) */
    Q4Writes *writes;
};

/* fp32 rows at hd 128 come through rings in shared memory while the launch is bound by latency, and straight into registers,
 * behind an append of its own, beyond this many rows of all units and kv heads together: through the ring every byte crosses
 * the load/store pipe twice.  us per launch, ring / registers, 2 kv heads: one unit of 24 576 rows 17.5 / 18.1, of 32 768
 * 21.7 / 19.2, of 262 144 103.7 / 85.7; 8 lists of 2051 11.8 / 14.0, 32 33.7 / 30.9; 8 sessions of 24 000 rows 90.5 / 74.
 * With more than 8 query heads per kv head the ring holds out longer, for one unit always (262 144 rows 103.7 / 123.0;
 * 4 sessions of 32 768 59.5 / 74.5, 8 of 24 000 122.3 / 79.8, 512 lists 353 / 315). */
constexpr uint64_t Q4_F32_RING_ROWS = 49152, Q4_F32_RING_ROWS_WIDE = 327680;
inline bool q4i_f32_direct(int kind, uint32_t hd, uint32_t n_head, uint32_t n_kvh, uint64_t units, uint32_t rows) {
    if (kind != Q4K_F32 || hd != 128) return false;
    return units * n_kvh * rows > Q4_F32_RING_ROWS && (n_head <= 8u * n_kvh || (units > 1 && units * n_kvh * rows > Q4_F32_RING_ROWS_WIDE));
}

struct Q4PtrList { void **p; uint32_t n; };

/* Device memory that a launch reads and writes.  bytes == 0: to the end of p's allocation (a row whose place the device
 * knows).  The status word, which launches only or bits into, and the library's scratch are left out. */
struct Q4Touch {
    struct { const void *p; uint64_t bytes; bool write; uint32_t newest; } r[12];   /* newest: of the rows at p the pooled block that the position word completes alone, of so many tokens */
    uint32_t n;
    void reads(const void *p, uint64_t bytes) { add(p, bytes, false); }
    void writes(const void *p, uint64_t bytes) { add(p, bytes, true); }
    void add(const void *p, uint64_t bytes, bool write) {
        if (!p) return;
        r[n].p = p; r[n].bytes = bytes; r[n].write = write; r[n].newest = 0;
        n++;
    }
};

/* runtime state (q4_runtime.cu) */
struct Q4State {
    bool ok;
    int device, sm_count;
    cudaStream_t own_stream, stream, copy_stream, down_stream;   /* compute, uploads, downloads */
    int capturing;
    int32_t *pos_d, *pos_h;
    uint32_t *err_d;             /* device-side sticky error bits */
    uint32_t err_h;
    uint32_t last_graph_nodes;
    /* What a kernel may read before it has waited for its predecessor in the stream (programmatic dependent launch).
     * Every kernel of the library either starts after its predecessor has finished, or waits for that before it lets its
     * successor start.  So what was written at least one library launch earlier is complete when a kernel starts:
     * `launches` counts them, the position word and the rows of a store remember the count at their last write, and
     * `unsettled` is the count at the last event behind which nothing is known (a graph launch, another stream).
     * A launch that runs apart (q4i_apart) is the exception: its successor may start before its predecessor has finished.
     * `settled` is the count at the last launch that did not: what was written before that one is complete. */
    uint64_t launches, settled, pos_written, unsettled;
    /* in a capture: what the launches since may still be at (those numbered `settled` and up), and the node that the last of
     * them left as the stream's only dependency */
    struct { uint64_t number; Q4Touch touch; } flight[4];
    uint32_t n_flight;
    cudaGraphNode_t last_node;
    uint32_t n_apart, last_graph_apart, n_ahead, last_graph_ahead;   /* launches apart, and with blocks read ahead, in this capture, in the last finished one */
    /* attention scratch: split-KV partial records + per-unit arrival counters */
    float *part;
    size_t part_floats;
    uint32_t *counters;
    size_t n_counters;
    /* An instantiated graph keeps the addresses its launches were captured with.  A workspace that a capture has used and
     * that then grows is kept until no graph is left (sizes grow by a quarter at least, so what is kept stays below four
     * times what is in use). */
    bool part_captured, counters_captured, stage_captured;
    Q4PtrList graphs, kept;      /* instantiated and not yet freed; workspaces that one of them may use */
};
extern Q4State g_q4;

bool q4i_fail(uint32_t bit, const char *what);
bool q4i_check(cudaError_t e, const char *what);
void q4i_in_capture(const Q4Touch *touch);
inline bool q4i_launched(bool ok, const Q4Touch *touch = nullptr, bool apart = false) {
    if (!ok) return false;
    g_q4.launches++;
    if (apart) g_q4.n_apart++;
    else g_q4.settled = g_q4.launches;
    if (g_q4.capturing) q4i_in_capture(touch);
    return true;
}
inline bool q4i_settled(uint64_t written) { return g_q4.settled > written && g_q4.settled > g_q4.unsettled; }
/* Whether the next launch, which will touch `touch`, may run beside the ones before it: it is captured right behind them, and
 * nothing that it writes is touched, and nothing that it reads is written, by any that may not have finished when it starts.
 * Such a kernel lets its successor start at once, does its work, and waits for its predecessor before it ends
 * (q4d_apart_begin / _end): whoever waits for it has waited for everything before it, as ever. */
bool q4i_apart(const Q4Touch &touch);
/* Whether the next launch may read the pooled blocks at p before it waits for the ones before it, but for the block of `ratio`
 * tokens that the position word completes (0: that one too, for a launch that has its position from elsewhere): captured likewise,
 * and nothing else in those bytes is written by any that may not have finished when it starts. */
bool q4i_blocks_ahead(const void *p, uint64_t bytes, uint32_t ratio);
inline void q4i_kv_written(q4_gpu_kv *kv, uint32_t layer) { kv->writes->at[layer] = g_q4.launches; }
bool q4i_scratch(size_t part_floats, size_t n_counters); /* grows outside capture, fails inside */
void q4i_give_back(void *p, bool captured);              /* cudaFree, now or with the last graph */

#define Q4_REQUIRE(cond, what)                    \
    do {                                          \
        if (!(cond)) return q4i_fail(Q4E_ARG, what); \
    } while (0)

#ifdef __CUDACC__
/* Programmatic dependent launch, kernel side: a block may become resident while the previous kernel of the stream drains;
 * only what is settled (q4i_settled) is read before this.  Then the next kernel's blocks may come in. */
__device__ __forceinline__ void q4d_pdl_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
/* A kernel that runs beside its predecessor (q4i_apart), in every thread, begin first and end last.  What it reads, the position
 * word and weights too, may have been written by the launch before last: by loads that do not look into L1. */
__device__ __forceinline__ void q4d_apart_begin() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void q4d_apart_end() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
/* host side: a launch that may start so (the kernel calls q4d_pdl_wait in every thread), in clusters of CLUSTER blocks */
template <uint32_t CLUSTER, typename K, typename... A>
bool q4i_launch_dep_in(const char *what, K kernel, dim3 grid, uint32_t threads, size_t smem, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = g_q4.stream;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = CLUSTER;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = CLUSTER > 1u ? 2 : 1;
    return q4i_check(cudaLaunchKernelEx(&cfg, kernel, args...), what);
}
template <typename K, typename... A>
bool q4i_launch_dep(const char *what, K kernel, dim3 grid, uint32_t threads, size_t smem, A... args) {
    return q4i_launch_dep_in<1>(what, kernel, grid, threads, smem, args...);
}
template <typename K, typename... A>
bool q4i_launch_pdl(const char *what, K kernel, dim3 grid, uint32_t threads, size_t smem, A... args) {
    return q4i_launched(q4i_launch_dep(what, kernel, grid, threads, smem, args...));
}
/* ---- the q8_0 quantiser, one copy for every kernel that writes a cache row.  8 lanes share a block
 * of 32 values (4 each): d = amax / 127 and id = 1 / d as IEEE fp32 divisions, codes =
 * clamp(rint(x * id), +-127), stored scale = fp16(d) (quantize_row_q8_0's arithmetic,
 * src/q4_quant.c / src/q4_rocm.cu f32_to_q8 kernels). */
__device__ __forceinline__ uint32_t q4d_quant4(const float4 x, float id) {
    int q0 = __float2int_rn(__fmul_rn(x.x, id)), q1 = __float2int_rn(__fmul_rn(x.y, id));
    int q2 = __float2int_rn(__fmul_rn(x.z, id)), q3 = __float2int_rn(__fmul_rn(x.w, id));
    q0 = max(-127, min(127, q0)); q1 = max(-127, min(127, q1));
    q2 = max(-127, min(127, q2)); q3 = max(-127, min(127, q3));
    return (uint32_t)(q0 & 0xff) | ((uint32_t)(q1 & 0xff) << 8) | ((uint32_t)(q2 & 0xff) << 16) |
           ((uint32_t)(q3 & 0xff) << 24);
}
/* amax over the 8 lanes that share a block (all 32 lanes of the warp must call), then d and 1/d */
__device__ __forceinline__ void q4d_block_scale(const float4 x, float &d, float &id) {
    float a = fmaxf(fmaxf(fabsf(x.x), fabsf(x.y)), fmaxf(fabsf(x.z), fabsf(x.w)));
    a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, 1));
    a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, 2));
    a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, 4));
    d = __fdiv_rn(a, 127.f);
    id = d > 0.f ? __fdiv_rn(1.f, d) : 0.f;
}
#endif

/* ---- record exchange between the ranks of a sequence-sharded decode -----------------------------
 * Every rank owns one window in its own memory that all peers can write.  It starts with this header;
 * the records follow at XCHG_REC_OFFSET: packet rec[2][units][world][slot_floats], one slot per
 * (parity of the call count, unit = kv head, writing rank).  A slot is the kernel's internal record
 * for the unit's heads, {acc[hd], m (log2 units, scale folded in), l, 2 pad} per head, each fp32
 * value stored as an 8-byte packet {value, epoch of the call that wrote it}. */
constexpr uint32_t XCHG_MAX_WORLD = 16, XCHG_MAX_UNITS = 16;
constexpr size_t XCHG_REC_OFFSET = 4096;
struct Q4XchgWin {
    uint32_t epoch[XCHG_MAX_UNITS];                       /* calls completed by the owner, per unit */
};
/* who and where, in the owner's device memory (never written by peers) */
struct Q4XchgDev {
    uint32_t rank, world, units, slot_floats;
    unsigned long long timeout_ns;
    Q4XchgWin *win[XCHG_MAX_WORLD];                       /* win[rank] is the local window */
};
enum { XCHG_FUSED = 0, XCHG_PUSH = 1, XCHG_MERGE = 2 };
struct q4_gpu_xchg {
    uint32_t n_head, n_kvh, hd;
    size_t win_bytes;
    Q4XchgWin *win;
    Q4XchgDev host, *dev;
    uint8_t attached[XCHG_MAX_WORLD];                     /* 1 = opened from an IPC handle, 2 = caller's pointer */
};
/* wait-and-merge half alone (q4_decode.cu): the records of the latest push on every rank -> out */
bool q4i_xchg_merge(const q4_gpu_xchg *x, const float *gate, float *out);

/* frees the prefill staging buffer (q4_prefill.cu) / the session-file staging (q4_sess.cu); called at shutdown */
void q4i_prefill_release();
void q4i_sess_release();

/* decode attention launcher (q4_decode.cu) */
struct Q4DecodeArgs {
    Q4Cache one;                 /* used when many == nullptr */
    const Q4Cache *many;         /* device array of cache views, one per session */
    int layout;                  /* LAY_* */
    uint32_t layer, n_units;     /* units = sessions (many) or tokens (one) */
    uint32_t n_head, n_kvh, hd;
    const void *q;
    int q_bf16;
    const float *gate;
    float *out, *part_out;
    const int32_t *idx;
    uint32_t width, idx_kvh_stride, idx_unit_stride;
    const int32_t *pos;          /* device positions: per session (many) or one word (one); may be null */
    uint32_t kv_base;            /* used when pos == nullptr: unit u attends kv_base + u + 1 rows */
    uint32_t hint_rows;          /* host's estimate of rows per unit, to size the split */
    int idx_bound_nkv;           /* list entries >= the unit's row count (newest + 1) are out of range (stores:
                                  * rows beyond it were never written); 0 = only max_kv bounds them (reference ABI) */
    float scale;
    /* optional caller-provided scratch (no-allocation entry point); null = library scratch */
    float *scratch_part;
    uint32_t *scratch_counters;
    size_t scratch_part_floats, scratch_n_counters;
    int scratch_clamp;           /* reduce the split count until the records fit the caller's scratch */
    /* sequence-sharded decode: leave the unit's record in the exchange window, push it to the peers and
     * (XCHG_FUSED) wait for theirs and write the merged output; null = single-rank decode */
    const Q4XchgDev *xchg;
    int xchg_phase;
    /* fused append (stores at hd 128 and 256): the new K and V rows [unit][n_kvh*hd] (fp32) are quantised or converted
     * and stored at each unit's position by the attention kernel itself before it reads the cache */
    const float *new_k, *new_v;
    int early_pos, early_rows;   /* the positions / the rows of a dense scan are settled (q4i_settled) */
};
bool q4i_decode(const Q4DecodeArgs &a);
bool q4i_decode_counters(uint64_t units);   /* the arrival counters that a decode of so many units x kv heads needs */

/* causal attention of n_tok > 1 query tokens on the tensor cores (q4_prefill.cu): hd 128 or 256 (a native q8_0 store:
 * 128), 1..16 query heads per kv head, scale > 0, 16-byte aligned operands.  1 = enqueued, 0 = failed, -1 = its
 * workspace is not to be had (it may not grow inside a capture, or no memory is left). */
struct Q4PrefillArgs {
    Q4Cache cache;
    int layout;
    uint32_t layer, n_head, n_kvh, hd;
    const void *q;               /* [n_tok][n_head][hd] bf16 or fp32 */
    int q_bf16;
    const float *gate;           /* or null */
    void *out;                   /* bf16 or fp32 */
    int out_bf16;
    uint32_t n_tok, kv_base;     /* token t attends rows [0, min(kv_base + t + 1, max_kv)) */
    float scale;
};
int q4i_prefill(const Q4PrefillArgs &a);
/* What block `block` of a prefill launch's list works on.  Items are kv head by kv head, each its n_groups groups of tokens with
 * the last tokens first; the first n_whole are one block each, the n_late behind them n_split blocks, range by range (what runs
 * at once reads the same tiles).  Divisions: a product with a rounded inverse is exact below 2^32 / n_groups items only, and a
 * chunk's length has no bound (8 kv heads: 23 254 groups); one is less than 0.1 us per block. */
struct Q4PfItem { uint32_t kh, group, range, ranges; };
__host__ __device__ inline Q4PfItem q4i_pf_item(uint32_t block, uint32_t n_groups, uint32_t n_whole, uint32_t n_late, uint32_t n_split) {
    Q4PfItem r = {0, 0, 0, 1};
    uint32_t item = block;
    if (block >= n_whole) {
        r.range = (block - n_whole) / n_late;
        r.ranges = n_split;
        item = block - r.range * n_late;
    }
    r.kh = item / n_groups;
    r.group = item - r.kh * n_groups;
    return r;
}

#endif
