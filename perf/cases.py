"""The attention steps that an engine host has libq4gpu do, as cases that can be timed and compared.

A case is one pass of a host's step over all attention layers of the model: a decoded token for one session or for a
batch, a prefill chunk, or a prefix restored and saved.  Paths:

  step           decode on library-owned stores: append + attention, dense or over 2051-entry lists that are given
                 ("lists") or produced by the indexer in the same step ("select"); one captured graph per step, the
                 position published before it
  prefill        a chunk of prompt: K norm + RoPE + append, then dense causal attention, bf16 queries and outputs
  sparse_prefill a slice of a long prompt: append, pool, score, select, one gathered list per token
  dropin_step    the unchanged C host's decode step through the reference ABI on caches of its own
  dropin_prefill the same host's prompt chunk: norm + RoPE, quantise / convert, attention in slices of 512 tokens
  snapshot       a session's prefix out of a device pool into its store, and back

Shapes are those of this repository's benchmark (16 query / 2 kv heads, head size 128) and of the engine's own model
(24 / 2 / 256, 64 rotary dims); 12 attention layers, 2051 = 512 blocks of 4 positions + 3 selected positions.
"""
import math
import os
import random
import sys

import torch

sys.path.insert(0, os.path.join(os.getcwd(), "suzuqu-engine-4exp_b200"))
import q4gpu  # noqa: E402

LAYERS, RATIO, K_BLK, WIDTH, IDX_HEADS, IDX_HD = 12, 4, 512, 2051, 4, 128
ROPE_BASE, EPS = 1e7, 1e-6
KINDS = {"q8_0": q4gpu.KIND_Q8, "f16": q4gpu.KIND_F16, "f32": q4gpu.KIND_F32}
SMALL = {"n_head": 16, "n_kvh": 2, "hd": 128}     # the benchmark's shape
MODEL = {"n_head": 24, "n_kvh": 2, "hd": 256}     # the engine's model


def step(sessions, lo, hi, mode, capacity=0, kind="q8_0", shape=SMALL, gate=True, contexts=7):
    """A decoded token for `sessions` sessions whose context lengths are spread evenly at random over [lo, hi]."""
    return dict(path="step", sessions=sessions, lo=lo, hi=hi, contexts=contexts, capacity=capacity or hi, mode=mode, kind=kind, gate=gate, **shape)


def listed():
    return [
        # a chat's first tokens: everything written so far is attended; the session was opened for 32768 tokens
        dict(step(1, 777, 777, "dense", capacity=32768), name="step_1_dense_777"),
        # one session at the end of the largest context, with the indexer: the engine's long-context token
        dict(step(1, 262144, 262144, "select"), name="step_1_select_262144"),
        # the benchmark's headline: 64 sessions, contexts up to 131072, lists at hand
        dict(step(64, 1024, 131072, "lists", gate=False), name="step_64_lists"),
        # a few long sessions decoding together, lists from the batched indexer
        dict(step(8, 8192, 131072, "select"), name="step_8_select"),
        # full attention over the largest context, and over an odd one in a 16-bit cache (Q4_KV=f16)
        dict(step(1, 262144, 262144, "dense", gate=False), name="step_1_dense_262144"),
        dict(step(1, 100003, 100003, "dense", capacity=131072, kind="f16", gate=False), name="step_1_dense_f16_100003"),
        # a long chunk behind a long prefix (the benchmark's prefill), and a short ragged prompt
        dict(path="prefill", n_tok=8192, base=16384, gate=False, name="prefill_8192_16384", **SMALL),
        dict(path="prefill", n_tok=333, base=0, gate=True, name="prefill_333", **SMALL),
        # one 512-token slice of a prompt that has reached 131072 tokens
        dict(path="sparse_prefill", n_tok=512, base=130560, name="sparse_prefill_512_131072", **SMALL),
        # the unchanged C host: a token at 32768, and its default chunk of 2048 tokens
        dict(path="dropin_step", ctx=32768, kind="q8_0", name="dropin_step_32768", **MODEL),
        dict(path="dropin_prefill", n_tok=2048, base=0, kind="q8_0", name="dropin_prefill_2048", **MODEL),
        # a cached prefix of 50001 tokens is put into a session, and saved from it after the turn
        dict(path="snapshot", rows=50001, kind="q8_0", name="snapshot_50001", **SMALL),
    ]


def draw(rng):
    def log(lo, hi):
        return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    path = rng.choice(["step", "step", "step", "prefill", "sparse_prefill", "dropin_step", "dropin_prefill", "snapshot"])
    kind = rng.choice(["q8_0", "q8_0", "q8_0", "f16", "f32"])
    shape = rng.choice([SMALL, SMALL, SMALL, MODEL])
    if path == "step":
        mode = rng.choice(["dense", "lists", "select"])
        sessions = rng.choice([1, log(2, 64)])
        if sessions == 1:
            lo = hi = log(64, 262144) if mode == "dense" else log(2100, 262144)
        else:
            # what the caches of all sessions take: an eighth of the card at most
            room = int(2e10 / (sessions * LAYERS * 2 * shape["n_kvh"] * row_bytes(kind, shape["hd"])))
            hi = min(log(256, 8192) if mode == "dense" else log(2100, 131072), max(2100, room))
            lo = max(32, hi // rng.choice([1, 4, 32]))
        return step(sessions, lo, hi, mode, capacity=max(hi, 1 << (hi * rng.choice([1, 2, 8]) - 1).bit_length()) if sessions == 1 and hi < 32768 else hi,
                    kind=kind, shape=shape, gate=rng.random() < 0.5, contexts=rng.randrange(1 << 20))
    if path == "prefill":
        return dict(path=path, n_tok=log(33, 8192), base=rng.choice([0, log(100, 16384)]), gate=rng.random() < 0.5, **SMALL)
    if path == "sparse_prefill":
        n_tok = log(64, 512)
        return dict(path=path, n_tok=n_tok, base=log(2100, 131072 - n_tok), **shape)
    if path == "dropin_step":
        return dict(path=path, ctx=log(64, 65536), kind=kind, **shape)
    if path == "dropin_prefill":
        n_tok = log(33, 2048)
        return dict(path=path, n_tok=n_tok, base=rng.randint(0, 2048 - n_tok), kind=kind, **shape)
    return dict(path="snapshot", rows=log(1000, 131072), kind=kind, **shape)


# ------------------------------------------------------------------------------------------- sizes
def row_bytes(kind, hd):
    """one K or V row of one kv head"""
    return hd // 32 * 34 if kind == "q8_0" else hd * (2 if kind == "f16" else 4)


def contexts(case):
    r = random.Random(case["contexts"])
    return [r.randint(case["lo"], case["hi"]) for _ in range(case["sessions"])]


def attended(case, ctx):
    return ctx if case.get("mode", "dense") == "dense" else min(ctx, WIDTH)


def work(case):
    nh, nkv, hd, path = case["n_head"], case["n_kvh"], case["hd"], case["path"]
    row = 2 * nkv * row_bytes(case.get("kind", "q8_0"), hd)         # K and V of one token and layer
    new = 2 * nkv * hd * 4                                          # the same as the projections leave it
    if path == "snapshot":
        return {"bytes": LAYERS * 4.0 * case["rows"] * row, "flops": 0}
    if path in ("step", "dropin_step"):
        b = f = 0.0
        own = path == "step"
        for ctx in contexts(case) if own else [case["ctx"]]:
            mode = case["mode"] if own else ("dense" if ctx <= WIDTH else "select")
            n = ctx if mode == "dense" else min(ctx, WIDTH)
            b += n * row + new + (nh * hd * (6 + (4 if case["gate"] else 0)) if own else nh * hd * 12)
            f += 4.0 * nh * hd * n
            if mode == "lists":
                b += 4 * nkv * WIDTH
            if mode == "select":
                b += ctx // RATIO * IDX_HD * 4 + IDX_HEADS * IDX_HD * 4 + 4 * WIDTH
                f += 2.0 * IDX_HEADS * IDX_HD * (ctx // RATIO)
        return {"bytes": LAYERS * b, "flops": LAYERS * f}
    n, base = case["n_tok"], case["base"]
    if path == "sparse_prefill":
        sel = sum(min(base + t + 1, WIDTH) for t in range(n))
        b = (base + n) * row + n * (new + nh * hd * 6 + IDX_HEADS * IDX_HD * 4 + 2 * IDX_HD + 4 * WIDTH) + (base + n) // RATIO * IDX_HD * 4
        f = 4.0 * nh * hd * sel + 2.0 * IDX_HEADS * IDX_HD * sum((base + t + 1) // RATIO for t in range(n))
        return {"bytes": LAYERS * b, "flops": LAYERS * f}
    pairs = n * base + n * (n + 1) / 2
    io = 4 + (4 if case["gate"] else 0) if path == "prefill" else 12
    return {"bytes": LAYERS * ((base + n) * row + n * (new + nh * hd * io)), "flops": LAYERS * 4.0 * nh * hd * pairs}


def tolerance(case):
    """Whole numbers (lists, cache bytes) are defined exactly.  Attention multiplies 16-bit queries and softmax weights
    (2^-11 each, rounded two or three times on the way) and adds in 32 bits: about 4e-4 of the result's norm; bf16
    outputs add 2^-9."""
    if case["path"] == "snapshot":
        return "exact"
    return {"rel": 5e-3} if case["path"] == "prefill" else {"rel": 1e-3}


# ------------------------------------------------------------------------------------------- states
class State:
    """What a host keeps for its step: stores, buffers, the captured graph."""

    def __init__(self, case, seed):
        self.case, self.L, self.graph = case, q4gpu.init(), None
        self.stream = torch.cuda.ExternalStream(self.L.q4_gpu_stream())
        self.gen = torch.Generator(device="cuda").manual_seed(seed)
        self.nh, self.nkv, self.hd = case["n_head"], case["n_kvh"], case["hd"]
        self.kind = KINDS[case.get("kind", "q8_0")]
        self.scale = 1.0 / math.sqrt(self.hd)
        self.n_rot = 64 if self.hd == 256 else self.hd
        q4gpu.check(self.L.q4_hip_qsa_topk_alloc(), "q4_hip_qsa_topk_alloc")

    def normal(self, *shape, dtype=torch.float32):
        return torch.randn(*shape, device="cuda", generator=self.gen).to(dtype)

    def empty(self, *shape, dtype=torch.float32):
        return torch.empty(*shape, device="cuda", dtype=dtype)

    def norm_weight(self, n):
        return 1.0 + 0.1 * self.normal(n)

    def store(self, capacity, rows):
        """a store whose first `rows` rows hold N(0,1) keys and values"""
        st = q4gpu.KVStore(LAYERS, self.nkv, self.hd, capacity, self.kind)
        for layer in range(LAYERS):
            for p in range(0, rows, 32768):
                n = min(32768, rows - p)
                st.append(layer, self.normal(n, self.nkv * self.hd), self.normal(n, self.nkv * self.hd), p, n)
        return st

    def capture(self, enqueue):
        enqueue()                                   # sizes the library's scratch; a capture may not allocate
        assert self.L.q4_hip_graph_begin() == 1
        enqueue()
        self.graph = self.L.q4_hip_graph_end()
        assert self.graph

    def __del__(self):
        if self.graph:
            self.L.q4_hip_graph_free(self.graph)


def selection(s, ctx):
    """4 first, 1024 newest and 1023 others of ctx positions, ascending; all of them in a shorter context"""
    out = torch.full((WIDTH,), -1, dtype=torch.int32, device="cuda")
    if ctx <= WIDTH:
        out[:ctx] = torch.arange(ctx, dtype=torch.int32, device="cuda")
        return out
    out[:4] = torch.arange(4, dtype=torch.int32, device="cuda")
    pick = torch.rand(ctx - 1028, device="cuda", generator=s.gen).topk(1023).indices
    out[4:1027] = (pick.sort().values + 4).to(torch.int32)
    out[1027:] = torch.arange(ctx - 1024, ctx, dtype=torch.int32, device="cuda")
    return out


def ok(done, what):
    if not done:
        raise RuntimeError(what + " failed")


def prepare_step(s):
    c, L = s.case, s.L
    ctxs = contexts(c)
    n, mode = len(ctxs), c["mode"]
    s.pos = [ctx - 1 for ctx in ctxs]
    s.stores = [s.store(max(ctx, c["capacity"]) if n == 1 else ctx, ctx - 1) for ctx in ctxs]
    s.k, s.v = s.normal(LAYERS, n, s.nkv * s.hd), s.normal(LAYERS, n, s.nkv * s.hd)
    s.q = s.normal(LAYERS, n, s.nh, s.hd, dtype=torch.bfloat16)
    s.gate = s.normal(LAYERS, n, s.nh, s.hd) if c["gate"] else None
    s.out = s.empty(LAYERS, n, s.nh, s.hd)
    s.outputs = {"out": s.out}
    at = dict(q_bf16=True)
    if mode == "lists":
        s.idx = torch.stack([torch.stack([torch.stack([selection(s, x) for _ in range(s.nkv)]) for x in ctxs]) for _ in range(LAYERS)])
        at.update(width=WIDTH, idx_kvh_stride=WIDTH)
        if n > 1:
            at.update(idx_sess_stride=s.nkv * WIDTH)
    elif mode == "select":
        s.sel = s.empty(LAYERS, n, WIDTH, dtype=torch.int32)
        s.outputs["sel"] = s.sel
        s.iq = s.normal(LAYERS, n, IDX_HEADS, IDX_HD)
        s.blocks = max(st.max_kv for st in s.stores) // RATIO
        s.score = s.empty(n, s.blocks)
        s.pools = [s.normal(LAYERS, st.max_kv // RATIO, IDX_HD) for st in s.stores]
        at.update(width=WIDTH)
        if n > 1:
            at.update(idx_sess_stride=WIDTH)
            s.pool_ptrs = torch.tensor([[p[layer].data_ptr() for p in s.pools] for layer in range(LAYERS)], dtype=torch.int64, device="cuda")
            s.pos_d = torch.tensor(s.pos, dtype=torch.int32, device="cuda")
        else:
            s.raw = s.normal(LAYERS, s.stores[0].max_kv, IDX_HD, dtype=torch.float16)
            s.iwn = s.norm_weight(IDX_HD)

    def idx(layer):
        return s.idx[layer] if mode == "lists" else s.sel[layer] if mode == "select" else None

    def gate(layer):
        return None if s.gate is None else s.gate[layer]

    def one():
        st = s.stores[0]
        for layer in range(LAYERS):
            if mode == "select":
                pool = s.pools[0][layer].data_ptr()
                ok(L.q4_hip_qsa_pool_d(s.raw[layer].data_ptr(), pool, s.iwn.data_ptr(), IDX_HD, RATIO, 64, ROPE_BASE, EPS), "pool")
                ok(L.q4_hip_qsa_score_d(s.iq[layer].data_ptr(), pool, s.score.data_ptr(), s.blocks, IDX_HEADS, IDX_HD, RATIO), "score")
                ok(L.q4_hip_qsa_topk_d(s.score.data_ptr(), s.sel[layer].data_ptr(), s.blocks, K_BLK, RATIO, WIDTH), "topk")
            st.append_decode_d(layer, s.k[layer], s.v[layer], s.q[layer], s.out[layer], s.nh, s.scale, gate=gate(layer), idx=idx(layer), **at)

    def many():
        for layer in range(LAYERS):
            if mode == "select":
                ok(L.q4_gpu_qsa_select_batch(s.pool_ptrs[layer].data_ptr(), s.pos_d.data_ptr(), s.iq[layer].data_ptr(), s.score.data_ptr(),
                                             s.sel[layer].data_ptr(), n, s.blocks, IDX_HEADS, IDX_HD, K_BLK, RATIO, WIDTH), "select")
            s.batch.append_decode(layer, s.k[layer], s.v[layer], s.q[layer], s.out[layer], s.nh, s.scale, gate=gate(layer), idx=idx(layer), **at)

    if n > 1:
        s.batch = q4gpu.Batch(s.stores)
        s.batch.set_pos(s.pos)
        s.capture(many)
    else:
        L.q4_hip_pos_push(s.pos[0])
        s.capture(one)


def run_step(s):
    if len(s.pos) > 1:
        s.batch.set_pos(s.pos)
    else:
        s.L.q4_hip_pos_push(s.pos[0])
    ok(s.L.q4_hip_graph_launch(s.graph), "graph")
    return s.outputs


def prepare_prefill(s):
    c = s.case
    n = c["n_tok"]
    s.st = s.store(c["base"] + n, c["base"])
    s.k, s.v = s.normal(LAYERS, n, s.nkv * s.hd), s.normal(LAYERS, n, s.nkv * s.hd)
    s.wn = s.norm_weight(s.hd)
    s.q = s.normal(LAYERS, n, s.nh, s.hd, dtype=torch.bfloat16)
    s.gate = s.normal(LAYERS, n, s.nh, s.hd) if c["gate"] else None
    s.out = s.empty(LAYERS, n, s.nh, s.hd, dtype=torch.bfloat16)


def run_prefill(s):
    L, n, base = s.L, s.case["n_tok"], s.case["base"]
    for layer in range(LAYERS):
        ok(L.q4_gpu_kv_prep_append(s.st.h, layer, s.k[layer].data_ptr(), s.v[layer].data_ptr(), s.wn.data_ptr(), s.n_rot, ROPE_BASE, EPS, base, n), "append")
        s.st.prefill(layer, s.q[layer], s.out[layer], s.nh, n, base, s.scale, gate=None if s.gate is None else s.gate[layer])
    return s.out


def prepare_sparse_prefill(s):
    c = s.case
    n, end = c["n_tok"], c["base"] + c["n_tok"]
    s.st = s.store(end, c["base"])
    s.k, s.v = s.normal(LAYERS, n, s.nkv * s.hd), s.normal(LAYERS, n, s.nkv * s.hd)
    s.wn, s.iwn = s.norm_weight(s.hd), s.norm_weight(IDX_HD)
    s.q = s.normal(LAYERS, n, s.nh, s.hd, dtype=torch.bfloat16)
    s.out = s.empty(LAYERS, n, s.nh, s.hd)
    s.iq = s.normal(LAYERS, n, IDX_HEADS, IDX_HD)
    s.raw = s.normal(LAYERS, end, IDX_HD, dtype=torch.float16)
    s.blocks = end // RATIO
    s.pool = s.normal(LAYERS, s.blocks, IDX_HD)
    s.score = s.empty(n, s.blocks)
    s.sel = s.empty(LAYERS, n, WIDTH, dtype=torch.int32)


def run_sparse_prefill(s):
    L, n, base = s.L, s.case["n_tok"], s.case["base"]
    for layer in range(LAYERS):
        pool, sel = s.pool[layer].data_ptr(), s.sel[layer].data_ptr()
        ok(L.q4_gpu_kv_prep_append(s.st.h, layer, s.k[layer].data_ptr(), s.v[layer].data_ptr(), s.wn.data_ptr(), s.n_rot, ROPE_BASE, EPS, base, n), "append")
        ok(L.q4_hip_qsa_pool(s.raw[layer].data_ptr(), pool, s.iwn.data_ptr(), IDX_HD, RATIO, base // RATIO, s.blocks, 64, ROPE_BASE, EPS), "pool")
        ok(L.q4_hip_qsa_score(s.iq[layer].data_ptr(), pool, s.score.data_ptr(), n, s.blocks, s.blocks, IDX_HEADS, IDX_HD, base, RATIO), "score")
        ok(L.q4_hip_qsa_topk(s.score.data_ptr(), sel, n, s.blocks, s.blocks, K_BLK, RATIO, base, WIDTH), "topk")
        s.st.decode_idx_n(layer, s.q[layer], s.out[layer], s.nh, s.scale, s.sel[layer], WIDTH, n, WIDTH, q_bf16=True)
    return {"out": s.out, "sel": s.sel}


def prepare_dropin(s, capacity, n, written):
    """caches [layer][token][kv head][row] of the host's own with `written` rows, and a chunk's projections"""
    c, L = s.case, s.L
    s.kvw = s.nkv * s.hd
    s.bpt = s.nkv * row_bytes(c["kind"], s.hd)
    s.kc, s.vc = s.empty(LAYERS, capacity, s.bpt, dtype=torch.uint8), s.empty(LAYERS, capacity, s.bpt, dtype=torch.uint8)
    for cache in (s.kc, s.vc):
        for layer in range(LAYERS):
            cache[layer].zero_()
            if written:
                dropin_write(s, cache[layer], 0, s.normal(written, s.kvw), written)
    s.qg, s.wq, s.wk = s.normal(LAYERS, n, s.nh, 2, s.hd), s.norm_weight(s.hd), s.norm_weight(s.hd)
    s.q, s.g = s.empty(n, s.nh, s.hd), s.empty(n, s.nh, s.hd)
    s.k_in, s.v = s.normal(LAYERS, n, s.kvw), s.normal(LAYERS, n, s.kvw)
    s.k = s.empty(LAYERS, n, s.kvw)
    s.out = s.empty(LAYERS, n, s.nh, s.hd)


def dropin_write(s, cache, pos, rows, n):
    dst, src = cache.data_ptr() + pos * s.bpt, rows.data_ptr()
    if s.kind == q4gpu.KIND_Q8:
        return s.L.q4_hip_f32_to_q8(dst, src, n * s.kvw)
    if s.kind == q4gpu.KIND_F16:
        return s.L.q4_hip_f32_to_f16(dst, src, n * s.kvw)
    return s.L.q4_hip_copy(dst, src, n * s.kvw)


def prepare_dropin_step(s):
    L, ctx = s.L, s.case["ctx"]
    s.pos = ctx - 1
    prepare_dropin(s, ctx, 1, s.pos)
    s.outputs = {"out": s.out, "k": s.kc, "v": s.vc}
    if ctx > WIDTH:
        s.blocks = ctx // RATIO
        s.raw, s.pool = s.normal(LAYERS, ctx, IDX_HD, dtype=torch.float16), s.normal(LAYERS, s.blocks, IDX_HD)
        s.ik, s.iq_in, s.iq = s.normal(LAYERS, IDX_HD), s.normal(LAYERS, IDX_HEADS, IDX_HD), s.empty(LAYERS, IDX_HEADS, IDX_HD)
        s.iwn, s.score, s.sel = s.norm_weight(IDX_HD), s.empty(s.blocks), s.empty(LAYERS, WIDTH, dtype=torch.int32)
        s.outputs["sel"] = s.sel

    def enqueue():
        # the projections' results land in the buffers that the host prepares in place
        ok(L.q4_hip_copy(s.k.data_ptr(), s.k_in.data_ptr(), s.k.numel()), "copy")
        if ctx > WIDTH:
            ok(L.q4_hip_copy(s.iq.data_ptr(), s.iq_in.data_ptr(), s.iq.numel()), "copy")
        for layer in range(LAYERS):
            k, kc, vc = s.k[layer].data_ptr(), s.kc[layer].data_ptr(), s.vc[layer].data_ptr()
            ok(L.q4_hip_qsa_q_prep_d(s.qg[layer].data_ptr(), s.wq.data_ptr(), s.q.data_ptr(), s.g.data_ptr(), s.nh, s.hd, s.n_rot, ROPE_BASE, EPS), "q_prep")
            ok(L.q4_hip_qsa_k_prep_d(k, s.wk.data_ptr(), s.nkv, s.hd, s.n_rot, ROPE_BASE, EPS), "k_prep")
            ok(L.q4_hip_kv_append_d(kc, vc, k, s.v[layer].data_ptr(), s.kvw, s.bpt, s.kind), "append")
            at = (s.q.data_ptr(), kc, vc, s.g.data_ptr(), s.out[layer].data_ptr())
            if ctx > WIDTH:
                iq, pool, sel = s.iq[layer].data_ptr(), s.pool[layer].data_ptr(), s.sel[layer].data_ptr()
                ok(L.q4_hip_f32_to_f16_d(s.raw[layer].data_ptr(), IDX_HD, s.ik[layer].data_ptr(), IDX_HD), "raw key")
                ok(L.q4_hip_qsa_pool_d(s.raw[layer].data_ptr(), pool, s.iwn.data_ptr(), IDX_HD, RATIO, 64, ROPE_BASE, EPS), "pool")
                ok(L.q4_hip_qsa_k_prep_d(iq, s.iwn.data_ptr(), IDX_HEADS, IDX_HD, 64, ROPE_BASE, EPS), "iq prep")
                ok(L.q4_hip_qsa_score_d(iq, pool, s.score.data_ptr(), s.blocks, IDX_HEADS, IDX_HD, RATIO), "score")
                ok(L.q4_hip_qsa_topk_d(s.score.data_ptr(), sel, s.blocks, K_BLK, RATIO, WIDTH), "topk")
                ok(L.q4_hip_qsa_decode_idx(*at, sel, WIDTH, s.nh, s.nkv, s.hd, 1, ctx, s.scale, s.kind), "decode_idx")
            else:
                ok(L.q4_hip_qsa_decode_n(*at, s.nh, s.nkv, s.hd, 1, s.pos, ctx, s.scale, s.kind), "decode_n")

    L.q4_hip_pos_push(s.pos)
    s.capture(enqueue)


def run_dropin_step(s):
    s.L.q4_hip_pos_push(s.pos)
    ok(s.L.q4_hip_graph_launch(s.graph), "graph")
    return s.outputs


def prepare_dropin_prefill(s):
    c = s.case
    prepare_dropin(s, c["base"] + c["n_tok"], c["n_tok"], c["base"])


def run_dropin_prefill(s):
    L, n, base = s.L, s.case["n_tok"], s.case["base"]
    ok(L.q4_hip_copy(s.k.data_ptr(), s.k_in.data_ptr(), s.k.numel()), "copy")
    for layer in range(LAYERS):
        k, kc, vc = s.k[layer], s.kc[layer], s.vc[layer]
        ok(L.q4_hip_qsa_q_prep_n(s.qg[layer].data_ptr(), s.wq.data_ptr(), s.q.data_ptr(), s.g.data_ptr(), s.nh, s.hd, s.n_rot, base, ROPE_BASE, EPS, n), "q_prep")
        ok(L.q4_hip_qsa_k_prep_n(k.data_ptr(), s.wk.data_ptr(), s.nkv, s.hd, s.n_rot, base, ROPE_BASE, EPS, n), "k_prep")
        ok(dropin_write(s, kc, base, k, n) and dropin_write(s, vc, base, s.v[layer], n), "kv_write")
        for t in range(0, n, 512):
            m, off = min(512, n - t), t * s.nh * s.hd * 4
            ok(L.q4_hip_qsa_decode_n(s.q.data_ptr() + off, kc.data_ptr(), vc.data_ptr(), s.g.data_ptr() + off, s.out[layer].data_ptr() + off,
                                     s.nh, s.nkv, s.hd, m, base + t, base + n, s.scale, s.kind), "decode_n")
    return {"out": s.out, "k": s.kc, "v": s.vc}


def prepare_snapshot(s):
    rows = s.case["rows"]
    s.st = s.store(rows + 4096, rows)
    size = s.st.snapshot_bytes(rows)
    s.saved, s.again = s.empty(size, dtype=torch.uint8), s.empty(size, dtype=torch.uint8)
    s.st.save(rows, s.saved)


def run_snapshot(s):
    s.st.restore(s.case["rows"], s.saved)
    s.st.save(s.case["rows"], s.again)
    return s.again


PREPARE = {"step": prepare_step, "prefill": prepare_prefill, "sparse_prefill": prepare_sparse_prefill, "dropin_step": prepare_dropin_step,
           "dropin_prefill": prepare_dropin_prefill, "snapshot": prepare_snapshot}
RUN = {"step": run_step, "prefill": run_prefill, "sparse_prefill": run_sparse_prefill, "dropin_step": run_dropin_step,
       "dropin_prefill": run_dropin_prefill, "snapshot": run_snapshot}


def prepare(case, seed):
    s = State(case, seed)
    with torch.cuda.stream(s.stream):
        PREPARE[case["path"]](s)
    s.stream.synchronize()
    return s


def run(s):
    return RUN[s.case["path"]](s)
