"""Captured launches that run beside the one before them (norms, the fp16 key, pooling): random sequences over a few buffers of
their own allocations, with every kind of dependence between neighbours (a buffer read after it is written, written after it
is read, written twice), copies between them, positions pushed inside the capture, and the attention that reads what they
wrote.  A replay leaves every buffer with the bytes that the same calls leave one by one, each waited for."""
import random

import numpy as np
import pytest
import torch

import q4gpu

pytestmark = pytest.mark.gpu

N_KVH, N_HEAD, HD, ROWS = 2, 8, 128, 64
KVW, QW = N_KVH * HD, N_HEAD * HD


class Buffers:
    """named device buffers of the library's own allocator, all in one state that can be set again"""

    def __init__(self, L, sizes, seed):
        self.L, rng = L, np.random.default_rng(seed)
        self.size, self.first = sizes, {}
        self.p = {n: L.q4_hip_malloc(b) for n, b in sizes.items()}
        for n, b in sizes.items():
            dt = np.float16 if n.startswith(("raw", "kc", "vc")) else np.float32
            self.first[n] = rng.standard_normal(b // dt().itemsize).astype(dt)

    def reset(self):
        for n, a in self.first.items():
            assert self.L.q4_hip_h2d(self.p[n], a.ctypes.data, self.size[n])

    def read(self):
        out = {}
        for n, b in self.size.items():
            out[n] = np.empty(b, np.uint8)
            assert self.L.q4_hip_d2h(out[n].ctypes.data, self.p[n], b)
        return out

    def free(self):
        for p in self.p.values():
            self.L.q4_hip_free(p)


def sequence(L, b, rng, n):
    p, ops = b.p, []
    two = lambda s: p[s + rng.choice("01")]
    for _ in range(n):
        kind = rng.choice(["q", "q", "k", "k", "iq", "append", "f16", "f16", "pool", "pool", "score", "topk", "attend", "copy", "push"])
        if kind == "q":
            a = (two("qg"), p["wn"], two("q"), two("g"), N_HEAD, HD, 64, 1e4, 1e-6)
            ops.append(lambda a=a: L.q4_hip_qsa_q_prep_d(*a))
        elif kind == "k":
            a = (two("k"), p["wn"], N_KVH, HD, 64, 1e4, 1e-6)
            ops.append(lambda a=a: L.q4_hip_qsa_k_prep_d(*a))
        elif kind == "iq":
            a = (two("q"), p["wn"], 4, HD, 64, 1e4, 1e-6)
            ops.append(lambda a=a: L.q4_hip_qsa_k_prep_d(*a))
        elif kind == "append":
            a = (two("kc"), two("vc"), two("k"), two("k"), KVW, KVW * 2, 1)
            ops.append(lambda a=a: L.q4_hip_kv_append_d(*a))
        elif kind == "f16":
            a = (two("raw"), HD, rng.choice([two("k"), two("q"), p["pool0"]]), HD)
            ops.append(lambda a=a: L.q4_hip_f32_to_f16_d(*a))
        elif kind == "pool":
            a = (two("raw"), two("pool"), p["wn"], HD, 4, 64, 1e4, 1e-6)
            ops.append(lambda a=a: L.q4_hip_qsa_pool_d(*a))
        elif kind == "score":
            a = (two("q"), two("pool"), p["score"], ROWS // 4, 4, HD, 4)
            ops.append(lambda a=a: L.q4_hip_qsa_score_d(*a))
        elif kind == "topk":
            a = (p["score"], p["sel"], ROWS // 4, 8, 4, 35)
            ops.append(lambda a=a: L.q4_hip_qsa_topk_d(*a))
        elif kind == "attend":
            a = (two("q"), two("kc"), two("vc"), two("g"), two("out"), N_HEAD, N_KVH, HD, 1, 40, ROWS, 0.09, 1)
            ops.append(lambda a=a: L.q4_hip_qsa_decode_n(*a))
        elif kind == "copy":
            a = (two("k"), two("q"), KVW)
            ops.append(lambda a=a: L.q4_hip_copy(*a))
        else:
            pos = rng.choice([3, 7, 31, 63, 40])
            ops.append(lambda pos=pos: L.q4_hip_pos_push(pos) or True)
    return ops


@pytest.mark.parametrize("seed", range(12))
def test_captured_sequences_leave_the_bytes_of_single_calls(seed):
    L = q4gpu.init()
    assert L.q4_gpu_set_stream(None) and L.q4_hip_qsa_topk_alloc()
    sizes = {"wn": HD * 4, "score": ROWS, "sel": 35 * 4}
    for i in "01":
        sizes.update({"qg" + i: QW * 8, "q" + i: QW * 4, "g" + i: QW * 4, "k" + i: KVW * 4, "kc" + i: ROWS * KVW * 2, "vc" + i: ROWS * KVW * 2,
                      "raw" + i: ROWS * HD * 2, "pool" + i: ROWS // 4 * HD * 4, "out" + i: QW * 4})
    b = Buffers(L, sizes, seed)
    ops = sequence(L, b, random.Random(seed), 60)
    b.reset()
    L.q4_hip_pos_push(11)
    for op in ops:
        assert op() and L.q4_hip_stream_sync()
    want = b.read()
    assert L.q4_hip_graph_begin() == 1
    for op in ops:
        assert op()
    graph = L.q4_hip_graph_end()
    assert graph
    for again in range(8):
        b.reset()
        L.q4_hip_pos_push(11)
        assert L.q4_hip_graph_launch(graph) and L.q4_hip_stream_sync()
        got = b.read()
        for n in sizes:
            assert np.array_equal(got[n], want[n]), (n, again)
    L.q4_hip_graph_free(graph)
    b.free()
    assert L.q4_gpu_last_error() == 0
    torch.cuda.synchronize()


def test_foreign_work_in_a_capture_is_waited_for():
    """a kernel of the host's between two launches writes what the second reads"""
    L = q4gpu.init()
    assert L.q4_gpu_set_stream(None)
    st = torch.cuda.ExternalStream(L.q4_gpu_stream())
    b = Buffers(L, {"wn": HD * 4, "raw0": ROWS * HD * 2, "pool0": ROWS // 4 * HD * 4}, 1)
    q, k, src = (torch.randn(1 << 20, device="cuda") for _ in range(3))
    torch.cuda.synchronize()
    L.q4_hip_pos_push(7)

    def calls():
        with torch.cuda.stream(st):
            assert L.q4_hip_qsa_k_prep_d(q.data_ptr(), b.p["wn"], N_KVH, HD, 64, 1e4, 1e-6)
            assert L.q4_hip_qsa_k_prep_d(q.data_ptr(), b.p["wn"], N_KVH, HD, 64, 1e4, 1e-6)
            k.copy_(src)
            k.mul_(2.0)
            assert L.q4_hip_f32_to_f16_d(b.p["raw0"], HD, k.data_ptr() + 4 * (k.numel() - HD), HD)
    calls()
    assert L.q4_hip_graph_begin() == 1
    calls()
    graph = L.q4_hip_graph_end()
    assert graph
    for i in range(8):
        with torch.cuda.stream(st):
            src.normal_()
            k.zero_()
        L.q4_hip_pos_push(7)
        assert L.q4_hip_graph_launch(graph) and L.q4_hip_stream_sync()
        row = b.read()["raw0"].view(np.float16).reshape(ROWS, HD)[7]
        assert np.array_equal(row, (src[-HD:] * 2).half().cpu().numpy()), i
    L.q4_hip_graph_free(graph)
    b.free()


def captured(L, calls, launches=1, before=None):
    """the calls as one graph, launched; how many of them may run beside their predecessor"""
    assert L.q4_hip_graph_begin() == 1
    for c in calls:
        assert c() in (True, None)
    graph = L.q4_hip_graph_end()
    assert graph
    n = L.q4_gpu_graph_apart()
    for _ in range(launches):
        if before:
            before()
        assert L.q4_hip_graph_launch(graph) and L.q4_hip_stream_sync()
    L.q4_hip_graph_free(graph)
    return n


def test_which_neighbours_run_apart():
    """independent neighbours do, up to four behind one that did not; every kind of conflict, foreign work and a position that is
    written meanwhile keep the order"""
    L = q4gpu.init()
    assert L.q4_gpu_set_stream(None)
    sizes = {"wn": HD * 4, "arena": 4 * KVW * 4 + 64}
    for i in "0123456":
        sizes.update({"k" + i: KVW * 4, "raw" + i: ROWS * HD * 2, "pool" + i: ROWS // 4 * HD * 4})
    b = Buffers(L, sizes, 5)
    b.reset()
    p = b.p
    L.q4_hip_pos_push(7)
    k_prep = lambda k: lambda: L.q4_hip_qsa_k_prep_d(k, p["wn"], N_KVH, HD, 64, 1e4, 1e-6)
    f16 = lambda raw, src: lambda: L.q4_hip_f32_to_f16_d(raw, HD, src, HD)
    pool = lambda raw, out: lambda: L.q4_hip_qsa_pool_d(raw, out, p["wn"], HD, 4, 64, 1e4, 1e-6)
    copy = lambda d, s: lambda: L.q4_hip_copy(d, s, HD)
    arena = p["arena"]
    assert captured(L, [k_prep(p["k0"]), f16(p["raw0"], p["k1"])]) == 1
    assert captured(L, [f16(p["raw0"], p["k1"]), pool(p["raw1"], p["pool0"])]) == 1
    assert captured(L, [k_prep(p["k0"]), f16(p["raw0"], p["k0"])]) == 0                                  # read after write
    assert captured(L, [f16(p["raw0"], p["k0"]), pool(p["raw0"], p["pool0"])]) == 0
    assert captured(L, [f16(p["raw0"], p["k0"]), k_prep(p["k0"])]) == 0                                  # write after read
    assert captured(L, [k_prep(p["k0"]), k_prep(p["k0"])]) == 0                                          # write after write
    assert captured(L, [k_prep(p["k0"]), k_prep(p["k1"]), f16(p["raw0"], p["k0"])]) == 1   # with the launch before last
    assert captured(L, [k_prep(p["k0"]), copy(p["k2"], p["k3"]), f16(p["raw0"], p["k1"])]) == 0          # another node between
    assert captured(L, [k_prep(p["k0"]), lambda: L.q4_hip_pos_push(7), f16(p["raw0"], p["k1"])]) == 0
    # rows of one allocation: next to each other, and one float of overlap
    assert captured(L, [k_prep(arena), k_prep(arena + KVW * 4)]) == 1
    assert captured(L, [k_prep(arena), k_prep(arena + KVW * 4 - 8)]) == 0
    assert captured(L, [k_prep(arena + KVW * 4), k_prep(arena + 8)]) == 0
    # a row whose place the device knows is taken to reach to the end of its allocation
    assert captured(L, [k_prep(arena + 2 * KVW * 4), f16(arena, p["k0"])]) == 0
    assert captured(L, [k_prep(arena), f16(arena + 2 * KVW * 4, p["k0"])]) == 1
    assert captured(L, [f16(p["raw" + i], p["k" + i]) for i in "012345"]) == 4                           # the sixth waits
    assert captured(L, [f16(p["raw" + i], p["k" + i]) for i in "0123456"]) == 5
    b.free()
    assert L.q4_gpu_last_error() == 0


def test_weights_and_position_written_by_the_launch_before_last():
    """read on every SM, written, a launch that is waited for, and then a launch apart that reads them"""
    L = q4gpu.init()
    assert L.q4_gpu_set_stream(None)
    wide = 8 * torch.cuda.get_device_properties(0).multi_processor_count
    b = Buffers(L, {"wn": HD * 4, "q0": wide * HD * 4, "q1": wide * HD * 4, "q2": wide * HD * 4, "k0": KVW * 4, "k1": KVW * 4}, 6)
    p = b.p

    def ops(pos):
        return [lambda: L.q4_hip_qsa_k_prep_d(p["q0"], p["wn"], wide, HD, 64, 1e4, 1e-6),
                lambda: L.q4_hip_qsa_k_prep_d(p["wn"], None, 1, HD, 64, 1e4, 1e-6),
                lambda: L.q4_hip_qsa_k_prep_d(p["k0"], p["wn"], N_KVH, HD, 64, 1e4, 1e-6),
                lambda: L.q4_hip_qsa_k_prep_d(p["q1"], p["wn"], wide, HD, 64, 1e4, 1e-6),
                lambda: L.q4_hip_pos_push(pos),
                lambda: L.q4_hip_qsa_k_prep_d(p["k1"], p["wn"], N_KVH, HD, 64, 1e4, 1e-6),
                lambda: L.q4_hip_qsa_k_prep_d(p["q2"], p["wn"], wide, HD, 64, 1e4, 1e-6)]

    b.reset()
    L.q4_hip_pos_push(11)
    for op in ops(5000):
        assert op() in (True, None) and L.q4_hip_stream_sync()
    want = b.read()
    results = []

    def before():
        results.append(b.read())
        b.reset()
        L.q4_hip_pos_push(11)
    assert captured(L, ops(5000), launches=12, before=before) == 2
    results.append(b.read())
    for got in results[1:]:
        for n in want:
            assert np.array_equal(got[n], want[n]), n
    b.free()
    assert L.q4_gpu_last_error() == 0


@pytest.mark.parametrize("dependent", [False, True])
def test_launch_behind_a_long_attention(dependent):
    """pooling runs beside a store's append + attention; the norm of the attention's output waits for it, long as that is"""
    L = q4gpu.init()
    assert L.q4_gpu_set_stream(None) and L.q4_hip_qsa_topk_alloc()
    rows = 60000
    b = Buffers(L, {"raw0": rows * HD * 2, "pool0": rows // 4 * HD * 4, "wn": HD * 4, "out0": QW * 4}, 7)
    p = b.p
    with torch.cuda.stream(torch.cuda.ExternalStream(L.q4_gpu_stream())):
        g = torch.Generator(device="cuda").manual_seed(3)
        st = q4gpu.KVStore(1, N_KVH, HD, rows, 2)
        st.append(0, torch.randn(rows - 1, KVW, device="cuda", generator=g), torch.randn(rows - 1, KVW, device="cuda", generator=g), 0, rows - 1)
        k, v, q = (torch.randn(n, device="cuda", generator=g) for n in (KVW, KVW, QW))
        L.q4_hip_pos_push(rows - 1)

        def attend():
            return L.q4_gpu_kv_append_decode_d(st.h, 0, k.data_ptr(), v.data_ptr(), q.data_ptr(), 0, None, p["out0"], N_HEAD, None, 0, 0, 0.09)

        def behind():
            if dependent:
                return L.q4_hip_qsa_k_prep_d(p["out0"], p["wn"], N_HEAD, HD, 64, 1e4, 1e-6)
            return L.q4_hip_qsa_pool_d(p["raw0"], p["pool0"], p["wn"], HD, 4, 64, 1e4, 1e-6)
        b.reset()
        assert attend() and L.q4_hip_stream_sync() and behind() and L.q4_hip_stream_sync()
        want = b.read()
        for _ in range(4):
            assert captured(L, [attend, behind], before=b.reset) == (0 if dependent else 1)
            got = b.read()
            assert all(np.array_equal(got[n], want[n]) for n in want)
        st.close()
    b.free()
    assert L.q4_gpu_last_error() == 0


def test_scores_that_read_their_blocks_ahead():
    """the score of a captured step requests all blocks but the newest before it waits: not where a launch that may still run
    writes an older one, and the block that pooling completes in the same step is waited for"""
    L = q4gpu.init()
    assert L.q4_gpu_set_stream(None) and L.q4_hip_qsa_topk_alloc()
    blocks = 9001
    b = Buffers(L, {"raw0": 4 * blocks * HD * 2, "raw1": 4 * blocks * HD * 2, "arena": 2 * blocks * HD * 4, "wn": HD * 4, "q0": 4 * HD * 4, "q1": 4 * HD * 4, "score": blocks * 4,
                    "k0": KVW * 4}, 8)
    p = b.p
    other = p["arena"] + blocks * HD * 4
    pool = lambda to, ratio=4: lambda: L.q4_hip_qsa_pool_d(p["raw0"], to, p["wn"], HD, ratio, 64, 1e4, 1e-6)
    score = lambda: L.q4_hip_qsa_score_d(p["q0"], p["arena"], p["score"], blocks, 4, HD, 4)
    at_host = lambda: L.q4_hip_qsa_score(p["q0"], p["arena"], p["score"], 1, blocks, blocks, 4, HD, 4 * blocks - 1, 4)
    norm = lambda x, heads: lambda: L.q4_hip_qsa_k_prep_d(x, p["wn"], heads, HD, 64, 1e4, 1e-6)
    many = lambda: L.q4_hip_qsa_pool(p["raw1"], p["arena"], p["wn"], HD, 4, 0, blocks, 64, 1e4, 1e-6)
    last = lambda: L.q4_hip_qsa_pool(p["raw1"], p["arena"], p["wn"], HD, 4, blocks - 1, blocks, 64, 1e4, 1e-6)
    old = lambda: L.q4_hip_copy(p["arena"], other, 64 * HD)
    row = lambda: L.q4_hip_qsa_k_prep_d(p["arena"] + 77 * HD * 4, p["wn"], 1, HD, 64, 1e4, 1e-6)
    for case, (calls, ahead) in enumerate([([norm(p["k0"], 2), pool(p["arena"]), score], 1),
                         ([norm(p["k0"], 2), pool(p["arena"]), norm(p["q0"], 4), score], 1),
                         ([pool(p["arena"]), norm(p["q0"], 4), score, pool(p["arena"]), score], 2),
                         ([score], 0),                                                    # nothing is known of what was before
                         ([norm(p["k0"], 2), pool(other), score], 1),                     # another layer's block, to the end of the allocation
                         ([norm(p["k0"], 2), pool(p["arena"], 2), score], 0),             # a block of other tokens
                         ([norm(p["k0"], 2), many, score], 0),
                         ([norm(p["k0"], 2), last, score], 0),
                         ([norm(p["k0"], 2), pool(p["arena"]), old, score], 0),           # a copy
                         ([norm(p["k0"], 2), row, score], 0),
                         ([row, norm(p["q0"], 4), score], 0),                             # the norm does not wait for the first
                         ([row, norm(p["q0"], 4), pool(p["arena"]), score], 1),           # pooling does: it writes there too
                         ([row, norm(p["q0"], 4), score, pool(p["arena"]), score], 1),
                         ([norm(p["k0"], 2), pool(p["arena"]), at_host], 0),              # the word's block is not the host position's newest
                         ([norm(p["k0"], 2), pool(other), at_host], 1)]):
        for pos in (4 * blocks - 1, 4 * blocks - 2, 4 * 8192 - 1, 3):
            b.reset()
            L.q4_hip_pos_push(pos)
            for call in calls:
                assert call() and L.q4_hip_stream_sync()
            want = b.read()
            captured(L, calls, before=b.reset)
            assert L.q4_gpu_graph_ahead() == ahead, case
            got = b.read()
            for n in want:
                assert np.array_equal(got[n], want[n]), (n, pos, case)
    b.free()
    assert L.q4_gpu_last_error() == 0
