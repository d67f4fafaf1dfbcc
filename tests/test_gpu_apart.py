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
