"""GPU parity of the tensor-core (tcgen05) causal prefill attention against the CPU oracle.
Outputs are bf16 by contract, so the comparison allows one bf16 rounding of the result on top of
the stated 2e-3 max-abs / 1e-3 relative tolerance."""
import ctypes

import numpy as np
import pytest
import torch

import q4gpu
from gpu_util import dev, host, lib

pytestmark = pytest.mark.gpu


def check(got, ref, what, out_scale=1.0):
    """2e-3 max-abs (times out_scale, the magnitude of the outputs, for the large-magnitude cases) + 1e-3
    relative, plus one bf16 rounding of the result"""
    got, ref = np.asarray(got, np.float64), np.asarray(ref, np.float64)
    assert np.isfinite(got).all(), what
    bound = 2e-3 * out_scale + (1e-3 + 2.0 ** -8) * np.abs(ref)
    err = np.abs(got - ref)
    worst = (err / bound).argmax()
    assert (err <= bound).all(), "%s: max abs err %.3e at ref %.3f; worst err %.3e against bound %.3e at ref %.3f" % (
        what, err.max(), ref.reshape(-1)[err.argmax()], err.reshape(-1)[worst], bound.reshape(-1)[worst], ref.reshape(-1)[worst])
    return err.max()


def run_case(oracle, n_tok, kv_base, n_head, n_kvh, seed, gate=True, rope=False):
    hd = 128
    ctx = kv_base + n_tok
    kvw = n_kvh * hd
    k = oracle.normal(seed, 0, ctx * kvw).reshape(ctx, kvw)
    v = oracle.normal(seed, 1, ctx * kvw).reshape(ctx, kvw)
    q = oracle.normal(seed, 2, n_tok * n_head * hd).reshape(n_tok, n_head, hd)
    if rope:
        k = oracle.rope_rows(k.reshape(ctx, n_kvh, hd), hd, 0, 1e7).reshape(ctx, kvw)
        q = oracle.rope_rows(q, hd, kv_base, 1e7)
    g = oracle.normal(seed, 3, n_tok * n_head * hd) if gate else None
    qb = oracle.f32_to_bf16(q)
    scale = 1.0 / np.sqrt(hd)
    st = q4gpu.KVStore(2, n_kvh, hd, ctx + 3, 2)
    st.append(1, dev(k), dev(v), 0, ctx)
    dq = torch.from_numpy(qb.view(np.int16).reshape(-1)).cuda()
    dout = torch.empty(n_tok * n_head * hd, dtype=torch.bfloat16, device="cuda")
    st.prefill(1, dq, dout, n_head, n_tok, kv_base, scale, gate=dev(g) if gate else None)
    got = host(dout.float()).reshape(n_tok, n_head, hd)
    ref = oracle.attn(oracle.bf16_to_f32(qb), oracle.kv_write(k, 2), oracle.kv_write(v, 2), g, n_head, n_kvh, hd,
                      n_tok, kv_base, ctx + 3, scale, 2, threads=8)
    st.close()
    return check(got, ref, "prefill n_tok %d kv_base %d heads %d/%d" % (n_tok, kv_base, n_head, n_kvh))


@pytest.mark.parametrize("n_tok,kv_base", [(1, 0), (2, 0), (16, 0), (17, 5), (33, 100), (64, 63), (50, 200), (130, 1)])
def test_prefill_small_ragged(oracle, n_tok, kv_base):
    lib()
    run_case(oracle, n_tok, kv_base, 16, 2, 1000 + n_tok)
    assert q4gpu.load().q4_gpu_last_error() == 0


@pytest.mark.parametrize("n_head,n_kvh", [(8, 1), (2, 2), (12, 1), (24, 2), (32, 2), (5, 1)])
def test_prefill_gqa_shapes(oracle, n_head, n_kvh):
    lib()
    run_case(oracle, 40, 77, n_head, n_kvh, 2000 + n_head, gate=(n_head % 2 == 0))


@pytest.mark.parametrize("n_head,n_kvh,n_tok,kv_base", [(64, 4, 297, 0), (64, 4, 313, 700), (9, 3, 1300, 5)])
def test_prefill_two_query_groups_per_block(oracle, n_head, n_kvh, n_tok, kv_base):
    """enough query groups to fill the SMs: two per block, the last of them partly or wholly padding"""
    lib()
    run_case(oracle, n_tok, kv_base, n_head, n_kvh, 3000 + n_tok)
    assert q4gpu.load().q4_gpu_last_error() == 0


@pytest.mark.parametrize("n_head,n_kvh,n_tok,kv_base", [(64, 4, 745, 0), (64, 4, 761, 130), (64, 4, 299, 3001), (16, 2, 37, 2950)])
def test_prefill_waves_and_ranges(oracle, n_head, n_kvh, n_tok, kv_base):
    """two query groups per block (above two and a half waves of one), and one group with its positions in ranges:
    several waves of blocks, and more ranges than tiles of one"""
    lib()
    run_case(oracle, n_tok, kv_base, n_head, n_kvh, 4000 + n_tok)
    assert q4gpu.load().q4_gpu_last_error() == 0


def test_prefill_chunk_over_existing_cache(oracle):
    """the chunked-prefill shape scaled down: 512 new tokens over a 1024-token cache, RoPE'd inputs"""
    lib()
    run_case(oracle, 512, 1024, 16, 2, 20261125 + 3, gate=False, rope=True)


def test_prefill_matches_decode_kernel(oracle):
    """the last query of a prefill chunk == the decode kernel's answer for the same rows"""
    lib()
    n_head, n_kvh, hd, ctx, n_tok = 16, 2, 128, 700, 90
    kvw = n_kvh * hd
    k = oracle.normal(5, 0, ctx * kvw).reshape(ctx, kvw)
    v = oracle.normal(5, 1, ctx * kvw).reshape(ctx, kvw)
    q = oracle.bf16_to_f32(oracle.f32_to_bf16(oracle.normal(5, 2, n_tok * n_head * hd))).reshape(n_tok, n_head, hd)
    st = q4gpu.KVStore(1, n_kvh, hd, ctx, 2)
    st.append(0, dev(k), dev(v), 0, ctx)
    dq = dev(q).to(torch.bfloat16)
    dout = torch.empty(n_tok, n_head, hd, dtype=torch.bfloat16, device="cuda")
    st.prefill(0, dq, dout, n_head, n_tok, ctx - n_tok, 0.0884)
    dd = torch.empty(n_head * hd, device="cuda")
    for t in (0, 45, n_tok - 1):
        st.decode(0, dq[t].contiguous(), dd, n_head, 0.0884, n_kv=ctx - n_tok + t + 1, q_bf16=True)
        check(host(dout[t].float()), host(dd).reshape(n_head, hd), "token %d" % t)
    st.close()


def test_prefill_rejects_unsupported(oracle):
    L = lib()
    st = q4gpu.KVStore(1, 2, 128, 64, 1)      # fp16 store: not the tensor-core path
    buf = torch.zeros(16 * 128, dtype=torch.bfloat16, device="cuda")
    assert not L.q4_gpu_kv_prefill(st.h, 0, buf.data_ptr(), None, buf.data_ptr(), 16, 1, 0, 0.1)
    assert L.q4_gpu_last_error() & 1
    st.close()


@pytest.mark.parametrize("mode", ["sigma8", "head_x50"])
def test_prefill_large_magnitude_queries(oracle, mode):
    """queries ~ N(0, 8^2), or one head of each kv group scaled by 50: scores of several hundred in the
    exponent, softmax close to one-hot.  This checks the running-max rescale, the fp16 weights and the
    accumulators at such magnitudes.  The tensor-core path stages K and V as fp16(code * scale) (the
    reference's own fp16 tile), a rounding that |q| multiplies; to keep it out of this check every 32-value
    block of the rows gets one element of magnitude 127/32, which makes its scale exactly 1/32 and every
    dequantised value exact in fp16 (the rounding itself is covered by the N(0,1) cases at the stated
    tolerance).  The absolute part of the tolerance is relative to the magnitude of the outputs."""
    lib()
    n_tok, kv_base, n_head, n_kvh, hd = 96, 400, 16, 2, 128
    ctx, kvw = kv_base + n_tok, n_kvh * hd

    def rows(stream):
        x = np.clip(oracle.normal(5200, stream, ctx * kvw), -3.9, 3.9).reshape(-1, 32)
        sign = np.where(x[:, 7] < 0, -1.0, 1.0).astype(np.float32)
        x[:, 7] = sign * np.float32(127.0 / 32.0)
        return x.reshape(ctx, kvw)
    k, v = rows(0), rows(1)
    q = oracle.normal(5200, 2, n_tok * n_head * hd).reshape(n_tok, n_head, hd).copy()
    if mode == "sigma8":
        q *= 8.0
    else:
        q[:, 3] *= 50.0
        q[:, 12] *= 50.0
    g = oracle.normal(5200, 3, n_tok * n_head * hd)
    qb = oracle.f32_to_bf16(q)
    scale = 1.0 / np.sqrt(hd)
    kc, vc = oracle.kv_write(k, 2), oracle.kv_write(v, 2)
    assert (kc.reshape(-1, 34)[:, :2].view(np.uint16) == 0x2800).all()      # every block scale is fp16 1/32
    st = q4gpu.KVStore(1, n_kvh, hd, ctx, 2)
    st.append(0, dev(k), dev(v), 0, ctx)
    dq = torch.from_numpy(qb.view(np.int16).reshape(-1)).cuda()
    dout = torch.empty(n_tok * n_head * hd, dtype=torch.bfloat16, device="cuda")
    st.prefill(0, dq, dout, n_head, n_tok, kv_base, scale, gate=dev(g))
    ref = oracle.attn(oracle.bf16_to_f32(qb), kc, vc, g, n_head, n_kvh, hd, n_tok, kv_base, ctx, scale, 2, threads=8)
    check(host(dout.float()).reshape(n_tok, n_head, hd), ref, "prefill, %s" % mode, out_scale=max(1.0, float(np.abs(ref).max())))
    st.close()


@pytest.mark.parametrize("kind", [2, 1, 0])
@pytest.mark.parametrize("n_head,n_kvh,hd,n_tok,kv_base,max_kv", [
    (24, 2, 256, 40, 0, 40), (24, 2, 256, 23, 1000, 1023), (4, 4, 256, 130, 127, 257), (16, 1, 256, 9, 640, 640),
    (16, 2, 128, 300, 500, 800), (16, 2, 128, 8, 2000, 2008), (3, 1, 128, 129, 0, 129), (16, 2, 128, 100, 30, 90), (64, 4, 128, 301, 200, 501),
    (24, 2, 256, 385, 2100, 2400), (24, 2, 256, 385, 2100, 2112)])   # pairs of blocks
def test_reference_abi_chunks_on_the_tensor_cores(oracle, kind, n_head, n_kvh, hd, n_tok, kv_base, max_kv):
    """q4_hip_qsa_decode_n with a prompt's slice on caches in the reference layout: every kind at both head sizes, group
    sizes that do not divide the 128-row tiles, tile edges, position ranges split over several blocks (few tokens
    behind many rows) and rows that max_kv cuts off; the tolerance is the fp32 oracle's"""
    from gpu_util import assert_close, dev_bytes
    L = lib()
    kvw = n_kvh * hd
    seed = 7000 + n_tok + hd
    rows = min(kv_base + n_tok, max_kv)
    k = oracle.normal(seed, 0, rows * kvw).reshape(rows, kvw)
    v = oracle.normal(seed, 1, rows * kvw).reshape(rows, kvw)
    q = oracle.normal(seed, 2, n_tok * n_head * hd)
    g = oracle.normal(seed, 3, n_tok * n_head * hd)
    kc, vc = oracle.kv_write(k, kind), oracle.kv_write(v, kind)
    out = torch.full((n_tok * n_head * hd,), float("nan"), device="cuda")
    scale = float(1.0 / np.sqrt(hd))
    assert L.q4_hip_qsa_decode_n(dev(q).data_ptr(), dev_bytes(kc).data_ptr(), dev_bytes(vc).data_ptr(), dev(g).data_ptr(), out.data_ptr(),
                                 n_head, n_kvh, hd, n_tok, kv_base, max_kv, scale, kind)
    ref = oracle.attn(q.reshape(n_tok, n_head, hd), kc, vc, g, n_head, n_kvh, hd, n_tok, kv_base, max_kv, scale, kind, threads=8)
    assert_close(host(out).reshape(ref.shape), ref, "kind %d %d/%d/%d" % (kind, n_head, n_kvh, hd))
    assert L.q4_gpu_last_error() == 0


def chunk_caches(L, seed, rows, kvw, kind=2):
    """caches of N(0,1) rows in the reference layout, quantised on the device"""
    g = torch.Generator(device="cuda").manual_seed(seed)
    bpt = {2: kvw // 32 * 34, 1: kvw * 2}[kind]
    out = []
    for _ in range(2):
        c = torch.empty(rows * bpt, dtype=torch.uint8, device="cuda")
        for p in range(0, rows, 65536):
            m = min(65536, rows - p)
            x = torch.randn(m * kvw, device="cuda", generator=g)
            f = L.q4_hip_f32_to_q8 if kind == 2 else L.q4_hip_f32_to_f16
            assert f(c.data_ptr() + p * bpt, x.data_ptr(), m * kvw)
        torch.cuda.synchronize()
        out.append(c)
    return out


def test_reference_abi_chunk_where_no_memory_is_left_for_operand_images():
    """12 tokens over 262144 rows want 1 GB of operand images: with 0.4 GB left on the card they are answered without, by the
    decode kernel, with no status bit, and the next launch is not taken for a failed one"""
    from gpu_util import assert_close
    L = lib()
    L.q4_hip_shutdown()                       # gives back what other tests made it reserve
    L = lib()
    n_head, n_kvh, hd, rows, n_tok = 24, 2, 256, 262144, 12
    kc, vc = chunk_caches(L, 11, rows, n_kvh * hd)
    g = torch.Generator(device="cuda").manual_seed(12)
    q, gate = torch.randn(n_tok, n_head, hd, device="cuda", generator=g), torch.randn(n_tok, n_head, hd, device="cuda", generator=g)
    out, want = torch.full_like(q, float("nan")), torch.empty_like(q)
    scale = 1.0 / 16.0
    for t in range(n_tok):
        assert L.q4_hip_qsa_decode_n(q[t].data_ptr(), kc.data_ptr(), vc.data_ptr(), gate[t].data_ptr(), want[t].data_ptr(), n_head, n_kvh, hd, 1,
                                     rows - n_tok + t, rows, scale, 2)
    # the chunk kernels, loaded while there is room
    assert L.q4_hip_qsa_decode_n(q.data_ptr(), kc.data_ptr(), vc.data_ptr(), gate.data_ptr(), out.data_ptr(), n_head, n_kvh, hd, n_tok, 0, 2048, scale, 2)
    row = torch.randn(n_kvh * hd + 4, device="cuda", generator=g)
    kf, vf = torch.zeros(4 * n_kvh * hd, device="cuda"), torch.zeros(4 * n_kvh * hd, device="cuda")
    L.q4_hip_pos_push(1)
    odd = (row.data_ptr() + 4, row.data_ptr() + 4, n_kvh * hd, 4 * n_kvh * hd, 0)
    assert L.q4_hip_kv_append_d(kf.data_ptr(), vf.data_ptr(), *odd)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    hog = L.q4_hip_malloc(torch.cuda.mem_get_info()[0] - (400 << 20))
    assert hog
    out.fill_(float("nan"))
    ok = L.q4_hip_qsa_decode_n(q.data_ptr(), kc.data_ptr(), vc.data_ptr(), gate.data_ptr(), out.data_ptr(), n_head, n_kvh, hd, n_tok, rows - n_tok, rows,
                               scale, 2)
    nxt = L.q4_hip_kv_append_d(kf.data_ptr(), vf.data_ptr(), *odd)
    got, err = host(out), L.q4_gpu_last_error()
    L.q4_hip_free(hog)
    assert ok and nxt and err == 0
    assert_close(got, host(want), "chunk without operand images")
    # the store's own prefill has no other form: refused, reported, and the next launch is sound
    st = q4gpu.KVStore(1, 2, 128, 262144, 2)
    bq = torch.zeros(8 * 16 * 128, dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    hog = L.q4_hip_malloc(torch.cuda.mem_get_info()[0] - (100 << 20))
    bad = L.q4_gpu_kv_prefill(st.h, 0, bq.data_ptr(), None, bq.data_ptr(), 16, 8, 262144 - 8, 0.1)
    nxt = L.q4_hip_kv_append_d(kf.data_ptr(), vf.data_ptr(), *odd)
    torch.cuda.synchronize()
    L.q4_hip_free(hog)
    assert not bad and nxt and L.q4_gpu_last_error() & 2
    st.close()


def test_captured_chunk_keeps_its_workspace_when_that_grows():
    """a captured slice, then a longer one that makes the operand images grow, memory of the old size taken by others, and the
    graph again; the same for a captured scan whose records lie in scratch.  With the last graph the old workspaces go back."""
    L = lib()
    L.q4_gpu_set_stream(None)                 # captures need a created stream
    L.q4_hip_shutdown()
    L = q4gpu.init()
    with torch.cuda.stream(torch.cuda.ExternalStream(L.q4_gpu_stream())):
        n_head, n_kvh, hd, n_tok, rows, more = 24, 2, 256, 16, 2048, 40000
        kc, vc = chunk_caches(L, 21, more, n_kvh * hd, 1)
        g = torch.Generator(device="cuda").manual_seed(22)
        q, gate = torch.randn(n_tok, n_head, hd, device="cuda", generator=g), torch.randn(n_tok, n_head, hd, device="cuda", generator=g)
        out, one = torch.empty_like(q), torch.empty(n_head, hd, device="cuda")

        def chunk(n, to):
            assert L.q4_hip_qsa_decode_n(q.data_ptr(), kc.data_ptr(), vc.data_ptr(), gate.data_ptr(), to.data_ptr(), n_head, n_kvh, hd, n_tok, n - n_tok, n,
                                         1.0 / 16.0, 1)

        def scan():
            assert L.q4_hip_qsa_decode_n(q.data_ptr(), kc.data_ptr(), vc.data_ptr(), gate.data_ptr(), one.data_ptr(), n_head, n_kvh, hd, 1, more - 1, more,
                                         1.0 / 16.0, 1)
        chunk(rows, out)
        scan()
        want, want_one = out.clone(), one.clone()
        assert L.q4_hip_graph_begin()
        chunk(rows, out)
        scan()
        graph = L.q4_hip_graph_end()
        assert graph
        chunk(more, torch.empty_like(out))    # operand images grow
        assert L.q4_hip_qsa_topk_alloc()      # scratch grows
        others = [torch.full((s << 20,), 0xff, dtype=torch.uint8, device="cuda") for s in (1, 2, 4, 8, 16, 32, 64)]
        out.zero_()
        one.zero_()
        for _ in range(3):
            assert L.q4_hip_graph_launch(graph)
        torch.cuda.synchronize()
        assert torch.equal(out, want) and torch.equal(one, want_one)
        assert all(bool((o == 0xff).all()) for o in others)
        assert L.q4_gpu_last_error() == 0
        del others
        torch.cuda.empty_cache()
        before = torch.cuda.mem_get_info()[0]
        L.q4_hip_graph_free(graph)
        assert torch.cuda.mem_get_info()[0] > before
    torch.cuda.synchronize()


def run_chunk(L, q, kc, vc, gate, n_head, n_kvh, hd, kv_base, max_kv, scale, kind):
    from gpu_util import dev_bytes
    n_tok = q.shape[0]
    out = torch.full((n_tok, n_head, hd), float("nan"), device="cuda")
    assert L.q4_hip_qsa_decode_n(dev(q).data_ptr(), dev_bytes(kc).data_ptr(), dev_bytes(vc).data_ptr(), dev(gate).data_ptr(), out.data_ptr(), n_head, n_kvh,
                                 hd, n_tok, kv_base, max_kv, scale, kind)
    return host(out)


@pytest.mark.parametrize("n_head,n_kvh,hd", [(24, 2, 256), (16, 2, 128)])
def test_first_token_of_a_reference_abi_chunk_is_its_value_row(oracle, n_head, n_kvh, hd):
    """a token that attends one row has weight 1 and gets codes x scales x sigmoid(gate) with no rounding to 16 bits: what is
    left is the gate's (2^-20); the values have 19 bits, a single fp16 image of them would be off by 2^-12"""
    L = lib()
    n, kvw = 208, n_kvh * hd          # tokens x rows x kv heads: on the tensor cores at both head sizes
    k, v = oracle.normal(41, 0, n * kvw).reshape(n, kvw), oracle.normal(41, 1, n * kvw).reshape(n, kvw)
    q, g = oracle.normal(41, 2, n * n_head * hd).reshape(n, n_head, hd), oracle.normal(41, 3, n * n_head * hd).reshape(n, n_head, hd)
    kc, vc = oracle.kv_write(k, 2), oracle.kv_write(v, 2)
    got = run_chunk(L, q, kc, vc, g, n_head, n_kvh, hd, 0, n, float(1.0 / np.sqrt(hd)), 2)[0].astype(np.float64)
    blocks = vc.reshape(n, n_kvh, hd // 32, 34)[0]
    rows = blocks[..., 2:].copy().view(np.int8).astype(np.float64) * blocks[..., :2].copy().view(np.float16).astype(np.float64)
    want = np.repeat(rows.reshape(n_kvh, hd), n_head // n_kvh, 0) / (1.0 + np.exp(-g[0].astype(np.float64)))
    assert (np.abs(got - want) <= 4e-6 * np.abs(want)).all(), np.abs(got / want - 1)[want != 0].max()


@pytest.mark.parametrize("kind,big", [(2, 900.0), (0, 1.0e5)])
@pytest.mark.parametrize("n_head,n_kvh,hd,n_tok,kv_base", [(24, 2, 256, 7, 300), (24, 2, 256, 40, 300), (16, 2, 128, 7, 300), (16, 2, 128, 140, 300),
                                                        (24, 2, 256, 385, 2100), (16, 2, 128, 610, 1600)])   # pairs of blocks
def test_reference_abi_chunk_of_rows_beyond_fp16(oracle, kind, big, n_head, n_kvh, hd, n_tok, kv_base):
    """values beyond 65504 in some rows of K and of V (q8_0: a block scale of 900 is a legal fp16; fp32: magnitudes of 1e5, in
    one dim that the queries leave out, since the decode form rounds fp32 rows to fp16): finite and right for few tokens and for
    many.  The rows of K with large values are turned away from the queries, those of V have ordinary keys.  An output is the
    large value times its weight, so its error is the weight's: 2^-11 from its own rounding, inside the 1e-3; queries, and the
    fp32 rows, are fp16 numbers here, or their rounding would move the scores by up to 1e-3 more (3.5 sigma of 2e-4)."""
    from gpu_util import assert_close
    L = lib()
    n, kvw = kv_base + n_tok, n_kvh * hd
    k, v = oracle.normal(51, 0, n * kvw).reshape(n, kvw).copy(), oracle.normal(51, 1, n * kvw).reshape(n, kvw).copy()
    q, g = oracle.normal(51, 2, n_tok * n_head * hd).reshape(n_tok, n_head, hd), oracle.normal(51, 3, n_tok * n_head * hd).reshape(n_tok, n_head, hd)
    q, k, v = (x.astype(np.float16).astype(np.float32) for x in (q, k, v))
    if kind == 2:
        q[..., :32] = np.abs(q[..., :32])
        for r in (3, 130, 290):
            k[r].reshape(n_kvh, hd)[:, :32] = -big * 127 * np.linspace(0.5, 1.0, 32, dtype=np.float32)
        v[100].reshape(n_kvh, hd)[:, 32:64] = big * 127 * np.linspace(-1.0, 1.0, 32, dtype=np.float32)
        kc, vc = oracle.kv_write(k, kind), oracle.kv_write(v, kind)
    else:
        q[..., 5] = 0.0
        if n_tok < 8:
            pytest.skip("the decode form rounds fp32 rows to fp16")
        k[130].reshape(n_kvh, hd)[:, 5] = big
        v[100].reshape(n_kvh, hd)[:, 40] = -big
        kc, vc = oracle.kv_write(k, kind), oracle.kv_write(v, kind)
    scale = float(1.0 / np.sqrt(hd))
    got = run_chunk(L, q, kc, vc, g, n_head, n_kvh, hd, kv_base, n, scale, kind)
    ref = oracle.attn(q, kc, vc, g, n_head, n_kvh, hd, n_tok, kv_base, n, scale, kind, threads=8)
    assert_close(got, ref, "kind %d" % kind)
    assert L.q4_gpu_last_error() == 0


@pytest.mark.parametrize("kind", [2, 1, 0])
@pytest.mark.parametrize("n_head,n_kvh,hd,n_tok,kv_base,at", [(24, 2, 256, 40, 200, 17), (16, 2, 128, 140, 200, 17),
                                                                (24, 2, 256, 385, 2100, 75), (24, 2, 256, 385, 2100, 76), (16, 2, 128, 610, 1600, 64)])   # pairs of blocks, both sides of a tile
def test_reference_abi_chunk_with_value_rows_that_are_not_finite(oracle, kind, n_head, n_kvh, hd, n_tok, kv_base, at):
    """a token's output depends on the rows up to its own: those before a row with an infinity or NaN in V stay as they are, the
    others get NaN"""
    from gpu_util import assert_close
    L = lib()
    kvw = n_kvh * hd
    n = kv_base + n_tok
    k, v = oracle.normal(61, 0, n * kvw).reshape(n, kvw), oracle.normal(61, 1, n * kvw).reshape(n, kvw).copy()
    q, g = oracle.normal(61, 2, n_tok * n_head * hd).reshape(n_tok, n_head, hd), oracle.normal(61, 3, n_tok * n_head * hd).reshape(n_tok, n_head, hd)
    kc, vc = oracle.kv_write(k, kind), oracle.kv_write(v, kind).copy()
    scale = float(1.0 / np.sqrt(hd))
    ref = oracle.attn(q, kc, vc, g, n_head, n_kvh, hd, n_tok, kv_base, n, scale, kind, threads=8)
    row = vc.reshape(n, -1)[kv_base + at]
    if kind == 2:
        row.view(np.uint16)[17 * 1] = 0x7C00                     # the second block's scale: infinity
    elif kind == 1:
        row.view(np.float16)[9] = np.inf
    else:
        row.view(np.float32)[9] = np.nan
    got = run_chunk(L, q, kc, vc, g, n_head, n_kvh, hd, kv_base, n, scale, kind)
    assert_close(got[:at], ref[:at], "tokens before the row")
    assert np.isnan(got[at:, :n_head // n_kvh]).any(axis=(1, 2)).all()
    assert_close(got[at:, n_head // n_kvh:], ref[at:, n_head // n_kvh:], "the other kv head")


@pytest.mark.parametrize("kind", [2, 1, 0])
@pytest.mark.parametrize("n_tok,rows", [(20, 2048), (20, 2049), (7, 8000), (8, 8000), (208, 208)])
def test_reference_abi_chunks_on_both_sides_of_the_decode_form(oracle, kind, n_tok, rows):
    """few tokens, and at hd 128 few tokens over few rows, are the decode kernel's; more are a chunk"""
    test_reference_abi_chunks_on_the_tensor_cores(oracle, kind, 16, 2, 128, n_tok, rows - n_tok, rows)


@pytest.mark.parametrize("sized_by", ["topk_alloc", "shorter_chunk"])
def test_chunk_captured_without_its_workspace_is_the_decode_kernels(oracle, sized_by):
    """operand images may not grow inside a capture: a chunk that was never run outside one, or only over fewer rows, is captured
    as decode launches"""
    from gpu_util import assert_close, dev_bytes
    L = lib()
    L.q4_gpu_set_stream(None)
    L.q4_hip_shutdown()                       # gives back what other tests made it reserve
    L = q4gpu.init()
    with torch.cuda.stream(torch.cuda.ExternalStream(L.q4_gpu_stream())):
        if sized_by == "topk_alloc":
            assert L.q4_hip_qsa_topk_alloc()
        n_head, n_kvh, hd, n_tok, kv_base = 24, 2, 256, 20, 300
        n, kvw = kv_base + n_tok, n_kvh * hd
        k, v = oracle.normal(95, 0, n * kvw).reshape(n, kvw), oracle.normal(95, 1, n * kvw).reshape(n, kvw)
        q, g = oracle.normal(95, 2, n_tok * n_head * hd).reshape(n_tok, n_head, hd), oracle.normal(95, 3, n_tok * n_head * hd)
        kc, vc = oracle.kv_write(k, 2), oracle.kv_write(v, 2)
        dq, dk, dv, dg = dev(q), dev_bytes(kc), dev_bytes(vc), dev(g)
        out = torch.full((n_tok, n_head, hd), float("nan"), device="cuda")
        torch.cuda.synchronize()

        def call(m, base=kv_base):
            return L.q4_hip_qsa_decode_n(dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), dg.data_ptr(), out.data_ptr(), n_head, n_kvh, hd, m, base, n, 1.0 / 16.0, 2)
        assert call(7)                        # the decode kernel, loaded outside the capture
        if sized_by == "shorter_chunk":
            assert call(n_tok, 100)
        out.fill_(float("nan"))
        assert L.q4_hip_graph_begin()
        ok = call(n_tok)
        graph = L.q4_hip_graph_end()
        assert ok and graph and L.q4_hip_graph_launch(graph)
        got = host(out)
        L.q4_hip_graph_free(graph)
    ref = oracle.attn(q, kc, vc, g, n_head, n_kvh, hd, n_tok, kv_base, n, 1.0 / 16.0, 2, threads=8)
    assert_close(got, ref, "captured chunk")
    assert L.q4_gpu_last_error() == 0


@pytest.mark.parametrize("n_head,n_kvh,n_tok,kv_base", [(16, 2, 3000, 0), (16, 2, 3000, 2100), (16, 2, 5003, 37), (16, 2, 1300, 1500), (16, 1, 4900, 300), (9, 3, 2600, 900),
                                                        (64, 4, 1205, 500)])
def test_last_wave_in_ranges_of_positions(n_head, n_kvh, n_tok, kv_base):
    """chunks of one to three waves of blocks and a remainder, over prefixes too short for the last wave to be split (it is in
    test_last_wave_split_over_positions); against chunks of 200 tokens, which are other blocks in other ranges, each within the
    tolerance of the oracle's tests.  And as many bytes again behind the output."""
    L = lib()
    hd, ctx = 128, kv_base + n_tok
    g = torch.Generator(device="cuda").manual_seed(n_tok)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    st = q4gpu.KVStore(1, n_kvh, hd, ctx, 2)
    st.append(0, rn(ctx, n_kvh * hd), rn(ctx, n_kvh * hd), 0, ctx)
    q, gate = rn(n_tok, n_head, hd).bfloat16(), rn(n_tok, n_head, hd)
    out = torch.full((2 * n_tok, n_head, hd), 7.0, dtype=torch.bfloat16, device="cuda")
    ref = torch.empty(n_tok, n_head, hd, dtype=torch.bfloat16, device="cuda")
    st.prefill(0, q, out, n_head, n_tok, kv_base, 1 / np.sqrt(hd), gate=gate)
    for t in range(0, n_tok, 200):
        m = min(200, n_tok - t)
        st.prefill(0, q[t:], ref[t:], n_head, m, kv_base + t, 1 / np.sqrt(hd), gate=gate[t:])
    got = host(out.float())
    check(got[:n_tok], host(ref.float()), "tail %d over %d" % (n_tok, kv_base))
    assert (got[n_tok:] == 7.0).all() and L.q4_gpu_last_error() == 0
    st.close()


def exact_attention(q, k, v, gate, n_head, n_kvh, kv_base, scale):
    """all tokens of a chunk, 64 bits; k and v are [row][kv head][hd]"""
    n, rows = q.shape[0], k.shape[0]
    ref = torch.empty(q.shape, dtype=torch.float64, device="cuda")
    for t in range(0, n, 1000):
        m = min(1000, n - t)
        hidden = torch.arange(rows, device="cuda")[None, :] > (kv_base + t + torch.arange(m, device="cuda"))[:, None]
        for h in range(n_head):
            s = (q[t:t + m, h].double() @ k[:, h // (n_head // n_kvh)].T * scale).masked_fill(hidden, float("-inf"))
            ref[t:t + m, h] = torch.softmax(s, -1) @ v[:, h // (n_head // n_kvh)]
    return host(ref * torch.sigmoid(gate.double()))


def rows_of(raw, n, n_kvh, hd, kind):
    """bytes in the reference's layout -> their values"""
    if kind == 2:
        b = raw.view(n, n_kvh, hd // 32, 34)
        return (b[..., 2:].contiguous().view(torch.int8).double() * b[..., :2].contiguous().view(torch.float16).double()).reshape(n, n_kvh, hd)
    return raw.view(torch.float16 if kind == 1 else torch.float32).view(n, n_kvh, hd).double()


def layout(L):
    a = (ctypes.c_uint32 * 3)()
    L.q4_gpu_prefill_layout(ctypes.byref(a, 0), ctypes.byref(a, 4), ctypes.byref(a, 8))
    return tuple(a)


on_148_sms = pytest.mark.skipif(torch.cuda.is_available() and torch.cuda.get_device_properties(0).multi_processor_count != 148,
                                reason="how a chunk is split depends on the number of SMs")


@on_148_sms
@pytest.mark.parametrize("n_head,n_kvh,n_tok,kv_base,want", [
    (16, 2, 3000, 6000, (148, 40, 3)), (64, 4, 766, 1000, (148, 44, 3)), (64, 4, 803, 2000, (148, 56, 2)), (64, 4, 1205, 3000, (296, 8, 9)),
    (16, 1, 4900, 12000, (296, 11, 12)), (9, 3, 2600, 6000, (148, 38, 3)),   # groups of tokens that do not fill their rows
    (16, 2, 1300, 4000, (148, 16, 9)),                                       # one query group per block
    (24, 8, 903, 8000, (148, 28, 5)),                                        # a last wave over the end of a kv head
    (16, 2, 3000, 2100, (188, 0, 1))])                                       # too short a prefix
def test_last_wave_split_over_positions(n_head, n_kvh, n_tok, kv_base, want):
    """the blocks of a chunk's last wave are split; all tokens against 64 bits, twice the same, and nothing is written behind the output"""
    L = lib()
    hd, ctx = 128, kv_base + n_tok
    g = torch.Generator(device="cuda").manual_seed(n_tok)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    st = q4gpu.KVStore(1, n_kvh, hd, ctx, 2)
    st.append(0, rn(ctx, n_kvh * hd), rn(ctx, n_kvh * hd), 0, ctx)
    q, gate = rn(n_tok, n_head, hd).bfloat16(), rn(n_tok, n_head, hd)
    outs = []
    for _ in range(2):
        out = torch.full((n_tok + 64, n_head, hd), 7.0, dtype=torch.bfloat16, device="cuda")
        st.prefill(0, q, out, n_head, n_tok, kv_base, 1 / np.sqrt(hd), gate=gate)
        assert layout(L) == want
        outs.append(out)
    assert torch.equal(outs[0], outs[1]) and (outs[0][n_tok:] == 7.0).all()
    raw = [torch.empty(ctx * st.token_bytes, dtype=torch.uint8, device="cuda") for _ in range(2)]
    for which in (0, 1):
        st.export(0, which, 0, ctx, raw[which])
    k, v = (rows_of(r, ctx, n_kvh, hd, 2) for r in raw)
    check(host(outs[0][:n_tok].float()), exact_attention(q, k, v, gate, n_head, n_kvh, kv_base, 1 / np.sqrt(hd)), "%d over %d" % (n_tok, kv_base))
    assert L.q4_gpu_last_error() == 0
    st.close()


@on_148_sms
@pytest.mark.parametrize("kind,n_head,hd,n_tok,kv_base,want", [
    (2, 24, 256, 800, 2048, (148, 12, 9)), (1, 24, 256, 800, 2048, (148, 12, 6)), (0, 24, 256, 1000, 4000, (148, 52, 2)),
    (2, 24, 256, 1000, 4000, (148, 52, 2)),
    (2, 16, 128, 1300, 4000, (148, 16, 9)),                                       # value and remainder
    (0, 16, 128, 1500, 4000, (148, 40, 3)), (1, 16, 128, 3000, 6000, (148, 40, 3))])   # one and two query groups per block, marks
def test_last_wave_split_over_positions_of_a_callers_cache(kind, n_head, hd, n_tok, kv_base, want):
    from gpu_util import assert_close
    L = lib()
    n_kvh, ctx = 2, kv_base + n_tok
    g = torch.Generator(device="cuda").manual_seed(n_tok + kind)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    raw = []
    for _ in range(2):
        x = rn(ctx, n_kvh * hd)
        r = torch.empty(ctx * n_kvh * {2: hd // 32 * 34, 1: hd * 2, 0: hd * 4}[kind], dtype=torch.uint8, device="cuda")
        if kind == 0:
            r.copy_(x.view(torch.uint8).view(-1))
        else:
            assert (L.q4_hip_f32_to_q8 if kind == 2 else L.q4_hip_f32_to_f16)(r.data_ptr(), x.data_ptr(), x.numel())
        raw.append(r)
    q, gate = rn(n_tok, n_head, hd), rn(n_tok, n_head, hd)
    scale = float(1 / np.sqrt(hd))
    outs = []
    for _ in range(2):
        out = torch.full((n_tok + 64, n_head, hd), 7.0, device="cuda")
        assert L.q4_hip_qsa_decode_n(q.data_ptr(), raw[0].data_ptr(), raw[1].data_ptr(), gate.data_ptr(), out.data_ptr(), n_head, n_kvh, hd, n_tok, kv_base, ctx, scale, kind)
        assert layout(L) == want
        outs.append(out)
    assert torch.equal(outs[0], outs[1]) and (outs[0][n_tok:] == 7.0).all()
    k, v = (rows_of(r, ctx, n_kvh, hd, kind) for r in raw)
    assert_close(host(outs[0][:n_tok]), exact_attention(q, k, v, gate, n_head, n_kvh, kv_base, scale), "%d over %d" % (n_tok, kv_base))
    assert L.q4_gpu_last_error() == 0


@on_148_sms
@pytest.mark.parametrize("kind,n_head,n_kvh,hd,n_tok,kv_base,blocks", [
    (2, 24, 2, 256, 241, 512, 50), (2, 24, 2, 256, 241, 511, 50),            # 25 groups of 10 tokens in two ranges: one block each
    (2, 24, 2, 256, 381, 512, 80), (2, 24, 2, 256, 381, 511, 78),            # 39 groups, the last pair's second one empty; one block each
    (2, 24, 2, 256, 250, 1000, 50), (2, 32, 2, 256, 199, 700, 50), (2, 24, 2, 256, 241, 3000, 52), (2, 32, 2, 256, 199, 2500, 52),   # pairs in ranges; 16 query heads per kv head
    (2, 16, 2, 128, 391, 1536, 50), (2, 16, 2, 128, 391, 1535, 50), (2, 16, 2, 128, 610, 1536, 80), (2, 16, 2, 128, 610, 1535, 78), (2, 16, 2, 128, 391, 2500, 52),
    (2, 16, 2, 128, 384, 5000, 48), (2, 9, 3, 128, 673, 1537, 54), (2, 1, 1, 128, 6100, 1700, 48),
    (2, 24, 2, 256, 512, 512, 104), (2, 24, 2, 256, 512, 1000, 104), (1, 24, 2, 256, 512, 4000, 104), (0, 24, 2, 256, 512, 4000, 104),   # whole: nothing to merge
    (1, 24, 2, 256, 241, 2048, 50), (1, 24, 2, 256, 241, 2047, 50), (1, 24, 2, 256, 381, 2048, 80), (1, 24, 2, 256, 381, 2047, 78),
    (0, 24, 2, 256, 250, 2100, 50), (0, 24, 2, 256, 250, 5000, 52), (0, 4, 1, 256, 1537, 2049, 49), (0, 4, 1, 256, 1601, 5000, 52),
    (2, 8, 1, 256, 770, 2048, 49), (2, 8, 1, 256, 850, 2048, 54), (2, 32, 2, 256, 290, 2048, 74),                # pairs would fill fewer places
    (-1, 16, 2, 128, 3010, 14336, 192), (-1, 16, 2, 128, 3010, 14335, 190), (-1, 32, 2, 128, 1510, 15000, 192)])   # the library's store: two groups per block
def test_pairs_of_blocks(kind, n_head, n_kvh, hd, n_tok, kv_base, blocks):
    """chunks behind a prefix on both sides of the line from which two blocks form one product: all tokens against 64 bits, twice and
    captured the same, nothing written behind the output, and the number of blocks (of a pair both count); one wave of pairs is not split"""
    from gpu_util import assert_close
    L = lib()
    ctx = kv_base + n_tok
    g = torch.Generator(device="cuda").manual_seed(n_tok + kind)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    scale = float(1 / np.sqrt(hd))
    q, gate = rn(n_tok, n_head, hd), rn(n_tok, n_head, hd)
    raw = []
    if kind < 0:
        q, dtype = q.bfloat16(), torch.bfloat16
        st = q4gpu.KVStore(1, n_kvh, hd, ctx, 2)
        st.append(0, rn(ctx, n_kvh * hd), rn(ctx, n_kvh * hd), 0, ctx)
        for which in (0, 1):
            raw.append(torch.empty(ctx * st.token_bytes, dtype=torch.uint8, device="cuda"))
            st.export(0, which, 0, ctx, raw[which])
        run = lambda out: st.prefill(0, q, out, n_head, n_tok, kv_base, scale, gate=gate)
    else:
        dtype = torch.float32
        for _ in range(2):
            x = rn(ctx, n_kvh * hd)
            r = torch.empty(ctx * n_kvh * {2: hd // 32 * 34, 1: hd * 2, 0: hd * 4}[kind], dtype=torch.uint8, device="cuda")
            if kind == 0:
                r.copy_(x.view(torch.uint8).view(-1))
            else:
                assert (L.q4_hip_f32_to_q8 if kind == 2 else L.q4_hip_f32_to_f16)(r.data_ptr(), x.data_ptr(), x.numel())
            raw.append(r)

        def run(out):
            assert L.q4_hip_qsa_decode_n(q.data_ptr(), raw[0].data_ptr(), raw[1].data_ptr(), gate.data_ptr(), out.data_ptr(), n_head, n_kvh, hd, n_tok, kv_base, ctx, scale, kind)
    outs = []
    for _ in range(2):
        out = torch.full((n_tok + 64, n_head, hd), 7.0, dtype=dtype, device="cuda")
        run(out)
        whole, late, ranges = layout(L)
        assert whole + late == blocks and (ranges == 1 or blocks != 104)
        outs.append(out)
    assert torch.equal(outs[0], outs[1]) and (outs[0][n_tok:] == 7.0).all()
    torch.cuda.synchronize()
    assert L.q4_gpu_set_stream(None) and L.q4_hip_graph_begin() == 1   # the library's own stream: the default one is not captured
    run(outs[1])
    graph = L.q4_hip_graph_end()
    outs[1].fill_(7.0)
    torch.cuda.synchronize()
    assert graph and L.q4_hip_graph_launch(graph) and L.q4_hip_stream_sync()
    assert torch.equal(outs[0], outs[1]) and layout(L)[0] + layout(L)[1] == blocks
    L.q4_hip_graph_free(graph)
    q4gpu.use_torch_stream()
    k, v = (rows_of(r, ctx, n_kvh, hd, 2 if kind < 0 else kind) for r in raw)
    ref = exact_attention(q, k, v, gate, n_head, n_kvh, kv_base, scale)
    (check if kind < 0 else assert_close)(host(outs[0][:n_tok].float()), ref, "%d over %d" % (n_tok, kv_base))
    assert L.q4_gpu_last_error() == 0
    if kind < 0:
        st.close()
