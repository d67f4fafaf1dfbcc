"""QSA indexer through the reference's entry points (q4_hip_qsa_pool / score / topk and their
device-position forms) against the oracle: pooled keys within fp32 libm tolerance (rsqrt, cos, sin
differ in the last bits between libm and the device), scores bit-exact on the same pool bytes, the
selection lists exactly equal -- including ties at the threshold, all-equal rows, the dense-prefix
case, a 65 536-block row (ctx 262 144) and several tokens per call."""
import numpy as np
import pytest
import torch

from gpu_util import dev, host, lib

pytestmark = pytest.mark.gpu

RATIO, N_ROT, BASE, EPS = 4, 64, 1e7, 1e-6


def make(oracle, seed, n_tok, n_head=4):
    raw = oracle.f32_to_f16(oracle.normal(seed, 0, n_tok * 128).reshape(n_tok, 128))
    wn = (1.0 + 0.1 * oracle.normal(seed, 1, 128)).astype(np.float32)
    return raw, wn


@pytest.mark.parametrize("n_tok", [4, 37, 4099])
def test_pool_matches_oracle(oracle, n_tok):
    L = lib()
    raw, wn = make(oracle, 50 + n_tok, n_tok)
    nb = n_tok // RATIO
    want = oracle.ix_pool(raw, wn, RATIO, 0, nb, N_ROT, BASE, EPS)
    d_raw = torch.from_numpy(raw.view(np.int16)).cuda()
    d_pool = torch.zeros(nb + 1, 128, device="cuda")
    # in two pieces, as a chunked prefill would
    mid = nb // 2
    if mid:
        assert L.q4_hip_qsa_pool(d_raw.data_ptr(), d_pool.data_ptr(), dev(wn).data_ptr(), 128, RATIO, 0, mid, N_ROT, BASE, EPS)
    assert L.q4_hip_qsa_pool(d_raw.data_ptr(), d_pool.data_ptr(), dev(wn).data_ptr(), 128, RATIO, mid, nb, N_ROT, BASE, EPS)
    got = host(d_pool)
    assert np.abs(got[:nb] - want).max() < 2e-3
    assert np.abs(got[:min(nb, 8)] - want[:min(nb, 8)]).max() < 2e-6
    assert (got[nb] == 0).all()
    # no weight: plain RMSNorm
    assert L.q4_hip_qsa_pool(d_raw.data_ptr(), d_pool.data_ptr(), None, 128, RATIO, 0, nb, N_ROT, BASE, EPS)
    assert np.abs(host(d_pool)[:nb] - oracle.ix_pool(raw, None, RATIO, 0, nb, N_ROT, BASE, EPS)).max() < 2e-3
    assert not L.q4_hip_qsa_pool(d_raw.data_ptr(), d_pool.data_ptr(), None, 64, RATIO, 0, nb, N_ROT, BASE, EPS)


def test_pool_d_completes_a_block_only_on_its_last_token(oracle):
    L = lib()
    n_tok = 23
    raw, wn = make(oracle, 61, n_tok)
    d_raw = torch.from_numpy(raw.view(np.int16)).cuda()
    d_pool = torch.zeros(n_tok // RATIO + 1, 128, device="cuda")
    want = oracle.ix_pool(raw, wn, RATIO, 0, n_tok // RATIO, N_ROT, BASE, EPS)
    for pos in range(n_tok):
        L.q4_hip_pos_push(pos)
        assert L.q4_hip_qsa_pool_d(d_raw.data_ptr(), d_pool.data_ptr(), dev(wn).data_ptr(), 128, RATIO, N_ROT, BASE, EPS)
        got = host(d_pool)
        done = (pos + 1) // RATIO
        assert np.abs(got[:done] - want[:done]).max() < 1e-5 if done else True
        assert (got[done:] == 0).all()


@pytest.mark.parametrize("n_head,n_tok,pos0", [(4, 1, 4098), (1, 1, 99), (3, 5, 700), (4, 3, 262141)])
def test_score_bit_exact_and_topk_exact(oracle, n_head, n_tok, pos0):
    """same pool bytes in, identical scores out (the dot product is one fused multiply-add per dim, in
    dim order); identical lists out"""
    L = lib()
    n_all = pos0 + n_tok
    nb = n_all // RATIO
    stride = nb + 7
    rng = np.random.default_rng(pos0)
    pool = rng.standard_normal((nb, 128)).astype(np.float32)
    q = rng.standard_normal((n_tok, n_head, 128)).astype(np.float32)
    want = oracle.ix_score(q, pool, n_tok, nb, stride, n_head, pos0, RATIO)
    d_score = torch.full((n_tok, stride), 7.0, device="cuda")
    assert L.q4_hip_qsa_score(dev(q).data_ptr(), dev(pool).data_ptr(), d_score.data_ptr(), n_tok, nb, stride, n_head, 128, pos0, RATIO)
    got = host(d_score)
    assert np.array_equal(got[:, :nb].view(np.uint32), want[:, :nb].view(np.uint32))
    assert (got[:, nb:] == 7.0).all()
    width, k_blk = 2051, 512
    d_sel = torch.zeros(n_tok, width, dtype=torch.int32, device="cuda")
    assert L.q4_hip_qsa_topk(d_score.data_ptr(), d_sel.data_ptr(), n_tok, nb, stride, k_blk, RATIO, pos0, width)
    want_sel = oracle.ix_topk(want, n_tok, stride, k_blk, RATIO, pos0, width)
    assert np.array_equal(host(d_sel), want_sel)


@pytest.mark.parametrize("n_tok,k_blk,width", [(4099, 512, 2051), (2051, 512, 2051), (2052, 512, 2051), (300, 16, 67),
                                                (70, 16, 67), (262144, 512, 2051)])
def test_topk_ties_and_degenerate_rows(oracle, n_tok, k_blk, width):
    L = lib()
    pos = n_tok - 1
    n_vis = (pos + 1) // RATIO
    stride = n_vis + 5
    rng = np.random.default_rng(n_tok)
    rows = [np.maximum(rng.standard_normal(stride), 0), np.round(np.maximum(rng.standard_normal(stride), 0) * 4) / 4,
            np.ones(stride), -np.abs(rng.standard_normal(stride)), np.where(np.arange(stride) % 3 == 0, 2.0, -1e30)]
    for i, row in enumerate(rows):
        row = row.astype(np.float32)[None, :]
        d_sel = torch.zeros(1, width, dtype=torch.int32, device="cuda")
        assert L.q4_hip_qsa_topk(dev(row).data_ptr(), d_sel.data_ptr(), 1, n_vis, stride, k_blk, RATIO, pos, width)
        want = oracle.ix_topk(row, 1, stride, k_blk, RATIO, pos, width)
        assert np.array_equal(host(d_sel), want), "row kind %d" % i


def test_device_position_forms_feed_the_sparse_decode(oracle):
    """score_d + topk_d at the position word == the host-position forms; the list is a valid input of the
    decode kernel (all entries <= pos or -1, no duplicates)"""
    L = lib()
    pos, n_head = 9001, 4
    nb = (pos + 1) // RATIO
    max_blocks = 4096
    rng = np.random.default_rng(7)
    pool = rng.standard_normal((max_blocks, 128)).astype(np.float32)
    q = rng.standard_normal((1, n_head, 128)).astype(np.float32)
    d_pool, d_q = dev(pool), dev(q)
    a_score, b_score = torch.zeros(1, max_blocks, device="cuda"), torch.zeros(1, max_blocks, device="cuda")
    a_sel = torch.zeros(2051, dtype=torch.int32, device="cuda")
    b_sel = torch.zeros_like(a_sel)
    assert L.q4_hip_qsa_score(d_q.data_ptr(), d_pool.data_ptr(), a_score.data_ptr(), 1, nb, max_blocks, n_head, 128, pos, RATIO)
    assert L.q4_hip_qsa_topk(a_score.data_ptr(), a_sel.data_ptr(), 1, nb, max_blocks, 512, RATIO, pos, 2051)
    L.q4_hip_pos_push(pos)
    assert L.q4_hip_qsa_score_d(d_q.data_ptr(), d_pool.data_ptr(), b_score.data_ptr(), max_blocks, n_head, 128, RATIO)
    assert L.q4_hip_qsa_topk_d(b_score.data_ptr(), b_sel.data_ptr(), max_blocks, 512, RATIO, 2051)
    assert np.array_equal(host(a_score)[0, :nb], host(b_score)[0, :nb])
    sel = host(b_sel)
    assert np.array_equal(sel, host(a_sel))
    live = sel[sel >= 0]
    assert live.max() <= pos and len(np.unique(live)) == len(live) == 2048 + (pos + 1) % RATIO
    assert L.q4_gpu_last_error() == 0


def test_batched_sessions_select_like_single_sessions(oracle):
    """q4_gpu_qsa_select_batch: every session has its own pool and position; scores bit-equal and lists
    equal to the oracle's per-session result (short rows, the dense-prefix case and a long row together)"""
    L = lib()
    n_head, width, k_blk = 4, 2051, 512
    positions = [4098, 99, 70001, 2050, 20000]          # 99 and 2050: every block fits (dense prefix)
    stride = max(p + 1 for p in positions) // RATIO + 3
    rng = np.random.default_rng(77)
    pools, d_pools, want_sc, want_sel = [], [], [], []
    q = rng.standard_normal((len(positions), n_head, 128)).astype(np.float32)
    for s_i, pos in enumerate(positions):
        nb = (pos + 1) // RATIO
        pool = rng.standard_normal((max(nb, 1), 128)).astype(np.float32)
        d_pools.append(dev(pool))
        sc = oracle.ix_score(q[s_i:s_i + 1], pool, 1, nb, stride, n_head, pos, RATIO)
        want_sc.append(sc)
        want_sel.append(oracle.ix_topk(sc, 1, stride, k_blk, RATIO, pos, width))
    ptrs = torch.tensor([t.data_ptr() for t in d_pools], dtype=torch.int64, device="cuda")
    d_pos = torch.tensor(positions, dtype=torch.int32, device="cuda")
    d_score = torch.zeros(len(positions), stride, device="cuda")
    d_sel = torch.zeros(len(positions), width, dtype=torch.int32, device="cuda")
    assert L.q4_gpu_qsa_select_batch(ptrs.data_ptr(), d_pos.data_ptr(), dev(q).data_ptr(), d_score.data_ptr(),
                                     d_sel.data_ptr(), len(positions), stride, n_head, 128, k_blk, RATIO, width)
    got_sc, got_sel = host(d_score), host(d_sel)
    for s_i, pos in enumerate(positions):
        nb = (pos + 1) // RATIO
        assert np.array_equal(got_sc[s_i, :nb].view(np.uint32), want_sc[s_i][0, :nb].view(np.uint32)), s_i
        assert np.array_equal(got_sel[s_i], want_sel[s_i][0]), s_i
    assert not L.q4_gpu_qsa_select_batch(None, d_pos.data_ptr(), dev(q).data_ptr(), d_score.data_ptr(), d_sel.data_ptr(),
                                         len(positions), stride, n_head, 128, k_blk, RATIO, width)
    L.q4_gpu_last_error()


def test_argument_checks():
    L = lib()
    z = torch.zeros(256, device="cuda")
    s = torch.zeros(64, dtype=torch.int32, device="cuda")
    assert not L.q4_hip_qsa_score(z.data_ptr(), z.data_ptr(), z.data_ptr(), 1, 1, 1, 5, 128, 3, 4)     # > 4 heads
    assert not L.q4_hip_qsa_score(z.data_ptr(), z.data_ptr(), z.data_ptr(), 1, 1, 1, 4, 64, 3, 4)      # hd != 128
    assert not L.q4_hip_qsa_topk(z.data_ptr(), s.data_ptr(), 1, 1, 1, 513, 4, 3, 64)                   # k_blk > 512
    assert not L.q4_hip_qsa_topk(None, s.data_ptr(), 1, 1, 1, 16, 4, 3, 64)


@pytest.mark.parametrize("n_head,n_tok,pos0,ratio", [(4, 33, 20000, 4), (3, 32, 40001, 4), (1, 97, 4003, 4), (4, 160, 2100, 4),
                                                     (2, 65, 2300, 1), (4, 16, 20, 4)])
def test_score_of_many_tokens_bit_exact(oracle, n_head, n_tok, pos0, ratio):
    """the tiled form (the last case: the scan): edges of its 32-token x 128-block tiles, fewer heads than four, blocks that
    only some of a tile's tokens see; nothing is written behind n_blocks, and nothing is read behind the blocks that
    the last token sees (NaN there)"""
    L = lib()
    nb = (pos0 + n_tok) // ratio
    n_blocks, stride = nb + 3, nb + 9
    rng = np.random.default_rng(n_tok * 1000 + pos0)
    pool = np.full((n_blocks, 128), np.nan, np.float32)
    pool[:nb] = rng.standard_normal((nb, 128)).astype(np.float32)
    q = rng.standard_normal((n_tok, n_head, 128)).astype(np.float32)
    want = oracle.ix_score(q, np.nan_to_num(pool), n_tok, n_blocks, stride, n_head, pos0, ratio)
    d_score = torch.full((n_tok, stride), 7.0, device="cuda")
    assert L.q4_hip_qsa_score(dev(q).data_ptr(), dev(pool).data_ptr(), d_score.data_ptr(), n_tok, n_blocks, stride, n_head, 128, pos0, ratio)
    got = host(d_score)
    assert np.array_equal(got[:, :n_blocks].view(np.uint32), want[:, :n_blocks].view(np.uint32))
    assert (got[:, n_blocks:] == 7.0).all()


@pytest.mark.parametrize("n_tok,n_vis,k_blk", [(3, 8192, 512), (1, 8193, 512), (2, 16389, 512), (1, 32773, 100), (160, 8200, 512),
                                               (80, 16390, 512), (40, 40000, 1)])
def test_topk_forms_and_their_edges(oracle, n_tok, n_vis, k_blk):
    """one block, clusters of 2 / 4 / 8, and the streaming form of many tokens (more clusters than fit at once), each on
    rows whose threshold bin is small, holds thousands of keys, and is all ties"""
    L = lib()
    ratio, width = 4, 4 * k_blk + 3
    pos0 = n_vis * ratio - n_tok
    stride = n_vis + 5
    rng = np.random.default_rng(n_vis + n_tok)
    rows = np.maximum(rng.standard_normal((n_tok, stride)), 0).astype(np.float32)
    rows[::3] = np.float32(1.0) + rng.integers(0, 1 << 14, rows[::3].shape).astype(np.float32) / (1 << 20)   # one 12-bit digit for all
    rows[2::3] = np.round(rows[2::3] * 4) / 4
    d_sel = torch.zeros(n_tok, width, dtype=torch.int32, device="cuda")
    assert L.q4_hip_qsa_topk(dev(rows).data_ptr(), d_sel.data_ptr(), n_tok, n_vis, stride, k_blk, ratio, pos0, width)
    want = oracle.ix_topk(rows, n_tok, stride, k_blk, ratio, pos0, width)
    assert np.array_equal(host(d_sel), want)


def test_batched_scores_of_many_uneven_sessions(oracle):
    """the sessions' tiles are shared equally among the blocks: 70 sessions (more than one warp's worth), some without a
    visible block, some of one row, one much longer than the others"""
    L = lib()
    n_head, ratio = 4, RATIO
    rng = np.random.default_rng(70)
    positions = [int(x) for x in rng.integers(0, 700, 70)]
    positions[0], positions[3], positions[33], positions[69], positions[40] = 0, 2, 3, 4099, 60003
    stride = max(positions) // ratio + 2
    q = rng.standard_normal((70, n_head, 128)).astype(np.float32)
    pools = [rng.standard_normal(((p + 1) // ratio + 1, 128)).astype(np.float32) for p in positions]
    d_pools = [dev(p) for p in pools]
    ptrs = torch.tensor([t.data_ptr() for t in d_pools], dtype=torch.int64, device="cuda")
    d_pos = torch.tensor(positions, dtype=torch.int32, device="cuda")
    d_score = torch.full((70, stride), 7.0, device="cuda")
    d_sel = torch.zeros(70, 67, dtype=torch.int32, device="cuda")
    assert L.q4_gpu_qsa_select_batch(ptrs.data_ptr(), d_pos.data_ptr(), dev(q).data_ptr(), d_score.data_ptr(), d_sel.data_ptr(), 70, stride,
                                     n_head, 128, 16, ratio, 67)
    got, sel = host(d_score), host(d_sel)
    for t, pos in enumerate(positions):
        nb = (pos + 1) // ratio
        want = oracle.ix_score(q[t:t + 1], pools[t], 1, nb, stride, n_head, pos, ratio) if nb else np.zeros((1, stride), np.float32)
        assert np.array_equal(got[t, :nb].view(np.uint32), want[0, :nb].view(np.uint32)), t
        assert (got[t, nb:] == 7.0).all(), t
        assert np.array_equal(sel[t], oracle.ix_topk(want, 1, stride, 16, ratio, pos, 67)[0]), t


@pytest.mark.parametrize("n_vis,slack", [(700, 2000), (8192, 1), (9000, 7000), (20000, 9000), (33000, 30000)])
@pytest.mark.parametrize("form", ["host", "host_3", "word", "word_settled"])
def test_topk_reads_visible_scores_only(oracle, n_vis, slack, form):
    """rows reach to `stride`, but of the last one only the visible scores exist: it ends with its allocation, as a host may lay
    it out that has sized its buffer for the blocks it has"""
    L = lib()
    n_tok = 3 if form == "host_3" else 1
    stride, pos0 = n_vis + slack, n_vis * RATIO
    n = (n_tok - 1) * stride + n_vis
    size = (4 * n + (2 << 20) - 1) // (2 << 20) * (2 << 20)          # whole pages of the device's memory
    base = L.q4_hip_malloc(size)
    score = base + size - 4 * n
    rng = np.random.default_rng(n_vis)
    rows = np.zeros((n_tok, stride), np.float32)
    rows[:, :n_vis] = np.maximum(rng.standard_normal((n_tok, n_vis)), 0)
    flat = np.ascontiguousarray(rows.reshape(-1)[:n])
    assert L.q4_hip_h2d(score, flat.ctypes.data, 4 * n)
    d_sel = torch.zeros(n_tok, 2051, dtype=torch.int32, device="cuda")
    if form.startswith("word"):
        L.q4_hip_pos_push(pos0)
        if form == "word_settled":
            d_copy = torch.empty(256, device="cuda")
            assert L.q4_hip_fill(d_copy.data_ptr(), 0.0, 256)
            assert L.q4_hip_qsa_topk_d(score, d_sel.data_ptr(), stride, 512, RATIO, 2051)
        assert L.q4_hip_qsa_topk_d(score, d_sel.data_ptr(), stride, 512, RATIO, 2051)
    else:
        assert L.q4_hip_qsa_topk(score, d_sel.data_ptr(), n_tok, n_vis, stride, 512, RATIO, pos0, 2051)
    want = oracle.ix_topk(rows, n_tok, stride, 512, RATIO, pos0, 2051)
    assert np.array_equal(host(d_sel), want)
    L.q4_hip_free(base)


@pytest.mark.parametrize("n_sess,positions", [(6, [4031 * 4 + 2, 3, 2, 255, 256, 4032 * 4 + 1]), (7, [4031 * 4 + 2, 3, 2, 255, 256, 4032 * 4 + 1, 700]),
                                              (1, [63]), (2, [64 * 4 - 1, 64 * 4 + 3])])
def test_batched_scores_with_and_without_a_block_for_every_two_tiles(oracle, n_sess, positions):
    """both sides of the line between a grid that gives every session its own blocks and one that shares all tiles out
    (6 sessions of 64 block pairs fit 444 blocks, 7 do not)"""
    L = lib()
    rng = np.random.default_rng(n_sess)
    stride = 4033 if n_sess > 2 else 65
    q = rng.standard_normal((n_sess, 4, 128)).astype(np.float32)
    pools = [rng.standard_normal((max((p + 1) // RATIO, 1), 128)).astype(np.float32) for p in positions]
    d_pools = [dev(p) for p in pools]
    ptrs = torch.tensor([t.data_ptr() for t in d_pools], dtype=torch.int64, device="cuda")
    d_pos = torch.tensor(positions, dtype=torch.int32, device="cuda")
    d_score = torch.full((n_sess, stride), 7.0, device="cuda")
    d_sel = torch.zeros(n_sess, 67, dtype=torch.int32, device="cuda")
    assert L.q4_gpu_qsa_select_batch(ptrs.data_ptr(), d_pos.data_ptr(), dev(q).data_ptr(), d_score.data_ptr(), d_sel.data_ptr(), n_sess, stride,
                                     4, 128, 16, RATIO, 67)
    got, sel = host(d_score), host(d_sel)
    for t, pos in enumerate(positions):
        nb = (pos + 1) // RATIO
        want = oracle.ix_score(q[t:t + 1], pools[t], 1, nb, stride, 4, pos, RATIO) if nb else np.zeros((1, stride), np.float32)
        assert np.array_equal(got[t, :nb].view(np.uint32), want[0, :nb].view(np.uint32)), t
        assert (got[t, nb:] == 7.0).all(), t
        assert np.array_equal(sel[t], oracle.ix_topk(want, 1, stride, 16, RATIO, pos, 67)[0]), t


@pytest.mark.parametrize("n_tok,blocks", [(4, 32768), (5, 65536), (8, 65536), (12, 8192), (12, 16384), (16, 8192)])
def test_scores_of_a_few_tokens_on_both_sides_of_the_product(n_tok, blocks):
    """whichever form the estimate picks, every token's row has the bits of a call of its own"""
    L = lib()
    g = torch.Generator(device="cuda").manual_seed(blocks + n_tok)
    pool = torch.randn(blocks, 128, device="cuda", generator=g)
    q = torch.randn(n_tok, 4, 128, device="cuda", generator=g)
    pos0 = blocks * RATIO - n_tok
    a, b = torch.zeros(n_tok, blocks, device="cuda"), torch.zeros(n_tok, blocks, device="cuda")
    assert L.q4_hip_qsa_score(q.data_ptr(), pool.data_ptr(), a.data_ptr(), n_tok, blocks, blocks, 4, 128, pos0, RATIO)
    for t in range(n_tok):
        assert L.q4_hip_qsa_score(q[t].data_ptr(), pool.data_ptr(), b[t].data_ptr(), 1, blocks, blocks, 4, 128, pos0 + t, RATIO)
    assert torch.equal(a.view(torch.int32), b.view(torch.int32))


@pytest.mark.parametrize("n_tok,n_head,blocks,slack", [(33, 4, 16389, 3), (40, 4, 16389, 0), (33, 3, 8193, 7), (64, 4, 4095, 1), (47, 2, 4098, 2), (130, 4, 16450, 2)])
def test_product_tiles_have_the_bits_of_the_scan(n_tok, n_head, blocks, slack):
    """wide (64 M = 256) and narrow (128) tiles: last columns of one to four blocks, rows that are stored 16 bytes at a time (stride
    a multiple of 4) and not, fewer heads than four, infinities, NaN, subnormals and negative zeros in the pool"""
    L = lib()
    g = torch.Generator(device="cuda").manual_seed(blocks + n_tok)
    pool = torch.randn(blocks, 128, device="cuda", generator=g)
    flat = pool.view(-1)
    for i, x in enumerate((float("inf"), float("-inf"), float("nan"), 1e-41, -0.0, 3e38)):
        flat[torch.randint(0, flat.numel(), (50,), device="cuda", generator=g)] = x
    pool[-1, 127] = float("inf")
    q = torch.randn(n_tok, n_head, 128, device="cuda", generator=g)
    q[1, 0, 5] = 0.0
    q[2, 0] = 1e-30
    pos0, stride = blocks * RATIO - n_tok, blocks + slack
    a, b = torch.full((n_tok, stride), 7.0, device="cuda"), torch.full((n_tok, stride), 7.0, device="cuda")
    assert L.q4_hip_qsa_score(q.data_ptr(), pool.data_ptr(), a.data_ptr(), n_tok, blocks, stride, n_head, 128, pos0, RATIO)
    for t in range(n_tok):
        assert L.q4_hip_qsa_score(q[t].data_ptr(), pool.data_ptr(), b[t].data_ptr(), 1, blocks, stride, n_head, 128, pos0 + t, RATIO)
    assert torch.equal(a.view(torch.int32), b.view(torch.int32))


@pytest.mark.parametrize("n_vis,stride,k_blk", [(16385, 16387, 512), (20000, 20000, 512), (32768, 32768, 512), (33001, 33004, 7), (65536, 65536, 512)])
def test_sampled_selection_of_many_tokens(oracle, n_vis, stride, k_blk):
    """rows long enough for a sample: ordinary ones, rows whose largest keys are exactly the sampled ones (the pivot is too
    high), rows whose sampled keys are the smallest, rows of ties and of zeros, large keys in one run, infinities; a row start
    on every 4-byte boundary"""
    L = lib()
    n_tok = 160
    rng = np.random.default_rng(n_vis)
    step = n_vis // 2048
    i = np.arange((n_vis + step - 1) // step, dtype=np.uint64)
    at = np.minimum(i * step + ((i * 0x9E3779B1 % 2**32) >> 16) % step, n_vis - 1)
    sc = np.zeros((n_tok, stride), np.float32)
    sc[:] = np.abs(rng.standard_normal((n_tok, stride))).astype(np.float32)
    sc[1::8, at] += 100
    sc[2::8, at] = 0
    sc[3::8] = np.round(sc[3::8] * 2)
    sc[4::8, 100:2000] += 7
    sc[5::8] = 50 + sc[5::8] * 1e-4
    sc[6::8, rng.integers(0, n_vis, 300)] = np.inf
    sc[7::8] = 0
    sc[15::16] = -1
    pos0, width = n_vis * RATIO - n_tok, k_blk * RATIO + 3
    d = torch.from_numpy(sc).cuda()
    d_sel = torch.full((n_tok, width), -7, dtype=torch.int32, device="cuda")
    assert L.q4_hip_qsa_topk(d.data_ptr(), d_sel.data_ptr(), n_tok, n_vis, stride, k_blk, RATIO, pos0, width)
    got = host(d_sel)
    for t in list(range(16)) + [n_tok - 1]:
        assert np.array_equal(got[t], oracle.ix_topk(sc[t:t + 1], 1, stride, k_blk, RATIO, pos0 + t, width)[0]), t


@pytest.mark.parametrize("per,more", [(0, 1), (0, 33), (1, 0), (32, -1), (32, 1), (128, 0), (128, 1), (224, 1), (448, 0), (448, 1)])
@pytest.mark.parametrize("n_head", [4, 3])
def test_scores_of_one_token_at_the_edges_of_a_blocks_share(oracle, per, more, n_head):
    """a block's share of the rows around one warp's, the line between one and two rows per lane, the last row that fits, and one
    more; host position with hidden blocks behind, and the position word over a longer pool; NaN behind the visible rows"""
    L = lib()
    rows = per * torch.cuda.get_device_properties(0).multi_processor_count + more
    rng = np.random.default_rng(rows)
    pool = np.full((rows + 5, 128), np.nan, np.float32)
    pool[:rows] = rng.standard_normal((rows, 128)).astype(np.float32)
    q = rng.standard_normal((1, n_head, 128)).astype(np.float32)
    pos = rows * RATIO + 2
    want = oracle.ix_score(q, np.nan_to_num(pool), 1, rows + 3, rows + 5, n_head, pos, RATIO)[0]
    d_q, d_pool = dev(q), dev(pool)
    a, b = torch.full((rows + 5,), 7.0, device="cuda"), torch.full((rows + 5,), 7.0, device="cuda")
    assert L.q4_hip_qsa_score(d_q.data_ptr(), d_pool.data_ptr(), a.data_ptr(), 1, rows + 3, rows + 5, n_head, 128, pos, RATIO)
    L.q4_hip_pos_push(pos)
    assert L.q4_hip_qsa_score_d(d_q.data_ptr(), d_pool.data_ptr(), b.data_ptr(), rows + 5, n_head, 128, RATIO)
    a, b = host(a), host(b)
    assert np.array_equal(a[:rows + 3].view(np.uint32), want[:rows + 3].view(np.uint32)) and (a[rows + 3:] == 7.0).all()
    assert np.array_equal(b[:rows].view(np.uint32), want[:rows].view(np.uint32)) and (b[rows:] == 7.0).all()


@pytest.mark.parametrize("n_tok,n_vis", [(3, 700), (3, 8192), (1, 9000), (2, 20000), (1, 40000), (1, 66000), (160, 8200), (160, 20000), (160, 33000), (300, 65536)])
def test_scores_that_are_not_numbers_are_ordered_by_their_bits(oracle, n_tok, n_vis):
    """every form: NaN above all numbers, NaN with a sign below them, infinities and zeros of both signs"""
    L = lib()
    rng = np.random.default_rng(n_vis)
    k_blk = 512 if n_vis > 4000 else 64
    sc = rng.standard_normal((n_tok, n_vis)).astype(np.float32)
    for t in range(n_tok):
        some, n = rng.permutation(n_vis), n_vis // 60 if n_vis < 16000 else 300
        sc[t, some[:n]] = np.nan
        sc[t, some[n:2 * n]] = -np.float32(np.nan)
        sc[t, some[2 * n:2 * n + 5]] = np.inf
        sc[t, some[2 * n + 5:3 * n]] = -np.inf
        sc[t, some[3 * n:5 * n]] = 0.0
        sc[t, some[5 * n:6 * n]] = -0.0
        if t % 3 == 2:
            sc[t] = np.minimum(sc[t], 0.0)   # keeps NaN
    pos0, width = n_vis * RATIO - n_tok, k_blk * RATIO + 3
    d = torch.from_numpy(sc).cuda()
    d_sel = torch.full((n_tok, width), -7, dtype=torch.int32, device="cuda")
    assert L.q4_hip_qsa_topk(d.data_ptr(), d_sel.data_ptr(), n_tok, n_vis, n_vis, k_blk, RATIO, pos0, width)
    got = host(d_sel)
    for t in list(range(min(n_tok, 6))) + [n_tok - 1]:
        assert np.array_equal(got[t], oracle.ix_topk(sc[t:t + 1], 1, n_vis, k_blk, RATIO, pos0 + t, width)[0]), t


@pytest.mark.parametrize("n_tok,n_vis", [(149, 24576), (149, 24577), (148, 40001), (300, 40001)])
def test_selection_where_many_keys_share_leading_bits(oracle, n_tok, n_vis):
    """on both sides of the sampled form's rule: rows whose threshold lies in the pivot's bin of 256 keys, whose last 8 bits then
    decide; exactly as many keys above the bin as are needed, one fewer, as many as there is room for, one more; a bin with too
    few keys behind it; NaN of both signs"""
    L = lib()
    k_blk, stride = 512, n_vis + 3
    rng = np.random.default_rng(n_vis + n_tok)
    step = n_vis // 2048
    i = np.arange(200, dtype=np.uint64)
    at = np.minimum(i * step + ((i * 0x9E3779B1 % 2**32) >> 16) % step, n_vis - 1)
    sc = np.zeros((n_tok, stride), np.float32)

    def near(x, n):   # one value's leading 24 bits, any last 8
        return (np.full(n, x, np.float32).view(np.uint32) & ~np.uint32(255) | rng.integers(0, 256, n, dtype=np.uint32)).view(np.float32)
    for t in range(n_tok):
        kind, some = t % 10, rng.permutation(n_vis)
        sc[t] = near(1.0, stride) if kind in (0, 1, 2) else 0.0
        if kind in (1, 2, 3, 4, 5, 6):
            above = {1: 511, 2: 512, 3: 511, 4: 512, 5: 2048, 6: 2049}[kind]
            sc[t, some[:above]] = 3 + rng.random(above)
        if kind == 7:
            sc[t] = np.abs(rng.standard_normal(stride)) * 0.1
            sc[t, at] = near(9.0, 200)
        if kind == 8:
            sc[t, some[:300]] = np.nan
            sc[t, some[300:600]] = -np.float32(np.nan)
            sc[t, some[600:2000]] = -0.0
        if kind == 9:
            sc[t] = near(-2.0, stride)
    pos0, width = n_vis * RATIO - n_tok, k_blk * RATIO + 3
    d = torch.from_numpy(sc).cuda()
    d_sel = torch.full((n_tok, width), -7, dtype=torch.int32, device="cuda")
    assert L.q4_hip_qsa_topk(d.data_ptr(), d_sel.data_ptr(), n_tok, n_vis, stride, k_blk, RATIO, pos0, width)
    got = host(d_sel)
    for t in list(range(10)) + [n_tok - 1]:
        assert np.array_equal(got[t], oracle.ix_topk(sc[t:t + 1], 1, stride, k_blk, RATIO, pos0 + t, width)[0]), t


@pytest.mark.parametrize("n_vis", [513, 1025, 2049, 8192, 8193, 16500, 40000, 65536])
def test_selection_from_the_threads_maxima(oracle, n_vis):
    """one block and clusters of 2, 4 and 8; rows whose pivot is negative, whose highest keys are a few threads' or one run, reach
    beyond the bins behind the pivot, share 24 bits with the threshold, are two values, or mostly NaN with a sign (a pivot of 0)"""
    L = lib()
    k_blk, kinds = 512, 10
    rng = np.random.default_rng(n_vis)
    sc = np.abs(rng.standard_normal((kinds, n_vis))).astype(np.float32)
    i = np.arange(n_vis)
    sc[1] = -1 - sc[1]
    sc[2] = np.exp(6 * rng.standard_normal(n_vis))
    sc[3, i % 1024 < 40] += 100
    sc[4, n_vis // 3:n_vis // 3 + 700] += 6
    some = rng.permutation(n_vis)
    sc[5], sc[5, some[:511]] = 0.25, 2 + rng.random(511)   # one short of ties
    sc[6, some[:480]] = 7 + rng.random(480)                 # the threshold among 40, then among 60 keys of the same 24 bits
    near = np.full(100, 5.0, np.float32).view(np.uint32) + rng.integers(0, 256, 100, dtype=np.uint32)
    sc[6, some[480:][:40]] = near.view(np.float32)[:len(some[480:][:40])]
    sc[7] = sc[6]
    sc[7, some[480:][:60]] = near.view(np.float32)[40:40 + len(some[480:][:60])]
    sc[8] = np.where(rng.random(n_vis) < 0.5, np.float32(-0.0), np.float32(0.0))
    sc[9, some[400:]] = (0xffffffff - rng.integers(0, 1 << 19, n_vis - 400, dtype=np.uint32)).view(np.float32)
    pos0, width = n_vis * RATIO - kinds, k_blk * RATIO + 3
    got = np.zeros((kinds, width), np.int32)
    for t in range(kinds):
        d, d_sel = torch.from_numpy(sc[t]).cuda(), torch.full((width,), -7, dtype=torch.int32, device="cuda")
        assert L.q4_hip_qsa_topk(d.data_ptr(), d_sel.data_ptr(), 1, n_vis, n_vis, k_blk, RATIO, pos0 + t, width)
        got[t] = host(d_sel)
        assert np.array_equal(got[t], oracle.ix_topk(sc[t:t + 1], 1, n_vis, k_blk, RATIO, pos0 + t, width)[0]), t
    d, d_sel = torch.from_numpy(sc).cuda(), torch.full((kinds, width), -7, dtype=torch.int32, device="cuda")
    assert L.q4_hip_qsa_topk(d.data_ptr(), d_sel.data_ptr(), kinds, n_vis, n_vis, k_blk, RATIO, pos0, width)
    assert np.array_equal(host(d_sel), got)


@pytest.mark.parametrize("n_vis", [600, 2100, 8192, 8193, 12000, 24576, 40000, 65536])
def test_selection_where_the_pivot_has_no_room(oracle, n_vis):
    """more keys reach the pivot than a block collects: ties at it with enough keys above it, one too few, or none; keys that share
    12, 24 or all bits with it; keys of a few threads far above it; the least and the largest key there is"""
    L = lib()
    k_blk = 512
    rng = np.random.default_rng(n_vis)
    i, some, x = np.arange(n_vis), rng.permutation(n_vis), rng.standard_normal(n_vis).astype(np.float32)

    def over_zeros(n):
        row = np.zeros(n_vis, np.float32)
        row[some[:n]] = 2 + rng.random(min(n, n_vis))
        return row

    def near(v):   # one value's leading 24 bits, any last 8
        return (v.astype(np.float32).view(np.uint32) & ~np.uint32(255) | rng.integers(0, 256, n_vis, dtype=np.uint32)).view(np.float32)
    rows = [over_zeros(n) for n in (511, 512, 513, 560, 1500)]
    rows += [np.round(x * q) / q for q in (1, 4, 16)]
    rows += [1000 + x / 2, -1000 - np.abs(x), near(np.ones(n_vis)), near(np.where(some % 3 == 0, 1.0, 1.0001)), near(-np.ones(n_vis))]
    rows += [np.where(x > c, 1.0, 0.0) for c in (1.0, 2.5)] + [np.where(x > 1, -1.0, -2.0)]
    rows += [np.where(i % 1024 < c, 100 + np.abs(x), np.abs(x)) for c in (70, 300)] + [np.where(i % 1024 < 300, 100 + x / 64, np.abs(x))]
    rows += [np.full(n_vis, v, np.uint32).view(np.float32) for v in (0xffffffff, 0x7fffffff)]
    rows += [np.where(x > c, np.float32(np.inf), x) for c in (0.0, 2.0)]
    tiny = over_zeros(300)
    tiny[some[300:]] = np.full(n_vis - 300 if n_vis > 300 else 0, 0xffffffff, np.uint32).view(np.float32)
    sc = np.stack([r.astype(np.float32) for r in rows] + [tiny])
    kinds, width = len(sc), k_blk * RATIO + 3
    pos0 = n_vis * RATIO - kinds
    got = np.zeros((kinds, width), np.int32)
    for t in range(kinds):
        d, d_sel = torch.from_numpy(sc[t]).cuda(), torch.full((width,), -7, dtype=torch.int32, device="cuda")
        assert L.q4_hip_qsa_topk(d.data_ptr(), d_sel.data_ptr(), 1, n_vis, n_vis, k_blk, RATIO, pos0 + t, width)
        got[t] = host(d_sel)
        assert np.array_equal(got[t], oracle.ix_topk(sc[t:t + 1], 1, n_vis, k_blk, RATIO, pos0 + t, width)[0]), t
    d, d_sel = torch.from_numpy(sc).cuda(), torch.full((kinds, width), -7, dtype=torch.int32, device="cuda")
    assert L.q4_hip_qsa_topk(d.data_ptr(), d_sel.data_ptr(), kinds, n_vis, n_vis, k_blk, RATIO, pos0, width)
    assert np.array_equal(host(d_sel), got)


@pytest.mark.parametrize("n_head", [1, 2, 3, 4])
def test_batched_scores_in_equal_shares(oracle, n_head):
    """sessions whose rows begin and end inside a warp's share, which is many tiles here (8 warps on each SM): tiles of 1 to 64 rows on
    both sides of 32, empty sessions between long ones; and shares of a few rows, of none"""
    L = lib()
    rng = np.random.default_rng(n_head)
    for blocks in ([40001, 0, 1, 33, 0, 65000, 64, 20007, 0, 31, 50003], [700, 0, 33, 1]):
        n, stride = len(blocks), 65001 if blocks[0] > 700 else 33000
        positions = [max(b * RATIO - 1 + i % 2 * 3, 0) for i, b in enumerate(blocks)]
        q = rng.standard_normal((n, n_head, 128)).astype(np.float32)
        pools = [rng.standard_normal((max(b, 1) + 1, 128)).astype(np.float32) for b in blocks]
        d_pools = [dev(p) for p in pools]
        ptrs = torch.tensor([t.data_ptr() for t in d_pools], dtype=torch.int64, device="cuda")
        d_pos = torch.tensor(positions, dtype=torch.int32, device="cuda")
        d_score = torch.full((n, stride), 7.0, device="cuda")
        d_sel = torch.zeros(n, 67, dtype=torch.int32, device="cuda")
        assert L.q4_gpu_qsa_select_batch(ptrs.data_ptr(), d_pos.data_ptr(), dev(q).data_ptr(), d_score.data_ptr(), d_sel.data_ptr(), n, stride, n_head,
                                         128, 16, RATIO, 67)
        got, sel = host(d_score), host(d_sel)
        for t, pos in enumerate(positions):
            nb = (pos + 1) // RATIO
            want = oracle.ix_score(q[t:t + 1], pools[t], 1, nb, stride, n_head, pos, RATIO) if nb else np.zeros((1, stride), np.float32)
            assert np.array_equal(got[t, :nb].view(np.uint32), want[0, :nb].view(np.uint32)), t
            assert (got[t, nb:] == 7.0).all(), t
            assert np.array_equal(sel[t], oracle.ix_topk(want, 1, stride, 16, RATIO, pos, 67)[0]), t
