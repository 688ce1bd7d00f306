"""The decode step where its launches differ: score rows at most top_k long (nothing to score), batches in which only some
sequences need a score, no sequence of 128 rows, and the selection's lone CTA at its edges; rows, pools and counts bit for
bit against the oracle, and the error word of each path."""
import numpy as np
import pytest
import torch

from oracle.workload import State, attend_close_ref, make_geom

pytestmark = pytest.mark.gpu


def dev(a):
    a = np.ascontiguousarray(a)
    if a.dtype in (np.uint16, np.uint32):
        a = a.view(np.int16 if a.dtype == np.uint16 else np.int32)
    return torch.from_numpy(a).cuda()


def _layer(st, fill=None):
    from rivoli_b200 import backend as be
    from rivoli_b200.layer import DsaDecodeLayer
    be.lib()
    g = make_geom(be.DsaGeom, **st.geom_kw)
    L = DsaDecodeLayer(g, st.B, max_ctx=int(st.seq_len.max()))
    for name in ("latent_pool", "latent_scale", "index_pool", "index_scale", "block_table"):
        getattr(L, name).copy_(dev(getattr(st, name)).view(getattr(L, name).shape))
    return be, g, L


def _step(L, st, **kw):
    return L.step(dev(st.new_latent), dev(st.new_key), dev(st.index_q), dev(st.index_w), dev(st.q), dev(st.row_pos), dev(st.seq_len), **kw)


CASES = {
    # all selected: below, at and (last) above top_k, with sequences of one row and of a page edge
    "all-below": dict(ctx_lens=[100, 255, 1, 64, 65], top_k=256),
    "all-at": dict(ctx_lens=[256, 130, 127, 128], top_k=256),
    "one-above": dict(ctx_lens=[257, 256, 1, 255], top_k=256),
    "below-wide-append": dict(ctx_lens=[40, 200], top_k=256, index_dim=512, kv_lora=512, rope_dim=128),
    "below-other-geometry": dict(ctx_lens=[40, 200, 33], top_k=256, index_dim=64, index_heads=8, kv_lora=256),
    "above-other-geometry": dict(ctx_lens=[400, 20, 333], top_k=256, index_dim=64, index_heads=8, kv_lora=256),
    # only the CUDA-core attention is launched
    "short": dict(ctx_lens=[127, 1, 64], top_k=2048),
    "short-top-k": dict(ctx_lens=[900, 127, 128], top_k=127),
    "not-short": dict(ctx_lens=[128, 1, 64], top_k=2048),
    # the selection's lone CTA and the first cluster
    "lone-cta": dict(ctx_lens=[8192, 300], top_k=300),
    "cluster": dict(ctx_lens=[8193, 301], top_k=300),
}


@pytest.mark.parametrize("name", list(CASES))
def test_step_matches_the_oracle(name):
    kw = dict(CASES[name])
    lens = kw.pop("ctx_lens")
    st = State(70, len(lens), lens, **kw)
    be, g, L = _layer(st)
    out = _step(L, st)
    be.device_sync(); L.check_status()
    want = st.oracle_step()
    n_sel = L.n_sel.cpu().numpy()
    np.testing.assert_array_equal(n_sel, want["n_sel"])
    for b in range(st.B):
        np.testing.assert_array_equal(L.rows[b, :n_sel[b]].cpu().numpy().view(np.uint32), want["rows"][b, :n_sel[b]])
    for k in ("latent_pool", "latent_scale", "index_pool", "index_scale"):
        np.testing.assert_array_equal(getattr(L, k).cpu().numpy().ravel().view(np.uint8), want[k].ravel().view(np.uint8))
    ok, worst, rms = attend_close_ref(out.view(torch.int16).cpu().numpy().view(np.uint16).reshape(want["out_f32"].shape), want["out_f32"])
    assert ok and rms <= 1e-2, (worst, rms)
    # the select operator alone takes the same rows
    rows = L.rows.clone()
    L.rows.fill_(-1)
    L.select(dev(st.index_q), dev(st.index_w), dev(st.seq_len))
    be.device_sync(); L.check_status()
    for b in range(st.B):
        assert torch.equal(L.rows[b, :n_sel[b]], rows[b, :n_sel[b]])


def test_short_batch_with_an_empty_sequence():
    st = State(71, 3, [100, 5, 64])
    be, g, L = _layer(st)
    seq_len = st.seq_len.copy()
    seq_len[1] = 0
    L.append(*[dev(getattr(st, k)[[0, 2]]) for k in ("new_latent", "new_key", "row_pos")], dev(np.array([0, 2], np.int32)))
    L.select(dev(st.index_q), dev(st.index_w), dev(seq_len))
    out = L.attend(dev(st.q))
    be.device_sync(); L.check_status()
    assert L.n_sel.tolist() == [100, 0, 64]
    assert not out[1].any() and bool(torch.isneginf(L.out_lse[1]).all())
    want = st.oracle_step()["out_f32"]
    ok, worst, rms = attend_close_ref(out.view(torch.int16).cpu().numpy().view(np.uint16).reshape(want.shape)[[0, 2]], want[[0, 2]])
    assert ok and rms <= 1e-2, (worst, rms)


@pytest.mark.parametrize("lens,top_k", [([200, 100], 256), ([400, 100], 256)])
def test_a_page_outside_the_pool_is_flagged_where_nothing_is_scored(lens, top_k):
    """Sequence 1 is selected whole: its bad page raises 1005, one past its length does not."""
    st = State(72, 2, lens, top_k=top_k)
    be, g, L = _layer(st)
    x = (dev(st.index_q), dev(st.index_w), dev(st.seq_len))
    for page, bad in ((1, True), (2, False)):
        bt = st.block_table.copy()
        bt[1, page] = g.n_pool_pages + 3
        L.block_table.copy_(dev(bt))
        L.select(*x)
        if bad:
            with pytest.raises(be.BackendError) as e:
                be.index_select_status(g, st.B, L.score_stride, L.select_scratch)
            assert e.value.code == 1005
        else:
            be.index_select_status(g, st.B, L.score_stride, L.select_scratch)


@pytest.mark.parametrize("cluster", [1, 2, 4, 8])
@pytest.mark.parametrize("kind", ["spread", "front", "ties", "equal"])
def test_selection_bands_of_every_cluster(cluster, kind):
    """Bands that end in each branch: a few tokens per CTA; hundreds in one CTA (more than its slots in the others' lists);
    thousands of ties; all scores equal. Token counts that leave the last step and the last CTA ragged, against exact scores
    with the exact top-k."""
    from rivoli_b200 import backend as be
    be.lib()
    n, k = 9001, 700
    st = State(73, 2, [n, 5000], top_k=k)
    g = make_geom(be.DsaGeom, **st.geom_kw)
    P = g.page_tokens
    rows = (st.block_table[0, np.arange(n) // P].astype(np.int64) * P + np.arange(n) % P)
    pool, scale = st.index_pool.reshape(-1, 128), st.index_scale
    if kind == "front":        # the first 600 tokens: the same key, at the cut
        pool[rows[100:700]] = pool[rows[100]]; scale[rows[100:700]] = scale[rows[100]]
        pool[rows[700:]] = pool[rows[1]]; scale[rows[700:]] = scale[rows[1]] * np.float32(1e-3)
        pool[rows[:100]] = pool[rows[100]]; scale[rows[:100]] = scale[rows[100]] * np.float32(1.5)
        st.index_w[0] = np.abs(st.index_w[0])
    elif kind == "ties":       # six thousand copies of one key
        pool[rows[1500:7500]] = pool[rows[1500]]; scale[rows[1500:7500]] = scale[rows[1500]]
    elif kind == "equal":
        pool[rows] = pool[rows[0]]; scale[rows] = scale[rows[0]]
    d = {m: dev(getattr(st, m)) for m in ("index_q", "index_w", "index_pool", "index_scale", "block_table", "seq_len")}
    got = torch.full((2, k), -1, dtype=torch.int32, device="cuda")
    n_sel = torch.zeros(2, dtype=torch.int32, device="cuda")
    scratch = torch.zeros(be.index_select_scratch_bytes(g, 2, n), dtype=torch.uint8, device="cuda")
    be.index_select_test_cluster(cluster)
    try:
        be.launch_index_select_paged(g, d["index_q"], d["index_w"], d["index_pool"], d["index_scale"], d["block_table"],
                                     d["seq_len"], 2, n, got, n_sel, scratch)
        be.index_select_status(g, 2, n, scratch)
    finally:
        be.index_select_test_cluster(0)
    codes = torch.zeros(2 * 32 * 128, dtype=torch.uint8, device="cuda")
    qs = torch.zeros(64, device="cuda")
    scores = torch.zeros((2, n), device="cuda")
    want, wn = torch.zeros_like(got), torch.zeros_like(n_sel)
    be.launch_index_q_quant(d["index_q"], 64, 128, codes, qs)
    be.launch_index_score_paged(g, codes, qs, d["index_w"], d["index_pool"], d["index_scale"], d["block_table"], d["seq_len"], 2, scores, n)
    s = scores.cpu().numpy()
    for b, m in enumerate((n, 5000)):
        order = np.lexsort((np.arange(m), -s[b, :m].astype(np.float64)))[:k]
        np.testing.assert_array_equal(got[b].cpu().numpy(), np.sort(order))


@pytest.mark.parametrize("lens,hint", [([300, 128, 700], 128), ([300, 5, 127], 0), ([64, 100], 0)])
def test_shared_layer_step_equals_its_operators(lens, hint):
    """Append and attention over another layer's rows in one call, bit for bit the two calls: hint taken, short sequences
    among long ones, only short ones."""
    st = State(74, len(lens), lens, top_k=256)
    outs = []
    for joint in (True, False):
        be, g, src = _layer(st)
        src.step(dev(st.new_latent), dev(st.new_key), dev(st.index_q), dev(st.index_w), dev(st.q), dev(st.row_pos), dev(st.seq_len))
        _, _, L = _layer(st)
        x = dev(st.new_latent).flip(0).contiguous(), dev(st.q).flip(0).contiguous(), dev(st.row_pos)
        for _ in range(3):          # back to back: each call starts under the one before it
            if joint:
                out = L.step_shared(*x, src, min_rows_hint=hint)
            else:
                L.append_latent_only(x[0], x[2])
                out = L.attend(x[1], rows_from=src)
        be.device_sync(); L.check_status()
        outs.append([t.cpu().contiguous().view(torch.uint8) for t in (out, L.out_lse, L.latent_pool, L.latent_scale, L.index_pool)])
    for a, b in zip(*outs):
        assert torch.equal(a, b)


@pytest.mark.parametrize("lens", [[257, 3, 300, 256, 128, 9000, 1], [257], [400] * 40, [385, 129] * 20])
def test_scorer_shares_of_ragged_batches(lens):
    """Shares of the tiles that begin and end anywhere: sequences without a score between others, more CTAs than tiles, one
    tile, shares over several sequences; rows against the unfused operators."""
    st = State(75, len(lens), lens, top_k=256)
    be, g, L = _layer(st)
    x = (dev(st.index_q), dev(st.index_w), dev(st.seq_len))
    L.select(*x)
    be.device_sync(); L.check_status()
    got, n = L.rows.clone(), L.n_sel.clone()
    L.select_unfused(*x)
    assert torch.equal(n, L.n_sel)
    for b, k in enumerate(n.tolist()):
        assert torch.equal(got[b, :k], L.rows[b, :k]), b


@pytest.mark.parametrize("lens", [[1, 64, 65, 128, 129, 192, 193], [255, 256, 257, 320, 321], [383, 385, 449, 640] * 19])
def test_attention_tiles_of_the_gather(lens):
    """Row counts around the tiles that the gather warps share and those they fill alone, in clusters and (76 sequences) with
    one CTA per sequence, against the CUDA-core kernel."""
    st = State(76, len(lens), lens)
    be, g, L = _layer(st)
    want = torch.empty_like(L.out)
    n = dev(st.seq_len)
    args = (dev(st.q), L.latent_pool, L.latent_scale, L.block_table, None, 0, n, st.B)
    be.attend_mma_test_hook(min_rows=0)
    try:
        be.launch_attend_paged_bf16(g, *args, L.out, L.out_m, L.out_lse, L.scratch)
        be.attend_paged_status(g, L.scratch)
    finally:
        be.attend_mma_test_hook()
    be.launch_attend_simt_paged_bf16(g, *args, want, None, None, None)
    a, b = L.out.float(), want.float()
    assert bool(((a - b).abs() <= 2e-2 * b.abs().amax(dim=(1, 2), keepdim=True) + 1e-3).all()), (a - b).abs().max().item()


@pytest.mark.parametrize("max_ctx", [16390, 131072, 131136])
@pytest.mark.parametrize("name", ["all-below", "one-above", "short", "short-top-k", "not-short", "lone-cta", "cluster", "above-other-geometry"])
def test_step_of_a_layer_built_for_far_longer_sequences(name, max_ctx):
    """A layer is built for the longest sequence that a server admits, not for the batch at hand: the launch plans follow that
    length (score rows that no 16-byte load fits, clusters most of whose CTAs have no token, score rows past what the tensor-core
    scorer takes), the results do not."""
    from rivoli_b200 import backend as be
    from rivoli_b200.layer import DsaDecodeLayer
    be.lib()
    kw = dict(CASES[name])
    lens = kw.pop("ctx_lens")
    st = State(74, len(lens), lens, **kw)
    g = make_geom(be.DsaGeom, **dict(st.geom_kw, max_pages_per_seq=-(-max_ctx // st.geom_kw["page_tokens"])))
    L = DsaDecodeLayer(g, st.B, max_ctx=max_ctx)
    for k in ("latent_pool", "latent_scale", "index_pool", "index_scale"):
        getattr(L, k).copy_(dev(getattr(st, k)).view(getattr(L, k).shape))
    L.block_table[:, :st.block_table.shape[1]] = dev(st.block_table)
    out = _step(L, st)
    be.device_sync(); L.check_status()
    want = st.oracle_step()
    n_sel = L.n_sel.cpu().numpy()
    np.testing.assert_array_equal(n_sel, want["n_sel"])
    for b in range(st.B):
        np.testing.assert_array_equal(L.rows[b, :n_sel[b]].cpu().numpy().view(np.uint32), want["rows"][b, :n_sel[b]])
    for k in ("latent_pool", "latent_scale", "index_pool", "index_scale"):
        np.testing.assert_array_equal(getattr(L, k).cpu().numpy().ravel().view(np.uint8), want[k].ravel().view(np.uint8))
    ok, worst, rms = attend_close_ref(out.view(torch.int16).cpu().numpy().view(np.uint16).reshape(want["out_f32"].shape), want["out_f32"])
    assert ok and rms <= 1e-2, (worst, rms)
