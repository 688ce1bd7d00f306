"""The selection's two ways of reading a score row, whole vectors and a score at a time: row lengths and bases on either side of the
16-byte rule, a lone CTA and clusters, given scores against the oracle and paged ones against each other."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc
from oracle.workload import State, make_geom
from tests.test_step_edges_gpu import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("n", [1025, 1028, 4096, 4099, 16384, 16385, 40001, 40004])
def test_given_scores(n, offset):
    from rivoli_b200 import backend as be
    be.lib()
    rng = np.random.default_rng(n + offset)
    b, k = 2, 700
    s = np.round(rng.standard_normal((b, n)) * 500).astype(np.float32) / 500      # ties at the cut
    lens = np.array([n, n - 3], np.int32)
    flat = torch.zeros(b * n + 1, device="cuda")
    d_s = flat[offset:offset + b * n]
    d_s.copy_(torch.from_numpy(s.ravel()))
    rows = torch.full((b, k), -1, dtype=torch.int32, device="cuda")
    n_sel = torch.full((b,), -1, dtype=torch.int32, device="cuda")
    be.launch_index_topk_batched(d_s, n, dev(lens), b, k, rows, n_sel)
    be.device_sync()
    want, want_n = orc.index_topk_batched(s, lens, k)
    assert n_sel.cpu().numpy().tolist() == want_n.tolist()
    np.testing.assert_array_equal(rows.cpu().numpy().view(np.uint32), want)


@pytest.mark.parametrize("cluster", [1, 2, 4, 8])
def test_paged_scores_in_rows_of_two_lengths(cluster):
    """The same sequences, the score rows a multiple of four long and not: the same rows are selected."""
    from rivoli_b200 import backend as be
    be.lib()
    n, k, got = 9001, 700, []
    st = State(75, 2, [n, 5000], top_k=k)
    g = make_geom(be.DsaGeom, **st.geom_kw)
    d = {m: dev(getattr(st, m)) for m in ("index_q", "index_w", "index_pool", "index_scale", "block_table", "seq_len")}
    be.index_select_test_cluster(cluster)
    try:
        for stride in (n, n + 3):
            rows = torch.full((2, k), -1, dtype=torch.int32, device="cuda")
            n_sel = torch.zeros(2, dtype=torch.int32, device="cuda")
            scratch = torch.zeros(be.index_select_scratch_bytes(g, 2, stride), dtype=torch.uint8, device="cuda")
            be.launch_index_select_paged(g, d["index_q"], d["index_w"], d["index_pool"], d["index_scale"], d["block_table"],
                                         d["seq_len"], 2, stride, rows, n_sel, scratch)
            be.index_select_status(g, 2, stride, scratch)
            got.append((rows, n_sel))
    finally:
        be.index_select_test_cluster(0)
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1]) and got[0][1].tolist() == [k, k]
