"""The selection over few given scores (a key per thread up to 768, the large kernel beyond) at the edges of its warps and of its range, against the
oracle: ties, zeros of both signs, infinities, counts of none, one, all but one and all."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def _scores(kind, b, n, rng):
    s = rng.standard_normal((b, n)).astype(np.float32)
    if kind == "ties":
        s = np.round(s)                            # zeros of both signs among them
    elif kind == "equal":
        s[:] = 0.25
    elif kind == "special":
        s.flat[::7] = np.inf
        s.flat[3::11] = -np.inf
        s.flat[5::13] = -0.0
        s.flat[6::17] = np.finfo(np.float32).min
    return s


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 257, 767, 768, 769, 1023, 1024, 1025])
@pytest.mark.parametrize("kind", ["spread", "ties", "equal", "special"])
def test_rows_of_few_scores(n, kind):
    from rivoli_b200 import backend as be
    be.lib()
    rng = np.random.default_rng(n)
    b = 3
    s = _scores(kind, b, n, rng)
    lens = np.array([n, max(n - 1, 0), n // 2], np.int32)
    d_s, d_l = torch.from_numpy(s).cuda(), torch.from_numpy(lens).cuda()
    for k in sorted({1, max(n // 3, 1), max(n - 1, 1), n, n + 5}):
        rows = torch.full((b, k), -1, dtype=torch.int32, device="cuda")
        n_sel = torch.full((b,), -1, dtype=torch.int32, device="cuda")
        be.launch_index_topk_batched(d_s, n, d_l, b, k, rows, n_sel)
        one = torch.full((k,), -1, dtype=torch.int32, device="cuda")
        be.launch_index_topk(d_s, n, k, one)
        be.device_sync()
        want, want_n = orc.index_topk_batched(s, lens, k)
        assert n_sel.cpu().numpy().tolist() == want_n.tolist()
        np.testing.assert_array_equal(rows.cpu().numpy().view(np.uint32), want)     # and nothing behind the selected
        first = orc.index_topk(s[0], k)
        np.testing.assert_array_equal(one.cpu().numpy().view(np.uint32)[:first.size], first)
