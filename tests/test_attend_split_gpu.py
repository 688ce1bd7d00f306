"""The tensor-core attention splits a sequence's rows by the batch alone: the same rows give the same bits whatever the length of
the list that holds them (a small top_k, a large one)."""
import numpy as np
import pytest
import torch

from oracle.workload import State, make_geom
from tests.test_step_edges_gpu import dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [1, 4, 10, 15, 20, 29, 40, 74, 75])   # clusters of eight down to two, and no split
@pytest.mark.parametrize("most", [128, 256, 512])
def test_rows_in_lists_of_two_lengths(batch, most):
    from rivoli_b200 import backend as be
    be.lib()
    st = State(60 + batch, batch, [most + 40] * batch, top_k=most)
    g = make_geom(be.DsaGeom, **st.geom_kw)
    assert be.attend_paged_uses_mma(g)
    rng = np.random.default_rng(batch)
    counts = np.array([most - 32 * (b % 4) for b in range(batch)], np.int32)
    rows = np.stack([np.sort(rng.choice(most + 40, most, replace=False)) for _ in range(batch)]).astype(np.int32)
    lp, ls, bt, n = dev(st.latent_pool), dev(st.latent_scale), dev(st.block_table), dev(counts)
    scratch = torch.zeros(be.attend_paged_scratch_bytes(g, batch), dtype=torch.uint8, device="cuda")
    got = []
    for stride in (most, 2048):
        lists = torch.zeros((batch, stride), dtype=torch.int32, device="cuda")
        lists[:, :most] = dev(rows)
        out = torch.zeros((batch, g.n_heads, g.kv_lora), dtype=torch.bfloat16, device="cuda")
        lse = torch.zeros((batch, g.n_heads), dtype=torch.float32, device="cuda")
        be.launch_attend_paged_bf16(g, dev(st.q), lp, ls, bt, lists, stride, n, batch, out, None, lse, scratch)
        be.attend_paged_status(g, scratch)
        got.append((out, lse))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
