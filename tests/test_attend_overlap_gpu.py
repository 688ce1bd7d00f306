"""The attention beside the append in front of it: a step that selects everything, and the step of a layer that shares a
selection, fetch rows while the token is still being appended. Bit for bit what the separate operators give, also where several
sequences map the same pages, so that a row of one is another's new token."""
import numpy as np
import pytest
import torch

from oracle.workload import State
from tests.test_step_edges_gpu import _layer, _step, dev

pytestmark = pytest.mark.gpu

# rows per sequence: up to four, to eight and over eight tiles of 64 in a CTA, cut over clusters of 8, 4, 2 and not at all; two
# batches that need the second mark of the gather's threads, one over what the marks hold
BATCHES = {"2": (2, 130, 2048), "9": (9, 128, 1030), "17": (17, 128, 2048), "40": (40, 129, 2048), "76": (76, 128, 700),
           "200": (200, 129, 500), "256": (256, 129, 260), "258": (258, 128, 200), "4-short": (4, 3, 400)}


def _hint(st, hinted):
    """What a host knows of the batch. With 128 rows or more in every sequence the attention is launched right behind the append;
    without, the CUDA-core kernel stands between them, and its blocks wait for the append before the attention gets an SM."""
    if not hinted:
        return 0
    hint = int(min(st.seq_len))
    if hint < 128:
        pytest.skip("a sequence of under 128 rows: the CUDA-core kernel is launched in any case")
    return hint


def _state(name, shared_pages):
    b, lo, hi = BATCHES[name]
    lens = [lo + (hi - lo) * i // (b - 1) for i in range(b)]
    if shared_pages:                               # sequence 2 i is 2 i + 1 a token earlier, in the same pages
        lens = [lens[i | 1] - (1 - (i & 1)) if (i | 1) < b else lens[i] for i in range(b)]
    st = State(90 + b, b, lens)
    if shared_pages:
        for i in range(0, b - 1, 2):
            st.block_table[i] = st.block_table[i + 1]
    return st


def _spoil(L, st):
    """What a read before the append would find: the rows of the new tokens, as large as codes get."""
    P = L.g.page_tokens
    rows = [int(st.block_table[b, p // P]) * P + int(p % P) for b, p in enumerate(st.row_pos)]
    assert 0 <= min(rows) and max(rows) < L.latent_scale.numel()
    rows = torch.tensor(rows, device="cuda")
    L.latent_pool.view(L.latent_scale.numel(), -1)[rows] = 0x7E
    L.latent_scale[rows] = 3.0


@pytest.mark.parametrize("hinted", [False, True])
@pytest.mark.parametrize("shared_pages", [False, True])
@pytest.mark.parametrize("name", list(BATCHES))
def test_a_step_that_selects_everything(name, shared_pages, hinted):
    st = _state(name, shared_pages)
    hint = _hint(st, hinted)
    be, g, L = _layer(st)
    for _ in range(3):
        _spoil(L, st)
        got = _step(L, st, min_rows_hint=hint).clone()
        lse = L.out_lse.clone()
        _spoil(L, st)
        L.append(dev(st.new_latent), dev(st.new_key), dev(st.row_pos))
        L.select(dev(st.index_q), dev(st.index_w), dev(st.seq_len))
        want = L.attend(dev(st.q))
        be.device_sync(); L.check_status()
        assert torch.equal(got, want) and torch.equal(lse, L.out_lse)


@pytest.mark.parametrize("hinted", [False, True])
@pytest.mark.parametrize("shared_pages", [False, True])
@pytest.mark.parametrize("name", list(BATCHES))
def test_a_step_that_shares_a_selection(name, shared_pages, hinted):
    st = _state(name, shared_pages)
    hint = _hint(st, hinted)
    be, g, L = _layer(st)
    _, _, F = _layer(st)
    _step(F, st)                                   # the selection: every row, the new token among them
    for _ in range(3):
        _spoil(L, st)
        got = L.step_shared(dev(st.new_latent), dev(st.q), dev(st.row_pos), F, min_rows_hint=hint).clone()
        lse = L.out_lse.clone()
        _spoil(L, st)
        L.append_latent_only(dev(st.new_latent), dev(st.row_pos))
        want = L.attend(dev(st.q), rows_from=F)
        be.device_sync(); L.check_status()
        assert torch.equal(got, want) and torch.equal(lse, L.out_lse)
