"""The block-compressed variant's prompt operators at the edges of their launches, against the oracle."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc
from tests.test_v4_gpu import _comp_fixture, _row_close, bits, dev

pytestmark = pytest.mark.gpu


def _be():
    from rivoli_b200 import backend
    backend.lib()
    return backend


@pytest.mark.parametrize("d,nblk,rd", [(512, 1, 64), (512, 742, 64), (256, 3, 2), (256, 1481, 64), (128, 5, 128), (128, 2961, 64), (192, 9, 64)])
def test_prefill_blocks_per_cta_and_grid(d, nblk, rd):
    be, rng = _be(), np.random.default_rng(nblk)
    op = orc.CompGeom.make(ratio=4, d=d, rd=rd)
    bp = be.CompGeom(*[getattr(op, n) for n, _ in orc.CompGeom._fields_])
    s = nblk * 4 + 3
    norm, freqs, ape = _comp_fixture(rng, op, s + 5)
    kv, sc = rng.standard_normal((s, op.cd)).astype(np.float32), rng.standard_normal((s, op.cd)).astype(np.float32)
    _, want = orc.v4_compress_prefill(kv, sc, ape, norm, freqs, op, nblk)
    out = torch.full((nblk + 1, d), 7.0, device="cuda")
    be.launch_kv_compress_prefill(dev(kv), dev(sc), dev(ape), dev(norm), dev(freqs), out, bp, nblk)
    got = out.cpu().numpy()
    assert all(_row_close(got[b], want[b]) for b in range(nblk))
    assert (got[nblk] == 7.0).all()


@pytest.mark.parametrize("rows,stride,n", [(1, 64, 64), (3, 448, 448), (37, 512, 448), (5, 132, 128), (2, 130, 64)])
def test_f8_prefix_rows_and_tails(rows, stride, n):
    be, rng = _be(), np.random.default_rng(rows)
    x = (rng.standard_normal((rows, stride)) * 10.0 ** rng.uniform(-9, 9, (rows, 1))).astype(np.float32)
    _, want = orc.act_quant_f8_prefix(x.reshape(-1), rows, stride, n, 64)
    t = dev(x.reshape(-1).copy())
    be.launch_act_quant_f8_prefix(t, t, rows, stride, n, 64)
    assert np.array_equal(bits(t.cpu().numpy()), bits(np.asarray(want).reshape(-1)))


@pytest.mark.parametrize("rows,d", [(1, 32), (9, 64), (7, 128), (17, 256)])
def test_spread_rows_per_cta(rows, d):
    be, rng = _be(), np.random.default_rng(d)
    x = (rng.standard_normal((rows, d)) * 2.0 ** rng.integers(-120, 100, (rows, 1)).astype(np.float32)).astype(np.float32)
    _, want = orc.v4_spread(x, d)
    t = dev(x.copy())
    be.launch_act_quant_f4_rotated(t, rows, d)
    assert np.array_equal(bits(t.cpu().numpy()), bits(want.reshape(rows, d)))


@pytest.mark.parametrize("b,cols", [(1, 1), (1, 63), (1, 64), (2, 65), (3, 640), (1, 1100), (9, 257), (74, 130), (75, 130), (150, 64)])
def test_sparse_attention_tiles_and_clusters(b, cols):
    """Column counts around the 64-row tile, batches of every cluster size and of more than one wave; masked slots, a wholly
    masked tile in front, and scores that keep growing (the reference maxima move in every tile)."""
    from rivoli_b200 import backend as be
    be.lib()
    g = be.V4Geom.make(max_comp=1024)
    gen = torch.Generator("cuda").manual_seed(1000 * b + cols)
    R = g.window + g.max_comp
    q = torch.randn((b, 64, 512), generator=gen, device="cuda").to(torch.bfloat16)
    kv = torch.randn((b, R, 512), generator=gen, device="cuda").to(torch.bfloat16)
    sink = torch.randn(64, generator=gen, device="cuda")
    sel = torch.stack([torch.randperm(R, generator=gen, device="cuda")[:cols] for _ in range(b)]).to(torch.int32)
    growth = torch.arange(cols, device="cuda", dtype=torch.float32) / max(cols, 1) * 4.0
    for i in range(0, b, 3):                                     # rows that align with head 0's query ever more
        rows = kv[i, sel[i].long()].float() + growth[:, None] * q[i, 0].float()[None, :]
        kv[i, sel[i].long()] = rows.to(torch.bfloat16)
    sel[torch.rand(sel.shape, generator=gen, device="cuda") < 0.2] = -1
    if cols > 64:
        sel[0, :64] = -1
    sel[:, -1] = 7
    out = torch.empty((b, 64, 512), dtype=torch.bfloat16, device="cuda")
    be.launch_v4_sparse_attend_bf16(g, b, q.view(torch.int16), kv.view(torch.int16), sink, sel, cols, out.view(torch.int16))
    be.v4_sparse_attend_status()
    for i in range(b):
        k = kv[i, sel[i].clamp(min=0).long()].double()
        s = (q[i].double() @ k.T) * g.softmax_scale
        s[:, sel[i] < 0] = -float("inf")
        s = torch.cat([s, sink.double()[:, None]], 1).softmax(-1)[:, :-1]
        want = s @ k
        err = (out[i].double() - want).abs()
        assert bool((err <= 1e-2 * want.abs() + 1e-2).all()), (i, err.max().item())
