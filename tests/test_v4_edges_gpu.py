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


@pytest.mark.parametrize("b,max_comp,heads", [(1, 127, 64), (1, 129, 3), (2, 2048, 64), (5, 500, 33), (37, 640, 64), (300, 130, 16)])
def test_packed_scorer_tiles_and_items(b, max_comp, heads):
    """Packed rows on the tensor cores against the ordered fold: scores, rows and flags for contexts around the 128-row tile,
    every item length, queries and single rows outside the integer form."""
    be = _be()
    g = be.V4Geom.make(max_comp=max_comp, index_heads=heads, index_topk=40)
    gen = torch.Generator("cuda").manual_seed(b)

    def spread(n):
        x = torch.randn((n, 128), generator=gen, device="cuda").to(torch.bfloat16).float()
        be.launch_act_quant_f4_rotated(x, n, 128)
        return x.to(torch.bfloat16)

    ikv, iq = spread(b * max_comp).view(b, max_comp, 128), spread(b * heads).view(b, heads, 128)
    iw = torch.randn((b, heads), generator=gen, device="cuda").to(torch.bfloat16).float()
    want_flags = torch.zeros(b, dtype=torch.int32)
    n_comp = torch.randint(30, max_comp + 1, (b,), generator=gen, device="cuda")
    n_comp[0] = max_comp
    if b > 2:
        n_comp[1], n_comp[2] = max_comp, 41
        iq[1, heads - 1, 5] = 0.3711
        ikv[2, 40, :32] *= 1024.0
        want_flags[1], want_flags[2] = 1, 2
    pos = (n_comp * 4).to(torch.int32)
    packed = torch.zeros((b, max_comp, 128), dtype=torch.uint8, device="cuda")
    pexp = torch.zeros((b, max_comp), dtype=torch.int32, device="cuda")
    be.launch_v4_index_pack_bf16(g, b, None, n_comp.to(torch.int32), max_comp, ikv.view(torch.int16), packed, pexp)
    res = []
    for fold, p in ((True, None), (False, packed), (False, None)):
        sel = torch.full((b, g.window + 40), -7, dtype=torch.int32, device="cuda")
        scratch = torch.full((be.v4_select_scratch_bytes(g, b) // 4,), 5.0, device="cuda")
        be.launch_v4_select_blocks_bf16(g, b, pos, iq.view(torch.int16), iw, ikv.view(torch.int16), sel, scratch, fold, p,
                                        None if p is None else pexp)
        be.v4_select_status()
        res.append((sel.cpu(), scratch[:b * max_comp].view(b, max_comp).cpu(), scratch[b * max_comp:].view(torch.int32).cpu()))
    for sel, sc, flags in res[1:]:
        assert torch.equal(sel, res[0][0])
        assert torch.equal(flags, want_flags)
        for i in range(b):
            n = int(n_comp[i])
            if n > 40:
                assert torch.equal(sc[i, :n].view(torch.int32), res[0][1][i, :n].view(torch.int32)), i


@pytest.mark.parametrize("b,d,idim,off", [(1, 512, 128, 0), (3, 512, 128, 0), (5, 256, 64, 0), (9, 128, 128, 0), (2, 192, 128, 0), (4, 512, 128, 1)])
def test_token_step_equals_its_operators(b, d, idim, off):
    """The joint call against the operators one by one, bit for bit, over a few tokens: every width of the joint launch, widths
    and alignments (``off`` floats off a 16-byte line) that go on their own in front of it."""
    be, rng = _be(), np.random.default_rng(7 * b + d)
    from rivoli_b200.v4 import V4Compressor, V4DecodeLayer, V4TokenStep
    runs = []
    for joint in (True, False):
        rng = np.random.default_rng(7 * b + d)
        f32 = lambda *s: dev(rng.standard_normal(s).astype(np.float32))
        bf = lambda *s: dev(orc.f32_to_bf16(rng.standard_normal(s).astype(np.float32)))
        g = be.V4Geom.make(n_heads=64 if d == 512 else 4, head_dim=d, window=8, index_heads=4, index_dim=idim, index_topk=3, max_comp=32)
        L = V4DecodeLayer(g, b)
        L.kv_cache.copy_(bf(*L.kv_cache.shape).view(torch.uint16))
        L.sink.copy_(f32(g.n_heads))
        comps = []
        for w, rotate in ((d, False), (idim, True)):
            p = be.CompGeom.make(ratio=4, d=w, rd=64 if w >= 128 else 32)
            norm, freqs, ape = _comp_fixture(rng, p, 64)
            c = V4Compressor(p, b, dev(ape), dev(norm), dev(freqs), rotate)
            c.kv_state.copy_(f32(*c.kv_state.shape)); c.score_state.copy_(f32(*c.score_state.shape))
            if off:
                c.ape = torch.cat([torch.zeros(off, device="cuda"), c.ape.flatten()])[off:]
            comps.append(c)
        step = V4TokenStep(L, *comps)
        pos0 = np.arange(b, dtype=np.int32) * 5 + 1
        outs = []
        for t in range(6):
            pos = dev(pos0 + t)
            x = (bf(b, d), (f32(b, 2 * d), f32(b, 2 * d)), (f32(b, 2 * idim), f32(b, 2 * idim)), bf(b, g.n_heads, d),
                 bf(b, 4, idim), f32(b, 4))
            if joint:
                out = step(pos, *x)
            else:
                comps[1].step(pos, *x[2], L.index_kv, g.max_comp, 0, L.packed, L.packed_exp)
                L.select(pos, x[4], x[5])
                L.kv_cache.view(torch.int16)[torch.arange(b, device="cuda"), (pos % 8).long()] = x[0].view(torch.int16)
                comps[0].step(pos, *x[1], L.kv_cache, L.kv_rows, g.window)
                out = L.attend(x[3])
            outs.append([a.clone().cpu().contiguous().view(torch.uint8) for a in (out, L.sel, L.kv_cache, L.index_kv) + tuple(
                s for c in comps for s in (c.kv_state, c.score_state))] + ([] if L.packed is None else [L.packed.cpu(), L.packed_exp.cpu()]))
        runs.append(outs)
    for t, (a, w) in enumerate(zip(*runs)):
        for i, (x, y) in enumerate(zip(a, w)):
            assert torch.equal(x, y), (t, i)


@pytest.mark.parametrize("d,nblk,rd", [(512, 1, 64), (512, 37, 64), (256, 70, 64), (128, 301, 64), (192, 9, 64)])
def test_prompt_blocks_are_the_decode_blocks(d, nblk, rd):
    """A block pooled from a prompt and the same block pooled token by token go through the same operations in the same order:
    every bit is the same. The values of an entry's two halves cancel, so that an order of its own would show in the result."""
    be, rng = _be(), np.random.default_rng(d + nblk)
    p = be.CompGeom.make(ratio=4, d=d, rd=rd)
    norm, freqs, ape = (dev(a) for a in _comp_fixture(rng, p, nblk * 4))
    ape *= 0.01
    kv = dev(rng.standard_normal((nblk * 4, 2, d)).astype(np.float32))
    kv[:, 0] += 300.0
    kv[:, 1] -= 300.0
    kv, sc = kv.reshape(nblk * 4, 2 * d).contiguous(), dev((0.01 * rng.standard_normal((nblk * 4, 2 * d))).astype(np.float32))
    want = torch.empty((nblk, d), device="cuda")
    be.launch_kv_compress_prefill(kv, sc, ape, norm, freqs, want, p, nblk)
    # every block is a sequence of its own: the block before it in the overlap half of its state, then its four tokens
    kv_state = torch.zeros((nblk, p.ents, p.cd), device="cuda")
    score_state = torch.full((nblk, p.ents, p.cd), float("-inf"), device="cuda")
    kb, sb = kv.view(nblk, 4, p.cd), sc.view(nblk, 4, p.cd)
    kv_state[1:, :4], score_state[1:, :4] = kb[:-1], (sb + ape)[:-1]
    one_kv, one_score = kv_state[-1].clone(), score_state[-1].clone()
    cache = torch.zeros((nblk, nblk, d), dtype=torch.uint16, device="cuda")
    pre = torch.empty((nblk, d), device="cuda")
    for t in range(4):
        pos = torch.arange(nblk, device="cuda", dtype=torch.int32) * 4 + t
        be.launch_v4_compress_step_bf16(p, nblk, pos, kb[:, t].contiguous(), sb[:, t].contiguous(), ape, kv_state, score_state, norm,
                                        freqs, False, cache, nblk, 0, pre)
    assert np.array_equal(bits(pre.cpu().numpy()), bits(want.cpu().numpy()))
    # and the operator of one sequence, which pools a whole state
    one_kv[4:], one_score[4:] = kb[-1], sb[-1] + ape
    one = torch.empty(d, device="cuda")
    be.launch_kv_compress_decode(one_kv, one_score, norm, freqs, one, p, nblk * 4 - 1)
    assert np.array_equal(bits(one.cpu().numpy()), bits(want[-1].cpu().numpy()))


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 3.4e38])
def test_quantisers_of_rows_that_are_not_finite(value):
    """A block whose largest magnitude is infinite has an infinite scale: nothing of it survives, and no finite number appears."""
    be, rng = _be(), np.random.default_rng(3)
    x = rng.standard_normal((5, 512)).astype(np.float32)
    x[1, 70], x[2, 64:128], x[3, 0], x[3, 447] = value, value, 0.0, value
    _, want = orc.act_quant_f8_prefix(x.reshape(-1), 5, 512, 448, 64)
    t = dev(x.reshape(-1).copy())
    be.launch_act_quant_f8_prefix(t, t, 5, 512, 448, 64)
    assert np.array_equal(t.cpu().numpy(), np.asarray(want).reshape(-1), equal_nan=True)
    for d in (32, 64, 128, 256):
        y = rng.standard_normal((4, d)).astype(np.float32)
        y[1, 5], y[2, 0], y[2, d - 1] = value, value, value
        _, want = orc.v4_spread(y, d)
        t = dev(y.copy())
        be.launch_act_quant_f4_rotated(t, 4, d)
        assert np.array_equal(t.cpu().numpy(), want.reshape(4, d), equal_nan=True), d


@pytest.mark.parametrize("as_address", [False, True])
def test_token_step_takes_a_strided_entry_in_the_order_of_its_stream(as_address):
    """The entry of a token as a slice of a wider tensor, on a stream that is not the current one, whose work is still pending."""
    be = _be()
    from rivoli_b200.v4 import V4Compressor, V4DecodeLayer, V4TokenStep
    g, b = be.V4Geom.make(max_comp=32, window=8, index_topk=8), 3
    gen = torch.Generator("cuda").manual_seed(0)
    f32 = lambda *s: torch.randn(s, generator=gen, device="cuda")
    bf = lambda *s: f32(*s).to(torch.bfloat16).view(torch.uint16)
    layer, rng = V4DecodeLayer(g, b), np.random.default_rng(0)
    comps = []
    for w, rotate in ((512, False), (128, True)):
        p = be.CompGeom.make(ratio=4, d=w, rd=64)
        norm, freqs, ape = _comp_fixture(rng, p, 64)
        comps.append(V4Compressor(p, b, dev(ape), dev(norm), dev(freqs), rotate))
    step = V4TokenStep(layer, *comps)
    wide, pos = bf(b, 3, 512), torch.tensor([4, 9, 17], dtype=torch.int32, device="cuda")
    x = ((f32(b, 1024), f32(b, 1024)), (f32(b, 256), f32(b, 256)), bf(b, 64, 512), bf(b, 64, 128), f32(b, 64))
    side = torch.cuda.Stream()
    step(pos, wide[:, 0].contiguous(), *x)                 # (the kernels are loaded)
    torch.cuda.synchronize()
    torch.cuda._sleep(100_000_000)                         # the current stream is busy for some 50 ms
    step(pos, wide[:, 1], *x, stream=side.cuda_stream if as_address else side)
    side.synchronize()
    with torch.cuda.stream(side):
        got = layer.kv_cache.view(torch.int16)[torch.arange(b, device="cuda"), (pos % 8).long()].cpu()
    assert torch.equal(got, wide.view(torch.int16)[:, 1].cpu())


def test_token_step_broadcasts_and_refuses_entries():
    """An entry that broadcasts to [B, head_dim] is every sequence's; one of another size, width or device is refused, on the host."""
    be = _be()
    from rivoli_b200.v4 import V4Compressor, V4DecodeLayer, V4TokenStep
    g, b = be.V4Geom.make(n_heads=4, max_comp=32, window=8, index_topk=8), 3
    gen, rng = torch.Generator("cuda").manual_seed(0), np.random.default_rng(0)
    f32 = lambda *s: torch.randn(s, generator=gen, device="cuda")
    bf = lambda *s: f32(*s).to(torch.bfloat16)
    layer, comps = V4DecodeLayer(g, b), []
    for w, rotate in ((512, False), (128, True)):
        p = be.CompGeom.make(ratio=4, d=w, rd=64)
        norm, freqs, ape = _comp_fixture(rng, p, 64)
        comps.append(V4Compressor(p, b, dev(ape), dev(norm), dev(freqs), rotate))
    step = V4TokenStep(layer, *comps)
    pos = torch.tensor([4, 9, 17], dtype=torch.int32, device="cuda")
    x = ((f32(b, 1024), f32(b, 1024)), (f32(b, 256), f32(b, 256)), bf(b, 4, 512).view(torch.uint16), bf(b, 64, 128).view(torch.uint16), f32(b, 64))
    ring = lambda: layer.kv_cache.view(torch.int16)[torch.arange(b, device="cuda"), (pos % 8).long()]
    for entry in (bf(1, 512), bf(512), bf(512, 3).T, bf(3, 512), bf(3, 512).view(torch.uint16)):
        step(pos, entry, *x)
        torch.cuda.synchronize()
        assert torch.equal(ring(), entry.view(torch.int16).expand(b, 512) if entry.stride(-1) == 1 else entry.contiguous().view(torch.int16))
    before = layer.kv_cache.view(torch.int16).clone()
    for entry in (bf(2, 512), bf(3, 256), bf(3, 513), f32(3, 512), bf(3, 512).cpu(), bf(1, 3, 512, 1)):
        with pytest.raises(RuntimeError):
            step(pos, entry, *x)
    torch.cuda.synchronize()
    assert torch.equal(layer.kv_cache.view(torch.int16), before)
