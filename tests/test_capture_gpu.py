"""Launches under stream capture, the first call of a geometry among them (plans and opt-ins are asked for inside the capture): a
replay after the inputs have changed gives what the calls give."""
import numpy as np
import pytest
import torch

from tests.test_v4_gpu import _comp_fixture, dev

pytestmark = pytest.mark.gpu


def _check(run, outputs, refill):
    """``run(stream)`` captured, replayed on refilled inputs and state; against a plain call on the same."""
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        run(stream)
    refill()
    before = [t.clone() for t in outputs()]
    graph.replay()
    torch.cuda.synchronize()
    got = [t.clone() for t in outputs()]
    for t, b in zip(outputs(), before):
        t.copy_(b)
    torch.cuda.synchronize()
    run(None)
    torch.cuda.synchronize()
    for g, w in zip(got, outputs()):
        assert torch.equal(g.contiguous().view(torch.uint8), w.contiguous().view(torch.uint8))


@pytest.mark.parametrize("b,n,top_k", [(5, 3001, 2048), (9, 1500, 2048), (150, 260, 256)])
def test_decode_step(b, n, top_k):
    from rivoli_b200 import backend as be
    from rivoli_b200.layer import DsaDecodeLayer
    gen = torch.Generator("cuda").manual_seed(b)
    bf = lambda *s: torch.randn(s, generator=gen, device="cuda").to(torch.bfloat16)
    pages = -(-n // 64)
    g = be.DsaGeom.make(top_k=top_k, max_pages_per_seq=pages, n_pool_pages=b * pages)
    L = DsaDecodeLayer(g, b, max_ctx=n)
    for i in range(b):
        L.reserve(i, n)
    L.upload_block_table()
    seq = torch.arange(b, device="cuda", dtype=torch.int32).repeat_interleave(n)
    L.append(bf(b * n, 576), bf(b * n, 128), torch.arange(n, device="cuda", dtype=torch.int32).repeat(b), seq)
    x = [bf(b, 576), bf(b, 128), bf(b, 32, 128), bf(b, 32).float(), bf(b, 64, 576)]
    pos = torch.full((b,), n - 1, dtype=torch.int32, device="cuda")

    def refill():
        for t in x:
            t.copy_(torch.randn(t.shape, generator=gen, device="cuda").to(torch.bfloat16))
    length = pos + 1
    _check(lambda s: L.step(*x, pos, length, stream=s),
           lambda: [L.out, L.out_lse, L.rows, L.n_sel, L.latent_pool, L.index_pool], refill)
    L.check_status()


@pytest.mark.parametrize("b", [1, 130])
def test_projections(b):
    from rivoli_b200 import backend as be
    from rivoli_b200.layer import IndexerFrontEnd, KvbProjection
    gen = torch.Generator("cuda").manual_seed(b)
    f32 = lambda *s: torch.randn(s, generator=gen, device="cuda")
    bf = lambda *s: f32(*s).to(torch.bfloat16)
    codes = lambda *s: f32(*s).to(torch.float8_e4m3fn).view(torch.uint8)
    scales = lambda r, c: f32(-(-r // 128) * -(-c // 128)).abs() * 0.01 + 0.002
    hidden, q_lora = 1024, 512
    w = {}
    for name, rows, cols in (("wk", 128, hidden), ("wq_b", 4096, q_lora), ("wproj", 32, hidden)):
        w[name], w[name + "_scale"] = codes(rows, cols), scales(rows, cols)
    w["knorm_w"], w["knorm_b"] = f32(128), f32(128)
    front = IndexerFrontEnd(be.IndexFrontGeom(hidden, q_lora, 32, 128, 0, 64, 128, 1e-6, 10000.0), b, w)
    kvb = KvbProjection(be.DsaGeom.make(max_pages_per_seq=1, n_pool_pages=1), b, codes(64 * 448, 512), scales(64 * 448, 512), 192, 256, 128)
    x, res, q, lat = bf(b, hidden), bf(b, q_lora), bf(b, 64, 256), bf(b, 64, 512)
    pos = torch.randint(0, 10000, (b,), generator=gen, device="cuda", dtype=torch.int32)

    def run(s):
        front.run(x, res, pos, stream=s)
        kvb.absorb(q, stream=s)
        kvb.value(lat, stream=s)

    def refill():
        for t in (x, res, q, lat):
            t.copy_(bf(*t.shape))
    _check(run, lambda: [front.index_key, front.index_q, front.index_w, kvb.q_abs, kvb.ctx], refill)


@pytest.mark.parametrize("b", [3, 80])
def test_v4_token(b):
    from rivoli_b200 import backend as be
    from rivoli_b200.v4 import V4Compressor, V4DecodeLayer, V4TokenStep
    g = be.V4Geom.make(max_comp=700)
    gen, rng = torch.Generator("cuda").manual_seed(b), np.random.default_rng(b)
    f32 = lambda *s: torch.randn(s, generator=gen, device="cuda")
    bf = lambda *s: f32(*s).to(torch.bfloat16).view(torch.uint16)
    L, comps = V4DecodeLayer(g, b), []
    L.kv_cache.copy_(bf(*L.kv_cache.shape))
    for d, rotate in ((512, False), (128, True)):
        p = be.CompGeom.make(ratio=4, d=d, rd=64)
        norm, freqs, ape = _comp_fixture(rng, p, 2800)
        comps.append(V4Compressor(p, b, dev(ape), dev(norm), dev(freqs), rotate))
        comps[-1].kv_state.copy_(f32(*comps[-1].kv_state.shape))
        comps[-1].score_state.copy_(f32(*comps[-1].score_state.shape))
    step = V4TokenStep(L, *comps)
    pos = torch.arange(b, dtype=torch.int32, device="cuda") + 2600
    entry, x = bf(b, 512), [f32(b, 1024), f32(b, 1024), f32(b, 256), f32(b, 256), bf(b, 64, 512), bf(b, 64, 128), f32(b, 64)]

    def refill():
        for t in [entry] + x:
            t.copy_(bf(*t.shape) if t.dtype == torch.uint16 else f32(*t.shape))
    _check(lambda s: step(pos, entry, (x[0], x[1]), (x[2], x[3]), x[4], x[5], x[6], stream=s),
           lambda: [L.out, L.sel, L.kv_cache, L.index_kv, L.packed, L.packed_exp] + [t for c in comps for t in (c.kv_state, c.score_state)],
           refill)
