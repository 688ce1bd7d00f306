"""Several host threads, each with a stream, a geometry and buffers of its own: every call succeeds and gives what it gives alone."""
import threading

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(workers, rounds):
    """Every worker ``rounds`` times, all at once; what went wrong."""
    wrong, start = [], threading.Barrier(len(workers))

    def body(i, work):
        try:
            start.wait()
            for _ in range(rounds):
                work()
        except Exception as e:                             # a thread's exception would only be printed
            wrong.append((i, e))

    threads = [threading.Thread(target=body, args=(i, w)) for i, w in enumerate(workers)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    return wrong


def test_selection_of_geometries_with_other_shared_memory():
    """The block selection's shared memory follows the geometry: a small one must not take a large one's opt-in away."""
    from rivoli_b200 import backend as be
    gen = torch.Generator("cuda").manual_seed(0)
    workers, checks = [], []
    for max_comp in (64, 8192, 128, 16384):
        g, b = be.V4Geom.make(max_comp=max_comp, index_topk=32), 2
        iq = torch.randn((b, 64, 128), generator=gen, device="cuda").to(torch.bfloat16)
        iw = torch.randn((b, 64), generator=gen, device="cuda")
        ikv = torch.randn((b, max_comp, 128), generator=gen, device="cuda").to(torch.bfloat16)
        pos = torch.full((b,), 4 * 60, dtype=torch.int32, device="cuda")
        stream = torch.cuda.Stream()
        out = [torch.full((b, g.window + 32), -7, dtype=torch.int32, device="cuda") for _ in range(2)]
        scratch = torch.zeros(be.v4_select_scratch_bytes(g, b), dtype=torch.uint8, device="cuda")

        def call(g=g, b=b, x=(pos, iq, iw, ikv), out=out, scratch=scratch, stream=stream, into=1):
            be.launch_v4_select_blocks_bf16(g, b, *x, out[into], scratch, True, stream=stream)
        call(into=0, stream=None)
        torch.cuda.synchronize()
        workers.append(call)
        checks.append(out)
    assert _run(workers, 300) == []
    for alone, together in checks:
        assert torch.equal(alone, together)


def test_decode_steps():
    """Layers of different batches and page sizes, the first calls included (plans are asked from the device once)."""
    from rivoli_b200 import backend as be
    from rivoli_b200.layer import DsaDecodeLayer
    gen = torch.Generator("cuda").manual_seed(1)
    bf = lambda *s: torch.randn(s, generator=gen, device="cuda").to(torch.bfloat16)
    workers, layers = [], []
    for b, n, page in ((1, 3000, 64), (7, 2500, 64), (3, 300, 16), (40, 2100, 32)):
        pages = -(-n // page)
        g = be.DsaGeom.make(page_tokens=page, max_pages_per_seq=pages, n_pool_pages=b * pages)
        pair = []
        for _ in range(2):
            L = DsaDecodeLayer(g, b, max_ctx=n)
            for i in range(b):
                L.reserve(i, n)
            L.upload_block_table()
            pair.append(L)
        seq = torch.arange(b, device="cuda", dtype=torch.int32).repeat_interleave(n)
        pos = torch.arange(n, device="cuda", dtype=torch.int32).repeat(b)
        latent, key = bf(b * n, 576), bf(b * n, 128)
        x = (bf(b, 576), bf(b, 128), bf(b, 32, 128), bf(b, 32).float(), bf(b, 64, 576),
             torch.full((b,), n - 1, dtype=torch.int32, device="cuda"), torch.full((b,), n, dtype=torch.int32, device="cuda"))
        for L in pair:
            L.append(latent, key, pos, seq)
        torch.cuda.synchronize()
        stream = torch.cuda.Stream()
        workers.append(lambda L=pair[1], x=x, stream=stream: L.step(*x, stream=stream))
        layers.append((pair, x))
    assert _run(workers, 50) == []
    for (alone, together), x in layers:
        alone.step(*x)
        torch.cuda.synchronize()
        together.check_status()
        for name in ("out", "out_lse", "n_sel", "latent_pool", "index_pool"):
            assert torch.equal(getattr(alone, name), getattr(together, name)), name
        n = int(alone.n_sel[0])
        assert np.array_equal(alone.rows[:, :n].cpu().numpy(), together.rows[:, :n].cpu().numpy())
