"""The single-sequence operators at the edges of their tiles, against the oracle: rows, columns, heads and tokens one
below, at and one above what a warp, a CTA, a staged chunk or a cluster takes, and inputs that forbid wide loads."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc

pytestmark = pytest.mark.gpu


def dev(a, shift=0):
    """On the GPU; ``shift`` elements into a larger buffer, so that the data starts off any wide alignment."""
    a = np.ascontiguousarray(a)
    a = a.view({np.uint16: np.int16, np.uint32: np.int32}.get(a.dtype.type, a.dtype))
    t = torch.zeros(a.size + shift, dtype=torch.from_numpy(a[:0].reshape(-1)).dtype, device="cuda")
    t[shift:] = torch.from_numpy(a.reshape(-1))
    return t[shift:]


def bits(a):
    return np.asarray(a, np.float32).view(np.uint32)


def _be():
    from rivoli_b200 import backend
    backend.lib()
    return backend


@pytest.mark.parametrize("o_dim,i_dim,block,nrow,shift", [
    (1, 1, 1, 1, 0), (33, 1024, 128, 1, 0), (17, 1028, 128, 2, 0), (149, 515, 4, 2, 0), (297, 2052, 128, 1, 0),
    (5, 6144, 128, 2, 0), (4737, 132, 128, 1, 0), (40, 1540, 128, 1, 1)])
def test_gemv_folds(o_dim, i_dim, block, nrow, shift):
    be, r = _be(), orc.Lcg(o_dim * 7919 + i_dim)
    packed = orc.f32_to_e4m3(r.draws(o_dim * i_dim))
    scale = (np.abs(r.draws((-(-o_dim // block)) * (-(-i_dim // block)))) + np.float32(0.01)).astype(np.float32)
    x = r.draws(nrow * i_dim)
    y = torch.zeros(nrow * o_dim, device="cuda")
    be.launch_gemv_fp8(dev(x, shift), dev(packed, shift), dev(scale), o_dim, i_dim, block, nrow, y)
    be.device_sync()
    for i in range(nrow):
        want = orc.gemv_fp8(x[i * i_dim:(i + 1) * i_dim], packed, scale, o_dim, i_dim, block)[0]
        np.testing.assert_array_equal(bits(y[i * o_dim:(i + 1) * o_dim].cpu().numpy()), bits(want))


@pytest.mark.parametrize("h,nope,vh,kvl,block,nrow,shift", [
    (3, 193, 33, 132, 4, 1, 0), (2, 192, 32, 128, 128, 2, 0), (5, 385, 31, 256, 128, 1, 0), (2, 64, 64, 516, 128, 2, 1)])
def test_absorb_and_value_folds(h, nope, vh, kvl, block, nrow, shift):
    be, r, qh = _be(), orc.Lcg(kvl + nope), nope + 8
    packed, scale = orc.kvb_fixture(r, h * (nope + vh), kvl, block)
    q, clat = r.draws(nrow * h * qh), r.draws(nrow * h * kvl)
    qabs, ctx = torch.zeros(nrow * h * kvl, device="cuda"), torch.zeros(nrow * h * vh, device="cuda")
    be.launch_mla_absorb(dev(q, shift), dev(packed, shift), dev(scale), h, qh, nope, vh, kvl, block, nrow, qabs)
    be.launch_mla_value(dev(clat, shift), dev(packed, shift), dev(scale), h, nope, vh, kvl, block, nrow, ctx)
    be.device_sync()
    for i in range(nrow):
        wa = orc.mla_absorb_fp8(q[i * h * qh:(i + 1) * h * qh], packed, scale, h, qh, nope, vh, kvl, block)[0]
        wv = orc.mla_value_fp8(clat[i * h * kvl:(i + 1) * h * kvl], packed, scale, h, nope, vh, kvl, block)[0]
        np.testing.assert_array_equal(bits(qabs[i * h * kvl:(i + 1) * h * kvl].cpu().numpy()), bits(wa))
        np.testing.assert_array_equal(bits(ctx[i * h * vh:(i + 1) * h * vh].cpu().numpy()), bits(wv))


@pytest.mark.parametrize("H,nr,kvl,rope,shift", [
    (1, 1, 512, 64, 0), (3, 2, 384, 64, 0), (64, 47, 512, 64, 0), (64, 97, 256, 64, 0), (2, 1537, 128, 64, 0),
    (5, 385, 512, 40, 0), (16, 33, 384, 128, 0), (64, 200, 512, 64, 1), (7, 70, 128, 5, 1)])
def test_attend_rows_heads_and_widths(H, nr, kvl, rope, shift):
    be, r, nb = _be(), orc.Lcg(H * 131 + nr), kvl // 128
    nt = nr + 5
    qabs, qrope = r.draws(H * kvl) * np.float32(4), r.draws(H * rope)
    lc8 = orc.f32_to_e4m3(r.draws(nt * kvl))
    lscale = (np.abs(r.draws(nt * nb)) + np.float32(0.01)).astype(np.float32)
    rc = orc.f32_to_bf16(r.draws(nt * rope))
    rows = np.sort(np.random.RandomState(nr).choice(nt, nr, replace=False)).astype(np.uint32)
    for sel in (rows, None):
        want = orc.mla_attend(qabs, qrope, lc8, lscale, rc, sel, H, nr, kvl, rope, nb, 0.25)
        out = torch.full((H * kvl,), float("nan"), device="cuda")
        be.launch_attend(dev(qabs, shift), dev(qrope, shift), dev(lc8, shift), dev(lscale), dev(rc, shift),
                         None if sel is None else dev(sel), H, nr, kvl, rope, nb, 0.25, out, None)
        be.device_sync()
        assert np.abs(out.cpu().numpy() - want).max() <= 2e-5 * np.abs(want).max()


@pytest.mark.parametrize("nt,nh,nact,shift", [(1, 1, 1, 0), (63, 32, 32, 0), (65, 33, 33, 0), (129, 64, 64, 0), (64, 64, 5, 0), (70, 65, 65, 0), (66, 32, 32, 1)])
def test_index_score_tokens_and_heads(nt, nh, nact, shift):
    be, r, hd = _be(), orc.Lcg(nt * 31 + nh), 128
    q, w, kc = r.draws(nh * hd), r.draws(nh), orc.f32_to_bf16(r.draws(nt * hd))
    heads = None if nact == nh else np.random.RandomState(nt).permutation(nh)[:nact].astype(np.uint32)
    want = orc.index_score(q, w, kc, heads, nt, nh, nact, hd, 0.75, 0.125)
    out = torch.zeros(nt, device="cuda")
    be.launch_index_score(dev(q), dev(w), dev(kc, shift), None if heads is None else dev(heads), nt, nh, nact, hd, 0.75, 0.125, out)
    be.device_sync()
    assert np.abs(out.cpu().numpy() - want).max() <= 1e-5 * np.abs(want).max()


@pytest.mark.parametrize("n", [4096, 4097, 8193, 16384, 16385, 131072, 131073])
@pytest.mark.parametrize("kind", ["normal", "ties", "infinite", "equal"])
def test_topk_lengths_ties_and_infinities(n, kind):
    be, rng = _be(), np.random.RandomState(n)
    s = rng.standard_normal(n).astype(np.float32)
    if kind == "ties":
        s = np.maximum(np.round(s * 4) / 4, 0).astype(np.float32)
        s[::7] = -0.0
    elif kind == "infinite":
        s[rng.rand(n) < 0.6] = -np.inf
        s[5] = np.inf
    elif kind == "equal":
        s[:] = 0.5
    for k in (1, n // 2, n - 1, n):
        rows = torch.full((n,), -1, dtype=torch.int32, device="cuda")
        be.launch_index_topk(dev(s), n, k, rows)
        be.device_sync()
        got = rows.cpu().numpy().view(np.uint32)
        np.testing.assert_array_equal(got[:k], orc.index_topk(s, k))
        assert (got[k:] == 0xFFFFFFFF).all()


@pytest.mark.parametrize("nr", [1, 2, 13, 96, 97, 1537])
@pytest.mark.parametrize("where", ["q", "row", "score"])
def test_attend_is_loud_about_values_that_are_not_numbers(nr, where):
    """A NaN (or a score that overflows) makes the whole output of the heads that see it NaN, and of no other head."""
    be, r, H, kvl, rope, nb = _be(), orc.Lcg(nr), 6, 512, 64, 4
    qabs, qrope = r.draws(H * kvl), r.draws(H * rope)
    lc8 = orc.f32_to_e4m3(r.draws(nr * kvl))
    lscale = (np.abs(r.draws(nr * nb)) + np.float32(0.01)).astype(np.float32)
    rc = orc.f32_to_bf16(r.draws(nr * rope))
    if where == "q":
        qabs[3 * kvl + 7] = np.nan
        bad = [3]
    elif where == "row":
        lc8[(nr // 2) * kvl + 100] = 0x7F
        bad = list(range(H))
    else:
        qabs[3 * kvl: 4 * kvl] = 0.0
        qrope[3 * rope: 4 * rope] = 3e38
        rc[(nr // 2) * rope: (nr // 2 + 1) * rope] = orc.f32_to_bf16(np.full(rope, 3e38, np.float32))
        qrope[:3 * rope] = 0.0
        qrope[4 * rope:] = 0.0
        bad = [3]
    out = torch.full((H * kvl,), 7.0, device="cuda")
    be.launch_attend(dev(qabs), dev(qrope), dev(lc8), dev(lscale), dev(rc), None, H, nr, kvl, rope, nb, 0.25, out, None)
    be.device_sync()
    nan = np.isnan(out.cpu().numpy().reshape(H, kvl))
    for h in range(H):
        assert nan[h].all() if h in bad else not nan[h].any(), h


@pytest.mark.parametrize("heads,nr", [(16, 1), (16, 97), (64, 40)])
def test_paged_attention_is_loud_about_values_that_are_not_numbers(heads, nr):
    """The same of the paged form, its own geometry and the short sequences of the 64-head one."""
    be = _be()
    g = be.DsaGeom.make(n_heads=heads, page_tokens=16, max_pages_per_seq=8, n_pool_pages=16)
    gen = torch.Generator("cuda").manual_seed(nr)
    pool = torch.randn(256 * 576, generator=gen, device="cuda").to(torch.float8_e4m3fn).view(torch.uint8)
    scale = torch.rand(256, generator=gen, device="cuda") + 0.01
    table = torch.arange(16, dtype=torch.int32, device="cuda").view(2, 8)
    q = torch.randn((2, heads, 576), generator=gen, device="cuda").to(torch.bfloat16)
    q[0, 5, 3] = float("nan")
    pool[(128 + nr - 1) * 576 + 20] = 0x7F                    # the last row of the second sequence
    out = torch.zeros((2, heads, 512), dtype=torch.bfloat16, device="cuda")
    n = torch.full((2,), nr, dtype=torch.int32, device="cuda")
    scratch = torch.zeros(max(16, be.attend_paged_scratch_bytes(g, 2)), dtype=torch.uint8, device="cuda")
    be.launch_attend_paged_bf16(g, q, pool, scale, table, None, 0, n, 2, out, None, None, scratch)
    be.device_sync()
    nan = out.float().isnan().cpu()
    for h in range(heads):
        assert bool(nan[0, h].all()) if h == 5 else not bool(nan[0, h].any()), h
    assert bool(nan[1].all())


@pytest.mark.parametrize("heads,nr", [(16, 0), (16, 2), (3, 97), (16, 700)])
def test_paged_attention_reports_the_largest_score(heads, nr):
    """out_m of the CUDA-core form is the largest score itself (the first score is below it by less than what makes the running
    reference follow), out_lse its log-sum-exp; -inf for an empty sequence."""
    be = _be()
    g = be.DsaGeom.make(n_heads=heads, page_tokens=16, max_pages_per_seq=64, n_pool_pages=128)
    gen = torch.Generator("cuda").manual_seed(nr)
    pool = torch.randn(2048 * 576, generator=gen, device="cuda").to(torch.float8_e4m3fn)
    scale = torch.rand(2048, generator=gen, device="cuda") * 0.1 + 0.01
    table = torch.arange(128, dtype=torch.int32, device="cuda").view(2, 64)
    q = torch.randn((2, heads, 576), generator=gen, device="cuda").to(torch.bfloat16)
    out, n = torch.zeros((2, heads, 512), dtype=torch.bfloat16, device="cuda"), torch.full((2,), nr, dtype=torch.int32, device="cuda")
    out_m, out_lse = torch.zeros((2, heads), device="cuda"), torch.zeros((2, heads), device="cuda")
    be.launch_attend_simt_paged_bf16(g, q, pool.view(torch.uint8), scale, table, None, 0, n, 2, out, out_m, out_lse, None)
    be.device_sync()
    if nr == 0:
        assert bool((out_m == -float("inf")).all() and (out_lse == -float("inf")).all() and (out == 0).all())
        return
    rows = pool.double().view(2048, 576) * scale.double()[:, None]
    s = torch.stack([q[b].double() @ rows[b * 1024:b * 1024 + nr].T for b in range(2)]) * g.softmax_scale
    # 576 products of f32 sums: 576 * 2^-24 of the largest partial sum, which is within a few of the scores' own size
    assert bool(((out_m.double() - s.amax(-1)).abs() <= 1e-4).all())
    assert bool(((out_lse.double() - s.logsumexp(-1)).abs() <= 1e-4).all())
