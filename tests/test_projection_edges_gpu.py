"""The batched projections where their tiles, splits and jobs differ, against float64 products of the dequantised weights."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _be():
    from rivoli_b200 import backend
    backend.lib()
    return backend


def _weights(gen, n, k):
    codes = (torch.randn((n, k), generator=gen, device="cuda") * 0.7).to(torch.float8_e4m3fn)
    scale = torch.rand((-(-n // 128), -(-k // 128)), generator=gen, device="cuda") * 0.02 + 0.004
    full = codes.double() * scale.double().repeat_interleave(128, 0)[:n].repeat_interleave(128, 1)[:, :k]
    return codes.view(torch.uint8), scale, full


def _close(got, want, rel):
    err = (got.double() - want).abs()
    assert bool((err <= rel * want.abs() + rel * want.abs().max()).all()), (err.max().item(), want.abs().max().item())


def _rotate(v, off, seg, pos, theta):
    j = torch.arange(seg // 2, device="cuda", dtype=torch.float64)
    ang = pos.double()[:, None] * theta ** (-2.0 * j / seg)
    cs, sn = [f(ang).view(len(pos), *([1] * (v.ndim - 2)), -1) for f in (torch.cos, torch.sin)]
    a, b = v[..., off:off + seg:2], v[..., off + 1:off + seg:2]
    return torch.cat([v[..., :off], a * cs - b * sn, b * cs + a * sn, v[..., off + seg:]], -1)


@pytest.mark.parametrize("B,hidden,q_lora,nh,hd,off,seg", [
    (1, 6144, 2048, 32, 128, 0, 64),       # one row
    (127, 6144, 2048, 32, 128, 0, 64), (129, 6144, 2048, 32, 128, 64, 64), (300, 512, 256, 32, 128, 3, 10),   # batch tiles
    (9, 128, 128, 16, 128, 0, 128),        # one split
    (9, 256, 8320, 16, 64, 0, 64),         # more chunks than stages, narrow joint tile of 80 columns (pieces by fours)
    (9, 1024, 512, 48, 128, 0, 64),        # key and weights too wide for one tile: three jobs
    (5, 640, 384, 16, 256, 0, 64),         # key of two tiles
    (6, 640, 384, 10, 128, 0, 64),         # CUDA cores
])
def test_front_end_jobs_and_splits(B, hidden, q_lora, nh, hd, off, seg):
    be = _be()
    from rivoli_b200.layer import IndexerFrontEnd
    gen = torch.Generator("cuda").manual_seed(B + hidden)
    wk, wk_s, wk_f = _weights(gen, hd, hidden)
    wq, wq_s, wq_f = _weights(gen, nh * hd, q_lora)
    wp, wp_s, wp_f = _weights(gen, nh, hidden)
    kn_w = torch.rand(hd, generator=gen, device="cuda") + 0.5
    kn_b = torch.randn(hd, generator=gen, device="cuda") * 0.05
    x = torch.randn((B, hidden), generator=gen, device="cuda").to(torch.bfloat16)
    qr = torch.randn((B, q_lora), generator=gen, device="cuda").to(torch.bfloat16)
    pos = torch.randint(0, 100000, (B,), generator=gen, device="cuda", dtype=torch.int32)
    fe = IndexerFrontEnd(be.IndexFrontGeom(hidden, q_lora, nh, hd, off, seg, 128, 1e-6, 10000.0), B, dict(
        wk=wk, wk_scale=wk_s, knorm_w=kn_w, knorm_b=kn_b, wq_b=wq, wq_b_scale=wq_s, wproj=wp, wproj_scale=wp_s))
    k = x.double() @ wk_f.T
    k = (k - k.mean(1, keepdim=True)) / (k.var(1, unbiased=False, keepdim=True) + 1e-6).sqrt() * kn_w + kn_b
    q = (qr.double() @ wq_f.T).view(B, nh, hd)
    for simt in (False, True):
        gk, gq, gw = fe.run(x, qr, pos, force_simt=simt)
        be.index_frontend_status()
        _close(gk.view(torch.bfloat16), _rotate(k, off, seg, pos, 10000.0), 2.0 ** -7)
        _close(gq.view(torch.bfloat16), _rotate(q, off, seg, pos, 10000.0), 2.0 ** -7)
        _close(gw, x.double() @ wp_f.T, 2.0 ** -8)


@pytest.mark.parametrize("B,H,nope,vh,kvl,rope", [(1, 64, 192, 256, 512, 64), (127, 2, 192, 256, 512, 64), (129, 3, 192, 256, 512, 64), (300, 5, 64, 128, 256, 8),
                                                  (7, 3, 128, 128, 256, 0), (8, 1, 256, 128, 512, 16)])
def test_kvb_tiles_and_runs(B, H, nope, vh, kvl, rope):
    """Batches around the 128-row tile, one to four chunks and runs of the contraction, every rope width class."""
    be = _be()
    gen = torch.Generator("cuda").manual_seed(B + nope)
    codes, scale, full = _weights(gen, H * (nope + vh), kvl)
    full = full.view(H, nope + vh, kvl)
    q = torch.randn((B, H, nope + rope), generator=gen, device="cuda").to(torch.bfloat16)
    lat = torch.randn((B, H, kvl), generator=gen, device="cuda").to(torch.bfloat16)
    q_abs = torch.zeros((B, H, kvl + rope), dtype=torch.bfloat16, device="cuda")
    ctx = torch.zeros((B, H, vh), dtype=torch.bfloat16, device="cuda")
    be.launch_mla_absorb_batched_bf16(q, codes, scale, H, nope + rope, nope, vh, kvl, rope, 128, B, q_abs)
    be.launch_mla_value_batched_bf16(lat, codes, scale, H, nope, vh, kvl, 128, B, ctx)
    be.kvb_proj_status()
    assert torch.equal(q_abs[..., kvl:], q[..., nope:])
    _close(q_abs[..., :kvl], torch.einsum("bhd,hdi->bhi", q[..., :nope].double(), full[:, :nope]), 2.0 ** -8)
    _close(ctx, torch.einsum("bhi,hji->bhj", lat.double(), full[:, nope:]), 2.0 ** -8)
