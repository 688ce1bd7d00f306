"""The paged append's quotients, codes and row layout at their edges, bit for bit against the oracle: every bf16 mantissa
under every bf16 absmax mantissa, magnitudes from subnormal to near overflow, zeros, infinities and NaNs, row counts around
a CTA's rows, and geometries of three and five chunk passes."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc
from oracle.workload import bf16_normal, make_geom

pytestmark = pytest.mark.gpu


def dev(a):
    a = np.ascontiguousarray(a)
    return torch.from_numpy(a.view(np.int16) if a.dtype == np.uint16 else a).cuda()


def _append_both(lat, key, **geom):
    from rivoli_b200 import backend as be
    be.lib()
    n, W, hd = lat.shape[0], lat.shape[1], key.shape[1]
    P = 16
    pages = -(-n // P) + 1
    kw = dict(page_tokens=P, max_pages_per_seq=pages, n_pool_pages=pages, **geom)
    table = np.random.RandomState(n).permutation(pages).astype(np.int32).reshape(1, pages)
    seq, pos = np.zeros(n, np.int32), np.arange(n, dtype=np.int32)
    rows = pages * P
    want = [np.zeros(rows * W, np.uint8), np.zeros(rows, np.float32), np.zeros(rows * hd, np.uint8), np.zeros(rows, np.float32)]
    assert orc.kv_append_paged(make_geom(orc.Geom, **kw), lat, key, seq, pos, table, *want) == 0
    got = [torch.zeros(rows * W, dtype=torch.uint8, device="cuda"), torch.zeros(rows, device="cuda"),
           torch.zeros(rows * hd, dtype=torch.uint8, device="cuda"), torch.zeros(rows, device="cuda")]
    be.launch_kv_append_paged(make_geom(be.DsaGeom, **kw), dev(lat), dev(key), dev(seq), dev(pos), n, dev(table), *got)
    be.device_sync()
    for g, w in zip(got, want):
        np.testing.assert_array_equal(g.cpu().numpy().view(np.uint8), w.view(np.uint8))


@pytest.mark.parametrize("exp", [-20, 0, 9])
def test_every_mantissa_pair(exp):
    """Row i: absmax mantissa i, the other values every mantissa at four exponents below it."""
    mant = np.arange(128, dtype=np.uint16)
    lat = np.zeros((128, 576), np.uint16)
    for i in range(128):
        top = np.uint16(((127 + exp) << 7) | i)
        lat[i, 0] = top
        for k in range(4):
            v = (((127 + exp - 1 - 2 * k) << 7) | mant).astype(np.uint16)
            lat[i, 1 + 128 * k:129 + 128 * k] = v | ((k & 1) << 15)
    key = np.ascontiguousarray(lat[:, :128])
    _append_both(lat, key)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 33])
def test_row_counts(n):
    rng = np.random.RandomState(n)
    _append_both(bf16_normal(rng, (n, 576)), bf16_normal(rng, (n, 128)))


def test_magnitudes_zeros_infinities_and_nans():
    rng = np.random.RandomState(3)
    x = rng.standard_normal((40, 576)) * 2.0 ** rng.randint(-140, 120, (40, 1)) * 2.0 ** -rng.randint(0, 16, (40, 576))
    lat = orc.f32_to_bf16(x.astype(np.float32))
    lat[0] = 0
    lat[1, ::2] = 0x8000
    lat[2, 5] = 0x7F80
    lat[3, 7] = 0x7FC0
    lat[4] = 0xFFC1
    lat[5] = rng.randint(0, 0x80, 576)
    lat[6, :] = 0x7F7F
    _append_both(lat, np.ascontiguousarray(lat[:, 448:]))


@pytest.mark.parametrize("kvl,rope,hd", [(128, 16, 16), (512, 128, 128), (512, 128, 512), (256, 64, 256), (512, 64, 192)])
def test_geometries(kvl, rope, hd):
    rng = np.random.RandomState(kvl + hd)
    _append_both(bf16_normal(rng, (19, kvl + rope)), bf16_normal(rng, (19, hd)), kv_lora=kvl, rope_dim=rope, index_dim=hd, index_heads=8)


@pytest.mark.parametrize("batch", [1, 4, 5, 117, 118, 119, 128, 129])    # few and many rows a block, the line between them at 148 SMs
def test_the_append_inside_a_step(batch):
    """The rows that a step with a selection appends beside its query preparation are those of the append alone."""
    from oracle.workload import State
    from tests.test_step_edges_gpu import _layer, _step, dev
    st = State(97, batch, [200 + b % 3 for b in range(batch)], top_k=64)
    be, g, a = _layer(st)
    _, _, b = _layer(st)
    _step(a, st)
    b.append(dev(st.new_latent), dev(st.new_key), dev(st.row_pos))
    be.device_sync(); a.check_status(); b.check_status()
    for name in ("latent_pool", "latent_scale", "index_pool", "index_scale"):
        assert torch.equal(getattr(a, name), getattr(b, name))
