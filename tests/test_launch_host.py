"""The native call path converts its arguments as ctypes does: same guard codes for the same values, on the CPU."""
import ctypes as C

import pytest
import torch

from rivoli_b200 import build

build.build()
from rivoli_b200 import backend as be  # noqa: E402


class Stream:
    cuda_stream = 0


T = torch.zeros(4)
G = be.DsaGeom.make(max_pages_per_seq=4, n_pool_pages=8)
COMP = be.CompGeom.make()


@pytest.mark.parametrize("name, args", [
    ("gemv_fp8", (T, T, T, 8, 8, 96, 1, T)),                       # not a power of two
    ("gemv_fp8", (T, T, T, 8, 8, 128, 3, T)),
    ("gemv_fp8", (T, T, T, (1 << 32) - 1, 8, 128, 1, T)),          # wraps to -1
    ("layernorm", (T, None, 0, 0, 1e-6, T)),
    ("rope_interleave", (T, 1, 8, 7, 3, 10000.0)),
    ("kv_append_paged", (None, T, T, None, T, 1, T, T, T, T, T, None, Stream())),
    ("kv_append_paged", (G, T, T, None, T, 0, T, T, T, T, T, None, None)),
    ("kv_compress_prefill", (T, T, T, be.CompFinish(0, 0, 0), COMP, 0, None)),
    ("kv_compress_prefill", (T, T, T, (T, T, T), COMP, 0, None)),
    ("kv_compress_deposit", (T, T, T, T, T, None, 1, 0, None)),
])
def test_guards_as_through_ctypes(name, args):
    plain = [a.data_ptr() if isinstance(a, torch.Tensor) else a.cuda_stream if isinstance(a, Stream) else
             C.addressof(a) if isinstance(a, C.Structure) else 0 if isinstance(a, tuple) else a for a in args]
    if any(isinstance(a, tuple) for a in args):
        plain[3] = C.addressof(be.CompFinish(*(t.data_ptr() for t in args[3])))
    want = getattr(be.lib(), "rivoli_" + name)(*plain)
    assert want > 0, "the case is one that the guard refuses"
    assert getattr(be._launch(), name)(*args) == want


def test_wrong_arguments_raise():
    n = be._launch()
    for args in ((T,), (T, T, T, 8, 8, 128, 1.5, T), ("x", T, T, 8, 8, 128, 1, T)):
        with pytest.raises((TypeError, AttributeError)):
            n.gemv_fp8(*args)
    with pytest.raises(TypeError):
        n.kv_compress_prefill(T, T, T, (T, T), COMP, 0, None)
    with pytest.raises(TypeError):
        n.kv_append_paged(COMP, T, T, None, T, 0, T, T, T, T, T, None, None)   # too small for the geometry
