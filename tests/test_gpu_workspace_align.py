"""Decompress in workspaces that start 8 bytes past a 16-byte boundary: the general decoder takes
them, and the outliers still land on their elements."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
import vecsz_gb300 as V
from vecsz_gb300 import _lib as L
from vecsz_gb300 import fields

pytestmark = pytest.mark.gpu


def decompress_at(cuda, data, shift, n, stale):
    d = V.parse_archive(data)
    o = L.DecompressOpts(1024, 8, 0, 0.0)
    ws = C.c_size_t(0)
    L.check(L.lib().vsz_decompress_bounds(C.byref(d), C.byref(o), C.byref(ws)), "decompress_bounds")
    buf = cuda.full((ws.value + 64,), stale, dtype=cuda.uint8, device="cuda")
    arch = cuda.from_numpy(np.frombuffer(data + bytes(64), np.uint8).copy()).cuda()
    out = cuda.empty(n, dtype=cuda.float32, device="cuda")
    status = cuda.zeros(1, dtype=cuda.int32, device="cuda")
    L.check(L.lib().vsz_decompress(C.byref(d), C.byref(o), C.c_void_p(arch.data_ptr()),
                                   C.c_void_p(buf.data_ptr() + shift), ws.value, C.c_void_p(out.data_ptr()),
                                   C.c_void_p(status.data_ptr()),
                                   C.c_void_p(cuda.cuda.current_stream().cuda_stream)), "decompress")
    assert int(status.item()) == 0
    return out.cpu().numpy()


@pytest.mark.parametrize("stale", [0, 1])
@pytest.mark.parametrize("dims,bs,eb,kind", [
    ((48, 40, 24), 8, 1e-3, "grf"),           # the wavefront pass
    ((64, 40, 24), 16, 1e-3, "grf"),          # the general reverse Lorenzo
    ((64, 40, 24), 8, 1e-6, "adversarial"),   # outliers nearly everywhere
    ((70_001,), 8, 0.5, "sparse"),            # one outlier in 2000
    ((300, 211), 8, 0.5, "sparse"),
    ((9,), 8, 0.5, "sparse"),
])
def test_unaligned_workspace(cuda, dims, bs, eb, kind, stale):
    n = int(np.prod(dims))
    if kind == "sparse":
        rng = np.random.default_rng(n)
        x = np.where(rng.random(n) < 0.0005, 9000, rng.integers(-9, 10, n)).astype(np.float32)
    else:
        x = (fields.grf_3d if kind == "grf" else fields.adversarial_3d)(*reversed(dims), seed=4).ravel()
    c = V.compress(x, dims, eb=eb, mode="abs", dict_size=1024, block_size=bs)
    want = O.decompress(c.data[: c.data_size], bs, 1024)
    for shift in (0, 8, 24):
        got = decompress_at(cuda, c.data, shift, n, stale)
        np.testing.assert_array_equal(got.view(np.uint32), want.view(np.uint32))
