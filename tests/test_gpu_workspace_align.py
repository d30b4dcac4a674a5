"""Workspaces that do not start on a 16-byte boundary: one field's decompress takes the general decoder,
and the outliers still land on their elements; a batch and a tree build lay them out from the next one."""
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


@pytest.mark.parametrize("shift", [8, 16, 200])
def test_batch_in_an_unaligned_workspace(cuda, shift):
    xs = [fields.grf_3d(24, 40, 48, seed=4).ravel(), fields.grf_3d(17, 23, 31, seed=5).ravel(), np.full(900, 2.0, np.float32)]
    dims = [(48, 40, 24), (31, 23, 17), (900,)]
    cs = [V.compress(x, d, eb=1e-3, mode="abs", dict_size=1024, block_size=8) for x, d in zip(xs, dims)]
    b = V.BatchDecompressor([c.data for c in cs])
    ws = cuda.full((b.ws.numel() + 256,), 1, dtype=cuda.uint8, device="cuda")
    b.close()
    h = C.c_void_p(0)
    L.check(L.lib().vsz_dbatch_create(b._arr, b.n, C.c_void_p(ws.data_ptr() + shift), b.ws.numel(),
                                      C.c_void_p(b.status.data_ptr()), C.byref(h)), "dbatch_create")
    b._h = h
    b.decompress()
    assert b.statuses() == [0, 0, 0]
    assert int((ws[: shift] != 1).sum()) == 0 and int((ws[shift + b.ws.numel():] != 1).sum()) == 0
    for c, o in zip(cs, b.outputs):
        want = O.decompress(c.data[: c.data_size], 8, 1024)
        np.testing.assert_array_equal(o.cpu().numpy().view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("dict_size", [1024, 16384])  # the replay in shared memory, in the scratch
def test_tree_build_in_unaligned_scratch(cuda, dict_size):
    rng = np.random.default_rng(dict_size)
    hist = rng.integers(0, 1000, dict_size).astype(np.uint64)
    lens, *_ = O.huffman_codebook(hist, dict_size)
    lib = L.lib()
    cb = cuda.zeros(lib.vsz_codebook_bytes(dict_size), dtype=cuda.uint8, device="cuda")
    head = cuda.zeros(lib.vsz_huff_head_max(dict_size) + 16, dtype=cuda.uint8, device="cuda")
    info = cuda.zeros(4, dtype=cuda.int32, device="cuda")
    dh = cuda.from_numpy(hist.astype(np.int64)).cuda()
    tb = lib.vsz_huffman_build_tmp_bytes(dict_size)
    tmp = cuda.full((tb + 64,), 1, dtype=cuda.uint8, device="cuda")
    L.check(lib.vsz_huffman_build(C.c_void_p(dh.data_ptr()), dict_size, C.c_void_p(cb.data_ptr()),
                                  C.c_void_p(head.data_ptr()), C.c_void_p(info.data_ptr()),
                                  C.c_void_p(tmp.data_ptr() + 8), tb,
                                  C.c_void_p(cuda.cuda.current_stream().cuda_stream)), "huffman_build")
    cuda.cuda.synchronize()
    assert int(tmp[8:12].view(cuda.int32).item()) == 0
    assert int((tmp[: 8] != 1).sum()) == 0 and int((tmp[8 + tb:] != 1).sum()) == 0
    np.testing.assert_array_equal(cb[8 * dict_size: 9 * dict_size].cpu().numpy(), np.minimum(lens, 255).astype(np.uint8))
