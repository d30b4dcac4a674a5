"""The device heap replay (k_huff_build) against the host's, on histograms with ties, gaps and long
chains (totals below 2^44, in 32 bits and beyond), at the heap sizes where its levels fill."""
import ctypes as C

import numpy as np
import pytest

import vecsz_gb300 as V
from vecsz_gb300 import api

pytestmark = pytest.mark.gpu


def host(hist):
    d = hist.size
    cb = np.zeros(9 * d + 64, np.uint8)
    head = np.zeros(V.lib().vsz_huff_head_max(d) + 16, np.uint8)
    info = (C.c_uint32 * 4)()
    assert V.lib().vsz_huffman_build_host(hist.ctypes.data_as(C.c_void_p), d, cb.ctypes.data_as(C.c_void_p),
                                          head.ctypes.data_as(C.c_void_p), info) == 0
    return cb, head, list(info)


def check(cuda, hist):
    d = hist.size
    cb, head, info = host(hist)
    gcb, ghead, ginfo = api.huffman_build(cuda.from_numpy(hist.view(np.int64)).cuda(), d)
    assert [int(v) for v in ginfo] == info
    n = 8 + info[1]
    np.testing.assert_array_equal(ghead.cpu().numpy()[:n], head[:n])
    np.testing.assert_array_equal(gcb.cpu().numpy()[: 9 * d], cb[: 9 * d])


@pytest.mark.parametrize("used", [1, 2, 3, 4, 15, 16, 17, 30, 31, 32, 33, 62, 63, 64, 65, 500, 1022, 1023, 1024])
@pytest.mark.parametrize("kind", ["ties", "random", "peak", "geometric"])
def test_matches_the_host_build(cuda, used, kind):
    rng = np.random.default_rng(used)
    if kind == "ties":
        f = rng.integers(1, 4, used)
    elif kind == "random":
        f = rng.integers(1, 1 << 30, used)
    elif kind == "peak":  # a smooth field's codes
        f = 1 + (1e9 * np.exp(-0.5 * ((np.arange(used) - used / 2) / (1 + used / 20)) ** 2)).astype(np.int64)
    else:
        f = 1 + (2.0 ** np.minimum(np.arange(used) * 0.7, 32)).astype(np.int64)
    hist = np.zeros(1024, np.uint64)
    hist[np.sort(rng.choice(1024, used, replace=False))] = f.astype(np.uint64)
    check(cuda, hist)


@pytest.mark.parametrize("dict_size", [2, 256, 4096, 16384, 65536])
def test_dictionaries(cuda, dict_size):
    rng = np.random.default_rng(dict_size)
    f = rng.integers(0, 50, dict_size).astype(np.uint64)
    f[0] = 7
    check(cuda, f)
