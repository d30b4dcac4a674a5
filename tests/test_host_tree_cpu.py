"""The host tree build against the oracle's codebook, at the symbol counts where levels of its heap fill
(short heaps take removals one after the other, longer ones both of a merge together)."""
import numpy as np
import pytest

import oracle as O
import vecsz_gb300 as V


@pytest.mark.parametrize("used", [2, 3, 5, 8, 9, 10, 11, 15, 16, 17, 18, 31, 33, 34, 64, 65, 66, 129, 700])
def test_heap_sizes(used):
    rng = np.random.default_rng(used)
    for top in (2, 40, 3000):  # ties everywhere, some, few
        hist = np.zeros(1024, np.uint64)
        hist[:used] = rng.integers(1, top, used)
        cb, head, info = np.zeros(9 * 1024, np.uint8), np.zeros(V.lib().vsz_huff_head_max(1024), np.uint8), np.zeros(4, np.uint32)
        assert V.lib().vsz_huffman_build_host(hist.ctypes.data, 1024, cb.ctypes.data, head.ctypes.data, info.ctypes.data) == 0
        lens, words, _, nodes = O.huffman_codebook(hist, 1024)
        assert int(info[0]) == nodes
        np.testing.assert_array_equal(cb[8 * 1024:], lens)
        fits = (lens > 0) & (lens <= 64)
        np.testing.assert_array_equal(cb[: 8 * 1024].view(np.uint64)[fits], words[fits] >> (64 - lens[fits].astype(np.uint64)))
