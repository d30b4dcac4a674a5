"""The decoders and reverse Lorenzo kernels that only larger calls reach: the window decoder and the
general indexed decoder of a single field, the batch's window and index decoders and its block, separable
and redo kernels (more than 2^13 chunks, more than 2^25 elements of 3D fields).  Against the oracle."""
import numpy as np
import pytest

import oracle as O
import vecsz_gb300 as V
from vecsz_gb300 import fields

pytestmark = pytest.mark.gpu


def from_residuals(r):
    """A 1D field with these Lorenzo residuals (blocks of 8 start from zero); bound 0.5 keeps them."""
    pad = np.zeros((r.size + 7) // 8 * 8, np.int64)
    pad[: r.size] = r
    return np.cumsum(pad.reshape(-1, 8), axis=1).reshape(-1)[: r.size].astype(np.float32)


def fibonacci():
    """34 Fibonacci counts, the rarest the largest code: codewords of up to 33 bits."""
    f = [1, 1]
    while len(f) < 34:
        f.append(f[-1] + f[-2])
    r = np.random.default_rng(0).permutation(np.repeat(33 - np.arange(34), f))
    return from_residuals(r), 256, (33, 64)


def rare_steps():
    """About 3 bits a code, the longest codewords past both tables."""
    rng = np.random.default_rng(78)
    n = (1 << 22) + 777
    k = np.minimum(rng.geometric(0.45, n) - 1, 30)
    return from_residuals(k * rng.choice(np.array([-1, 1]), n)), 1024, (21, 32)


def wide():
    """16 K symbols: more secondary entries than the window decoder keeps in shared memory."""
    rng = np.random.default_rng(1)
    n = (1 << 22) + 777
    return from_residuals(np.rint(rng.laplace(0, 1000, n)).clip(-30000, 30000).astype(np.int64)), 65536, (21, 32)


def longest(x, dict_size):
    code = O.dualquant(x, (x.size,), 8, dict_size, 0.5)[0]
    return int(O.huffman_codebook(np.bincount(code, minlength=dict_size).astype(np.uint64), dict_size)[0].max())


@pytest.mark.parametrize("make", [rare_steps, wide, fibonacci])
def test_single_field_decoders(cuda, make):
    x, dict_size, lens = make()
    assert lens[0] <= longest(x, dict_size) <= lens[1]
    ref, _ = O.compress(x, (x.size,), 8, dict_size, 0.5, False)
    c = V.compress(x, (x.size,), 0.5, "abs", dict_size, 8)
    assert c.data[: c.data_size] == ref
    np.testing.assert_array_equal(V.decompress(c).view(np.uint32), O.decompress(ref, 8, dict_size).view(np.uint32))


def steps_3d(dims, share, seed):
    """Small integers, and at `share` of the elements values past 2^21: outliers, and blocks that the
    separable pass leaves to the reference-order kernel."""
    rng = np.random.default_rng(seed)
    n = int(np.prod(dims))
    x = rng.integers(-4, 5, n).astype(np.float32)
    at = rng.random(n) < share
    x[at] = rng.integers(1 << 21, 1 << 23, int(at.sum()))
    return x


def test_batch_past_both_limits(cuda):
    f = [(steps_3d((384, 384, 256), 0.0005, 1), (384, 384, 256), 1024)]              # separable, with redo units
    f += [(steps_3d((264, 41, 19), 0.002, 2), (264, 41, 19), 1024)]                  # the same, rows of two segments
    f += [(steps_3d(d, 0.05, 3 + i), d, 1024) for i, d in enumerate(((64, 40, 24), (16, 100, 9), (101, 67, 45), (23, 50, 17), (136, 33, 12), (139, 33, 12)))]
    f += [(fields.grf_3d(40, 61, 83, seed=5).ravel() * 1000, (83, 61, 40), 4096)]
    for i, d in enumerate(((640, 300), (641, 300), (24, 500), (31, 77))):
        f.append((fields.bump_field_2d(d[1], d[0], seed=20 + i).ravel() * 4000, d, 1024))
    rng = np.random.default_rng(9)
    for n in (70_000, 70_003, 1):
        f.append((from_residuals(np.rint(rng.standard_normal(n) * 60).astype(np.int64)), (n,), 1024))
    f.append((np.full(5000, 3.0, np.float32), (5000,), 1024))                          # one symbol
    for make in (rare_steps, wide, fibonacci):                                         # fibonacci: past 32 bits
        x, dict_size, _ = make()
        f.append((x, (x.size,), dict_size))
    assert sum(x.size for x, d, _ in f if len(d) == 3) > 1 << 25
    refs, archives = [], []
    for x, dims, dict_size in f:
        c = V.compress(x, dims, 0.5, "abs", dict_size, 8)
        refs.append(O.compress(x, dims, 8, dict_size, 0.5, False)[0])
        assert c.data[: c.data_size] == refs[-1]
        archives.append(c.data)
    d = [V.parse_archive(a) for a in archives]
    assert 0 < d[0].n_outlier * 64 < f[0][0].size and 0 < d[1].n_outlier * 64 < f[1][0].size
    assert sum(int(v.n_chunks) for v in d) > 1 << 13
    b = V.BatchDecompressor(archives)
    for _ in range(2):  # the redo counts and task counters are cleared by each call
        for o in b.outputs:
            o.fill_(float("nan"))
        b.decompress()
        assert b.statuses() == [0] * len(f)
    for (x, dims, dict_size), ref, out in zip(f, refs, b.outputs):
        want = O.decompress(ref, 8, dict_size)
        np.testing.assert_array_equal(out.cpu().numpy().view(np.uint32), want.view(np.uint32), err_msg=str(dims))


# chunks at the ends of one, two and three rounds of the split decoder, and trees on either side of its rule
@pytest.mark.parametrize("chunks", [1 << 13, 19456, 30000])
@pytest.mark.parametrize("over", [0, 1])
@pytest.mark.parametrize("sigma,dict_size", [(60, 1024), (1500, 16384)])
def test_where_the_decoder_changes(cuda, chunks, over, sigma, dict_size):
    rng = np.random.default_rng(chunks + over)
    r = np.rint(rng.standard_normal(chunks * 512 + over) * sigma).astype(np.int64)
    x = from_residuals(np.clip(r, 1 - dict_size // 2, dict_size // 2 - 1))
    c = V.compress(x, (x.size,), 0.5, "abs", dict_size, 8)
    np.testing.assert_array_equal(V.decompress(c), x)


# largest tree of a batch on either side of its rule
@pytest.mark.parametrize("width", [1400, 1900])
def test_where_the_batch_decoder_changes(cuda, width):
    rng = np.random.default_rng(width)
    xs = [from_residuals(rng.integers(-w, w + 1, n)) for w, n in ((width // 2, 200_000), (3, 40_001), (90, 513))]
    cs = [V.compress(x, (x.size,), 0.5, "abs", 4096, 8) for x in xs]
    nodes = V.parse_archive(cs[0].data).node_count
    assert (nodes <= 3072) == (width == 1400) and 2500 < nodes < 4000
    b = V.BatchDecompressor([c.data for c in cs])
    b.decompress()
    assert b.statuses() == [0, 0, 0]
    for x, o in zip(xs, b.outputs):
        np.testing.assert_array_equal(o.cpu().numpy(), x)


# more than 2^13 chunks, small trees: the window decoder with its secondary table in shared memory; at 152
# SMs 456 tasks of 256 chunks are one round of that form, 608 of the other
@pytest.mark.parametrize("tasks", [40, 500])
def test_batch_of_small_trees(cuda, tasks):
    rng = np.random.default_rng(tasks)
    r = np.rint(rng.laplace(0, 40, tasks * 256 * 512 - 77)).clip(-500, 500).astype(np.int64)
    xs = [from_residuals(r), from_residuals(rng.integers(-3, 4, 70_003)), np.full(600, 2.0, np.float32)]
    b = V.BatchDecompressor([V.compress(x, (x.size,), 0.5, "abs", 1024, 8).data for x in xs])
    assert sum(int(d.n_chunks) for d in b.descs) > 1 << 13 and max(int(d.node_count) for d in b.descs) < 3000
    b.decompress()
    assert b.statuses() == [0, 0, 0]
    for x, o in zip(xs, b.outputs):
        np.testing.assert_array_equal(o.cpu().numpy(), x)
