"""The split Huffman decoder (several lanes per 512-code chunk, fields of up to 2^13 chunks; more where
its rule says so): streams that start out of step, at the edges of chunks and warps and about the range that takes it.  Fields hold
integers and the bound is 0.5, so the reconstruction is the field itself."""
import numpy as np
import pytest

import vecsz_gb300 as V

pytestmark = pytest.mark.gpu


def residuals(kind, n, rng):
    if kind == "runs":      # one codeword nearly everywhere: parts start in or out of its phase
        return np.where(rng.random(n) < 0.002, rng.integers(-300, 300, n), 0)
    if kind == "wide":      # above 10 bits a code: the words do not fit the warp's buffer
        return rng.integers(-30000, 30000, n)
    if kind == "long":      # Fibonacci counts: codewords longer than both tables
        f = [1, 1]
        while sum(f) < n:
            f.append(f[-1] + f[-2])
        r = np.repeat(np.arange(len(f)), f)[:n]
        return rng.permutation(r) - 5
    return np.rint(rng.standard_normal(n) * 9).astype(np.int64)  # "smooth": a few bits a code


def field(kind, n, seed):
    """A 1D field with these Lorenzo residuals (blocks of 8 start from zero)."""
    r = residuals(kind, n, np.random.default_rng(seed))
    pad = np.zeros((n + 7) // 8 * 8, np.int64)
    pad[:n] = r
    return np.cumsum(pad.reshape(-1, 8), axis=1).reshape(-1)[:n].astype(np.float32)


def roundtrip(cuda, x, dict_size, damage=None):
    codec = V.DeviceCodec((x.size,), eb=0.5, mode="abs", dict_size=dict_size)
    codec.compress(cuda.from_numpy(x).cuda())
    codec.prepare_decompress(codec.archive_bytes())
    if damage:
        damage(codec)
    out = cuda.empty(x.size, dtype=cuda.float32, device="cuda")
    codec.decompress(codec.archive, out)
    return codec.decompress_status(), out.cpu().numpy()


@pytest.mark.parametrize("kind,dict_size", [("smooth", 1024), ("runs", 1024), ("wide", 65536), ("long", 256)])
@pytest.mark.parametrize("n", [1, 31, 511, 512, 513, 1027, 16 * 1024 + 9, 400_003])
def test_roundtrip(cuda, kind, dict_size, n):
    x = field(kind, n, n)
    status, out = roundtrip(cuda, x, dict_size)
    assert status == 0
    np.testing.assert_array_equal(out, x)


# 2^12 chunks: a warp for each; more: half a warp
@pytest.mark.parametrize("kind,dict_size", [("smooth", 1024), ("runs", 1024), ("wide", 65536), ("long", 256)])
@pytest.mark.parametrize("n", [(1 << 21) - 3, 1 << 21, (1 << 21) + 1, (1 << 21) + 513])
def test_where_the_lanes_per_chunk_change(cuda, kind, dict_size, n):
    x = field(kind, n, n)
    status, out = roundtrip(cuda, x, dict_size)
    assert status == 0
    np.testing.assert_array_equal(out, x)


@pytest.mark.parametrize("kind,n", [("smooth", 1 << 24), ("smooth", (1 << 24) + 1), ("runs", 1 << 22), ("runs", (1 << 22) + 1)])
def test_last_field_that_takes_it(cuda, kind, n):
    x = field(kind, n, 3)
    status, out = roundtrip(cuda, x, 1024)
    assert status == 0
    np.testing.assert_array_equal(out, x)


def test_damaged_index(cuda):
    def damage(codec):  # a chunk one bit shorter, the next one longer: both end off their mark
        d = codec._desc
        idx = codec.archive[d.index_offset: d.index_offset + 2 * d.n_chunks].view(cuda.int16)
        idx[3] -= 1
        idx[4] += 1
    status, _ = roundtrip(cuda, field("smooth", 20_000, 1), 1024, damage)
    assert status == 3  # VSZ_ERR_CORRUPT
