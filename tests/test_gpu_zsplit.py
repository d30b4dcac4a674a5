"""Dual-quant units split along z (fields with fewer warp tiles than fill the GPU): every split from
whole blocks to single planes, at every block size, on ragged and aligned rows, against the oracle's
archive; and the outlier copy over groups of 32 row segments."""
import numpy as np
import pytest

import oracle as O
import vecsz_gb300 as V

pytestmark = pytest.mark.gpu


def smooth(dims, seed, spikes=0.0):
    z, y, x = (np.linspace(0, 9, d, dtype=np.float32) for d in reversed(dims))
    rng = np.random.default_rng(seed)
    f = np.sin(x)[None, None, :] * np.cos(y)[None, :, None] + np.sin(z)[:, None, None]
    f = f + rng.standard_normal(f.shape, dtype=np.float32) * np.float32(0.01)
    if spikes:
        f = np.where(rng.random(f.shape, dtype=np.float32) < spikes, f * 1e3, f)
    return np.ascontiguousarray(f, np.float32).reshape(-1)


def check(cuda, x, dims, bs, eb=1e-3):
    ref, _ = O.compress(x, dims, bs, 1024, eb, False)
    codec = V.DeviceCodec(dims, eb=eb, mode="abs", dict_size=1024, block_size=bs)
    codec.compress(cuda.from_numpy(x).cuda())
    arch = codec.archive_bytes()
    assert arch[: len(ref)] == ref


@pytest.mark.parametrize("bs", [8, 16, 32, 64])
@pytest.mark.parametrize("dims", [(40, 24, 70), (37, 21, 67), (129, 9, 17)])
def test_single_planes(cuda, dims, bs):
    check(cuda, smooth(dims, 1, 0.01), dims, bs)


# about 3, 7, 14 and 30 million elements: one, two, four and eight planes of a block of 8 to a unit
@pytest.mark.parametrize("dims", [(128, 152, 151), (256, 170, 161), (255, 171, 320), (320, 300, 315)])
@pytest.mark.parametrize("bs", [8, 32])
def test_splits(cuda, dims, bs):
    check(cuda, smooth(dims, 2), dims, bs)


@pytest.mark.parametrize("spikes", [0.002, 0.3])
def test_batch_of_splits(cuda, spikes):
    """One launch over fields of every dimensionality, alignment and block size, outliers included."""
    shapes = [((5000,), 8), ((4096,), 64), ((37, 90), 8), ((64, 48), 16), ((60, 50), 8), ((40, 24, 70), 8),
              ((37, 21, 67), 8), ((36, 11, 9), 16), ((129, 9, 17), 8), ((64, 64, 33), 32)]
    rng = np.random.default_rng(5)
    fields, host = [], []
    for dims, bs in shapes:
        n = int(np.prod(dims))
        x = np.cumsum(rng.standard_normal(n) * 1e-2).astype(np.float32)
        x = np.where(rng.random(n) < spikes, x + 50, x).astype(np.float32)
        host.append(x)
        fields.append({"x": cuda.from_numpy(x).cuda(), "dims": dims, "eb": 1e-3, "mode": "abs", "dict_size": 1024,
                       "block_size": bs})
    b = V.BatchCompressor(fields)
    b.compress()
    for i, (dims, bs) in enumerate(shapes):
        ref, _ = O.compress(host[i], dims, bs, 1024, 1e-3, False)
        assert b.archive_bytes(i)[: len(ref)] == ref, dims


@pytest.mark.parametrize("eb", [1e-3, 0.37, 7.1e-7, 1.3e5, 3e-25, 2e32])
def test_tail_columns_near_halves(cuda, eb):
    """3D tail columns round half away in double; their FP32 form must agree beside every half."""
    dims = (15, 40, 40)
    n = int(np.prod(dims))
    rng = np.random.default_rng(9)
    k = np.where(rng.random(n) < 0.5, rng.integers(-300, 300, n), rng.integers(-(1 << 23), 1 << 23, n))
    with np.errstate(over="ignore"):
        x = ((k + 0.5) * 2 * eb).astype(np.float32)
    x = (x.view(np.int32) + rng.integers(-2, 3, n).astype(np.int32)).view(np.float32)
    x[::97] = -0.0
    x[1::97] = (rng.standard_normal(x[1::97].size) * eb).astype(np.float32)
    x[2::197] = 3e38
    x = np.where(np.isfinite(x), x, np.float32(1.0)).astype(np.float32)
    check(cuda, x, dims, 8, eb)


@pytest.mark.parametrize("d0", [1, 3, 7, 8, 9, 16, 23, 31, 33, 40, 50, 56, 60, 63, 64, 65])
@pytest.mark.parametrize("rest", [(1,), (7,), (50,), (9, 3), (37, 17)])
def test_narrow_rows(cuda, d0, rest):
    """Rows of at most 64 columns: several groups of 8 rows to a warp."""
    dims = (d0,) + rest
    check(cuda, smooth(dims, d0, 0.02) if len(dims) == 3 else smooth(dims + (1,), d0, 0.02), dims, 8)
