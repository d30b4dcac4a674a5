"""Outlier placement (k_outlier_scatter): outliers written to their elements of the output before the
reverse Lorenzo, at every density, at the ends of 512-code chunks and at every alignment of the
archive's outlier section; and the separable pass's redo units, which read the archive instead."""
import numpy as np
import pytest

import oracle as O
import vecsz_gb300 as V

pytestmark = pytest.mark.gpu


def check(cuda, x, dims, dict_size=256, eb=0.5):
    ref, _ = O.compress(x, dims, 8, dict_size, eb, False)
    codec = V.DeviceCodec(dims, eb=eb, mode="abs", dict_size=dict_size)
    codec.compress(cuda.from_numpy(x).cuda())
    arch = codec.archive_bytes()
    assert arch[: len(ref)] == ref
    codec.prepare_decompress(arch)
    out = cuda.empty(x.size, dtype=cuda.float32, device="cuda")
    codec.decompress(codec.archive, out)
    assert codec.decompress_status() == 0
    xr = O.decompress(ref, 8, dict_size, 0.0)
    np.testing.assert_array_equal(out.cpu().numpy().view(np.uint32), xr.view(np.uint32))
    return codec


@pytest.mark.parametrize("density", [0.0, 0.001, 0.05, 0.6, 1.0])
@pytest.mark.parametrize("dims", [(511,), (513,), (70001,), (37, 65), (64, 48), (19, 23, 29), (40, 17, 24)])
def test_density(cuda, dims, density):
    n = int(np.prod(dims))
    rng = np.random.default_rng(n)
    x = np.where(rng.random(n) < density, rng.integers(1000, 100000, n), rng.integers(-4, 5, n)).astype(np.float32)
    check(cuda, x, dims)


def test_every_alignment_of_the_section(cuda):
    seen = set()
    for n in range(1000, 1040):
        rng = np.random.default_rng(n)
        x = np.where(rng.random(n) < 0.1, 5000, rng.integers(-20, 21, n)).astype(np.float32)
        seen.add(check(cuda, x, (n,))._desc.outlier_offset % 4)
    assert seen == {0, 1, 2, 3}


@pytest.mark.parametrize("dims", [(264, 9, 17), (64, 40, 24)])
def test_redo_units_with_outliers(cuda, monkeypatch, dims):
    """Values past 2^21 send blocks of the separable pass to the reference-order kernel."""
    monkeypatch.setenv("VSZ_DQ_NO_WAVEFRONT", "1")
    n = int(np.prod(dims))
    rng = np.random.default_rng(n)
    x = rng.integers(-4, 5, n).astype(np.float32)
    at = rng.random(n) < 0.002
    x[at] = rng.integers(1 << 21, 1 << 23, int(at.sum()))
    codec = check(cuda, x, dims, dict_size=1024)
    assert 0 < codec._desc.n_outlier * 64 < n


@pytest.mark.parametrize("density", [0.0, 0.001, 0.3, 1.0])
@pytest.mark.parametrize("dims", [(511,), (513,), (70001,), (300, 211), (40, 37, 24)])
def test_without_the_index(cuda, dims, density):
    """Archives as the reference writes them: the self-synchronising decoder's streams cut chunks of 512
    codes anywhere, and it counts their zero codes."""
    n = int(np.prod(dims))
    rng = np.random.default_rng(n + 1)
    x = np.where(rng.random(n) < density, rng.integers(1000, 100000, n), rng.integers(-4, 5, n)).astype(np.float32)
    ref, _ = O.compress(x, dims, 8, 256, 0.5, False)
    y = V.decompress(ref, len(ref), 0, 256, 8)
    np.testing.assert_array_equal(y.view(np.uint32), O.decompress(ref, 8, 256, 0.0).view(np.uint32))


@pytest.mark.parametrize("shift", [0, 1, 8])  # codes on a 16-byte boundary, off it, 16 bytes further
@pytest.mark.parametrize("dims", [(511,), (512,), (513,), (5000,), (64, 40, 24), (37, 65)])
def test_stage_call(cuda, dims, shift):
    """vsz_dualquant_decompress: codes that no decoder of this library counted."""
    from vecsz_gb300 import api
    n = int(np.prod(dims))
    rng = np.random.default_rng(n + shift)
    x = np.where(rng.random(n) < 0.1, rng.integers(1000, 100000, n), rng.integers(-4, 5, n)).astype(np.float32)
    code, dense = O.dualquant(x, dims, 8, 256, 0.5)
    outliers = O.gather_outliers(code, dense)
    consts, _, _ = api.eb_setup(cuda.from_numpy(x).cuda(), 0.5)
    d_code = cuda.zeros(n + 16, dtype=cuda.int16, device="cuda")[shift: shift + n]
    d_code.copy_(cuda.from_numpy(code.astype(np.uint16).view(np.int16)))
    got = api.dualquant_decompress(dims, 8, 256, d_code, cuda.from_numpy(outliers).cuda(), consts)
    want = O.xlorenzo(code, O.scatter_outliers(code, outliers), dims, 8, 256, 0.5)
    np.testing.assert_array_equal(got.cpu().numpy().ravel()[:n].view(np.uint32), want.view(np.uint32))
