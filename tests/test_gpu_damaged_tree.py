"""Archives whose tree says its root is a leaf although the header counts several nodes (one byte of
the leaf flags), or whose header counts one node where the parsed description had more: nothing to
decode by, so every decoder reports VSZ_ERR_CORRUPT, whatever an earlier call left in its workspace."""
import numpy as np
import pytest

import vecsz_gb300 as V
from vecsz_gb300 import _lib as L

pytestmark = pytest.mark.gpu


def archive(n, dtype="f32"):
    x = (np.arange(n) * 7 % 13).astype(np.float32)  # few distinct residuals: a tree of well under 256 nodes
    c = V.compress(x, (n,), eb=0.5, mode="abs", dict_size=1024, block_size=8, dtype=dtype)
    d = V.parse_archive(c.data)
    assert 2 < d.node_count <= 256 and d.has_trailer
    return x, c.data, d


def root_flag(data, d):
    b = bytearray(data)
    at = d.huff_offset + 9 + 6 * d.node_count  # [count][dict][width][L][R][C u32][leaf flags]
    assert b[at] == 0
    b[at] = 1
    return bytes(b)


def one_node(data, d):
    b = bytearray(data)
    h = d.huff_offset
    b[h:h + 4] = (1).to_bytes(4, "big")
    b[h + 9:h + 16] = bytes([0, 0, 5, 0, 0, 0, 1])  # L, R, C = 5, a leaf
    return bytes(b)


# under the split decoder's limit, and past it
@pytest.mark.parametrize("damage", [root_flag, one_node])
@pytest.mark.parametrize("n", [700, 40_003, (1 << 22) + 600])
def test_single_after_a_good_one(cuda, n, damage):
    x, data, d = archive(n)
    codec = V.DeviceCodec((n,), eb=0.5, mode="abs", dict_size=1024)
    codec.prepare_decompress(data)
    out = cuda.empty(n, dtype=cuda.float32, device="cuda")
    for buf, status in ((data, 0), (damage(data, d), L.VSZ_ERR_CORRUPT), (data, 0)):
        dev = cuda.from_numpy(np.frombuffer(buf + bytes(64), np.uint8).copy()).cuda()
        codec.decompress(dev, out)
        assert codec.decompress_status() == status
    np.testing.assert_array_equal(out.cpu().numpy(), x)


@pytest.mark.parametrize("damage", [root_flag, one_node])
@pytest.mark.parametrize("n", [40_003, (1 << 22) + 600])
def test_batch_fails_that_field_alone(cuda, n, damage):
    good = [archive(n), archive(5000)]
    b = V.BatchDecompressor([good[0][1], good[1][1]])
    for _ in range(2):  # tables of the first pass are in the workspace in the second
        b.d_archives[0].copy_(cuda.from_numpy(np.frombuffer(good[0][1] + bytes(64), np.uint8).copy()))
        b.decompress()
        assert b.statuses() == [0, 0]
        b.d_archives[0].copy_(cuda.from_numpy(np.frombuffer(damage(good[0][1], good[0][2]) + bytes(64), np.uint8).copy()))
        b.decompress()
        assert b.statuses() == [L.VSZ_ERR_CORRUPT, 0]
        np.testing.assert_array_equal(b.outputs[1].cpu().numpy(), good[1][0])


@pytest.mark.parametrize("dtype", ["f32", "f64"])
def test_host_entry_points(cuda, dtype):
    x, data, d = archive(40_003, dtype)
    np.testing.assert_allclose(V.decompress(data, d.data_size), x, rtol=0, atol=0.5)
    with pytest.raises(L.VszError) as e:
        V.decompress(root_flag(data, d), d.data_size)
    assert e.value.status == L.VSZ_ERR_CORRUPT


def test_without_the_index(cuda):
    """The packed block alone: the self-synchronising decoder."""
    x, data, d = archive(40_003)
    with pytest.raises(L.VszError) as e:
        V.decompress(root_flag(data, d)[: d.data_size], d.data_size, 0, 1024, 8)
    assert e.value.status == L.VSZ_ERR_CORRUPT
