"""Trees built within a batch's dual-quant launch (dictionaries up to 1024 symbols) and by their own:
fields at that limit and past it, of one unit and of many, in one task and in many, repeated calls."""
import numpy as np
import pytest

import vecsz_gb300 as V
from vecsz_gb300 import fields

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("units", [8, 4096])
def test_dictionaries_at_the_limit(cuda, units):
    fs = []
    for i, (dims, dict_size) in enumerate([((9,), 1024), ((64, 33), 1026), ((70, 65, 40), 1024), ((70, 65, 40), 1026),
                                           ((300, 200), 2), ((64, 64, 64), 512), ((1000,), 4096), ((40, 8, 3), 65536)]):
        n = int(np.prod(dims))
        x = fields.grf_3d(1, 1, n, seed=i).ravel() if len(dims) == 1 else fields.grf_3d(*(dims + (1,))[:3], seed=i).ravel()
        fs.append({"x": cuda.from_numpy(np.ascontiguousarray(x, np.float32)).cuda(), "dims": dims, "eb": 10.0 ** -(2 + i % 4),
                   "mode": "r2r", "dict_size": dict_size, "block_size": 8 if i % 3 else 16})
    b = V.BatchCompressor(fs)
    b.set_task_sizes(units, 64)
    for _ in range(2):
        b.compress()
        cuda.cuda.synchronize()
        for i, f in enumerate(fs):
            codec = V.DeviceCodec(f["dims"], eb=f["eb"], mode="r2r", dict_size=f["dict_size"], block_size=f["block_size"])
            codec.compress(f["x"])
            assert b.archive_bytes(i) == codec.archive_bytes(), f"field {i}"
    b.close()
