"""Performance cases of the library: what its users have it do, through its public entry points.

A case is a dict of plain values.  "op" says which call is made:

  compress           DeviceCodec.compress: a resident field to its archive
  decompress         DeviceCodec.decompress: a resident archive to its field
  batch_compress     BatchCompressor.compress: many uneven fields in one call
  batch_decompress   BatchDecompressor.decompress: many archives in one call
  host_compress      HostOp.compress and wait: a field in pinned host memory to its archive there

"dims" is the reference's order (x fastest) written "AxBxC".  Fields are the three kinds the
benchmark uses: "grf" a log-normal random field with a k^-11/3 power spectrum over four decades
(cosmology-like densities), "bump" smooth 2D bumps with a little noise in [0, 1] (climate-like
fields), "spiky" the first with 5 % Cauchy spikes (nearly every value an outlier at a tight bound).
"""
import ctypes
import math
import random

import torch

import vecsz_gb300 as V
from vecsz_gb300 import _lib as L

DEV = "cuda"


# ---- the cases --------------------------------------------------------------------------------

def listed():
    nyx = {"dims": "512x512x512", "kind": "grf", "mode": "r2r", "eb": 1e-4, "dict": 1024}
    climate = {"dims": "3600x1800", "kind": "bump", "mode": "abs", "eb": 1e-4, "dict": 1024}
    small = {"dims": "64x64x64", "kind": "grf", "mode": "r2r", "eb": 1e-3, "dict": 1024}
    ragged = {"dims": "333x241x187", "kind": "grf", "mode": "r2r", "eb": 1e-4, "dict": 1024}
    spiky = {"dims": "384x384x256", "kind": "spiky", "mode": "abs", "eb": 1e-6, "dict": 1024}
    batch = {"fields": 60, "n_min": 1 << 14, "n_max": 1 << 22, "shape_seed": 11, "dict": 1024}
    return [
        # the smallest requests a server or an in-situ loop makes: launches and latency
        dict(small, name="compress_small", op="compress"),
        dict(small, name="decompress_small", op="decompress"),
        # one 2D climate variable
        dict(climate, name="compress_2d", op="compress"),
        dict(climate, name="decompress_2d", op="decompress"),
        # a 3D field whose rows are aligned to nothing, as a subdomain of a decomposed grid is
        dict(ragged, name="compress_ragged", op="compress"),
        dict(ragged, name="decompress_ragged", op="decompress"),
        # the benchmark's large 3D snapshot
        dict(nyx, name="compress_large", op="compress"),
        dict(nyx, name="decompress_large", op="decompress"),
        # a field that hardly compresses: outliers everywhere, long codewords
        dict(spiky, name="decompress_spiky", op="decompress"),
        # a mixed set of 1D, 2D and 3D fields (particle arrays among them), each with its own bound
        dict(batch, name="compress_batch", op="batch_compress"),
        dict(batch, name="decompress_batch", op="batch_decompress"),
        # a field in the caller's host memory, there and back over the link
        {"name": "compress_host", "op": "host_compress", "dims": "256x256x256", "kind": "grf", "mode": "r2r",
         "eb": 1e-3, "dict": 1024},
    ]


def _dims_of(nd, n, u):
    """About n elements in nd dimensions at aspect ratios drawn by u(a, b)."""
    if nd == 1:
        return (n,)
    if nd == 2:
        d0 = max(1, round(n ** u(0.25, 0.75)))
        return (d0, max(1, round(n / d0)))
    w = [u(0.5, 1.5) for _ in range(3)]
    d0, d1 = (max(1, round(n ** (v / sum(w)))) for v in w[:2])
    return (d0, d1, max(1, round(n / (d0 * d1))))


def _log_uniform(u, a, b):
    return math.exp(u(math.log(a), math.log(b)))


def draw(rng):
    u = rng.uniform
    op = rng.choice(["compress"] * 4 + ["decompress"] * 4 + ["batch_compress", "batch_decompress", "host_compress"])
    if op.startswith("batch"):
        return {"op": op, "fields": rng.randint(4, 60), "n_min": 1 << 14, "n_max": round(_log_uniform(u, 1 << 17, 1 << 22)),
                "shape_seed": rng.randrange(1 << 20), "dict": 1024}
    nd = rng.choice([1, 2, 2, 3, 3, 3])
    n = round(_log_uniform(u, 1 << 16, 1 << (24 if op == "host_compress" else 26)))
    # the wide dictionary and the loose bounds are for fields of some size
    c = {"op": op, "dims": "x".join(map(str, _dims_of(nd, n, u))), "kind": "grf", "mode": "r2r",
         "eb": round(_log_uniform(u, 1e-5, 1e-2 if n >= 1 << 19 else 3e-4), 8),
         "dict": rng.choice([1024, 1024, 4096]) if n >= 1 << 21 else 1024}
    if nd == 2 and n >= 1 << 19 and rng.random() < 0.5:
        c.update(kind="bump", mode="abs", eb=max(c["eb"], 1e-4))
    elif nd == 3 and rng.random() < 0.1:
        c.update(kind="spiky", mode="abs", eb=1e-6)
    return c


def _dims(case):
    return tuple(int(v) for v in case["dims"].split("x"))


def _batch_cases(case):
    """The fields of a batch: 1D / 2D / 3D at 20 / 40 / 40 %, sizes and bounds log-uniform."""
    r = random.Random(case["shape_seed"])
    out = []
    for _ in range(case["fields"]):
        nd = r.choice([1, 2, 2, 3, 3])
        n = round(_log_uniform(r.uniform, case["n_min"], case["n_max"]))
        out.append({"dims": "x".join(map(str, _dims_of(nd, n, r.uniform))),
                    "kind": "bump" if nd == 2 and r.random() < 0.5 else "grf", "mode": "r2r",
                    "eb": _log_uniform(r.uniform, 1e-5, 1e-2), "dict": case["dict"]})
    return out


def _elements(case):
    if "fields" in case:
        return sum(_elements(c) for c in _batch_cases(case))
    return math.prod(_dims(case))


def work(case):
    # a field is 4 bytes a value; its archive 4 where nothing compresses, else 6 to 8 bits a value
    n = _elements(case)
    return {"bytes": n * (8 if case.get("kind") == "spiky" else 5), "flops": 0}


# ---- inputs -----------------------------------------------------------------------------------

def _fft_size(n):
    """The next size with no prime factor above 7 (fast transforms)."""
    while True:
        m = n
        for p in (2, 3, 5, 7):
            while m % p == 0:
                m //= p
        if m == 1:
            return n
        n += 1


def _grf(shape, gen):
    full = [_fft_size(max(2, v)) for v in shape]
    k2 = torch.zeros((), device=DEV)
    for ax, m in enumerate(full):
        f = torch.fft.rfftfreq(m, device=DEV) if ax == len(full) - 1 else torch.fft.fftfreq(m, device=DEV)
        k2 = k2 + f.view([-1 if i == ax else 1 for i in range(len(full))]) ** 2
    k2.view(-1)[0] = 1.0
    amp = k2 ** (-11.0 / 12.0)
    amp.view(-1)[0] = 0.0
    spec = torch.complex(amp * torch.randn(amp.shape, generator=gen, device=DEV),
                         amp * torch.randn(amp.shape, generator=gen, device=DEV))
    g = torch.fft.irfftn(spec, s=full)[tuple(slice(0, v) for v in shape)]
    span = (g.max() - g.min()).clamp_min(1e-30)
    return torch.exp(g * (4.0 * math.log(10.0) / span))


def _bump(shape, gen):
    ny, nx = shape
    p = torch.rand((4, 64, 1, 1), generator=gen, device=DEV)
    yy = torch.arange(ny, device=DEV, dtype=torch.float32)[None, :, None]
    xx = torch.arange(nx, device=DEV, dtype=torch.float32)[None, None, :]
    s2 = 2 * (20 + 380 * p[2]) ** 2
    gy = torch.exp(-(yy - ny * p[0]) ** 2 / s2)[:, :, 0]
    gx = torch.exp(-(xx - nx * p[1]) ** 2 / s2)[:, 0, :] * torch.randn((64, 1), generator=gen, device=DEV)
    f = torch.zeros(shape, device=DEV)
    for i in range(64):
        f += gy[i][:, None] * gx[i][None, :]
    f += torch.rand(shape, generator=gen, device=DEV) * 1e-5
    return (f - f.min()) / (f.max() - f.min()).clamp_min(1e-30)


def _field(case, seed):
    """The case's field, flat, x fastest."""
    gen = torch.Generator(device=DEV).manual_seed(seed)
    shape = tuple(reversed(_dims(case)))
    if case["kind"] == "bump":
        return _bump(shape, gen).reshape(-1).contiguous()
    f = _grf(shape, gen).reshape(-1).contiguous()
    if case["kind"] == "spiky":
        at = torch.rand(f.shape, generator=gen, device=DEV) < 0.05
        f = torch.where(at, torch.tan(math.pi * (torch.rand(f.shape, generator=gen, device=DEV) - 0.5)) * 100 * f.std(), f)
    return f


# ---- the calls --------------------------------------------------------------------------------

def _codec(case):
    return V.DeviceCodec(_dims(case), eb=case["eb"], mode=case["mode"], dict_size=case["dict"])


def _batch(case, seed):
    fields = [{"x": _field(c, seed * 1009 + i), "dims": _dims(c), "eb": c["eb"], "mode": c["mode"], "dict_size": c["dict"]}
              for i, c in enumerate(_batch_cases(case))]
    return V.BatchCompressor(fields)


def prepare(case, seed):
    op = case["op"]
    if op == "compress":
        return {"op": op, "codec": _codec(case), "x": _field(case, seed), "front": _front_bytes(case)}
    if op == "decompress":
        codec = _codec(case)
        codec.compress(_field(case, seed))
        codec.prepare_decompress(codec.archive_bytes())
        return {"op": op, "codec": codec, "out": torch.empty(codec.n, dtype=torch.float32, device=DEV)}
    if op == "batch_compress":
        return {"op": op, "batch": _batch(case, seed), "front": [_front_bytes(c) for c in _batch_cases(case)]}
    if op == "batch_decompress":
        b = _batch(case, seed)
        b.compress()
        return {"op": op, "batch": V.BatchDecompressor([b.archive_bytes(i) for i in range(b.n)])}
    dims = _dims(case)
    p = V.make_params(case["eb"], case["mode"], case["dict"])
    cap = ctypes.c_size_t(0)
    L.check(L.lib().vsz_compress_host_bound(ctypes.byref(p), len(dims), L.dims_arg(dims), ctypes.byref(cap)))
    return {"op": op, "host": V.HostOp(), "params": p, "dims": dims, "front": _front_bytes(case),
            "x": _field(case, seed).cpu().pin_memory(),
            "archive": torch.zeros(cap.value, dtype=torch.uint8, pin_memory=True),
            "result": torch.zeros(8, dtype=torch.int64, pin_memory=True)}


def _front_bytes(case):
    """The front of an archive buffer that holds the whole archive: the buffers are sized for the
    worst case, 12 bytes a value; the archives take 1 to 10 bits a value, and more than two bytes
    only where outliers are common (tight bounds, spikes)."""
    n = math.prod(_dims(case))
    return (2 if case["eb"] >= 1e-4 else 6) * n // 8 * 8 + 65536


def _front(archive, nbytes):
    return archive[: min(archive.numel() // 8 * 8, nbytes)].view(torch.int64)


def run(state):
    op = state["op"]
    if op == "compress":
        c = state["codec"]
        c.compress(state["x"])
        return {"archive": _front(c.archive, state["front"]), "result": c.result}
    if op == "decompress":
        state["codec"].decompress(state["codec"].archive, state["out"])
        return state["out"]
    if op == "batch_compress":
        b = state["batch"]
        b.compress()
        return {"archives": [_front(a, n) for a, n in zip(b.archives, state["front"])], "results": b.results}
    if op == "batch_decompress":
        state["batch"].decompress()
        return list(state["batch"].outputs)
    h = state["host"]
    h.compress(state["params"], state["dims"], state["x"].data_ptr(), state["archive"].data_ptr(),
               state["archive"].numel(), state["result"].data_ptr())
    h.wait()  # the result record and the archive are on the host now
    return {"archive": _front(state["archive"], state["front"]), "result": state["result"]}


def _exact_field(case, seed):
    """The reconstruction in 64 bits: the format's quantization cell of each value times the cell
    width.  Cells are chosen by the format's rules: a single-precision product and rint, but the
    double product and round-half-away in the partial last group of 8 columns of a 3D row; the
    partial last group of a 2D row is stored as 0."""
    x = _field(case, seed)
    dims = _dims(case)
    eb = case["eb"]
    if case["mode"] == "r2r":
        eb = eb * float(x.max() - x.min())
    r = 1.0 / (2.0 * eb)
    s = torch.round(x * torch.tensor(r, dtype=torch.float32, device=DEV)).double().view(-1, dims[0])
    tail = dims[0] & ~7
    if len(dims) == 2:
        s[:, tail:] = 0
    elif len(dims) == 3:
        t = x.view(-1, dims[0])[:, tail:].double() * r
        s[:, tail:] = torch.sign(t) * torch.floor(t.abs() + 0.5)
    return (s * (2.0 * eb)).view(-1)


def exact(case, seed):
    if case["op"] == "decompress":
        return _exact_field(case, seed)
    if case["op"] == "batch_decompress":
        return [_exact_field(c, seed * 1009 + i) for i, c in enumerate(_batch_cases(case))]
    return None  # archives are bytes
