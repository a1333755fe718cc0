"""Performance cases of the cubelet compression path.

Each case is one call pattern of a program that uses the library: a single
cubelet compressed or restored (latency), a batch of them (throughput), a
large volume cut into overlapping cubelets, or a short stream of requests to
the serving loop.  listed() is the fixed set, draw() gives further cases of
the same ranges.

A case is a plain dict.  "kind" selects the call:

  compress       Context.compress (host array) or compress_device
  batch          Context.compress_prepared over `count` cubelets in HBM
  split          Context.compress_split over a device-resident volume
  restore        Context.decompress (host array) or decompress_batch of one
  restore_batch  Context.run_decompress over `count` results into HBM
  serve          Server.submit_* / wait over `count` requests

Shapes, types and parameters come from the case alone (`layout` seeds the
shapes of a batch), the contents from the seed, so a program that compresses
the same geometry again and again is what a repeated pass stands for.
"""
import ctypes
import functools
import math
import random

import numpy as np
import torch

from wavelets_gb300 import lib, params as P

WAVELETS = {"haar": P.HAAR, "cdf97": P.CDF97}
QUANTS = {"uniform": P.UNIFORM, "log": P.LOG, "lloyd": P.LLOYD}
TYPES = {"u8": lib.WL_U8, "u16": lib.WL_U16, "f32": lib.WL_F32}
ITEM = {"u8": 1, "u16": 2, "f32": 4}
AXES = (16, 32, 48, 64, 96, 128, 256)  # axis lengths of the mixed batch


# ---- the cases ---------------------------------------------------------------

def _one(kind, z, y, x, dtype, steps, wavelet="cdf97", quant="log", bins=256, keep=0.1,
         at="device", exact=False, two_d=False):
    return {"kind": kind, "z": z, "y": y, "x": x, "dtype": dtype, "sx": steps[0], "sy": steps[1],
            "sz": steps[2], "wavelet": wavelet, "quant": quant, "bins": bins, "keep": keep,
            "at": at, "exact_order": exact, "two_d": two_d}


def listed():
    return [
        # the smallest call: a 64 x 64 image tile in host memory, the library's
        # default parameters (a thumbnail, one tile of an interactive viewer)
        dict(_one("compress", 1, 64, 64, "u8", (-1, -1, -1), keep=0.5, at="host"),
             name="tile_64"),
        # one 2048 x 2048 8-bit image, eleven levels, already on the GPU
        dict(_one("compress", 1, 2048, 2048, "u8", (11, 11, 0)), name="image_2048"),
        # one float32 simulation volume, uniform quantizer
        dict(_one("compress", 256, 256, 256, "f32", (3, 3, 3), quant="uniform", bins=1024,
                  keep=0.05), name="volume_256"),
        # a microscope stack of no convenient size, 16-bit, from host memory
        dict(_one("compress", 93, 181, 147, "u16", (4, 4, 4), bins=512, at="host"),
             name="ragged_u16"),
        # the reference's float order (byte-identical files for an archive
        # that the reference must reproduce)
        dict(_one("compress", 160, 128, 192, "u8", (3, 3, 3), exact=True), name="reference_order"),
        # the mixed batch: 512 cubelets of uneven size and type, Lloyd quantizer
        {"name": "mixed_512", "kind": "batch", "count": 512, "layout": 20261205, "axes": "mixed",
         "low": 16, "high": 256, "quant": "lloyd", "bins": 256, "keep": 0.1},
        # a small batch of odd sizes, log quantizer: what a server collects
        {"name": "ragged_40", "kind": "batch", "count": 40, "layout": 40, "axes": "any",
         "low": 16, "high": 200, "quant": "log", "bins": 256, "keep": 0.1},
        # a 2 GiB scan cut into 128^3 cubelets with 8 voxels of overlap
        {"name": "split_1024", "kind": "split", "side": 1024, "cube": 128, "overlap": 8,
         "steps": 4, "quant": "log", "bins": 512, "keep": 0.03},
        # restoring the image into a host array, the volume into HBM, and the
        # mixed batch into HBM
        dict(_one("restore", 1, 2048, 2048, "u8", (11, 11, 0), at="host"), name="restore_image"),
        dict(_one("restore", 256, 256, 256, "f32", (3, 3, 3), quant="uniform", bins=1024,
                  keep=0.05), name="restore_volume"),
        {"name": "restore_512", "kind": "restore_batch", "count": 512, "layout": 20261205,
         "axes": "mixed", "low": 16, "high": 256, "quant": "lloyd", "bins": 256, "keep": 0.1},
        # the serving loop: 24 requests of different sizes, a fifth of them
        # decompressions, submitted together and waited for
        {"name": "serve_24", "kind": "serve", "count": 24, "layout": 24, "low": 16, "high": 256,
         "quant": "log", "bins": 256, "keep": 0.1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("image", "compress", "compress", "batch", "batch", "split", "restore",
                       "restore_batch", "serve"))
    quant = rng.choice(("log", "log", "uniform", "lloyd"))
    bins = rng.choice((64, 100, 256, 512, 1024)) + rng.randrange(3)
    keep = rng.choice((0.03, 0.05, 0.1, 0.1, 0.2, 0.5))
    wavelet = rng.choice(("haar", "cdf97", "cdf97"))
    if kind == "image" or (kind == "restore" and rng.random() < 0.5):
        y, x = _log(rng, 64, 2048), _log(rng, 64, 2048)
        return _one("restore" if kind == "restore" else "compress", 1, y, x,
                    rng.choice(("u8", "u8", "u16", "f32")),
                    rng.choice(((-1, -1, 0), (4, 4, 0), (3, 2, 0))), wavelet, quant, bins, keep,
                    rng.choice(("host", "device")),
                    kind == "image" and rng.random() < 0.15, rng.random() < 0.2)
    if kind in ("compress", "restore"):
        z, y, x = (_log(rng, 16, 300) for _ in range(3))
        s = tuple(rng.randrange(1, 5) for _ in range(3))
        return _one(kind, z, y, x, rng.choice(("u8", "u16", "f32")), s, wavelet, quant, bins, keep,
                    rng.choice(("host", "device")), kind == "compress" and rng.random() < 0.15)
    if kind == "split":
        cube = rng.choice((64, 96, 128))
        return {"kind": "split", "side": _log(rng, 160, 800), "cube": cube, "overlap": 8,
                "steps": rng.randrange(2, 5), "quant": rng.choice(("log", "uniform")),
                "bins": bins, "keep": keep}
    if kind == "serve":
        return {"kind": "serve", "count": rng.randrange(6, 25), "layout": rng.randrange(1 << 30),
                "low": 16, "high": _log(rng, 64, 256), "quant": "log", "bins": bins, "keep": keep}
    axes = rng.choice(("mixed", "any"))
    return {"kind": kind, "count": _log(rng, 4, 400 if axes == "mixed" else 120),
            "layout": rng.randrange(1 << 30), "axes": axes, "low": 16,
            "high": 256 if axes == "mixed" else _log(rng, 48, 256), "quant": quant, "bins": bins,
            "keep": keep}


# ---- shapes and contents -----------------------------------------------------

def _params(wavelet, steps, quant, bins, keep, exact=False, two_d=False):
    return P.Params(steps=tuple(steps), wavelet=WAVELETS[wavelet],
                    threshold_fraction=float(np.float32(1.0 - keep)), bin_count=bins,
                    quant_alg=QUANTS[quant], exact_transform=exact, transform_2d=two_d)


def _layout(case):
    """(shape (z, y, x), type, wavelet, steps) of every cubelet of a batch or
    request of a stream."""
    r = random.Random(case["layout"])
    out = []
    for i in range(case["count"]):
        if case["kind"] == "serve":
            shape = tuple(_log(r, case["low"], case["high"]) for _ in range(3))
            out.append((shape, ("u8", "u16", "f32")[i % 3], "cdf97", (3, 3, 3)))
            continue
        if case["axes"] == "mixed":
            shape = tuple(r.choice(AXES) for _ in range(3))
        else:
            shape = tuple(_log(r, case["low"], case["high"]) for _ in range(3))
        u = r.random()
        s = int(math.floor(math.log2(min(shape)))) - 2
        out.append((shape, "u8" if u < 0.5 else "u16" if u < 0.8 else "f32",
                    r.choice(("haar", "cdf97")), (s, s, s)))
    return out


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7fffffffffffffff)
    return g


def _blobs(g, shape, count, sigma, amp, noise):
    """Sum of `count` axis-aligned Gaussian blobs plus white noise, float32."""
    f = []
    for n in shape:
        c = torch.rand(count, 1, generator=g, device="cuda") * n
        s = sigma[0] + (sigma[1] - sigma[0]) * torch.rand(count, 1, generator=g, device="cuda")
        f.append(torch.exp(-0.5 * ((torch.arange(n, device="cuda") - c) / s) ** 2))
    a = amp[0] + (amp[1] - amp[0]) * torch.rand(count, 1, generator=g, device="cuda")
    zy = ((a * f[0])[:, :, None] * f[1][:, None, :]).reshape(count, -1)
    v = (zy.T @ f[2]).reshape(shape)
    return v.add_(torch.randn(shape, generator=g, device="cuda"), alpha=noise)


def _typed(v, dtype, scale):
    """The volume in its type; integers scaled to the type's range, or (scale
    False) rounded and clipped.  16-bit values are kept as int16 bits."""
    if dtype == "f32":
        return v.contiguous()
    top = 255.0 if dtype == "u8" else 65535.0
    if scale:
        lo, hi = v.min(), v.max()
        v = (v - lo) * (top / (hi - lo).clamp_min(1e-20))
    v = v.round_().clamp_(0.0, top)
    return v.to(torch.uint8) if dtype == "u8" else v.to(torch.int32).to(torch.int16)


def _contents(shape, dtype, seed):
    """One cubelet on the GPU: an image of blobs, a gradient and noise, or a
    volume of blobs and noise scaled to its type."""
    g = _gen(seed)
    if shape[0] == 1:
        n = max(shape)
        v = _blobs(g, shape, 64, (n / 256.0, n / 8.0), (20.0, 120.0), 3.0)
        ramp = torch.rand(2, generator=g, device="cuda") * 80.0 - 40.0
        v += ramp[0] * torch.linspace(0, 1, shape[1], device="cuda")[None, :, None]
        v += ramp[1] * torch.linspace(0, 1, shape[2], device="cuda")[None, None, :]
        if dtype == "u16":
            v *= 256.0
        return _typed(v, dtype, False)
    small = min(shape)
    return _typed(_blobs(g, shape, 12 if small < 200 else 200,
                         (2.0, max(2.0, small / (2.0 if small < 200 else 4.0))), (-1.0, 1.0), 0.01),
                  dtype, True)


def _phantom(side, seed):
    """Forty ellipsoids of constant density, later ones over earlier ones, plus
    noise; unsigned 16-bit values as int16 bits."""
    g = _gen(seed)
    r = random.Random(seed)
    v = torch.zeros((side,) * 3, device="cuda")
    for _ in range(40):
        c = [r.uniform(0.15, 0.85) * side for _ in range(3)]
        d = [r.uniform(0.03, 0.3) * side for _ in range(3)]
        lo = [max(0, int(a - b)) for a, b in zip(c, d)]
        hi = [min(side, int(a + b) + 2) for a, b in zip(c, d)]
        q = [((torch.arange(l, h, device="cuda") - a) / b) ** 2
             for l, h, a, b in zip(lo, hi, c, d)]
        inside = q[0][:, None, None] + q[1][None, :, None] + q[2][None, None, :] <= 1.0
        v[lo[0]:hi[0], lo[1]:hi[1], lo[2]:hi[2]].masked_fill_(inside, r.uniform(0, 4095))
    out = torch.empty((side,) * 3, dtype=torch.int16, device="cuda")
    for z in range(0, side, 64):
        part = v[z:z + 64]
        part += 20.0 * torch.randn(part.shape, generator=g, device="cuda")
        out[z:z + 64] = part.round_().clamp_(0, 65535).to(torch.int32).to(torch.int16)
    return out


def _host(t):
    """The tensor as the numpy array a caller holds (unsigned 16-bit view)."""
    a = t.cpu().numpy()
    return a.view(np.uint16) if a.dtype == np.int16 else a


def _batch_tensors(case, seed):
    return [_contents(shape, dt, seed * 4099 + i)
            for i, (shape, dt, _, _) in enumerate(_layout(case))]


def _split_origins(case):
    """Offset and length of the cubelets along one axis."""
    n, c, o = case["side"], case["cube"], case["overlap"]
    return [(k * (c - o), min(c, n - k * (c - o))) for k in range((n - o - 1) // (c - o) + 1)]


# ---- states ------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _context():
    return lib.Context(0)


@functools.lru_cache(maxsize=None)
def _server():
    # three lanes, one of them for small requests, bounded batches: the
    # configuration that the serving benchmark uses
    return lib.Server(lanes=3, max_batch_bytes=32 << 20, express_lanes=1)


def _case_params(case):
    return _params(case["wavelet"], (case["sx"], case["sy"], case["sz"]), case["quant"],
                   case["bins"], case["keep"], case["exact_order"], case["two_d"])


def _batch_items(case, tensors):
    return [(t.data_ptr(), TYPES[dt], shape[::-1],
             _params(w, steps, case["quant"], case["bins"], case["keep"]))
            for t, (shape, dt, w, steps) in zip(tensors, _layout(case))]


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "ctx": _context()}
    if kind not in ("restore", "restore_batch"):
        s["words"] = np.zeros(_room(case), np.int32)
        count = len(_split_origins(case)) ** 3 if kind == "split" else case.get("count", 1)
        s["tables"] = np.zeros(count * (6 * case["bins"] + 8), np.int32)
    if kind in ("compress", "restore"):
        t = _contents((case["z"], case["y"], case["x"]), case["dtype"], seed)
        s["params"] = _case_params(case)
        s["at"] = case["at"]
        if kind == "compress" and case["at"] == "host":
            s["array"] = _host(t)
        else:
            s["data"], s["dtype"] = t, TYPES[case["dtype"]]
            s["size"] = (case["x"], case["y"], case["z"])
        torch.cuda.synchronize()
        if kind == "restore":
            s["packed"] = s["ctx"].compress_device(t.data_ptr(), s["dtype"], s["size"], s["params"])
            s["out"] = torch.zeros_like(s.pop("data"))
    elif kind in ("batch", "restore_batch"):
        tensors = _batch_tensors(case, seed)
        torch.cuda.synchronize()
        pb = s["ctx"].prepare_batch(_batch_items(case, tensors), on_device=True)
        if kind == "batch":
            s["data"], s["batch"] = tensors, pb
        else:
            # one buffer for each type, the cubelets back to back in it
            types = [dt for _, dt, _, _ in _layout(case)]
            sizes = [(t.numel() * t.element_size() + 255) // 256 * 256 for t in tensors]
            at = {"u8": 0, "u16": 0, "f32": 0}
            where = []
            for dt, n in zip(types, sizes):
                where.append(at[dt])
                at[dt] += n
            tensors = None
            out = {dt: torch.zeros(n, dtype=torch.uint8, device="cuda") for dt, n in at.items() if n}
            s["packed"] = s["ctx"].compress_prepared(pb)
            s["prepared"] = s["ctx"].prepare_decompress(
                s["packed"], device_outs=[out[dt].data_ptr() + w for dt, w in zip(types, where)])
            s["out"] = {dt: o.view(torch.float32) if dt == "f32" else
                        o.view(torch.int16) if dt == "u16" else o for dt, o in out.items()}
            torch.cuda.synchronize()
    elif kind == "split":
        s["data"] = _phantom(case["side"], seed)
        # compress_split takes the geometry from an array and the data from ptr
        s["shape"] = np.broadcast_to(np.zeros((), np.uint16), (case["side"],) * 3)
        s["params"] = _params("cdf97", (case["steps"],) * 3, case["quant"], case["bins"],
                              case["keep"])
        s["cube"], s["overlap"] = (case["cube"],) * 3, case["overlap"]
    else:  # serve
        s["server"] = _server()
        tensors = _batch_tensors(case, seed)
        torch.cuda.synchronize()
        s["requests"] = []
        for i, (t, (shape, dt, w, steps)) in enumerate(zip(tensors, _layout(case))):
            p = _params(w, steps, case["quant"], case["bins"], case["keep"])
            a = _host(t)
            # page-locked, as a server's receive buffers are
            view = torch.zeros(a.nbytes, dtype=torch.uint8, pin_memory=True).numpy()
            view = view.view(a.dtype).reshape(a.shape)
            if i % 5 == 4:
                c = s["ctx"].compress_device(t.data_ptr(), TYPES[dt], shape[::-1], p)
                s["requests"].append(("restore", c, view))
            else:
                view[...] = a
                s["requests"].append(("compress", view, p))
    return s


# ---- passes ------------------------------------------------------------------
# A program takes the compressed words out of the library's storage into a
# buffer of its own (an archive block, a send buffer) and lets the results go.
# The buffers are sized for any contents of the geometry and start as zeros.

class _Storage:
    """Bytes [lo, hi) of the results' storage as int32; holds the results."""

    def __init__(self, lo, hi, owner):
        self.owner = owner
        self.__array_interface__ = {"version": 3, "shape": ((hi - lo) // 4,), "typestr": "<i4",
                                    "data": (lo, False)}


def _room(case):
    """int32 words set aside for the codes of a case: 24 bits for each kept
    coefficient and one for each voxel."""
    return int(_voxels(case) * (0.75 * case["keep"] + 0.03125)) + 8192


def _take(state, name, array):
    """`array` at the start of the state's buffer of that name."""
    buf, n = state[name], array.size
    if n < 1 << 20:
        buf[:n] = array
    else:  # copied by several host threads
        torch.from_numpy(buf)[:n].copy_(torch.from_numpy(array))
    return buf


def _span(arrays, owner):
    """The arrays after each other: a view where the library left them that
    way, else a copy."""
    total = sum(a.nbytes for a in arrays)
    lo = arrays[0].__array_interface__["data"][0]
    hi = arrays[-1].__array_interface__["data"][0] + arrays[-1].nbytes
    if hi - lo == total:
        return np.asarray(_Storage(lo, hi, owner))
    return np.concatenate([a.view(np.int32) for a in arrays])


_FIELDS = np.dtype({
    "names": ["words", "n_words", "decode", "n_decode", "n_boundaries", "n_values", "threshold",
              "max_value", "min_coef", "max_coef", "longest", "zero_bin"],
    "formats": ["u8", "i4", "u8", "i4", "i4", "i4"] + ["f4"] * 4 + ["i4"] * 2,
    "offsets": [getattr(lib.WlResult, f).offset for f in (
        "words", "n_words", "decode", "n_decode", "n_boundaries", "n_values", "threshold_value",
        "max_value", "min_coef", "max_coef", "longest_code", "zero_bin")],
    "itemsize": ctypes.sizeof(lib.WlResult)})


def _regions(rec, name, sizes, owner):
    """Per-cubelet regions of `sizes` int32 from the pointers in rec[name],
    after each other."""
    p, n = rec[name], sizes.astype(np.uint64) * 4
    lo, hi = int(p[0]), int(p[-1] + n[-1])
    if hi - lo == int(n.sum()):
        return np.asarray(_Storage(lo, hi, owner))
    return np.concatenate([np.asarray(_Storage(int(a), int(a + b), owner)) for a, b in zip(p, n)])


def _packed(state, c):
    """One compressed cubelet: words, decode table, codebook, numbers."""
    return {"words": _take(state, "words", c.words.view(np.int32)),
            "tables": _take(state, "tables", np.concatenate(
                [c.decode, c.boundaries.view(np.int32), c.values.view(np.int32)])),
            "stats": np.array([c.threshold_value, c.max_value, c.min_coef, c.max_coef], np.float32),
            "whole": np.array([c.words.size, c.decode.size, c.longest_code, c.zero_bin])}


def _packed_batch(state, rb):
    """A batch's results, read from the library's structs."""
    rec = np.frombuffer(rb.outs, _FIELDS, count=len(rb))
    tables = rec["n_decode"] + rec["n_boundaries"] + rec["n_values"]  # one region per cubelet
    return {"words": _take(state, "words", _regions(rec, "words", rec["n_words"], rb)),
            "tables": _take(state, "tables", _regions(rec, "decode", tables, rb)),
            "stats": np.stack([rec["threshold"], rec["max_value"], rec["min_coef"],
                               rec["max_coef"]], 1),
            "whole": np.stack([rec["n_words"], rec["n_decode"], rec["longest"],
                               rec["zero_bin"]], 1)}


def _packed_list(state, res):
    """A batch's results from Compressed objects (no codebooks)."""
    return {"words": _take(state, "words", _span([c.words for c in res], res)),
            "tables": _take(state, "tables", _span([c.decode for c in res], res)),
            "stats": np.array([(c.threshold_value, c.max_value, c.min_coef, c.max_coef)
                               for c in res], np.float32),
            "whole": np.array([(c.words.size, c.decode.size, c.longest_code, c.zero_bin)
                               for c in res])}


def run(state):
    kind, ctx = state["kind"], state["ctx"]
    if kind == "compress":
        if state["at"] == "host":
            return _packed(state, ctx.compress(state["array"], state["params"]))
        return _packed(state, ctx.compress_device(state["data"].data_ptr(), state["dtype"],
                                                  state["size"], state["params"]))
    if kind == "batch":
        return _packed_batch(state, ctx.compress_prepared(state["batch"], lazy=True))
    if kind == "split":
        _, res = ctx.compress_split(state["shape"], state["cube"], state["overlap"],
                                    state["params"], ptr=state["data"].data_ptr(), on_device=True)
        return _packed_list(state, res)
    if kind == "restore":
        if state["at"] == "host":
            out = ctx.decompress(state["packed"])
            return out.view(np.int16) if out.dtype == np.uint16 else out
        ctx.decompress_batch([state["packed"]], device_outs=[state["out"].data_ptr()])
        return state["out"]
    if kind == "restore_batch":
        ctx.run_decompress(state["prepared"])
        return state["out"]
    srv = state["server"]
    tickets = [srv.submit_compress(r[1], r[2]) if r[0] == "compress" else
               srv.submit_decompress(r[1], r[2]) for r in state["requests"]]
    got = [srv.wait(t)[0] for t in tickets]
    got = [c for c in got if c is not None]
    return dict(_packed_list(state, got),
                restored=[r[2].view(np.int16) if r[2].dtype == np.uint16 else r[2]
                          for r in state["requests"] if r[0] == "restore"])


# ---- what a pass cannot do without -------------------------------------------

def _cost(voxels, nbytes, keep):
    # about one byte of code for each kept coefficient and a quarter of one
    # for the zero runs between them; per axis and level a lifting pair is
    # four multiply-adds with an addition, and a scale, over a geometric
    # series of levels
    return {"bytes": nbytes + 1.25 * keep * voxels, "flops": 42.0 * voxels}


def _voxels(case):
    if case["kind"] in ("compress", "restore"):
        return case["z"] * case["y"] * case["x"]
    if case["kind"] == "split":
        return sum(n for _, n in _split_origins(case)) ** 3
    return sum(math.prod(shape) for shape, _, _, _ in _layout(case))


def work(case):
    kind = case["kind"]
    if kind in ("compress", "restore"):
        v = _voxels(case)
        return _cost(v, v * ITEM[case["dtype"]], case["keep"])
    if kind == "split":
        return _cost(_voxels(case), 2 * case["side"] ** 3, case["keep"])
    items = [(math.prod(shape), ITEM[dt]) for shape, dt, _, _ in _layout(case)]
    return _cost(sum(v for v, _ in items), sum(v * b for v, b in items), case["keep"])


# ---- 64-bit values -----------------------------------------------------------

def _axis64(v, steps, wavelet):
    """`steps` analysis levels along the last axis, in float64: four lifting
    steps with whole-sample mirroring and the scale K, or the orthonormal
    Haar butterfly."""
    n = v.shape[-1]
    for _ in range(steps):
        e, o = v[..., 0:n:2].clone(), v[..., 1:n:2].clone()
        if wavelet == "haar":
            lo, hi = (e + o) * math.sqrt(0.5), (e - o) * math.sqrt(0.5)
        else:
            after = lambda a: torch.cat([a[..., 1:], a[..., -1:]], -1)    # noqa: E731
            before = lambda a: torch.cat([a[..., :1], a[..., :-1]], -1)   # noqa: E731
            o += -1.586134342059924 * (e + after(e))
            e += -0.052980118572961 * (before(o) + o)
            o += 0.882911075530934 * (e + after(e))
            e += 0.443506852043971 * (before(o) + o)
            lo, hi = e * 1.149604398860241, o * (-1.0 / 1.149604398860241)
        v[..., :n // 2] = lo
        v[..., n // 2:n] = hi
        n //= 2
    return v


def _stats64(t, dtype, wavelet, steps, keep, two_d=False):
    """Threshold, largest |c|, smallest and largest coefficient of the
    transform of `t` in float64."""
    v = t.to(torch.float64)
    if dtype == "u16":
        v = torch.where(v < 0, v + 65536.0, v)
    most = [max(0, (n - 1).bit_length()) for n in v.shape[::-1]]
    st = [m if s < 0 or s > m else s for s, m in zip(steps, most)]
    for axis, s in zip((2, 1, 0), st):
        n = v.shape[axis]
        pad = (-n) % (1 << s)
        if pad:
            v = torch.cat([v, v.narrow(axis, n - 1, 1).expand(
                *[pad if a == axis else -1 for a in range(3)])], axis)
    for axis, s in zip((2, 1, 0), st):
        if s and not (two_d and axis == 0):
            v = _axis64(v.movedim(axis, 2).contiguous(), s, wavelet).movedim(2, axis)
    v = v.reshape(-1)
    a = v.abs().sort().values
    k = min(int(np.float32(np.float32(1.0 - keep)) * np.float32(a.numel())), a.numel() - 1)
    return torch.stack([a[k], a[-1], v.min(), v.max()]).cpu().numpy()


def _none(stats, **more):
    return dict(more, words=None, tables=None, stats=stats, whole=None)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("restore", "restore_batch"):
        return None
    if kind == "compress":
        t = _contents((case["z"], case["y"], case["x"]), case["dtype"], seed)
        return _none(_stats64(t, case["dtype"], case["wavelet"],
                              (case["sx"], case["sy"], case["sz"]), case["keep"], case["two_d"]))
    if kind == "split":
        v, at = _phantom(case["side"], seed), _split_origins(case)
        rows = [_stats64(v[z:z + d, y:y + h, x:x + w], "u16", "cdf97", (case["steps"],) * 3,
                         case["keep"]) for z, d in at for y, h in at for x, w in at]
        return _none(np.stack(rows))
    rows = [_stats64(_contents(shape, dt, seed * 4099 + i), dt, w, steps, case["keep"])
            for i, (shape, dt, w, steps) in enumerate(_layout(case))
            if kind != "serve" or i % 5 != 4]
    return _none(np.stack(rows), **({"restored": None} if kind == "serve" else {}))
