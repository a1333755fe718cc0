"""Python binding of libwlgpu's C ABI (include/wlgpu.h) through ctypes.

Arrays follow the reference's cube layout: a numpy array of shape
(depth, height, width) holds a cubelet whose x (width) index is fastest,
i.e. size = (X, Y, Z) = (shape[2], shape[1], shape[0]).

The compute path is the CUDA library only: if ``libwlgpu.so`` is missing or
no GPU is visible, these calls raise -- there is no CPU fallback.
"""
from __future__ import annotations

import ctypes
import dataclasses
import os
import struct
from typing import List, Optional, Sequence

import numpy as np

from . import params as P

HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(HERE, "_lib", "libwlgpu.so")

WL_OK, WL_EINVAL, WL_ENOMEM, WL_ETIMEOUT, WL_EFORMAT, WL_ECUDA, WL_EIO = range(7)
WL_U8, WL_I32, WL_F32, WL_U16 = 1, 2, 3, 4
STATUS_NAMES = {0: "OK", 1: "EINVAL", 2: "ENOMEM", 3: "ETIMEOUT", 4: "EFORMAT",
                5: "ECUDA", 6: "EIO"}

NP_TO_WL = {np.dtype(np.uint8): WL_U8, np.dtype(np.int32): WL_I32,
            np.dtype(np.float32): WL_F32, np.dtype(np.uint16): WL_U16}
WL_TO_NP = {v: k for k, v in NP_TO_WL.items()}


class WlParams(ctypes.Structure):
    _fields_ = [("steps", ctypes.c_int * 3), ("wavelet", ctypes.c_int),
                ("threshold_fraction", ctypes.c_float), ("bin_count", ctypes.c_int),
                ("quant_alg", ctypes.c_int), ("compress_zeros", ctypes.c_int),
                ("lloyd_iters", ctypes.c_int), ("exact_transform", ctypes.c_int),
                ("transform_2d", ctypes.c_int)]


class WlResult(ctypes.Structure):
    _fields_ = [("size", ctypes.c_int * 3), ("original_size", ctypes.c_int * 3),
                ("original_dtype", ctypes.c_int), ("steps", ctypes.c_int * 3),
                ("wavelet", ctypes.c_int), ("quant_alg", ctypes.c_int),
                ("bin_count", ctypes.c_int), ("threshold_fraction", ctypes.c_float),
                ("threshold_value", ctypes.c_float), ("max_value", ctypes.c_float),
                ("min_coef", ctypes.c_float), ("max_coef", ctypes.c_float),
                ("zero_bin", ctypes.c_int), ("dup_key", ctypes.c_int),
                ("dup_value", ctypes.c_int), ("longest_code", ctypes.c_int),
                ("n_words", ctypes.c_int), ("words", ctypes.POINTER(ctypes.c_uint32)),
                ("n_decode", ctypes.c_int), ("decode", ctypes.POINTER(ctypes.c_int32)),
                ("n_boundaries", ctypes.c_int), ("n_values", ctypes.c_int),
                ("boundaries", ctypes.POINTER(ctypes.c_float)),
                ("values", ctypes.POINTER(ctypes.c_float)),
                ("owner", ctypes.c_void_p), ("transform_2d", ctypes.c_int)]


class WlCubelet(ctypes.Structure):
    _fields_ = [("data", ctypes.c_void_p), ("dtype", ctypes.c_int),
                ("size", ctypes.c_int * 3), ("params", WlParams),
                ("row_pitch", ctypes.c_longlong), ("slice_pitch", ctypes.c_longlong)]


REQ_COMPRESS, REQ_DECOMPRESS = 1, 2


class WlServeConfig(ctypes.Structure):
    _fields_ = [("lanes", ctypes.c_int), ("memory_budget", ctypes.c_size_t),
                ("max_batch", ctypes.c_int), ("stage_host_inputs", ctypes.c_int),
                ("max_batch_bytes", ctypes.c_size_t), ("express_lanes", ctypes.c_int),
                ("small_request_bytes", ctypes.c_size_t), ("express_priority", ctypes.c_int)]


class WlRequest(ctypes.Structure):
    _fields_ = [("kind", ctypes.c_int), ("cubelet", WlCubelet),
                ("compressed", ctypes.POINTER(WlResult)), ("out_dtype", ctypes.c_int),
                ("out", ctypes.c_void_p), ("out_on_device", ctypes.c_int)]


class WlContainerStats(ctypes.Structure):
    _fields_ = [("cubelets", ctypes.c_int), ("copied", ctypes.c_int),
                ("bytes_in", ctypes.c_ulonglong), ("bytes_out", ctypes.c_ulonglong),
                ("seconds", ctypes.c_double), ("read_seconds", ctypes.c_double),
                ("compute_seconds", ctypes.c_double), ("write_seconds", ctypes.c_double)]


class WlOptPoint(ctypes.Structure):
    _fields_ = [("threshold_fraction", ctypes.c_float), ("bin_count", ctypes.c_int),
                ("size_bytes", ctypes.c_int), ("psnr", ctypes.c_float)]


class WlErrorStats(ctypes.Structure):
    _fields_ = [("count", ctypes.c_longlong), ("average_error", ctypes.c_float),
                ("l1", ctypes.c_float), ("l2", ctypes.c_float), ("mse", ctypes.c_float),
                ("psnr", ctypes.c_float), ("relative_error", ctypes.c_float),
                ("sum_value", ctypes.c_double), ("sum_value_squared", ctypes.c_double),
                ("sum_diff", ctypes.c_double), ("sum_diff_squared", ctypes.c_double)]

    def as_dict(self):
        return {k: getattr(self, k) for k, _ in self._fields_}


class WlRequestInfo(ctypes.Structure):
    _fields_ = [("status", ctypes.c_int), ("queue_ms", ctypes.c_double),
                ("service_ms", ctypes.c_double), ("total_ms", ctypes.c_double),
                ("batch_size", ctypes.c_int), ("lane", ctypes.c_int)]


EXPORTS = {
    "wl_params_default": (None, [ctypes.POINTER(WlParams)]),
    "wl_result_free": (None, [ctypes.POINTER(WlResult)]),
    "wl_init": (ctypes.c_int, [ctypes.c_int, ctypes.POINTER(ctypes.c_void_p)]),
    "wl_destroy": (None, [ctypes.c_void_p]),
    "wl_last_error": (ctypes.c_char_p, [ctypes.c_void_p]),
    "wl_compress_cubelet": (ctypes.c_int, [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int,
                                           ctypes.POINTER(ctypes.c_int), ctypes.c_int,
                                           ctypes.POINTER(WlParams), ctypes.POINTER(WlResult)]),
    "wl_compress_batch": (ctypes.c_int, [ctypes.c_void_p, ctypes.POINTER(WlCubelet), ctypes.c_int,
                                         ctypes.c_int, ctypes.POINTER(WlResult)]),
    "wl_decompress_cubelet": (ctypes.c_int, [ctypes.c_void_p, ctypes.POINTER(WlResult),
                                             ctypes.c_int, ctypes.c_void_p, ctypes.c_int]),
    "wl_compress_file": (ctypes.c_int, [ctypes.c_void_p, ctypes.c_char_p, ctypes.c_char_p,
                                        ctypes.POINTER(WlParams)]),
    "wl_decompress_file": (ctypes.c_int, [ctypes.c_void_p, ctypes.c_char_p, ctypes.c_char_p]),
    "wl_encode_cube": (ctypes.c_int, [ctypes.POINTER(WlResult), ctypes.c_int,
                                      ctypes.POINTER(ctypes.POINTER(ctypes.c_uint8)),
                                      ctypes.POINTER(ctypes.c_size_t)]),
    "wl_free": (None, [ctypes.c_void_p]),
    "wl_last_timings": (ctypes.c_int, [ctypes.c_void_p, ctypes.POINTER(ctypes.c_float)]),
    "wl_sync": (ctypes.c_int, [ctypes.c_void_p]),
    "wl_forward_transform": (ctypes.c_int, [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int,
                                            ctypes.POINTER(ctypes.c_int), ctypes.POINTER(WlParams),
                                            ctypes.c_void_p, ctypes.c_size_t,
                                            ctypes.POINTER(ctypes.c_int)]),
    "wl_inverse_transform": (ctypes.c_int, [ctypes.c_void_p, ctypes.c_void_p,
                                            ctypes.POINTER(ctypes.c_int), ctypes.POINTER(ctypes.c_int),
                                            ctypes.c_int, ctypes.POINTER(ctypes.c_int),
                                            ctypes.c_int, ctypes.c_void_p]),
    "wl_device_alloc": (ctypes.c_void_p, [ctypes.c_size_t]),
    "wl_device_free": (None, [ctypes.c_void_p]),
    "wl_copy_to_device": (ctypes.c_int, [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_size_t]),
    "wl_copy_to_host": (ctypes.c_int, [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_size_t]),
    "wl_last_launch_count": (ctypes.c_int, [ctypes.c_void_p]),
    "wl_set_profiling": (ctypes.c_int, [ctypes.c_void_p, ctypes.c_int]),
    "wl_kernel_timings": (ctypes.c_int, [ctypes.c_void_p, ctypes.POINTER(ctypes.c_float)]),
    "wl_select_threshold_noalloc": (ctypes.c_int, [ctypes.c_void_p, ctypes.c_longlong,
                                                   ctypes.c_float, ctypes.c_void_p,
                                                   ctypes.c_void_p]),
    "wl_host_alloc": (ctypes.c_void_p, [ctypes.c_size_t]),
    "wl_host_free": (None, [ctypes.c_void_p]),
    "wl_serve_config_default": (None, [ctypes.POINTER(WlServeConfig)]),
    "wl_serve_create": (ctypes.c_int, [ctypes.c_int, ctypes.POINTER(WlServeConfig),
                                       ctypes.POINTER(ctypes.c_void_p)]),
    "wl_serve_submit": (ctypes.c_int, [ctypes.c_void_p, ctypes.POINTER(WlRequest),
                                       ctypes.POINTER(ctypes.c_ulonglong)]),
    "wl_serve_wait": (ctypes.c_int, [ctypes.c_void_p, ctypes.c_ulonglong, ctypes.c_int,
                                     ctypes.POINTER(WlResult), ctypes.POINTER(WlRequestInfo)]),
    "wl_serve_submit_batch": (ctypes.c_int, [ctypes.c_void_p, ctypes.POINTER(WlRequest),
                                             ctypes.c_int, ctypes.POINTER(ctypes.c_ulonglong)]),
    "wl_serve_wait_batch": (ctypes.c_int, [ctypes.c_void_p, ctypes.POINTER(ctypes.c_ulonglong),
                                           ctypes.c_int, ctypes.POINTER(WlResult),
                                           ctypes.POINTER(ctypes.c_int)]),
    "wl_set_host_input_mode": (ctypes.c_int, [ctypes.c_void_p, ctypes.c_int]),
    "wl_serve_last_error": (ctypes.c_char_p, [ctypes.c_void_p]),
    "wl_serve_destroy": (None, [ctypes.c_void_p]),
    "wl_results_free": (None, [ctypes.POINTER(WlResult), ctypes.c_int]),
    "wl_decompress_batch": (ctypes.c_int, [ctypes.c_void_p, ctypes.POINTER(WlResult), ctypes.c_int,
                                           ctypes.POINTER(ctypes.c_int),
                                           ctypes.POINTER(ctypes.c_void_p), ctypes.c_int]),
    "wl_compress_container": (ctypes.c_int, [ctypes.c_void_p, ctypes.c_char_p, ctypes.c_char_p,
                                             ctypes.POINTER(WlParams), ctypes.c_size_t,
                                             ctypes.POINTER(WlContainerStats)]),
    "wl_decompress_container": (ctypes.c_int, [ctypes.c_void_p, ctypes.c_char_p,
                                               ctypes.c_char_p, ctypes.c_size_t,
                                               ctypes.POINTER(WlContainerStats)]),
    "wl_optimize": (ctypes.c_int, [ctypes.c_void_p, ctypes.c_void_p, ctypes.POINTER(ctypes.c_int),
                                   ctypes.c_int, ctypes.POINTER(WlParams),
                                   ctypes.POINTER(WlOptPoint), ctypes.c_int,
                                   ctypes.POINTER(ctypes.c_int)]),
    "wl_optimize_file": (ctypes.c_int, [ctypes.c_void_p, ctypes.c_char_p,
                                        ctypes.POINTER(WlParams), ctypes.POINTER(WlOptPoint),
                                        ctypes.c_int, ctypes.POINTER(ctypes.c_int)]),
    "wl_autotune": (ctypes.c_int, [ctypes.c_void_p, ctypes.c_int, ctypes.c_int]),
    "wl_tune_export": (ctypes.c_int, [ctypes.c_char_p, ctypes.c_size_t,
                                      ctypes.POINTER(ctypes.c_size_t)]),
    "wl_tune_import": (ctypes.c_int, [ctypes.c_char_p]),
    "wl_tune_reset": (None, []),
    "wl_set_graph_mode": (ctypes.c_int, [ctypes.c_void_p, ctypes.c_int]),
    "wl_set_encode_slices": (ctypes.c_int, [ctypes.c_void_p, ctypes.c_int]),
    "wl_set_token_chunk": (ctypes.c_int, [ctypes.c_void_p, ctypes.c_int]),
    "wl_graph_stats": (ctypes.c_int, [ctypes.c_void_p, ctypes.POINTER(ctypes.c_longlong)]),
    "wl_graph_error": (ctypes.c_char_p, [ctypes.c_void_p]),
    "wl_error_metrics": (ctypes.c_int, [ctypes.c_void_p, ctypes.POINTER(WlResult),
                                        ctypes.c_void_p, ctypes.c_int, ctypes.c_int,
                                        ctypes.c_float, ctypes.POINTER(WlErrorStats)]),
    "wl_set_memory_limit": (ctypes.c_int, [ctypes.c_void_p, ctypes.c_size_t]),
    "wl_set_stream_priority": (ctypes.c_int, [ctypes.c_void_p, ctypes.c_int]),
    "wl_memory_held": (ctypes.c_size_t, [ctypes.c_void_p]),
    "wl_error_metrics_file": (ctypes.c_int, [ctypes.c_void_p, ctypes.c_char_p, ctypes.c_char_p,
                                             ctypes.POINTER(WlErrorStats)]),
}

_lib = None


def load(path: str = LIB_PATH):
    """Load libwlgpu.so (built by wavelets_gb300.build.build())."""
    global _lib
    if _lib is not None:
        return _lib
    if not os.path.exists(path):
        raise RuntimeError(f"libwlgpu.so not built ({path}); run wavelets_gb300.build.build()")
    lib = ctypes.CDLL(path)
    for name, (res, args) in EXPORTS.items():
        fn = getattr(lib, name)
        fn.restype = res
        fn.argtypes = args
    _lib = lib
    return lib


class WlError(RuntimeError):
    def __init__(self, status, msg):
        super().__init__(f"{STATUS_NAMES.get(status, status)}: {msg}")
        self.status = status


def make_params(p: Optional[P.Params] = None) -> WlParams:
    p = p or P.Params()
    w = WlParams()
    w.steps[:] = [int(s) for s in p.steps]
    w.wavelet = int(p.wavelet)
    w.threshold_fraction = float(p.threshold_fraction)
    w.bin_count = int(p.bin_count)
    w.quant_alg = int(p.quant_alg)
    w.compress_zeros = 1 if p.compress_zeros else 0
    w.lloyd_iters = int(p.lloyd_iters)
    w.exact_transform = 1 if p.exact_transform else 0
    w.transform_2d = 1 if getattr(p, "transform_2d", False) else 0
    return w


class _ParamsBytes:
    """make_params as bytes, made once for items in a row with the same object
    and the same values (items of one call often share their parameters, and
    an object may change between items)."""

    def __init__(self):
        self.p, self.values, self.made = self, None, b""

    def __call__(self, p: Optional[P.Params]) -> bytes:
        if p is self.p and (p is None or vars(p) == self.values):
            return self.made
        self.made = bytes(make_params(p))
        # values that can change in place are not compared
        fixed = p is None or (type(p) is P.Params and type(p.steps) is tuple)
        self.p, self.values = (p if fixed else self), (dict(vars(p)) if fixed and p else None)
        return self.made


def _addr(a: np.ndarray) -> int:
    return a.__array_interface__["data"][0]


@dataclasses.dataclass
class Compressed:
    """A compressed cubelet (copy of a wl_result)."""
    size: tuple              # stored (rotated) width, height, depth
    original_size: tuple     # X, Y, Z
    original_dtype: int
    steps: tuple
    wavelet: int
    quant_alg: int
    bin_count: int
    threshold_fraction: float
    threshold_value: float
    max_value: float
    min_coef: float
    max_coef: float
    zero_bin: int
    dup_key: int
    dup_value: int
    longest_code: int
    words: np.ndarray
    decode: np.ndarray
    boundaries: np.ndarray
    values: np.ndarray
    transform_2d: bool = False  # 2-D mode: size is the padded (x, y, z), not rotated

    @classmethod
    def from_struct(cls, r: WlResult) -> "Compressed":
        def arr(ptr, n, dt):
            if n <= 0 or not ptr:
                return np.zeros(0, dt)
            a = np.empty(n, dt)
            ctypes.memmove(a.ctypes.data, ctypes.cast(ptr, ctypes.c_void_p).value, a.nbytes)
            return a
        return cls(tuple(r.size), tuple(r.original_size), r.original_dtype, tuple(r.steps),
                   r.wavelet, r.quant_alg, r.bin_count, r.threshold_fraction,
                   r.threshold_value, r.max_value, r.min_coef, r.max_coef, r.zero_bin,
                   r.dup_key, r.dup_value, r.longest_code,
                   arr(r.words, r.n_words, np.uint32), arr(r.decode, r.n_decode, np.int32),
                   arr(r.boundaries, r.n_boundaries, np.float32),
                   arr(r.values, r.n_values, np.float32), bool(r.transform_2d))

    def _record(self):
        """The WlResult field values over this object's arrays, and those
        arrays."""
        keep = w, d, b, v = (np.ascontiguousarray(self.words, np.uint32),
                             np.ascontiguousarray(self.decode, np.int32),
                             np.ascontiguousarray(self.boundaries, np.float32),
                             np.ascontiguousarray(self.values, np.float32))
        return (self.size, self.original_size, self.original_dtype,
                self.steps, self.wavelet, self.quant_alg, self.bin_count,
                self.threshold_fraction, self.threshold_value, self.max_value, self.min_coef,
                self.max_coef, self.zero_bin, self.dup_key, self.dup_value, self.longest_code,
                w.size, _addr(w), d.size, _addr(d), b.size, v.size, _addr(b),
                _addr(v), 0, 1 if self.transform_2d else 0), keep

    def to_struct(self):
        """A WlResult pointing into this object's arrays (keep self alive)."""
        rec, self._keep = self._record()
        return _result_array([rec])[0]

    @property
    def compressed_bytes(self) -> int:
        return int(self.words.size) * 4


def _size_of(arr: np.ndarray):
    a = arr if arr.ndim == 3 else arr.reshape((1,) * (3 - arr.ndim) + arr.shape)
    Z, Y, X = a.shape
    return (X, Y, Z)


class _ResultsOwner:
    """Releases the library results whose arrays numpy views point into."""

    def __init__(self, lib, outs, n):
        self.lib, self.outs, self.n = lib, outs, n

    def __del__(self):
        try:
            self.lib.wl_results_free(self.outs, self.n)
        except Exception:
            pass


class PreparedBatch:
    """A batch description (the wl_cubelet array) built once and compressed
    any number of times: inputs that stay at the same addresses -- pinned
    staging buffers, device arrays -- are described once, so a call costs
    only the library's own work."""

    def __init__(self, cubs, n, on_device, keep):
        self.cubs, self.n, self.on_device, self._keep = cubs, n, on_device, keep


class ResultBatch:
    """The results of one compression call, left in the library's structs
    until asked for: results() makes the Compressed objects (zero-copy),
    release() frees them without looking."""

    def __init__(self, lib, outs, n):
        self.lib, self.outs, self.n = lib, outs, n
        self._live = True

    def __len__(self):
        return self.n

    def compressed_bytes(self) -> int:
        rec = np.frombuffer(self.outs, _result_dtype_cached(), count=self.n)
        return int(rec["n_words"].astype(np.int64).sum()) * 4

    def results(self) -> List["Compressed"]:
        assert self._live, "results already taken or released"
        self._live = False
        return adopt_results(self.lib, self.outs, self.n)

    def release(self):
        if self._live:
            self._live = False
            self.lib.wl_results_free(self.outs, self.n)

    def __del__(self):
        try:
            self.release()
        except Exception:
            pass


def _result_dtype():
    """numpy mirror of WlResult for vectorised field access."""
    names, formats, offsets = [], [], []
    for name, ct in WlResult._fields_:
        f = getattr(WlResult, name)
        if name in ("words", "decode", "boundaries", "values", "owner"):
            fmt = np.uint64
        elif isinstance(ct, type) and issubclass(ct, ctypes.Array):
            fmt = (np.int32, (ct._length_,))
        elif ct is ctypes.c_float:
            fmt = np.float32
        else:
            fmt = np.int32
        names.append(name)
        formats.append(fmt)
        offsets.append(f.offset)
    return np.dtype({"names": names, "formats": formats, "offsets": offsets,
                     "itemsize": ctypes.sizeof(WlResult)})


_RESULT_DT = None
def _packer(t) -> struct.Struct:
    """The layout of a ctypes structure as a struct format: a pointer is an
    address, an array its elements, a structure its bytes."""
    codes = {ctypes.c_int: "i", ctypes.c_float: "f", ctypes.c_longlong: "q"}
    fmt, end = "=", 0
    for name, ct in t._fields_:
        f = getattr(t, name)
        if issubclass(ct, ctypes.Array):
            code = codes[ct._type_] * ct._length_
        elif issubclass(ct, ctypes.Structure):
            code = f"{ctypes.sizeof(ct)}s"
        else:
            code = codes.get(ct, "Q")
        fmt += f"{f.offset - end}x{code}"
        end = f.offset + f.size
    return struct.Struct(fmt + f"{ctypes.sizeof(t) - end}x")


_PACK_CUBELET, _PACK_RESULT = _packer(WlCubelet).pack, _packer(WlResult).pack


def _cubelet_array(rows):
    """The WlCubelet array of (data, dtype, size, params bytes, row pitch,
    slice pitch) rows.  Integers are packed at once; anything else goes in
    field by field, which takes and refuses what ctypes does (pointer objects
    and None, no fractions, no sizes of another length)."""
    n = len(rows)
    try:
        return (WlCubelet * n).from_buffer(bytearray().join(
            [_PACK_CUBELET(d, t, x, y, z, p, r, s) for d, t, (x, y, z), p, r, s in rows]))
    except (struct.error, OverflowError, TypeError, ValueError):
        pass
    cubs = (WlCubelet * n)()
    for c, (ptr, dt, size, prm, row_pitch, slice_pitch) in zip(cubs, rows):
        c.data, c.dtype = ptr, dt
        c.size[:] = size
        c.params = WlParams.from_buffer_copy(prm)
        c.row_pitch, c.slice_pitch = row_pitch, slice_pitch
    return cubs


def _result_array(recs):
    """The WlResult array of Compressed._record values (see _cubelet_array)."""
    n = len(recs)
    try:
        return (WlResult * n).from_buffer(bytearray().join(
            [_PACK_RESULT(x, y, z, ox, oy, oz, t, sx, sy, sz, *rest)
             for (x, y, z), (ox, oy, oz), t, (sx, sy, sz), *rest in recs]))
    except (struct.error, OverflowError, TypeError, ValueError):
        pass
    rs = (WlResult * n)()
    for r, rec in zip(rs, recs):
        for (name, ct), value in zip(WlResult._fields_, rec):
            if issubclass(ct, ctypes.Array):
                getattr(r, name)[:] = value
            elif issubclass(ct, ctypes._Pointer):
                setattr(r, name, ctypes.cast(value, ct))
            else:
                setattr(r, name, value)
    return rs


def _result_dtype_cached():
    global _RESULT_DT
    if _RESULT_DT is None:
        _RESULT_DT = _result_dtype()
    return _RESULT_DT


_SCALARS = ("original_dtype", "wavelet", "quant_alg", "bin_count", "threshold_fraction",
            "threshold_value", "max_value", "min_coef", "max_coef", "zero_bin", "dup_key",
            "dup_value", "longest_code")


def _int32_view(lo, hi, owner):
    """The bytes [lo, hi) at an address as int32; the array holds owner."""
    buf = (ctypes.c_char * (hi - lo)).from_address(lo)
    buf._owner = owner
    return np.frombuffer(buf, np.int32)


def adopt_results(lib, outs, n) -> List["Compressed"]:
    """Compressed objects over the results' arrays without copying them.  The
    library keeps a batch's arrays in one block; the numpy views hold a
    reference that releases the results when the last view goes away."""
    rec = np.frombuffer(outs, _result_dtype_cached(), count=n)
    cnts = np.stack([rec["n_words"], rec["n_decode"], rec["n_boundaries"], rec["n_values"]],
                    1).astype(np.uint64)
    ptrs = np.stack([rec["words"], rec["decode"], rec["boundaries"], rec["values"]], 1)
    used = (cnts > 0) & (ptrs != 0)
    slab = rec["owner"]
    if n == 0 or not used.any() or not slab.all():
        res = [Compressed.from_struct(outs[i]) for i in range(n)]
        lib.wl_results_free(outs, n)
        return res
    # one view per storage block (a pipelined batch has several); all views
    # share the owner that releases the batch's results
    owner = _ResultsOwner(lib, outs, n)
    starts = np.where(used, ptrs, np.uint64(1 << 63))
    ends = np.where(used, ptrs + 4 * cnts, np.uint64(0))
    base, rows = [], np.empty(n, np.uint64)
    for sid in dict.fromkeys(slab.tolist()):
        sel = slab == sid
        lo, hi = int(starts[sel].min()), int(ends[sel].max())
        view = _int32_view(lo, hi, owner) if hi > lo else np.zeros(0, np.int32)
        base.append((view.view(np.uint32), view, view.view(np.float32)))
        rows[sel] = lo
        if sel.all():
            block = [0] * n
            break
        if len(base) == 1:
            block = np.zeros(n, np.int64)
        block[sel] = len(base) - 1
    first = np.where(used, (ptrs - rows[:, None]) // 4, 0).astype(np.int64)
    last = first + np.where(used, cnts, 0).astype(np.int64)

    def views(kind, column):  # the arrays of one kind, a slice each
        if not used[:, column].any():
            return [base[0][kind][:0]] * n
        lo, hi = first[:, column].tolist(), last[:, column].tolist()
        if len(base) == 1:
            v = base[0][kind]
            return [v[x:y] for x, y in zip(lo, hi)]
        return [base[k][kind][x:y] for k, x, y in zip(block, lo, hi)]

    cols = [rec[k].tolist() for k in _SCALARS]
    sizes, originals, steps = (map(tuple, rec[k].tolist())
                               for k in ("size", "original_size", "steps"))
    return list(map(Compressed, sizes, originals, cols[0], steps, *cols[1:], views(0, 0),
                    views(1, 1), views(2, 2), views(2, 3), rec["transform_2d"].astype(bool).tolist()))


def _adopt_one(lib, r: WlResult) -> "Compressed":
    """adopt_results for one result, without the array work of a batch."""
    n = (r.n_words, r.n_decode, r.n_boundaries, r.n_values)
    outs = (WlResult * 1).from_buffer(r)
    rec = np.frombuffer(r, _result_dtype_cached())
    p = rec[["words", "decode", "boundaries", "values"]].item()
    if not r.owner or not any(n):
        res = Compressed.from_struct(r)
        lib.wl_results_free(outs, 1)
        return res
    owner = _ResultsOwner(lib, outs, 1)
    a = [_int32_view(q, q + 4 * k, owner) if k > 0 and q else _EMPTY for q, k in zip(p, n)]
    c = Compressed.__new__(Compressed)
    d = c.__dict__
    for k in _SCALARS:
        d[k] = getattr(r, k)
    d["size"], d["original_size"] = tuple(r.size), tuple(r.original_size)
    d["steps"], d["transform_2d"] = tuple(r.steps), bool(r.transform_2d)
    d["words"], d["decode"] = a[0].view(np.uint32), a[1]
    d["boundaries"], d["values"] = a[2].view(np.float32), a[3].view(np.float32)
    return c


_EMPTY = np.zeros(0, np.int32)


class Context:
    """A libwlgpu context (one CUDA stream + device workspace) on one GPU."""

    def __init__(self, device: int = 0):
        self.lib = load()
        h = ctypes.c_void_p()
        st = self.lib.wl_init(device, ctypes.byref(h))
        if st != WL_OK:
            raise WlError(st, f"wl_init(device={device}) failed")
        self.h = h

    def close(self):
        if getattr(self, "h", None):
            self.lib.wl_destroy(self.h)
            self.h = None

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass

    def _check(self, st):
        if st != WL_OK:
            raise WlError(st, self.lib.wl_last_error(self.h).decode())

    def compress(self, arr, params: Optional[P.Params] = None, ptr: Optional[int] = None,
                 dtype: Optional[int] = None, size=None) -> Compressed:
        """Compress one cubelet given as a numpy array, or as a raw pointer
        (host or device: set ``ptr`` plus ``dtype``/``size`` and pass
        ``arr=None``; device pointers use compress_device)."""
        return self._compress(arr, params, ptr, dtype, size, on_device=False)

    def compress_device(self, ptr: int, dtype: int, size, params=None) -> Compressed:
        return self._compress(None, params, ptr, dtype, size, on_device=True)

    def _compress(self, arr, params, ptr, dtype, size, on_device):
        if arr is not None:
            a = np.ascontiguousarray(arr)
            dtype = NP_TO_WL[a.dtype]
            size = _size_of(a)
            ptr = a.ctypes.data
        sz = (ctypes.c_int * 3)(*size)
        res = WlResult()
        st = self.lib.wl_compress_cubelet(self.h, ctypes.c_void_p(ptr), dtype, sz,
                                          1 if on_device else 0, ctypes.byref(make_params(params)),
                                          ctypes.byref(res))
        self._check(st)
        return _adopt_one(self.lib, res)

    def prepare_batch(self, items: Sequence, params=None, on_device: bool = False,
                      raw: bool = False) -> PreparedBatch:
        """Describe a batch once (see compress_batch for items)."""
        n = len(items)
        keep, rows, params_bytes = [], [], _ParamsBytes()
        for it in items:
            pitch = (0, 0)
            if raw or on_device:
                ptr, dt, size, prm = it[:4]
                if len(it) > 4:  # (row pitch, slice pitch) of a sub-volume
                    pitch = it[4]
            else:
                if isinstance(it, tuple):
                    a, prm = it
                else:
                    a, prm = it, params
                a = np.ascontiguousarray(a)
                keep.append(a)
                ptr, dt, size = a.ctypes.data, NP_TO_WL[a.dtype], _size_of(a)
            prm = prm if prm is not None else params
            rows.append((ptr, dt, tuple(size), params_bytes(prm), pitch[0], pitch[1]))
        return PreparedBatch(_cubelet_array(rows), n, on_device, keep)

    def compress_prepared(self, pb: PreparedBatch, lazy: bool = False):
        """Compress a prepared batch; lazy returns a ResultBatch."""
        outs = (WlResult * pb.n)()
        st = self.lib.wl_compress_batch(self.h, pb.cubs, pb.n, 1 if pb.on_device else 0, outs)
        self._check(st)
        rb = ResultBatch(self.lib, outs, pb.n)
        return rb if lazy else rb.results()

    def compress_batch(self, items: Sequence, params=None, on_device: bool = False,
                       raw: bool = False) -> List[Compressed]:
        """items: list of numpy arrays, or (array, Params) pairs, or, with
        on_device/raw, (ptr, dtype, size, Params) tuples."""
        return self.compress_prepared(self.prepare_batch(items, params, on_device, raw))

    def compress_split(self, volume, cube=(128, 128, 128), overlap=8, params=None,
                       ptr=None, on_device=False):
        """Split a (Z, Y, X) volume into overlapping cubelets (the reference's
        `cube split`) and compress them in one batch, reading each cubelet in
        place from the volume (numpy array, or `ptr` to device / page-locked
        memory holding it).  Returns (grid, results) in the reference's
        cubelet order; grid holds (offset, size) in x, y, z order."""
        from wavelets_gb300.split import split_grid
        a = volume
        Z, Y, X = a.shape
        es = a.dtype.itemsize
        if ptr is None and not a.flags.c_contiguous:
            raise ValueError("volume must be C-contiguous")
        base = ptr if ptr is not None else a.ctypes.data
        grid = split_grid((X, Y, Z), cube, overlap)
        items = []
        for (ox, oy, oz), size in grid:
            off = (ox + X * (oy + Y * oz)) * es
            items.append((base + off, NP_TO_WL[a.dtype], size, params, (X, X * Y)))
        return grid, self.compress_batch(items, on_device=on_device, raw=not on_device)

    def decompress(self, c: Compressed, dtype=None) -> np.ndarray:
        """Restore a cubelet; dtype defaults to the original."""
        wl_dt = NP_TO_WL[np.dtype(dtype)] if dtype is not None else c.original_dtype
        X, Y, Z = c.original_size
        out = np.empty((Z, Y, X), WL_TO_NP[wl_dt])
        r = c.to_struct()
        st = self.lib.wl_decompress_cubelet(self.h, ctypes.byref(r), wl_dt,
                                            ctypes.c_void_p(out.ctypes.data), 0)
        self._check(st)
        return out

    def prepare_decompress(self, cs: Sequence[Compressed], dtypes=None, device_outs=None):
        """The wl_decompress_batch arguments for these results (reusable:
        run_decompress(prep) restores them again without rebuilding them)."""
        n = len(cs)
        recs = [c._record() for c in cs]
        rs = _result_array([rec for rec, _ in recs])
        keep = [arrays for _, arrays in recs]  # that the records point into
        outs, ptrs = [], (ctypes.c_void_p * n)()
        dts = (ctypes.c_int * n)()
        for i, c in enumerate(cs):
            wl_dt = (NP_TO_WL[np.dtype(dtypes[i])] if dtypes is not None and dtypes[i] is not None
                     else c.original_dtype)
            if device_outs is not None:
                ptrs[i] = device_outs[i]
            else:
                X, Y, Z = c.original_size
                o = np.empty((Z, Y, X), WL_TO_NP[wl_dt])
                outs.append(o)
                ptrs[i] = o.ctypes.data
            dts[i] = wl_dt
        return {"n": n, "rs": rs, "dts": dts, "ptrs": ptrs, "outs": outs, "keep": keep,
                "on_device": device_outs is not None}

    def run_decompress(self, prep):
        """One wl_decompress_batch call with prepared arguments."""
        self._check(self.lib.wl_decompress_batch(self.h, prep["rs"], prep["n"], prep["dts"],
                                                 prep["ptrs"], 1 if prep["on_device"] else 0))
        return None if prep["on_device"] else prep["outs"]

    def decompress_batch(self, cs: Sequence[Compressed], dtypes=None, device_outs=None):
        """Restore many cubelets in one batched call (dtypes default to each
        one's original).  With device_outs (one device address per cubelet,
        original_size elements of its type each) the cubelets are restored
        into device memory and nothing is returned; else into new arrays."""
        return self.run_decompress(self.prepare_decompress(cs, dtypes, device_outs))

    def forward_transform(self, arr, params: Optional[P.Params] = None):
        """Coefficients of the forward transform in the stored (rotated) order
        and the stored size (width, height, depth)."""
        a = np.ascontiguousarray(arr)
        size = _size_of(a)
        prm = params or P.Params()
        steps = P.clamp_steps(prm.steps, size)
        n = 1
        for s, L in zip(steps, size):
            n *= P.padded_length(L, s)
        out = np.empty(n, np.float32)
        stored = (ctypes.c_int * 3)()
        st = self.lib.wl_forward_transform(self.h, ctypes.c_void_p(a.ctypes.data),
                                           NP_TO_WL[a.dtype], (ctypes.c_int * 3)(*size),
                                           ctypes.byref(make_params(prm)),
                                           ctypes.c_void_p(out.ctypes.data), n, stored)
        self._check(st)
        return out, tuple(stored)

    def inverse_transform(self, coeffs, stored_size, steps, wavelet, original_size,
                          dtype=np.float32):
        c = np.ascontiguousarray(coeffs, np.float32)
        X, Y, Z = original_size
        out = np.empty((Z, Y, X), dtype)
        st = self.lib.wl_inverse_transform(self.h, ctypes.c_void_p(c.ctypes.data),
                                           (ctypes.c_int * 3)(*stored_size),
                                           (ctypes.c_int * 3)(*steps), int(wavelet),
                                           (ctypes.c_int * 3)(*original_size),
                                           NP_TO_WL[np.dtype(dtype)],
                                           ctypes.c_void_p(out.ctypes.data))
        self._check(st)
        return out

    def error_metrics(self, c: Compressed, original: np.ndarray, max_possible: float = 0.0):
        """The reference's -err metrics of a compressed cubelet against its
        original array (wl_error_metrics)."""
        a = np.ascontiguousarray(original)
        st = WlErrorStats()
        r = c.to_struct()
        self._check(self.lib.wl_error_metrics(self.h, ctypes.byref(r),
                                              ctypes.c_void_p(a.ctypes.data),
                                              NP_TO_WL[a.dtype], 0, ctypes.c_float(max_possible),
                                              ctypes.byref(st)))
        return st.as_dict()

    def error_metrics_file(self, original_path: str, compressed_path: str):
        st = WlErrorStats()
        self._check(self.lib.wl_error_metrics_file(self.h, original_path.encode(),
                                                   compressed_path.encode(), ctypes.byref(st)))
        return st.as_dict()

    def compress_file(self, inp: str, out: str, params: Optional[P.Params] = None):
        self._check(self.lib.wl_compress_file(self.h, inp.encode(), out.encode(),
                                              ctypes.byref(make_params(params))))

    def decompress_file(self, inp: str, out: str):
        self._check(self.lib.wl_decompress_file(self.h, inp.encode(), out.encode()))

    def timings(self):
        """Device time (ms) of the last compress: transform, select,
        quantize+count, Huffman build, encode, total."""
        t = (ctypes.c_float * 6)()
        self._check(self.lib.wl_last_timings(self.h, t))
        return list(t)

    def launch_count(self) -> int:
        return int(self.lib.wl_last_launch_count(self.h))

    def set_profiling(self, on: bool):
        self._check(self.lib.wl_set_profiling(self.h, 1 if on else 0))

    KERNEL_GROUPS = ("dwt_x", "dwt_y", "dwt_z", "select", "quant_setup", "quantize",
                     "runs", "huffman_build", "encode")

    def kernel_timings(self):
        t = (ctypes.c_float * 9)()
        self._check(self.lib.wl_kernel_timings(self.h, t))
        return dict(zip(self.KERNEL_GROUPS, list(t)))

    def sync(self):
        self._check(self.lib.wl_sync(self.h))

    def autotune(self, max_len: int = 0, reps: int = 0) -> str:
        """Time every tile height of every column-transform size class on
        this context's device and keep the fastest (process-wide); returns
        the table as text (see tune_table)."""
        self._check(self.lib.wl_autotune(self.h, int(max_len), int(reps)))
        return tune_table()

    def optimize(self, arr: np.ndarray, params: Optional[P.Params] = None):
        """The reference's -opt sweep on an 8-bit cubelet: a list of
        (threshold fraction, bin count, size in bytes, PSNR)."""
        a = np.ascontiguousarray(arr, np.uint8)
        sz = (ctypes.c_int * 3)(*_size_of(a))
        n = ctypes.c_int()
        prm = make_params(params)
        self._check(self.lib.wl_optimize(self.h, ctypes.c_void_p(a.ctypes.data), sz, 0,
                                         ctypes.byref(prm), None, 0, ctypes.byref(n)))
        pts = (WlOptPoint * n.value)()
        self._check(self.lib.wl_optimize(self.h, ctypes.c_void_p(a.ctypes.data), sz, 0,
                                         ctypes.byref(prm), pts, n.value, ctypes.byref(n)))
        return [(p.threshold_fraction, p.bin_count, p.size_bytes, p.psnr) for p in pts]

    def compress_container(self, in_path: str, out_path: str, params=None,
                           batch_bytes: int = 0) -> dict:
        """Compress every cubelet of a .cube file into a new .cube file
        (reading, GPU work and writing overlapped); returns the stage times."""
        st = WlContainerStats()
        self._check(self.lib.wl_compress_container(self.h, in_path.encode(), out_path.encode(),
                                                   ctypes.byref(make_params(params)),
                                                   int(batch_bytes), ctypes.byref(st)))
        return {k: getattr(st, k) for k, _ in WlContainerStats._fields_}

    def decompress_container(self, in_path: str, out_path: str, batch_bytes: int = 0) -> dict:
        """Restore every compressed cubelet of a .cube file into a new one."""
        st = WlContainerStats()
        self._check(self.lib.wl_decompress_container(self.h, in_path.encode(), out_path.encode(),
                                                     int(batch_bytes), ctypes.byref(st)))
        return {k: getattr(st, k) for k, _ in WlContainerStats._fields_}

    def set_host_input_mode(self, mode: int):
        """0: read page-locked host inputs in place; 1: copy them with the
        copy engine first."""
        self._check(self.lib.wl_set_host_input_mode(self.h, int(mode)))

    def set_memory_limit(self, nbytes: int):
        """Cap the context's device workspace (0: no cap); see wl_set_memory_limit."""
        self._check(self.lib.wl_set_memory_limit(self.h, nbytes))

    def memory_held(self) -> int:
        return self.lib.wl_memory_held(self.h)

    def set_encode_slices(self, slices: int):
        """Bit-packer lanes per 4096-element chunk (1, 2, 4, 8, 16, 32);
        0 = chunks and lanes chosen from the batch size.  The output does not depend on it."""
        self._check(self.lib.wl_set_encode_slices(self.h, int(slices)))

    def set_token_chunk(self, elements: int):
        """Elements per chunk of the quantizer and the bit packer (512, 1024,
        2048, 4096); 0 = by the size of the call.  The output does not depend
        on it."""
        self._check(self.lib.wl_set_token_chunk(self.h, int(elements)))

    def set_graph_mode(self, mode: int):
        """1: capture a batch geometry seen twice in a row as a CUDA graph
        and replay it; 0: always launch directly."""
        self._check(self.lib.wl_set_graph_mode(self.h, int(mode)))

    def graph_stats(self):
        t = (ctypes.c_longlong * 4)()
        self._check(self.lib.wl_graph_stats(self.h, t))
        out = dict(zip(("direct", "captures", "replays", "failed"), [int(x) for x in t]))
        err = self.lib.wl_graph_error(self.h)
        if err:
            out["error"] = err.decode()
        return out


TUNE_PASSES = ("fwd_x", "fwd_y", "fwd_z", "inv_z", "inv_y", "inv_x")


def tune_table() -> str:
    """The process-wide tile table: one line per tuned size class,
    "pass type class rows warps" and the microseconds of the six candidate
    shapes (TILE_SHAPES)."""
    lib = load()
    n = ctypes.c_size_t()
    st = lib.wl_tune_export(None, 0, ctypes.byref(n))
    if st:
        raise WlError(st, "tune export")
    buf = ctypes.create_string_buffer(n.value + 1)
    st = lib.wl_tune_export(buf, n.value + 1, ctypes.byref(n))
    if st:
        raise WlError(st, "tune export")
    return buf.value.decode()


def tune_load(text: str):
    """Install tile-table lines (as tune_table returns them)."""
    st = load().wl_tune_import(text.encode())
    if st:
        raise WlError(st, "malformed tile table")


def tune_reset():
    load().wl_tune_reset()


TILE_SHAPES = ((32, 4), (64, 4), (128, 4), (32, 8), (64, 8), (128, 8))


def tune_rows(text: str):
    """Parse a tile table: {(pass, type, class): ((rows, warps), times)} with
    the microseconds of the TILE_SHAPES candidates (0 = not measured)."""
    out = {}
    for ln in text.splitlines():
        f = ln.split()
        if len(f) >= 5:
            out[(int(f[0]), int(f[1]), int(f[2]))] = (
                (int(f[3]), int(f[4])), tuple(float(x) for x in f[5:11]))
    return out


def encode_cube(c: Compressed, footer: bool = False) -> bytes:
    """The .cube file bytes the reference would write for this cubelet."""
    lib = load()
    r = c.to_struct()
    buf = ctypes.POINTER(ctypes.c_uint8)()
    n = ctypes.c_size_t()
    st = lib.wl_encode_cube(ctypes.byref(r), 1 if footer else 0, ctypes.byref(buf), ctypes.byref(n))
    if st != WL_OK:
        raise WlError(st, "wl_encode_cube failed")
    data = ctypes.string_at(buf, n.value)
    lib.wl_free(buf)
    return data


class DeviceBuffer:
    """Device memory from wl_device_alloc."""

    def __init__(self, nbytes: int):
        self.lib = load()
        self.nbytes = nbytes
        self.ptr = self.lib.wl_device_alloc(nbytes)
        if not self.ptr:
            raise MemoryError("wl_device_alloc failed")

    def upload(self, arr: np.ndarray, offset: int = 0):
        a = np.ascontiguousarray(arr)
        assert offset + a.nbytes <= self.nbytes
        st = self.lib.wl_copy_to_device(ctypes.c_void_p(self.ptr + offset),
                                        ctypes.c_void_p(a.ctypes.data), a.nbytes)
        if st != WL_OK:
            raise WlError(st, "upload failed")

    def download(self, shape, dtype, offset: int = 0) -> np.ndarray:
        """A host copy of the bytes at offset as an array of shape and dtype."""
        out = np.empty(shape, dtype)
        assert offset + out.nbytes <= self.nbytes
        st = self.lib.wl_copy_to_host(ctypes.c_void_p(out.ctypes.data),
                                      ctypes.c_void_p(self.ptr + offset), out.nbytes)
        if st != WL_OK:
            raise WlError(st, "download failed")
        return out

    def free(self):
        if self.ptr:
            self.lib.wl_device_free(self.ptr)
            self.ptr = None

    def __del__(self):
        try:
            self.free()
        except Exception:
            pass


class PinnedBuffer:
    """Page-locked host memory from wl_host_alloc, viewable as numpy."""

    def __init__(self, nbytes: int):
        self.lib = load()
        self.nbytes = nbytes
        self.ptr = self.lib.wl_host_alloc(nbytes)
        if not self.ptr:
            raise MemoryError("wl_host_alloc failed")

    def array(self, dtype, shape):
        n = int(np.prod(shape)) * np.dtype(dtype).itemsize
        assert n <= self.nbytes
        buf = (ctypes.c_uint8 * n).from_address(self.ptr)
        return np.frombuffer(buf, dtype).reshape(shape)

    def free(self):
        if self.ptr:
            self.lib.wl_host_free(self.ptr)
            self.ptr = None

    def __del__(self):
        try:
            self.free()
        except Exception:
            pass


class Server:
    """The serving loop of libwlgpu: compress and decompress requests admitted
    as they arrive, batched continuously onto `lanes` concurrent lanes, gated
    by a device working-memory budget.  Inputs and outputs are kept alive here
    until their request has been waited for."""

    def __init__(self, lanes: int = 2, memory_budget: int = 16 << 30, max_batch: int = 1024,
                 device: int = 0, stage_host_inputs: bool = True, max_batch_bytes: int = 0,
                 express_lanes: int = 0, small_request_bytes: int = 4 << 20,
                 express_priority: bool = False):
        self.lib = load()
        cfg = WlServeConfig()
        self.lib.wl_serve_config_default(ctypes.byref(cfg))
        cfg.lanes, cfg.memory_budget, cfg.max_batch = lanes, memory_budget, max_batch
        cfg.stage_host_inputs = 1 if stage_host_inputs else 0
        cfg.max_batch_bytes = max_batch_bytes
        cfg.express_lanes = express_lanes
        cfg.small_request_bytes = small_request_bytes
        cfg.express_priority = 1 if express_priority else 0
        h = ctypes.c_void_p()
        st = self.lib.wl_serve_create(device, ctypes.byref(cfg), ctypes.byref(h))
        if st != WL_OK:
            raise WlError(st, f"wl_serve_create(device={device}) failed")
        self.h = h
        self._keep = {}

    def _submit(self, req, keep):
        t = ctypes.c_ulonglong()
        st = self.lib.wl_serve_submit(self.h, ctypes.byref(req), ctypes.byref(t))
        if st != WL_OK:
            raise WlError(st, self.lib.wl_serve_last_error(self.h).decode())
        self._keep[t.value] = (req, keep)
        return t.value

    def submit_compress(self, arr=None, params=None, ptr=None, dtype=None, size=None) -> int:
        """Compress a numpy array (host) or a raw (ptr, wl dtype, size) input."""
        req = WlRequest()
        req.kind = REQ_COMPRESS
        keep = None
        if arr is not None:
            keep = np.ascontiguousarray(arr)
            ptr, dtype, size = keep.ctypes.data, NP_TO_WL[keep.dtype], _size_of(keep)
        req.cubelet.data = ptr
        req.cubelet.dtype = dtype
        req.cubelet.size[:] = size
        req.cubelet.params = make_params(params)
        return self._submit(req, keep)

    def submit_batch(self, pb: "PreparedBatch") -> np.ndarray:
        """Queue every cubelet of a prepared batch back to back (a free lane
        takes them together); returns their tickets."""
        reqs = getattr(pb, "_reqs", None)
        if reqs is None:
            reqs = (WlRequest * pb.n)()
            for i in range(pb.n):
                reqs[i].kind = REQ_COMPRESS
                reqs[i].cubelet = pb.cubs[i]
            pb._reqs = reqs
        t = (ctypes.c_ulonglong * pb.n)()
        st = self.lib.wl_serve_submit_batch(self.h, reqs, pb.n, t)
        if st != WL_OK:
            raise WlError(st, self.lib.wl_serve_last_error(self.h).decode())
        return t

    def wait_batch(self, tickets) -> "ResultBatch":
        """Wait for the tickets of submit_batch; the results as a ResultBatch."""
        n = len(tickets)
        outs = (WlResult * n)()
        sts = (ctypes.c_int * n)()
        st = self.lib.wl_serve_wait_batch(self.h, tickets, n, outs, sts)
        rb = ResultBatch(self.lib, outs, n)
        if st != WL_OK:
            rb.release()
            raise WlError(st, self.lib.wl_serve_last_error(self.h).decode())
        return rb

    def submit_decompress(self, c: "Compressed", out: np.ndarray) -> int:
        """Restore `c` into the host array `out` (original size, any dtype)."""
        req = WlRequest()
        req.kind = REQ_DECOMPRESS
        r = c.to_struct()
        req.compressed = ctypes.pointer(r)
        req.out_dtype = NP_TO_WL[out.dtype]
        req.out = out.ctypes.data
        req.out_on_device = 0
        return self._submit(req, (c, r, out))

    def wait(self, ticket: int, timeout_ms: int = -1):
        """(Compressed or None, info dict); None while a poll finds it pending."""
        res = WlResult()
        info = WlRequestInfo()
        st = self.lib.wl_serve_wait(self.h, ticket, timeout_ms, ctypes.byref(res),
                                    ctypes.byref(info))
        if st == WL_ETIMEOUT:
            return None, None
        req, _ = self._keep.pop(ticket)
        if st != WL_OK:
            raise WlError(st, self.lib.wl_serve_last_error(self.h).decode())
        d = {k: getattr(info, k) for k, _ in WlRequestInfo._fields_}
        if req.kind == REQ_COMPRESS:
            return _adopt_one(self.lib, res), d
        return None, d

    def close(self):
        if getattr(self, "h", None):
            self.lib.wl_serve_destroy(self.h)
            self.h = None

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass
