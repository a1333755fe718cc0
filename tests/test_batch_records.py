"""Descriptions that the Python binding builds for the library, without a GPU:
the records hold what the items say, whatever object says it."""
import ctypes

import numpy as np
import pytest

from wavelets_gb300 import lib, params as P


@pytest.fixture(scope="module")
def ctx():
    return lib.Context.__new__(lib.Context)  # describing needs no device


class Lazy:
    """A sequence that makes its items when they are asked for."""

    def __init__(self, n, make):
        self.n, self.make = n, make

    def __len__(self):
        return self.n

    def __getitem__(self, i):
        if i >= self.n:
            raise IndexError(i)
        return self.make(i)


def test_parameters_made_per_item(ctx):
    pb = ctx.prepare_batch(Lazy(50, lambda i: (4096, lib.WL_F32, (8, 8, 8),
                                               P.Params(bin_count=10 + i, steps=[i, 1, 2]))),
                           raw=True)
    assert [c.params.bin_count for c in pb.cubs] == list(range(10, 60))
    assert [list(c.params.steps) for c in pb.cubs] == [[i, 1, 2] for i in range(50)]
    pb = ctx.prepare_batch(Lazy(50, lambda i: (4096, lib.WL_F32, (8, 8, 8),
                                               P.Params(bin_count=10 + i))), raw=True)
    assert [c.params.bin_count for c in pb.cubs] == list(range(10, 60))


def test_parameters_changed_between_items(ctx):
    p = P.Params()

    def item(i):
        p.threshold_fraction = i / 50
        return 4096, lib.WL_F32, (8, 8, 8), p
    pb = ctx.prepare_batch(Lazy(50, item), raw=True)
    assert [c.params.threshold_fraction for c in pb.cubs] == [np.float32(i / 50) for i in range(50)]


def test_default_and_shared_parameters(ctx):
    q = P.Params(bin_count=33)
    a = np.zeros((2, 3, 4), np.uint8)
    pb = ctx.prepare_batch([(a, q), (a, None), a, (a, q)], params=P.Params(bin_count=44))
    assert [c.params.bin_count for c in pb.cubs] == [33, 44, 44, 33]
    assert [c.params.bin_count for c in ctx.prepare_batch([a, a]).cubs] == [256, 256]


def test_pointers_and_pitches(ctx):
    """Pointer objects and None are taken beside addresses, as ctypes takes
    them; every field reaches its place."""
    q = P.Params(bin_count=99)
    big = (1 << 64) - 4096
    pb = ctx.prepare_batch([(ctypes.c_void_p(8192), lib.WL_U8, (1, 2, 3), q),
                            (None, lib.WL_F32, [4, 5, 6], q),
                            (12288, lib.WL_U16, (7, 8, 9), q, (1 << 33, 1 << 40))], raw=True)
    assert [c.data for c in pb.cubs] == [8192, None, 12288]
    assert [c.dtype for c in pb.cubs] == [lib.WL_U8, lib.WL_F32, lib.WL_U16]
    assert [list(c.size) for c in pb.cubs] == [[1, 2, 3], [4, 5, 6], [7, 8, 9]]
    assert [(c.row_pitch, c.slice_pitch) for c in pb.cubs] == [(0, 0), (0, 0), (1 << 33, 1 << 40)]
    pb = ctx.prepare_batch([(big, lib.WL_I32, (1, 2, 3), q), (0, lib.WL_U8, (4, 5, 6), None)],
                           raw=True)
    assert [c.data for c in pb.cubs] == [big, None]
    assert [c.params.bin_count for c in pb.cubs] == [99, 256]
    assert [list(c.size) for c in pb.cubs] == [[1, 2, 3], [4, 5, 6]]


@pytest.mark.parametrize("item", [(4096, lib.WL_U8, (8.5, 8, 8)), (4096, lib.WL_U8, (8, 8)),
                                  (4096, lib.WL_U8, (8,)), (4096, lib.WL_U8, (8, 8, 8, 8)),
                                  (4096, 1.5, (8, 8, 8)), (4096.5, lib.WL_U8, (8, 8, 8)),
                                  ("4096", lib.WL_U8, (8, 8, 8)),
                                  (4096, lib.WL_U8, (8, 8, 8), None, (8.5, 64))])
def test_other_values_are_refused(ctx, item):
    q = P.Params()
    item = item if len(item) > 3 else item + (q,)
    good = (4096, lib.WL_U8, (8, 8, 8), q)
    for items in ([item], [good, item, good]):
        with pytest.raises((TypeError, ValueError)):
            ctx.prepare_batch(items, raw=True)


def compressed(**over):
    f = dict(size=(4, 5, 6), original_size=(6, 4, 5), original_dtype=lib.WL_F32, steps=(1, 2, 3),
             wavelet=P.CDF97, quant_alg=P.LLOYD, bin_count=9, threshold_fraction=0.5,
             threshold_value=0.25, max_value=3.5, min_coef=-2.5, max_coef=3.25, zero_bin=4,
             dup_key=9, dup_value=4, longest_code=7, words=np.arange(11, dtype=np.uint32),
             decode=np.arange(34, dtype=np.int32), boundaries=np.arange(8, dtype=np.float32),
             values=np.arange(9, dtype=np.float32), transform_2d=True)
    return lib.Compressed(**{**f, **over})


def fields(r):
    """A WlResult's values, its arrays as lists."""
    out = {}
    for name, ct in lib.WlResult._fields_:
        v = getattr(r, name)
        n = {"words": r.n_words, "decode": r.n_decode, "boundaries": r.n_boundaries,
             "values": r.n_values}.get(name)
        out[name] = v[:n] if n is not None else list(v) if hasattr(v, "__len__") else v
    return out


def test_result_records(ctx):
    c = compressed()
    got = fields(c.to_struct())
    assert got.pop("owner") is None
    for name, v in got.items():
        if name.startswith("n_"):
            assert v == getattr(c, {"n_words": "words", "n_decode": "decode",
                                    "n_boundaries": "boundaries", "n_values": "values"}[name]).size
        elif isinstance(v, list):
            assert v == [x for x in getattr(c, name)]
        else:
            assert v == getattr(c, name)
    rs = ctx.prepare_decompress([c, compressed(dup_key=-1, size=[7, 8, 9]), c])["rs"]
    assert fields(rs[0]) == fields(rs[2]) == fields(c.to_struct())
    assert rs[1].dup_key == -1 and list(rs[1].size) == [7, 8, 9]


@pytest.mark.parametrize("over", [dict(size=(4.5, 5, 6)), dict(size=(4, 5)), dict(steps=(1,)),
                                  dict(bin_count=8.5), dict(dup_key=None), dict(wavelet="2"),
                                  dict(threshold_value=None), dict(original_size=(1, 2, 3, 4))])
def test_result_values_refused(ctx, over):
    with pytest.raises((TypeError, ValueError)):
        compressed(**over).to_struct()


def test_converted_arrays_stay_alive(ctx):
    """Arrays of other types are converted; the copies live as long as the
    description, also of a result described twice."""
    c = compressed(words=list(range(11)), decode=np.arange(34.0), values=np.arange(18)[::2])
    prep = ctx.prepare_decompress([c, c], device_outs=[0, 0])
    c.to_struct()
    live = {a.__array_interface__["data"][0] for arrays in prep["keep"] for a in arrays}
    for r in prep["rs"]:
        for name in ("words", "decode", "boundaries", "values"):
            assert ctypes.cast(getattr(r, name), ctypes.c_void_p).value in live
        assert r.words[:11] == list(range(11)) and r.decode[:34] == list(range(34))
        assert r.values[:9] == [2.0 * k for k in range(9)]
