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
