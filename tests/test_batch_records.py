"""Descriptions that the Python binding builds for the library, without a GPU:
the records hold what the items say, whatever object says it."""
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
