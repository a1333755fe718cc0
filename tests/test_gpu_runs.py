"""Zero runs that cross chunks (4096 coefficients) and the ranges of 256 chunks
that one CTA joins: sparse cubelets of several such ranges, the tokens and the
stream exact against the oracle (huffman.h:31-57, 278-296)."""
import numpy as np
import pytest

from oracle import oracle
from wavelets_gb300 import lib, params as P

pytestmark = pytest.mark.gpu

C = 4096          # coefficients per chunk
R = 256 * C       # coefficients per CTA range
SHAPE = (5501, 9, 64)
N = 5501 * 9 * 64  # three ranges, five chunks and a partial one
assert N == 3 * R + 5 * C + 64 * 37

PLACES = {
    "first": [0],
    "last": [N - 1],
    "ends": [0, N - 1],
    "range_edges": [R - 1, R, 2 * R - 1, 2 * R, 3 * R],
    "before_edge": [R - 1, 3 * R - 1],
    "after_edge": [R, 3 * R],
    "far_apart": [5, 2 * R + 17],
    "one_per_range": [7, R + 9, 2 * R + 1030, 3 * R + C],
    "chunk_edges": [k * C for k in range(0, 700, 3)] + [k * C - 1 for k in range(1, 700, 5)],
    "eights": [R - 9, R, R + 9, R + 18, 2 * R - 8, 2 * R + 1, 2 * R + 10],
}


@pytest.fixture(scope="module")
def ctx():
    from wavelets_gb300 import build
    build.build()
    c = lib.Context(0)
    yield c
    c.close()


def _check(got, arr, p):
    want = oracle.encode(arr, p.threshold_fraction, p.bin_count, oracle.UNIFORM, True)
    assert list(got.decode) == list(want["decode"])
    assert np.array_equal(got.words, want["words"])


def _case(name):
    arr = np.zeros(N, np.float32)
    at = sorted(set(PLACES[name]))
    arr[at] = np.linspace(1.0, 2.0, len(at), dtype=np.float32)
    return arr.reshape(SHAPE)


PRM = P.Params(steps=(0, 0, 0), threshold_fraction=0.5, quant_alg=P.UNIFORM, bin_count=64)


@pytest.mark.parametrize("name", sorted(PLACES))
def test_sparse_cubelet(ctx, name):
    arr = _case(name)
    _check(ctx.compress(arr, PRM), arr, PRM)


def test_batch_of_uneven_cubelets(ctx):
    """CTA ranges of small cubelets beside those of a large one."""
    small, tiny = np.zeros((3, 5, 64), np.float32), np.zeros((1, 1, 7), np.float32)
    small[1, 2, 3] = 1.0
    tiny[0, 0, 6] = 2.0
    items = [(small, PRM), (_case("one_per_range"), PRM), (tiny, PRM)]
    for (arr, p), got in zip(items, ctx.compress_batch(items)):
        _check(got, arr, p)
