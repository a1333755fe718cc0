"""The Huffman tree build against the oracle's priority queue
(huffman.cc:42-97): alphabets around the sizes where the build changes shape
(powers of two of the sort, the list one warp merges, the wide-CTA limit, one to
a few symbols) with
counts that tie, that grow geometrically (long codes, many merge rounds) and
that are random.  Decode table, longest code and stream are exact."""
import numpy as np
import pytest

from oracle import oracle
from wavelets_gb300 import lib, params as P

pytestmark = pytest.mark.gpu

BINS = (2, 3, 31, 32, 33, 63, 64, 65, 255, 256, 257, 511, 599, 600, 1023, 1024, 2047, 4096)


@pytest.fixture(scope="module")
def ctx():
    from wavelets_gb300 import build
    build.build()
    c = lib.Context(0)
    yield c
    c.close()


def _values(bins, counts, seed):
    """A float cubelet with about `bins` distinct values, value k counts[k] times."""
    rng = np.random.default_rng(seed)
    centre = -1.0 + 2.0 * (np.arange(bins) + 0.5) / bins
    v = np.repeat(centre, counts).astype(np.float32)
    rng.shuffle(v)
    return v.reshape(1, 1, -1)


def _counts(kind, bins, seed):
    rng = np.random.default_rng(seed)
    if kind == "ties":        # equal counts: only the index order decides
        return np.full(bins, 3)
    if kind == "few":         # small counts, many ties among leaves and merged nodes
        return rng.integers(0, 4, bins) + (np.arange(bins) == 0)
    if kind == "geometric":   # about Fibonacci: one pair or two a round
        return np.maximum(1, (1.5 ** rng.permutation(np.minimum(np.arange(bins), 26))).astype(int))
    return rng.integers(1, 200, bins)


@pytest.mark.parametrize("kind", ["ties", "few", "geometric", "random"])
@pytest.mark.parametrize("bins", BINS)
def test_tree_matches_oracle(ctx, bins, kind):
    arr = _values(bins, _counts(kind, bins, bins), bins)[..., :16000]
    for zeros in (True, False):
        p = P.Params(steps=(0, 0, 0), threshold_fraction=0.0, quant_alg=P.UNIFORM, bin_count=bins,
                     compress_zeros=zeros)
        got = ctx.compress(arr, p)
        want = oracle.encode(arr, 0.0, bins, oracle.UNIFORM, zeros)
        assert list(got.decode) == list(want["decode"])
        assert got.longest_code == want["longest"]
        assert np.array_equal(got.words, want["words"])


def test_batch_of_alphabets(ctx):
    """One call with every alphabet size: shared memory is sized for the
    largest, each cubelet builds its own."""
    items = []
    for i, bins in enumerate(BINS):
        arr = _values(bins, _counts("random", bins, i), i)[..., :16000]
        items.append((arr, P.Params(steps=(0, 0, 0), threshold_fraction=0.0, quant_alg=P.UNIFORM,
                                    bin_count=bins)))
    for (arr, p), got in zip(items, ctx.compress_batch(items)):
        want = oracle.encode(arr, 0.0, p.bin_count, oracle.UNIFORM, True)
        assert list(got.decode) == list(want["decode"])
        assert np.array_equal(got.words, want["words"])
