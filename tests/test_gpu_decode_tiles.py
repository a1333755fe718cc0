"""The tiled Huffman decoder on streams made by hand: code shapes that
resynchronise at once, late or never, codes longer than the lookup tables,
zero runs, and lengths around the tile (255 x 256 bits) and subsequence (256
bits) edges.  Expected values come from the oracle's bit-by-bit walk
(huffman.h:96-131); with no transform steps the restored floats are the
codebook values themselves, so they are compared exactly."""
import functools

import numpy as np
import pytest

from oracle import oracle
from wavelets_gb300 import lib, params as P

pytestmark = pytest.mark.gpu

TILE = 255 * 256  # bits


@pytest.fixture(scope="module")
def ctx():
    from wavelets_gb300 import build
    build.build()
    c = lib.Context(0)
    yield c
    c.close()


def _tree(shape):
    """Nested pairs with leaf numbers in left-to-right order."""
    kind, k = shape
    if kind == "flat":      # every code k bits: wrong starts never resynchronise
        def full(d, at):
            return at if d == 0 else (full(d - 1, at), full(d - 1, at + (1 << (d - 1))))
        return full(k, 0), 1 << k
    if kind == "comb":      # codes of 1, 2, .. k bits, two of k
        t = k
        for i in range(k - 1, -1, -1):
            t = (i, t)
        return t, k + 1
    if kind == "keys":      # the zero-run key (last leaf) has the one-bit code
        t = 0
        for i in range(1, k + 1):
            t = (i, t)
        return t, k + 1
    # mixed: a random tree of k leaves
    rng = np.random.default_rng(k)
    nodes = list(range(k))
    while len(nodes) > 1:
        i, j = rng.choice(min(len(nodes), 9), 2, replace=False)
        a, b = nodes[i], nodes[j]
        nodes = [x for m, x in enumerate(nodes) if m not in (i, j)] + [(a, b)]
    return nodes[0], k


@functools.lru_cache(maxsize=None)
def _code(shape):
    """Breadth-first decode table (computeDecodeTable), codes, leaf count."""
    tree, leaves = _tree(shape)
    order, codes, dec = [(tree, ())], {}, []
    h = 0
    while h < len(order):
        nd, path = order[h]
        if isinstance(nd, tuple):
            dec += [len(order), len(order) + 1]
            order += [(nd[0], path + (0,)), (nd[1], path + (1,))]
        else:
            dec += [0, nd]
            codes[nd] = np.array(path, np.uint8)
        h += 1
    return np.array(dec, np.int32), codes, leaves


def _stream(shape, bits, runs, seed):
    """A compressed cubelet of about `bits` bits of random symbols, and its bins."""
    dec, codes, leaves = _code(shape)
    bins = leaves - 1 if runs else leaves
    key = bins if runs else -1
    zero = bins // 2 if runs else -1
    rng = np.random.default_rng(seed)
    mean = np.mean([len(c) for c in codes.values()])
    syms = rng.integers(0, leaves, max(1, int(bits / mean)))
    if shape[0] == "keys":  # mostly runs: a tile covers millions of elements
        syms[rng.random(syms.size) < 0.9] = leaves - 1
    parts = []
    n = 0
    for s in syms:
        parts.append(codes[s])
        if s == key:
            v = int(rng.integers(0, 8)) if runs == "long" else 0
            parts.append(np.array([v & 1, v >> 1 & 1, v >> 2 & 1], np.uint8))
            n += 1 << (v + 3)
        else:
            n += 1
    b = np.concatenate(parts)
    words = np.packbits(np.pad(b, (0, -len(b) % 32)), bitorder="little").view(np.uint32)
    values = np.linspace(-3.0, 5.0, bins).astype(np.float32)
    # the largest box the stream has values for
    x = min(n, 64)
    y = min(n // x, 1024)
    z = n // (x * y)
    c = lib.Compressed((x, y, z), (x, y, z), lib.WL_F32, (0, 0, 0), P.CDF97,
                       P.LLOYD, bins, 0.5, 0.1, 5.0, -3.0, 5.0, max(zero, 0), key, zero,
                       max(len(x) for x in codes.values()), words, dec, values[:-1], values)
    want = oracle.huffman_decode(words, dec, key, zero, n)
    assert want.size == n
    return c, values[want][:x * y * z].reshape(z, y, x)


SHAPES = [("flat", 9), ("flat", 8), ("comb", 20), ("comb", 57), ("keys", 8), ("mixed", 300),
          ("mixed", 4096)]
LENGTHS = [1, 256, 300, TILE - 40, TILE + 90, 2 * TILE + 5000]


@pytest.mark.parametrize("runs", [None, "short", "long"])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: f"{s[0]}{s[1]}")
def test_streams(ctx, shape, runs):
    made = [_stream(shape, bits, runs, i) for i, bits in enumerate(LENGTHS)]
    for c, want in made:
        assert np.array_equal(ctx.decompress(c), want)
    for got, (_, want) in zip(ctx.decompress_batch([c for c, _ in made]), made):
        assert np.array_equal(got, want)


def test_short_and_long_streams_refused(ctx):
    """A stream with fewer values than its cubelet is refused, alone and in a
    batch; the context decodes the next one."""
    c, want = _stream(("mixed", 300), TILE + 90, None, 3)
    x, y, z = c.size
    good = c.size
    c.size = c.original_size = (x, y, z + 2)
    for call in (lambda: ctx.decompress(c), lambda: ctx.decompress_batch([c, c])):
        with pytest.raises(lib.WlError) as e:
            call()
        assert e.value.status == lib.WL_EFORMAT
    c.size = c.original_size = good
    assert np.array_equal(ctx.decompress(c), want)
