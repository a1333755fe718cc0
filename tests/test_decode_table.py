"""The host's rule for Huffman decode tables: trees pass, in the reference's
breadth-first layout or any other that lists children after their parent;
anything that would give the decoder a token without an end or a length is
refused before a launch.  CPU only."""
import ctypes
import glob
import os

import numpy as np
import pytest

from conftest import GOLDEN
from wavelets_gb300 import cubefile

LONGEST = 60


@pytest.fixture(scope="module")
def steps():
    from wavelets_gb300 import build
    fn = ctypes.CDLL(build.build()).wl_internal_decode_table_steps
    fn.argtypes = [ctypes.c_void_p, ctypes.c_int, ctypes.c_int, ctypes.c_int]

    def call(table, bins, key=-1):
        t = np.ascontiguousarray(table, np.int32)
        return fn(t.ctypes.data, t.size, bins, key)
    return call


@pytest.fixture(scope="module")
def ok(steps):
    return lambda *a: steps(*a) >= 0


def comb(bits):
    """Codes of 1, 2, .. bits bits, two of the longest, breadth first."""
    t = []
    for i in range(bits):
        t += [2 * i + 1, 2 * i + 2] if i == 0 else [0, i - 1, 2 * i + 1, 2 * i + 2]
    return t + [0, bits - 1, 0, bits]


def comb_depth_first(bits):
    """The same codes, every inner node followed by its leaf."""
    t = []
    for i in range(bits):
        t += [2 * i + 1, 2 * i + 2, 0, i]
    return t + [0, bits]


def random_tree(rng, leaves):
    """Breadth-first table of a random tree."""
    nodes = [(s,) for s in range(leaves)]
    while len(nodes) > 1:
        i, j = sorted(rng.choice(len(nodes), 2, replace=False))
        b, a = nodes.pop(j), nodes.pop(i)
        nodes.append((a, b))
    order, t = [nodes[0]], []
    for nd in order:
        if len(nd) == 2:
            t += [len(order), len(order) + 1]
            order += list(nd)
        else:
            t += [0, nd[0]]
    return t


def test_reference_files_pass(ok):
    seen = 0
    for path in sorted(glob.glob(os.path.join(GOLDEN, "*.cube"))):
        for c in cubefile.read_file(path):
            if c.params is None or not c.params.huffman_decode_table:
                continue
            key = c.params.huffman_dup_key
            assert ok(c.params.huffman_decode_table, c.params.bin_count,
                      -1 if key is None else key), path
            seen += 1
    assert seen > 20


def test_trees_pass(ok):
    rng = np.random.default_rng(0)
    for leaves in (2, 3, 17, 256, 1025):
        assert ok(random_tree(rng, leaves), leaves)
        assert ok(random_tree(rng, leaves), leaves - 1, leaves - 1)  # one leaf the key
    assert ok(comb(LONGEST), LONGEST + 1)
    assert ok([0, 3], 4) and ok([0, 4], 4, 4)  # one symbol, without a bit
    # children not next to each other
    assert ok([1, 4, 2, 3, 0, 0, 0, 1, 0, 2], 3)
    assert ok(comb_depth_first(LONGEST), LONGEST + 1)


REFUSED = {
    "a node its own child": [1, 2, 0, 0, 2, 3, 0, 1],
    "the root a left child": [1, 2, 0, 0, 3, 4, 0, 1, 0, 0, 0, 0, 5],
    "the root a right child": [1, 2, 0, 0, 3, 0, 0, 1],
    "root its own right child": [1, 0, 0, 1],
    "child before its parent": [1, 2, 3, 4, 1, 4, 0, 0, 0, 1],
    "one child twice": [1, 1, 0, 0],
    "shared child": [1, 2, 3, 4, 4, 5, 0, 0, 0, 1, 0, 2],
    "node nothing reaches": [1, 2, 0, 0, 0, 1, 0, 2],
    "tree nothing reaches": [1, 2, 0, 0, 0, 1, 4, 5, 0, 0, 0, 1],
    "leaf root and more": [0, 0, 0, 1],
    "61-bit code": comb(LONGEST + 1),
    "61-bit code, depth first": comb_depth_first(LONGEST + 1),
    "child past the end": [1, 3, 0, 0, 0, 1],
    "negative child": [-1, 2, 0, 0, 0, 1],
    "negative right child": [1, -2, 0, 0, 0, 1],
    "symbol past the bins": [1, 2, 0, 0, 0, 9],
    "negative symbol": [1, 2, 0, 0, 0, -1],
    "half an entry": [1, 2, 0, 0, 0],
    "nothing": [],
}


@pytest.mark.parametrize("name", sorted(REFUSED))
def test_refused(ok, name):
    assert not ok(REFUSED[name], 8 if "symbol" in name else 80)


def walk_ok(t, bins, key):
    """Every node reached once from the root, by codes of at most 60 bits."""
    nodes, todo, seen = len(t) // 2, [(0, 0)], set()
    while todo:
        i, d = todo.pop()
        if i in seen or not 0 <= i < nodes or d > LONGEST:
            return False
        seen.add(i)
        a, b = t[2 * i], t[2 * i + 1]
        if a == 0:
            if not (0 <= b < bins or (b == key and b >= 0)) or (i == 0 and nodes > 1):
                return False
        else:
            todo += [(a, d + 1), (b, d + 1)]
    return len(seen) == nodes


def test_accepted_tables_are_trees(ok):
    """Tables with entries changed at random: what passes is a tree."""
    rng = np.random.default_rng(1)
    passed = 0
    for _ in range(4000):
        leaves = int(rng.integers(2, 12))
        t = random_tree(rng, leaves)
        for _ in range(int(rng.integers(1, 3))):
            t[int(rng.integers(0, len(t)))] = int(rng.integers(-1, len(t) // 2 + 1))
        if ok(t, leaves - 1, leaves - 1):
            assert walk_ok(t, leaves - 1, leaves - 1), t
            passed += 1
    assert passed > 100


def test_step_tables(steps):
    """One per inner node at depth 12, 16, 20 .."""
    rng = np.random.default_rng(2)

    def shuffled(t):
        """The same tree with its nodes numbered depth first."""
        out = []

        def place(i):
            k = len(out)
            out.append((0, t[2 * i + 1]))
            if t[2 * i]:
                out[k] = (place(t[2 * i]), place(t[2 * i + 1]))
            return k
        place(0)
        return [x for p in out for x in p]
    trees = [comb(k) for k in (1, 11, 12, 13, 16, 17, 40, LONGEST)]
    trees += [random_tree(rng, k) for k in (2, 300, 5000)]
    for t in trees:
        want, todo = 0, [(0, 0)]
        while todo:
            i, d = todo.pop()
            if t[2 * i]:
                want += d >= 12 and (d - 12) % 4 == 0
                todo += [(t[2 * i], d + 1), (t[2 * i + 1], d + 1)]
        assert steps(t, 5000) == want
        assert steps(shuffled(t), 5000) == want
