"""Device workspace of a decompression: step tables are laid out for the inner
nodes that need one, not for every inner node, so that cubelets with large
alphabets are restored within the limit that they always were."""
import numpy as np
import pytest

from wavelets_gb300 import lib, params as P

pytestmark = pytest.mark.gpu

# bytes that restoring the batch below held, without a limit, when a stream had
# one lookup table and its bins in 32 bits
LIMIT = 31_029_390


def test_large_alphabets_within_the_limit():
    from wavelets_gb300 import build
    build.build()
    rng = np.random.default_rng(0)
    p = P.Params(steps=(1, 1, 1), threshold_fraction=0.0, bin_count=4096)
    items = [(rng.integers(0, 65536, (16, 16, 16)).astype(np.uint16), p) for _ in range(200)]
    a, b = lib.Context(0), lib.Context(0)
    try:
        cs = a.compress_batch(items)
        assert min(c.decode.size for c in cs) > 4000
        want = a.decompress_batch(cs)
        b.set_memory_limit(LIMIT)
        for x, y in zip(b.decompress_batch(cs), want):
            assert np.array_equal(x, y)
        assert b.memory_held() <= LIMIT
    finally:
        a.close()
        b.close()
