"""A forced slice count is lanes per 4096 elements whatever the call's size:
the call is then cut into chunks of 4096, which shows in the per-chunk
workspace of a fresh context, and the bits are the default's."""
import numpy as np
import pytest

from wavelets_gb300 import lib, params as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slices", [1, 8, 32])
def test_forced_count_is_per_4096_elements(slices):
    from wavelets_gb300 import build
    build.build()
    a = np.random.default_rng(1).normal(0, 1, (64, 128, 128)).astype(np.float32)  # 512-element chunks by default
    p = P.Params(steps=(2, 2, 2), threshold_fraction=0.8, quant_alg=P.UNIFORM)
    held, words = [], []
    for f in (0, slices):
        ctx = lib.Context(0)
        try:
            ctx.set_encode_slices(f)
            c = ctx.compress(a, p)
            held.append(ctx.memory_held())
            words.append((np.array(c.words), np.array(c.decode)))
        finally:
            ctx.close()
    # 128 bytes of slice offsets a chunk alone, with a quarter's slack
    chunks = a.size // 512, a.size // 4096
    assert held[0] - held[1] >= 128 * 1.25 * (chunks[0] - chunks[1])
    for x, y in zip(*words):
        assert np.array_equal(x, y)
