"""Page-locked storage that a result holds: a small result made after a large
one does not keep storage of the large one's size."""
import ctypes

import numpy as np
import pytest

from wavelets_gb300 import lib, params as P

pytestmark = pytest.mark.gpu

MiB = 1 << 20


def storage(r):
    """Bytes of the block that a result's arrays lie in (ResultSlab: reference
    count, address, size)."""
    base, cap = (ctypes.c_size_t * 2).from_address(r.owner + 8)
    assert base <= ctypes.cast(r.words, ctypes.c_void_p).value < base + cap
    return cap


def test_small_after_large():
    from wavelets_gb300 import build
    build.build()
    rng = np.random.default_rng(2)
    noise = rng.integers(0, 65536, (128, 160, 160)).astype(np.uint16)
    sparse = np.zeros_like(noise)
    sparse[::16, 5, 7] = 900
    p = P.Params(steps=(1, 1, 1), threshold_fraction=0.05, bin_count=1024, quant_alg=P.UNIFORM)
    ctx = lib.Context(0)
    held = []

    def call(a):
        pb = ctx.prepare_batch([(a, p)])
        r = (lib.WlResult * 1)()
        assert ctx.lib.wl_compress_batch(ctx.h, pb.cubs, 1, 0, r) == lib.WL_OK
        return r

    def words(r):
        return np.array(r[0].words[:r[0].n_words], np.uint32)
    try:
        free = call(sparse)
        want = words(free)
        ctx.lib.wl_results_free(free, 1)  # a block of the smallest size to take
        for _ in range(3):
            held.append(call(noise))
            large = storage(held[-1][0])
            assert held[-1][0].n_words * 4 > 2 * MiB and large == 4 * MiB
            held.append(call(sparse))
            assert held[-1][0].n_words * 4 < MiB // 4
            assert storage(held[-1][0]) <= MiB
            assert np.array_equal(words(held[-1]), want)
            held.append(call(sparse))
            assert storage(held[-1][0]) <= MiB
            assert np.array_equal(words(held[-1]), want)
    finally:
        for r in held:
            ctx.lib.wl_results_free(r, 1)
        ctx.close()
