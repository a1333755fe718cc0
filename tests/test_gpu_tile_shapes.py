"""Every tile shape of the column-tile kernels gives the same results, on
passes that these kernels take: lengths that are neither a power of two, 48, 96
or 192 nor 8, 16 or 32 times at most 16 (those go to the register kernels: 136,
152, 200, 250, 6, 10, 50 do not), and y and x passes of an odd number of
layers; inputs from pageable, page-locked and device memory, forward against
the float64 yardstick, inverse back to every type."""
import numpy as np
import pytest

from oracle import lifting64
from test_gpu_tune import _forced, _same
from wavelets_gb300 import lib, params as P, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from wavelets_gb300 import build
    build.build()
    c = lib.Context(0)
    c.set_graph_mode(0)
    yield c
    lib.tune_reset()
    c.close()


# (z, y, x), steps: three odd or ragged axes of every length class
SHAPES = [((9, 136, 152), (3, 3, 0)), ((5, 200, 10), (3, 3, 0)), ((136, 6, 152), (3, 1, 3)),
          ((50, 50, 50), (1, 1, 1)), ((7, 64, 128), (4, 3, 0)), ((152, 9, 33), (0, 0, 3)),
          ((250, 10, 6), (1, 1, 1)), ((3, 500, 35), (0, 2, 0)), ((3, 35, 500), (2, 0, 0)),
          ((1, 151, 249), (3, 3, 0)), ((20, 20, 20), (2, 2, 2)), ((3, 512, 40), (3, 9, 0))]
TYPES = [np.uint8, np.uint16, np.float32, np.int32]


def _items():
    rng = np.random.default_rng(8)
    out = []
    for i, (shape, steps) in enumerate(SHAPES):
        for k in range(2):
            p = P.Params(steps=steps, wavelet=P.HAAR if (i + k) % 3 == 0 else P.CDF97,
                         quant_alg=[P.LOG, P.UNIFORM, P.LLOYD][(i + k) % 3], bin_count=255,
                         threshold_fraction=0.8)
            a = synth.scaled_blob_cubelet(rng, shape, TYPES[(i + 2 * k) % 4])
            out.append((np.ascontiguousarray(a), p))
    return out


def test_every_shape_gives_the_same_results(ctx):
    import torch
    items = _items()
    pinned = [torch.from_numpy(a.view(np.uint8).reshape(-1).copy()).pin_memory() for a, _ in items]
    device = [t.cuda() for t in pinned]
    torch.cuda.synchronize()

    def raw(bufs):
        return [(t.data_ptr(), lib.NP_TO_WL[a.dtype], a.shape[::-1], p)
                for t, (a, p) in zip(bufs, items)]
    ref = None
    try:
        for shape in lib.TILE_SHAPES:
            lib.tune_load(_forced(*shape))
            comp = ctx.compress_batch(items)
            for bufs, on_device in ((pinned, False), (device, True)):
                other = ctx.compress_batch(raw(bufs), on_device=on_device, raw=True)
                assert all(map(_same, comp, other))
            back = ctx.decompress_batch(comp) + ctx.decompress_batch(comp,
                                                                     [np.float32] * len(comp))
            if ref is None:
                ref = comp, back
                continue
            for i, (x, y) in enumerate(zip(comp, ref[0])):
                assert _same(x, y), (shape, i)
            for i, (x, y) in enumerate(zip(back, ref[1])):
                assert np.array_equal(x, y), (shape, i)
    finally:
        lib.tune_reset()


@pytest.mark.parametrize("tile", lib.TILE_SHAPES, ids=lambda t: f"{t[0]}x{t[1]}")
def test_transforms_against_float64(ctx, tile):
    rng = np.random.default_rng(9)
    try:
        lib.tune_load(_forced(*tile))
        for shape, steps in SHAPES:
            a = rng.normal(0, 100, shape).astype(np.float32)
            for wavelet in (P.HAAR, P.CDF97):
                got, stored = ctx.forward_transform(a, P.Params(steps=steps, wavelet=wavelet))
                want, _ = lifting64.forward(a, steps, wavelet)
                assert np.abs(got.ravel() - want).max() <= 2e-6 * np.abs(want).max()
                back = ctx.inverse_transform(got, stored, steps, wavelet, shape[::-1])
                assert np.abs(back - a).max() <= 4e-6 * np.abs(a).max()
    finally:
        lib.tune_reset()
