"""The register kernel of the y passes (row pairs packed in two floats) against
the tile kernels: with an even number of z layers the rows pair up, with an
odd number they go to the tile kernels, and the transforms of the layers both
volumes share are the same to the bit, forward and inverse.  Forward also
against the float64 yardstick."""
import numpy as np
import pytest

from oracle import lifting64
from wavelets_gb300 import lib, params as P

pytestmark = pytest.mark.gpu

# most levels in the register kernel
LEVELS = {16: 4, 32: 5, 48: 4, 64: 6, 96: 4, 128: 7, 192: 4, 256: 8, 512: 9, 1024: 10, 2048: 11}
CASES = [(L, s) for L, most in LEVELS.items() for s in sorted({1, 2, 4, 5, most - 1, most, most + 1})
         if L % (1 << s) == 0 and s <= (L - 1).bit_length()]

# lengths whose lanes a row are not a power of two: 8, 16 and 32 elements a
# lane at most 16 times, and just beyond
LEVELS_ANY = {8: 3, 24: 3, 40: 3, 80: 4, 112: 4, 120: 3, 136: 3, 144: 4, 160: 5, 208: 4, 224: 5,
              240: 4, 272: 4, 480: 5, 544: 5}
ANY = [(L, s) for L, most in LEVELS_ANY.items() for s in sorted({1, 2, most, most + 1})
       if L % (1 << s) == 0 and s <= (L - 1).bit_length()]
CASES += ANY


@pytest.fixture(scope="module")
def ctx():
    from wavelets_gb300 import build
    build.build()
    c = lib.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("wavelet", [P.HAAR, P.CDF97])
@pytest.mark.parametrize("L,s", CASES)
def test_even_and_odd_layer_counts_agree(ctx, L, s, wavelet):
    X, Z = 10, 38  # pairs do not fill the last block
    vol = np.random.default_rng(L + s).normal(0, 100, (Z, L, X)).astype(np.float32)
    p = P.Params(steps=(1, s, 0), wavelet=wavelet)
    even, stored = ctx.forward_transform(vol, p)
    odd, _ = ctx.forward_transform(vol[:Z - 1], p)
    assert tuple(stored) == (Z, X, L)
    even, odd = even.reshape(L, X, Z), odd.reshape(L, X, Z - 1)
    assert np.array_equal(even[:, :, :Z - 1], odd)
    ref, _ = lifting64.forward(vol, (1, s, 0), wavelet)
    assert np.abs(even.ravel() - ref).max() <= 2e-6 * np.abs(ref).max()
    back = ctx.inverse_transform(even, (Z, X, L), (1, s, 0), wavelet, (X, L, Z))
    back_odd = ctx.inverse_transform(odd, (Z - 1, X, L), (1, s, 0), wavelet, (X, L, Z - 1))
    assert np.array_equal(back[:Z - 1], back_odd)
    assert np.abs(back - vol).max() <= 4e-6 * np.abs(vol).max()


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.int32, np.float32])
@pytest.mark.parametrize("L,s", CASES)
def test_x_rows_of_every_type(ctx, L, s, dtype):
    """The x passes: whole rows, rows cut short by the real length (REPEAT
    padding and crop) and rows that start off the lane vectors."""
    Y, Z = 6, 38
    rng = np.random.default_rng(L * s)
    for X in sorted({L, L - (1 << s) // 2, L - 1}):
        if P.clamp_steps((s, 1, 0), (X, Y, Z)) != (s, 1, 0) or P.padded_length(X, s) != L:
            continue
        if dtype == np.float32:
            vol = rng.normal(0, 100, (Z, Y, X)).astype(np.float32)
        else:
            vol = rng.integers(0, min(np.iinfo(dtype).max, 1 << 20) + 1, (Z, Y, X)).astype(dtype)
        for wavelet in (P.HAAR, P.CDF97):
            p = P.Params(steps=(s, 1, 0), wavelet=wavelet)
            even, stored = ctx.forward_transform(vol, p)
            odd, _ = ctx.forward_transform(vol[:Z - 1], p)
            assert tuple(stored) == (Z, L, Y)
            even, odd = even.reshape(Y, L, Z), odd.reshape(Y, L, Z - 1)
            assert np.array_equal(even[:, :, :Z - 1], odd)
            ref, _ = lifting64.forward(vol, (s, 1, 0), wavelet)
            assert np.abs(even.ravel() - ref).max() <= 2e-6 * np.abs(ref).max()
            back = ctx.inverse_transform(even, (Z, L, Y), (s, 1, 0), wavelet, (X, Y, Z), dtype)
            back_odd = ctx.inverse_transform(odd, (Z - 1, L, Y), (s, 1, 0), wavelet,
                                             (X, Y, Z - 1), dtype)
            assert np.array_equal(back[:Z - 1], back_odd)


@pytest.mark.parametrize("dtype", [np.uint8, np.float32])
@pytest.mark.parametrize("Y,X,steps", [(64, 64, (-1, -1)), (128, 256, (-1, -1)), (256, 48, (3, 5)),
                                       (512, 96, (4, 9)), (96, 512, (7, 4)), (1024, 64, (6, 10)),
                                       (2048, 128, (-1, -1)), (32, 2048, (11, 5)),
                                       (1024, 2048, (3, 2)), (600, 1000, (-1, -1)),
                                       (2048, 1023, (10, 1))])
def test_images(ctx, Y, X, steps, dtype):
    """One layer (rows paired along the other axis) against the middle one of
    three layers, which the other kernels take; deep levels, long axes, cut
    rows; integers restored the same."""
    rng = np.random.default_rng(Y + X)
    img = rng.normal(128, 60, (1, Y, X))
    img = img.astype(np.float32) if dtype == np.float32 else np.clip(img, 0, 255).astype(dtype)
    three = np.repeat(img, 3, 0)
    for wavelet in (P.HAAR, P.CDF97):
        p = P.Params(steps=(steps[0], steps[1], 0), wavelet=wavelet)
        one, (_, Xp, Yp) = ctx.forward_transform(img, p)
        all3, _ = ctx.forward_transform(three, p)
        one, all3 = one.reshape(Yp, Xp), all3.reshape(Yp, Xp, 3)
        assert np.array_equal(one, all3[:, :, 1])
        st = P.clamp_steps(p.steps, (X, Y, 1))
        back = ctx.inverse_transform(one, (1, Xp, Yp), st, wavelet, (X, Y, 1), dtype)
        back3 = ctx.inverse_transform(all3, (3, Xp, Yp), st, wavelet, (X, Y, 3), dtype)
        assert np.array_equal(back[0], back3[1])


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.int32, np.float32])
def test_rows_at_any_address(ctx, dtype):
    """Cubelets in device memory that start off the lane vectors and have rows
    of odd length, several lengths in one launch: as alone from the host, where
    they start at an aligned address."""
    import torch
    rng = np.random.default_rng(5)
    p = P.Params(steps=(3, 2, 1), threshold_fraction=0.7, bin_count=64)
    es = np.dtype(dtype).itemsize
    vols, items, keep = [], [], []
    for k, x in enumerate((77, 80, 113, 120, 161, 131, 131, 255)):
        v = rng.integers(0, 200, (16, 20, x)).astype(dtype)
        buf = torch.zeros(v.nbytes + 16 * es, dtype=torch.uint8, device="cuda")
        buf[k * es:k * es + v.nbytes] = torch.from_numpy(v.reshape(-1).view(np.uint8)).cuda()
        vols.append(v)
        keep.append(buf)
        items.append((buf.data_ptr() + k * es, lib.NP_TO_WL[np.dtype(dtype)], (x, 20, 16), p))
    torch.cuda.synchronize()
    for v, c in zip(vols, ctx.compress_batch(items, on_device=True, raw=True)):
        want = ctx.compress(v, p)
        assert np.array_equal(c.words, want.words)
        assert (c.threshold_value, c.max_value) == (want.threshold_value, want.max_value)


@pytest.mark.parametrize("wavelet", [P.HAAR, P.CDF97])
@pytest.mark.parametrize("L,s", ANY + [(512, 5), (512, 6)])
def test_z_rows(ctx, L, s, wavelet):
    """z passes of the same lengths, an odd number of rows: against the float64
    yardstick, back again, and the extremes gathered on the way."""
    X, Y = 13, 11
    vol = np.random.default_rng(L * s).normal(0, 100, (L, Y, X)).astype(np.float32)
    p = P.Params(steps=(0, 0, s), wavelet=wavelet, threshold_fraction=0.5, bin_count=64)
    got, stored = ctx.forward_transform(vol, p)
    ref, _ = lifting64.forward(vol, (0, 0, s), wavelet)
    assert np.abs(got.ravel() - ref).max() <= 2e-6 * np.abs(ref).max()
    back = ctx.inverse_transform(got, stored, (0, 0, s), wavelet, (X, Y, L))
    assert np.abs(back - vol).max() <= 4e-6 * np.abs(vol).max()
    c = ctx.compress(vol, p)
    a = np.sort(np.abs(got.ravel()))
    assert (c.min_coef, c.max_coef, c.max_value) == (got.min(), got.max(), a[-1])
    assert c.threshold_value in a and abs(np.searchsorted(a, c.threshold_value) - a.size / 2) <= 2
