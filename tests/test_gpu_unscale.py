"""Inverse passes in registers whose scale is undone by a division, on values
where the corrected quotient would not be one: minus zeros, subnormal and tiny
numbers, numbers near the largest, infinities and NaN beside ordinary ones.
Bit for bit what the tile kernels give, which divide: an odd number of layers
sends the same rows there."""
import numpy as np
import pytest

from wavelets_gb300 import lib, params as P

pytestmark = pytest.mark.gpu

LENGTHS = [(40, 3), (48, 4), (144, 2), (160, 5), (192, 4), (512, 9), (512, 2)]


@pytest.fixture(scope="module")
def ctx():
    from wavelets_gb300 import build
    build.build()
    c = lib.Context(0)
    yield c
    c.close()


def rows(kind, n, L):
    """n rows of L values; a kind per eight rows where it is `mixed`."""
    rng = np.random.default_rng(L)
    v = rng.normal(0, 1, (n, L)).astype(np.float32)
    scale = {"tiny": 1e-39, "subnormal": 3e-44, "small": 1e-31, "huge": 2e38, "plain": 1.0}
    with np.errstate(over="ignore", under="ignore"):
        if kind in scale:
            v = (v.astype(np.float64) * scale[kind]).astype(np.float32)
        elif kind == "minus zeros":
            v[rng.random((n, L)) < 0.97] = -0.0
            v[: n // 2] = -0.0
        elif kind == "specials":
            at = rng.random((n, L))
            v[at < 0.01] = np.inf
            v[(at > 0.01) & (at < 0.02)] = -np.inf
            v[(at > 0.02) & (at < 0.03)] = np.nan
            v[:4] = 0.0
        else:
            v = (v.astype(np.float64) * 10.0 ** rng.integers(-45, 38, (n, L))).astype(np.float32)
    return v


def same(a, b):
    nan = np.isnan(a)
    assert np.array_equal(nan, np.isnan(b))
    assert np.array_equal(np.where(nan, 0, a).view(np.uint32), np.where(nan, 0, b).view(np.uint32))


KINDS = ["plain", "tiny", "subnormal", "small", "huge", "minus zeros", "specials", "mixed"]


@pytest.mark.parametrize("wavelet", [P.HAAR, P.CDF97])
@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("L,s", LENGTHS)
def test_y_x_and_z_rows(ctx, L, s, kind, wavelet):
    X, Z = 6, 8
    v = rows(kind, X * Z, L).reshape(X, Z, L)
    y = np.ascontiguousarray(v.transpose(2, 0, 1))  # stored (y, x, z)
    even = ctx.inverse_transform(y, (Z, X, L), (0, s, 0), wavelet, (X, L, Z))
    odd = ctx.inverse_transform(np.ascontiguousarray(y[:, :, :Z - 1]), (Z - 1, X, L), (0, s, 0),
                                wavelet, (X, L, Z - 1))
    same(even[:Z - 1], odd)
    x = np.ascontiguousarray(v.transpose(0, 2, 1))  # the same rows along x
    even_x = ctx.inverse_transform(x, (Z, L, X), (s, 0, 0), wavelet, (L, X, Z))
    odd_x = ctx.inverse_transform(np.ascontiguousarray(x[:, :, :Z - 1]), (Z - 1, L, X),
                                  (s, 0, 0), wavelet, (L, X, Z - 1))
    same(even_x[:Z - 1], odd_x)
    # and along z: stored (y, x, z) as it is
    z = ctx.inverse_transform(v[:, :Z - 1], (L, Z - 1, X), (0, 0, s), wavelet, (Z - 1, X, L))
    same(z, np.ascontiguousarray(odd.transpose(1, 2, 0)))


@pytest.mark.parametrize("kind", KINDS)
def test_long_images(ctx, kind):
    """Both axes of an image, one above the column tiles' limit."""
    Y, X, st = 1024, 96, (4, 10, 0)
    v = rows(kind, Y, X)
    one = ctx.inverse_transform(v.reshape(Y, X, 1), (1, X, Y), st, P.CDF97, (X, Y, 1))
    three = ctx.inverse_transform(np.repeat(v.reshape(Y, X, 1), 3, 2), (3, X, Y), st, P.CDF97,
                                  (X, Y, 3))
    same(one[0], three[1])
