"""The quotient that the register passes form where a scale is undone by a
division (dwt_strided.cuh Unscale): v times the reciprocal and one correction
step, with fused multiply-adds, is the correctly rounded v / s for every scale
of the lifting transform and every significand.  CPU only, in float64: the
products of two floats are exact there, sums are rounded with the part that
they lose known."""
import numpy as np
import pytest

K = 1.149604398860241
LEVELS = 14
SCALES = sorted({float(np.float32(K ** t)) for t in range(LEVELS + 1)} |
                {float(np.float32(-K ** t / K)) for t in range(LEVELS)})
CHUNK = 1 << 20


def fma(a, b, c):
    """float32(a * b + c), one rounding; float32 arrays."""
    p = a.astype(np.float64) * b.astype(np.float64)  # exact
    c = c.astype(np.float64)
    s = p + c
    t = s - c
    lost = (c - (s - t)) + (p - t)  # two-sum: s + lost = p + c
    tie = ((s.view(np.int64) & 0x1fffffff) == 0x10000000) & (lost != 0)
    return np.where(tie, np.nextafter(s, np.copysign(np.inf, lost)), s).astype(np.float32)


def quotient(v, s):
    s = np.full_like(v, s)
    r = np.float32(1) / s
    q = v * r
    # |s| q - v, or |s| q + v with a negative scale, times -|r|
    rest = fma(q, np.abs(s), np.where(s > 0, -v, v))
    return fma(rest, -np.abs(r), q)


@pytest.mark.parametrize("s", SCALES)
def test_every_significand(s):
    s = np.float32(s)
    for at in range(0, 1 << 23, CHUNK):
        v = (np.arange(at, at + CHUNK, dtype=np.uint32) | 0x3f800000).view(np.float32)
        assert np.array_equal(quotient(v, s), v / s)


@pytest.mark.parametrize("e", [-99, -60, 60, 126])
def test_ends_of_the_range(e):
    """Quotients near 2^-100 and 2^126, where the kernel still relies on it."""
    rng = np.random.default_rng(e & 0xff)
    for s in SCALES:
        q = (rng.integers(0, 1 << 23, 4096).astype(np.uint32) | 0x3f800000).view(np.float32)
        v = (q * np.float32(s)).astype(np.float64) * 2.0 ** e
        v = v[np.abs(v) < np.finfo(np.float32).max].astype(np.float32)
        want = v / np.float32(s)
        keep = (np.abs(want) >= 2.0 ** -100) & (np.abs(want) <= 2.0 ** 126)
        assert np.array_equal(quotient(v[keep], np.float32(s)), want[keep])


@pytest.mark.parametrize("v", [0.0, -0.0])
def test_zeros_keep_their_sign(v):
    v = np.array([v], np.float32)
    for s in SCALES:
        assert np.signbit(quotient(v, np.float32(s)))[0] == np.signbit(v / np.float32(s))[0]
