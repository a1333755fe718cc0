"""The quantizer's candidate queue and token staging against the oracle:
lengths around a lane's run (16), a block (512) and a chunk (4096), densities
from one value to every element, values in clusters with gaps above 1024
between them, with and without zero runs, all three quantizers."""
import numpy as np
import pytest

from oracle import oracle
from wavelets_gb300 import lib, params as P

pytestmark = pytest.mark.gpu

LENGTHS = (15, 16, 17, 31, 511, 512, 513, 530, 1024, 4095, 4096, 4097, 9000, 16384)


@pytest.fixture(scope="module")
def ctx():
    from wavelets_gb300 import build
    build.build()
    c = lib.Context(0)
    yield c
    c.close()


def _values(kind, n, rng):
    v = rng.normal(0, 1, n).astype(np.float32)
    if kind == "clusters":    # 40 values, then nothing for up to 3000 elements
        keep = np.zeros(n, bool)
        at = 0
        while at < n:
            keep[at:at + int(rng.integers(1, 41))] = True
            at += int(rng.integers(60, 3000))
        v[~keep] = 0
    elif kind == "gaps":      # every gap length in turn
        keep = np.cumsum(np.arange(1, 200) + 1)
        v[np.setdiff1d(np.arange(n), keep[keep < n])] = 0
    return v.reshape(1, 1, n)


# (kind, threshold fraction)
KINDS = [("dense", 0.0), ("dense", 0.5), ("dense", 0.9), ("dense", 0.99), ("clusters", 0.5),
         ("gaps", 0.5)]


@pytest.mark.parametrize("zeros", [True, False])
@pytest.mark.parametrize("alg", [P.UNIFORM, P.LOG, P.LLOYD])
@pytest.mark.parametrize("kind,frac", KINDS)
def test_tokens_match_oracle(ctx, kind, frac, alg, zeros):
    rng = np.random.default_rng(17)
    items = [(_values(kind, n, rng), P.Params(steps=(0, 0, 0), threshold_fraction=frac,
                                              quant_alg=alg, bin_count=[256, 65][n % 2],
                                              compress_zeros=zeros)) for n in LENGTHS]
    many = ctx.compress_batch(items)
    for (arr, p), got in zip(items, many):
        one = ctx.compress(arr, p)
        assert np.array_equal(one.words, got.words) and np.array_equal(one.decode, got.decode)
        qalg = {P.UNIFORM: oracle.UNIFORM, P.LOG: oracle.LOG, P.LLOYD: oracle.LLOYD}[alg]
        bins = oracle.quantize(arr, qalg, p.bin_count, got.threshold_value, got.max_value,
                               got.boundaries if alg == P.LLOYD else None)
        want = oracle.huffman_encode(bins, p.bin_count, got.zero_bin if zeros else -1)
        assert list(got.decode) == list(want["decode"])
        assert np.array_equal(got.words, want["words"])
