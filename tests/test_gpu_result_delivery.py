"""Results of a call reach the host by a kernel (small ones, into storage set
aside from the last call's size), by the copy engine after they did not fit,
or by the copy engine from the start (large ones): the same bytes each way,
also with captured graphs replayed, and the stage times stay sensible."""
import numpy as np
import pytest

from oracle import oracle
from wavelets_gb300 import lib, params as P

pytestmark = pytest.mark.gpu

# (shape, bins): results of a few KB, about 1.5 MB (above the 1 MiB first set
# aside), and above the 8 MiB a kernel delivers
SIZES = {"tiny": ((2, 9, 17), 64), "middle": ((96, 96, 128), 4096), "large": ((160, 200, 250), 4096)}
ORDER = ["tiny", "middle", "middle", "middle", "tiny", "large", "large", "tiny", "middle"]


@pytest.fixture(scope="module")
def ctx():
    from wavelets_gb300 import build
    build.build()
    c = lib.Context(0)
    yield c
    c.close()


def _item(name):
    shape, bins = SIZES[name]
    arr = np.random.default_rng(len(name)).integers(0, 65536, shape).astype(np.uint16)
    return arr, P.Params(steps=(1, 1, 1), threshold_fraction=0.05, bin_count=bins,
                         quant_alg=P.UNIFORM)


@pytest.mark.parametrize("quant", [P.UNIFORM, P.LOG, P.LLOYD])
def test_every_route_gives_the_same_results(ctx, quant):
    first = {}
    for name in ORDER:
        arr, p = _item(name)
        p.quant_alg = quant
        got = ctx.compress(arr, p)
        if name not in first:
            first[name] = got
            if quant == P.UNIFORM:
                coeffs, _ = ctx.forward_transform(arr, p)
                want = oracle.encode(coeffs, p.threshold_fraction, p.bin_count, oracle.UNIFORM)
                assert np.array_equal(got.words, want["words"])
                assert list(got.decode) == list(want["decode"])
        for field in ("words", "decode", "boundaries", "values"):
            assert np.array_equal(getattr(got, field), getattr(first[name], field)), (name, field)
        assert got.threshold_value == first[name].threshold_value
        t = ctx.timings()
        assert all(x >= 0 for x in t) and 0 < sum(t[:5]) < 1.5 * t[5] + 1.0
    if quant == P.UNIFORM:
        assert first["middle"].words.nbytes > 1 << 20
        assert first["large"].words.nbytes > 8 << 20
