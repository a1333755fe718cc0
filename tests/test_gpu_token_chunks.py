"""The quantizer, the zero-run join and the bit packer with every chunk size
forced: the tests of their edges (tests/test_gpu_quantize_blocks.py, 4096-element
chunk and 256-chunk range edges of tests/test_gpu_runs.py, every slice count of
tests/test_gpu_encode_slices.py), whose calls are so small that they would be
cut into chunks of 512."""
import numpy as np
import pytest

from test_gpu_encode_slices import (_batch, _same, test_every_slice_count_packs_the_same_bits,
                                    test_single_cubelet_every_slice_count)
from test_gpu_quantize_blocks import test_tokens_match_oracle
from test_gpu_runs import test_batch_of_uneven_cubelets, test_sparse_cubelet
from wavelets_gb300 import lib

pytestmark = pytest.mark.gpu

CHUNKS = (512, 1024, 2048, 4096)


@pytest.fixture(scope="module", params=CHUNKS)
def ctx(request):
    from wavelets_gb300 import build
    build.build()
    c = lib.Context(0)
    c.set_token_chunk(request.param)
    yield c
    c.close()


def test_chunk_sizes_and_slices_give_the_same_bits():
    """Changing both on one context, with a graph captured for each."""
    items = _batch(13)
    c = lib.Context(0)
    try:
        want = c.compress_batch(items)
        for chunk in CHUNKS:
            c.set_token_chunk(chunk)
            for slices in (0, 1, 16):
                c.set_encode_slices(slices)
                for _ in range(3):
                    for w, g in zip(want, c.compress_batch(items)):
                        _same(w, g)
        for bad in (-512, 1, 256, 513, 3000, 8192):
            with pytest.raises(lib.WlError):
                c.set_token_chunk(bad)
    finally:
        c.close()


def test_chunk_size_shows_in_the_workspace():
    """128 bytes of slice offsets a chunk, among others."""
    a = np.random.default_rng(1).normal(0, 1, (64, 64, 64)).astype(np.float32)
    held = []
    for chunk in CHUNKS:
        c = lib.Context(0)
        c.set_token_chunk(chunk)
        c.compress(a)
        held.append(c.memory_held())
        c.close()
    for k in range(3):
        assert held[k] - held[k + 1] >= 128 * (a.size // CHUNKS[k] - a.size // CHUNKS[k + 1])
