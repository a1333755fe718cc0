"""Compressed cubelets whose Huffman table or stream is malformed: refused with
WL_EFORMAT alone and in a batch, host and device outputs, and the context
decodes the next one.  The tables are refused on the host, before a launch
(tests/test_decode_table.py has the rule)."""
import ctypes
import dataclasses

import numpy as np
import pytest

from test_decode_table import LONGEST, REFUSED, comb
from wavelets_gb300 import lib, params as P

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from wavelets_gb300 import build
    build.build()
    c = lib.Context(0)
    yield c
    c.close()


@pytest.fixture(scope="module")
def good(ctx):
    a = np.random.default_rng(3).normal(0, 1, (24, 40, 48)).astype(np.float32)
    return ctx.compress(a, P.Params(steps=(3, 3, 3), threshold_fraction=0.6, bin_count=80))


def refused(call):
    with pytest.raises(lib.WlError) as e:
        call()
    assert e.value.status == lib.WL_EFORMAT


@pytest.mark.parametrize("name", sorted(REFUSED))
def test_malformed_table(ctx, good, name):
    want = ctx.decompress(good)
    bad = dataclasses.replace(good, decode=np.array(REFUSED[name], np.int32))
    if "symbol" in name:
        bad.bin_count, bad.quant_alg = 8, P.LLOYD
        bad.boundaries, bad.values = np.zeros(7, np.float32), np.zeros(8, np.float32)
        bad.dup_key = bad.dup_value = -1
    refused(lambda: ctx.decompress(bad))
    refused(lambda: ctx.decompress_batch([good, bad, good]))
    assert np.array_equal(ctx.decompress(good), want)


def test_longest_code(ctx, good):
    """60 bits are decoded: the symbols of a comb, from the longest code down."""
    t = comb(LONGEST)
    bins = LONGEST + 1
    bits = []
    for s in (LONGEST, LONGEST - 1, 0, 7):
        bits += [1] * s + ([0] if s < LONGEST else [])
    words = np.packbits(np.array(bits + [0] * (-len(bits) % 32), np.uint8),
                        bitorder="little").view(np.uint32)
    values = np.linspace(-1, 1, bins).astype(np.float32)
    c = dataclasses.replace(good, size=(4, 1, 1), original_size=(4, 1, 1), steps=(0, 0, 0),
                            bin_count=bins, quant_alg=P.LLOYD, words=words,
                            decode=np.array(t, np.int32), boundaries=values[:-1], values=values,
                            dup_key=-1, dup_value=-1)
    assert np.array_equal(ctx.decompress(c).ravel(), values[[LONGEST, LONGEST - 1, 0, 7]])


def short(c):
    """The same cubelet with less than its stream."""
    return dataclasses.replace(c, words=np.array(c.words[:c.words.size // 3]))


@pytest.mark.parametrize("shape,steps", [((24, 40, 48), (3, 3, 3)), ((1, 300, 200), (2, 2, 0)),
                                         ((6, 64, 50), (0, 0, 0))])
def test_refused_stream_leaves_the_outputs(ctx, shape, steps):
    """A short stream is found on the GPU: nothing of it, of its neighbours in
    the batch or of an earlier call reaches the caller's memory."""
    a = np.random.default_rng(4).normal(0, 1, shape).astype(np.float32)
    c = ctx.compress(a, P.Params(steps=steps, threshold_fraction=0.6, bin_count=80))
    want = ctx.decompress(c)
    batch = [c, short(c), c]
    prep = (lib.WlResult * 3)()
    for k, x in enumerate(batch):
        ctypes.memmove(ctypes.byref(prep, k * ctypes.sizeof(lib.WlResult)),
                       ctypes.byref(x.to_struct()), ctypes.sizeof(lib.WlResult))
    mark = np.random.default_rng(5).normal(0, 1, shape).astype(np.float32)
    for on_device in (0, 1):
        host = [mark.copy() for _ in batch]
        dev = [lib.DeviceBuffer(a.nbytes) for _ in batch]
        for d in dev:
            d.upload(mark)
        outs = (ctypes.c_void_p * 3)(*([d.ptr for d in dev] if on_device
                                       else [h.ctypes.data for h in host]))
        assert ctx.lib.wl_decompress_batch(ctx.h, prep, 3, None, outs, on_device) == lib.WL_EFORMAT
        assert ctx.lib.wl_decompress_cubelet(ctx.h, ctypes.byref(prep[1]), lib.WL_F32,
                                             outs[0], on_device) == lib.WL_EFORMAT
        for h, d in zip(host, dev):
            if on_device:
                h[...] = d.download(shape, np.float32)
            assert np.array_equal(h, mark)
            d.free()
    assert np.array_equal(ctx.decompress(c), want)
