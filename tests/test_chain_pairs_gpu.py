"""Chained layers on CTA pairs (conv_tcgen05.cu): filters resident beside columns, beside tiles of a filter row
and beside tiles of all filter rows, streamed filters with one and two filter tiles, the plain ring; odd rows,
partly empty chunks, accumulators that share columns, filters that end inside a tile
and inside a byte's pair, an odd number of position tiles, fewer tiles than SMs; and layers that stay on single
CTAs. test_chain_pairs_cpu.py pins which are which. Against the oracle, layer by layer: the next layer's sums
bit for bit, its A within rounding of a reordered sum, floats to the parity contract's 1e-4."""
import numpy as np
import pytest

import xnor_nn_b200 as xb
from oracle.pyoracle import Shape
from xnor_nn_b200 import synth

pytestmark = pytest.mark.gpu

# name: mb, ic, oc, ih, iw, kh, kw, ph, pw of the first layer; the second has 16 filters of 3 x 3
PAIRS = {
    "columns": (1601, 96, 256, 4, 4, 5, 5, 2, 2),
    "rows_of_all_filter_rows": (801, 480, 256, 8, 4, 4, 1, 0, 0),
    "rows_of_a_filter_row": (900, 480, 224, 9, 3, 5, 1, 0, 0),
    "streamed": (801, 320, 250, 4, 4, 3, 3, 1, 1),
    "streamed_two_filter_tiles": (830, 384, 512, 4, 4, 3, 3, 1, 1),
    "streamed_four_tiles_odd_filters": (801, 288, 1023, 4, 4, 3, 3, 1, 1),
    "streamed_192_filters": (801, 480, 192, 4, 4, 3, 3, 1, 1),
    "ring": (1101, 350, 511, 5, 4, 3, 1, 0, 0),
    "part_chunk_fewer_tiles_than_sms": (41, 384, 256, 4, 4, 3, 3, 1, 1),
    "fewer_tiles_than_sms": (41, 288, 256, 4, 4, 3, 3, 1, 1),
}
SINGLE = {
    "even_rows_whole_chunks": (801, 256, 256, 4, 4, 3, 3, 1, 1),
    "part_chunk_64_filters": (801, 384, 64, 4, 4, 3, 3, 1, 1),
    "short_tiles": (801, 288, 160, 4, 4, 3, 3, 1, 1),
    "one_filter_row": (1200, 480, 512, 4, 4, 1, 1, 0, 0),
}


@pytest.mark.parametrize("name", list(PAIRS) + list(SINGLE))
def test_chain_against_the_oracle(oracle, name):
    mb, ic, oc, ih, iw, kh, kw, ph, pw = {**PAIRS, **SINGLE}[name]
    oh, ow = ih + 2 * ph - kh + 1, iw + 2 * pw - kw + 1
    layers = [(mb, oc, ic, ih, iw, kh, kw, 1, 1, ph, pw), (mb, 16, oc, oh, ow, 3, 3, 1, 1, 1, 1)]
    src = synth.normal(len(name), mb * ic * ih * iw)
    src[: ic * ih * iw] = 0.0  # K = 0: results are +-0
    x, convs = src, []
    for i, d in enumerate(layers):
        w = synth.normal(5 + i, d[1] * d[2] * d[5] * d[6], 0.05)
        convs.append(xb.Convolution(xb.ALGORITHM_BCAST, xb.NCHW, xb.OIHW, xb.NCHW, *d, w))
        want = oracle.convolution(Shape.make(*d, 0, 0, 0), x, w)
        if i == 0:
            k = want["k"]
        x = want["dst"]
    got = np.full(x.size, np.nan, np.float32)
    for _ in range(2):
        xb.forward_chain(convs, src, got)
        assert np.array_equal(convs[1].forward_sums(), want["sums"])
        assert np.array_equal(convs[0].read(xb.SLOT_K, np.float32), k)
        a = convs[1].read(xb.SLOT_A, np.float32)
        # at most 1023 terms of one sign in 32 bits, in another order: 1023 * 2^-24 each way
        assert np.all(np.abs(a - want["a"]) <= 2 * 1023 * 2.0 ** -24 * want["a"])
        assert np.all(np.abs(got - x) <= 1e-4 * np.abs(x))
        assert np.array_equal(got == 0, x == 0)
    for conv in convs:
        conv.close()
