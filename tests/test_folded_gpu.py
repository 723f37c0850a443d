"""Strided layers on the tensor cores: the packer folds filter columns and the rows of a stride into
channels, so what can go wrong are the edges of that folding (filters lower than the stride,
strides that do not divide the filter, borders, uneven paddings, channel groups, both layouts).
Sums, alpha, A and K bit for bit against the oracle, floats to the parity contract's 1e-4."""
import numpy as np
import pytest

import cases
import xnor_nn_b200 as xb

pytestmark = pytest.mark.gpu


def _c(name, *args, **kw):
    return cases._c(name, *args, **kw)


FOLDED = [
    _c("conv1_like", 3, 96, 3, 63, 59, 11, 11, sh=4, sw=4),
    _c("conv1_padded", 2, 20, 3, 40, 41, 7, 7, sh=2, sw=2, ph=3, pw=3),
    _c("resnet_3x3", 5, 72, 64, 14, 14, 3, 3, sh=2, sw=2, ph=1, pw=1),
    _c("projection_1x1", 4, 40, 100, 15, 13, 1, 1, sh=2, sw=2),
    _c("stride_beyond_filter", 2, 24, 9, 17, 19, 2, 2, sh=3, sw=3),
    _c("strides_differ", 2, 33, 21, 18, 23, 3, 5, sh=2, sw=3, ph=1, pw=1),
    _c("one_stride_only", 2, 16, 12, 9, 30, 3, 3, sh=1, sw=2, ph=1, pw=1),
    _c("uneven_padding", 2, 16, 5, 12, 12, 3, 3, sh=2, sw=2, ph=0, pw=1),
    _c("padding_of_the_filter", 1, 16, 6, 9, 9, 3, 3, sh=2, sw=2, ph=3, pw=3),
    # 200 channels x 4 rows x 221 columns do not fit the packer's stage: two groups of channels
    _c("channel_groups", 1, 16, 200, 26, 221, 4, 5, sh=4, sw=4),
    _c("seven_channels", 2, 24, 7, 20, 22, 9, 9, sh=3, sw=3, ph=4, pw=4),
    _c("eight_channels", 2, 24, 8, 20, 22, 9, 9, sh=3, sw=3, ph=4, pw=4),
    _c("single_channel", 2, 260, 1, 28, 28, 5, 5, sh=2, sw=2, ph=2, pw=2),
    _c("two_channels_one_word_a_row", 3, 24, 2, 31, 70, 7, 7, sh=2, sw=2, ph=3, pw=3),
    _c("four_channels_two_words_a_row", 3, 24, 4, 33, 34, 10, 10, sh=3, sw=2, ph=9, pw=9),
    _c("three_channels_three_words_a_row", 2, 24, 3, 40, 71, 18, 18, sh=5, sw=5, ph=2, pw=2),
    # seven channels: rows of 1000 values, and the largest stage there is (48048 bytes of bits)
    _c("seven_channels_wide", 1, 8, 7, 17, 1000, 8, 8, sh=8, sw=8),
    _c("seven_channels_wide_border", 1, 8, 7, 11, 1117, 11, 11, sh=11, sw=11, ph=1900, pw=1900),
    _c("channels_last", 3, 40, 37, 16, 17, 3, 3, sh=2, sw=2, ph=1, pw=1, fmt=(1, 1, 1)),
    _c("channels_last_conv1", 2, 36, 3, 47, 51, 11, 11, sh=4, sw=4, fmt=(1, 1, 0)),
    _c("many_tiles", 70, 48, 3, 61, 61, 3, 3, sh=2, sw=2, ph=1, pw=1),
]


@pytest.mark.parametrize("case", FOLDED, ids=[c[0] for c in FOLDED])
def test_folded_layer_against_the_oracle(oracle, case):
    _, d, _, fmt = case
    src, w = cases.make_inputs(case)
    want = oracle.convolution(cases.oracle_shape(case), src, w)
    conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NHWC if fmt[0] else xb.NCHW,
                          xb.HWIO if fmt[1] else xb.OIHW, xb.NHWC if fmt[2] else xb.NCHW,
                          d["mb"], d["oc"], d["ic"], d["ih"], d["iw"], d["kh"], d["kw"], d["sh"],
                          d["sw"], d["ph"], d["pw"], w)
    assert conv.kernel == xb.KERNEL_TCGEN05_I8
    for call in (conv.forward, conv.forward_stepwise):
        dst = np.full(want["dst"].size, np.nan, np.float32)
        call(src, dst)
        assert np.array_equal(conv.forward_sums(), want["sums"])
        assert np.array_equal(conv.read(xb.SLOT_ALPHA, np.float32), want["alpha"])
        assert np.array_equal(conv.read(xb.SLOT_A, np.float32), want["a"])
        assert np.array_equal(conv.read(xb.SLOT_K, np.float32), want["k"])
        assert np.all(np.abs(dst - want["dst"]) <= 1e-4 * np.abs(want["dst"]))
    conv.close()
