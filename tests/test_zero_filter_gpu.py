"""A filter whose weights are all zero (pruned, dead) has alpha 0, and its results are zeros whose
sign is the sign of the integer sum: (S * alpha) * K is -0 for a negative S and +0 otherwise, as
upstream multiplies (src/default/bcast_convolution_default.cpp:60-103). The sign matters: the next
layer's packer reads the sign bit. Signs of all results and the next layer's integer sums against
the oracle, on every store path of every kernel."""
import numpy as np
import pytest

import cases
import xnor_nn_b200 as xb
from oracle.pyoracle import Shape
from xnor_nn_b200 import synth

pytestmark = pytest.mark.gpu

_c = cases._c
LAYERS = [
    (_c("zero_nchw", 2, 48, 40, 9, 11, 3, 3, ph=1, pw=1), xb.KERNEL_TCGEN05_I8),
    (_c("zero_nhwc", 2, 48, 40, 9, 11, 3, 3, ph=1, pw=1, fmt=(0, 0, 1)), xb.KERNEL_TCGEN05_I8),
    (_c("zero_nhwc_16_bytes", 2, 20, 40, 9, 11, 3, 3, ph=1, pw=1, fmt=(0, 0, 1)), xb.KERNEL_TCGEN05_I8),
    (_c("zero_nhwc_odd", 2, 13, 40, 9, 11, 3, 3, ph=1, pw=1, fmt=(0, 0, 1)), xb.KERNEL_TCGEN05_I8),
    (_c("zero_pairs", 2140, 32, 40, 2, 2, 3, 3, ph=1, pw=1), xb.KERNEL_TCGEN05_I8),
    (_c("zero_folded", 2, 24, 3, 40, 41, 7, 7, sh=2, sw=2, ph=3, pw=3), xb.KERNEL_AUTO),
    (_c("zero_rows_nchw", 2, 48, 40, 9, 11, 3, 3, ph=1, pw=1), xb.KERNEL_TCGEN05_I8_ROWS),
    (_c("zero_rows_nhwc", 2, 48, 40, 9, 11, 3, 3, ph=1, pw=1, fmt=(0, 0, 1)), xb.KERNEL_TCGEN05_I8_ROWS),
    # outputs that see no input pixel: S = 0, the result +0
    (_c("zero_padding_of_the_filter", 2, 24, 20, 5, 6, 3, 3, ph=3, pw=3), xb.KERNEL_AUTO),
    (_c("zero_popc", 2, 48, 40, 9, 11, 3, 3, ph=1, pw=1), xb.KERNEL_POPC),
]


def _zero_filter(w, oc, hwio, filters):
    if hwio:
        w[..., filters] = 0.0
    else:
        w.reshape(oc, -1)[filters] = 0.0
    return w


@pytest.mark.parametrize("layer", LAYERS, ids=[c[0][0] for c in LAYERS])
def test_sign_of_a_zero_result(oracle, layer):
    case, kernel = layer
    _, d, _, fmt = case
    src, w = cases.make_inputs(case)
    _zero_filter(w, d["oc"], fmt[1], [0, 5, d["oc"] - 1])
    want = oracle.convolution(cases.oracle_shape(case), src, w)
    zeros = want["dst"] == 0
    assert np.signbit(want["dst"][zeros]).any()  # the case has what it is about
    conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NHWC if fmt[0] else xb.NCHW,
                          xb.HWIO if fmt[1] else xb.OIHW, xb.NHWC if fmt[2] else xb.NCHW, d["mb"],
                          d["oc"], d["ic"], d["ih"], d["iw"], d["kh"], d["kw"], d["sh"], d["sw"],
                          d["ph"], d["pw"], w, kernel=kernel)
    dst = np.full(want["dst"].size, np.nan, np.float32)
    conv.forward(src, dst)
    assert np.array_equal(dst == 0, zeros)
    assert np.array_equal(np.signbit(dst), np.signbit(want["dst"]))
    conv.close()


@pytest.mark.parametrize("kernel", [xb.KERNEL_TCGEN05_I8, xb.KERNEL_TCGEN05_I8_ROWS],
                         ids=["tiles", "rows"])
def test_next_layer_after_a_zero_filter(oracle, kernel):
    """40 -> 48 -> 24 channels, filter 7 of the first layer all zero: the second layer's sums, the
    layers run one after the other and (position tiles) chained."""
    mb, h, w_ = 2, 9, 11
    w0 = synth.normal(11, 48 * 40 * 9, 0.05).reshape(48, 40, 3, 3)
    w1 = synth.normal(12, 24 * 48 * 9, 0.05).reshape(24, 48, 3, 3)
    w0[7] = 0.0
    src = synth.normal(13, mb * 40 * h * w_)
    s0 = Shape.make(mb, 48, 40, h, w_, 3, 3, 1, 1, 1, 1)
    s1 = Shape.make(mb, 24, 48, h, w_, 3, 3, 1, 1, 1, 1)
    mid = oracle.convolution(s0, src, w0)["dst"]
    want = oracle.convolution(s1, mid, w1)
    convs = [xb.Convolution(xb.ALGORITHM_BCAST, xb.NCHW, xb.OIHW, xb.NCHW, mb, oc, ic, h, w_, 3, 3,
                            1, 1, 1, 1, wt, kernel=kernel)
             for oc, ic, wt in ((48, 40, w0), (24, 48, w1))]
    x = np.empty(mid.size, np.float32)
    y = np.empty(want["dst"].size, np.float32)
    convs[0].forward(src, x)
    convs[1].forward(x, y)
    assert np.array_equal(convs[1].forward_sums(), want["sums"])
    xb.forward_chain(convs, src, y)
    assert np.array_equal(convs[1].forward_sums(), want["sums"])
    for cv in convs:
        cv.close()
