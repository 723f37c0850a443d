"""Positions of more than 128 bytes start on 64-byte boundaries (Plan::icp), and filter rows that hold several
columns (Plan::tap_pitch): every kernel that writes or reads such rows, at the least and the most that lies
between them: the one-launch pass, both convolutions, both orders of the source and the weights, the upstream
calls one by one, a chain into such rows, and frames left over from other values. Against the oracle: sums, A and
K bit for bit, floats to the parity contract's 1e-4."""
import numpy as np
import pytest

import cases
import xnor_nn_b200 as xb
from oracle.pyoracle import Shape
from xnor_nn_b200 import synth

pytestmark = pytest.mark.gpu

LAYERS = [  # channels of 144, 160, 176 and 192 bytes, 208 and 256
    cases._c("one_launch_257", 2, 40, 257, 6, 7, 3, 3, ph=1, pw=1),
    cases._c("one_launch_nhwc_hwio_320", 3, 33, 320, 5, 5, 3, 3, ph=1, pw=1, fmt=(1, 1, 1)),
    cases._c("two_launches_352", 180, 96, 352, 13, 12, 3, 3, ph=1, pw=1),
    cases._c("two_launches_nhwc_hwio_390", 150, 48, 390, 11, 13, 2, 3, fmt=(1, 1, 0)),
    cases._c("filter_rows_of_240_bytes", 2, 33, 96, 7, 8, 5, 5, ph=2, pw=2),
    cases._c("filter_rows_of_144_bytes_hwio", 300, 40, 90, 9, 8, 3, 3, ph=1, pw=1, fmt=(1, 1, 1)),
    cases._c("filter_rows_of_560_bytes", 60, 24, 150, 12, 14, 7, 7, ph=3, pw=3),
    cases._c("two_launches_512", 60, 64, 512, 14, 13, 3, 3, ph=1, pw=1),
]


@pytest.mark.parametrize("kernel", [xb.KERNEL_TCGEN05_I8, xb.KERNEL_TCGEN05_I8_ROWS], ids=["tiles", "rows"])
@pytest.mark.parametrize("case", LAYERS, ids=[c[0] for c in LAYERS])
def test_layer_against_the_oracle(oracle, case, kernel):
    _, d, _, fmt = case
    src, w = cases.make_inputs(case)
    conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NHWC if fmt[0] else xb.NCHW, xb.HWIO if fmt[1] else xb.OIHW,
                          xb.NHWC if fmt[2] else xb.NCHW, d["mb"], d["oc"], d["ic"], d["ih"], d["iw"], d["kh"],
                          d["kw"], d["sh"], d["sw"], d["ph"], d["pw"], w, kernel=kernel)
    assert conv.kernel == kernel
    got = np.full(int(np.prod(conv.out_shape)), np.nan, np.float32)
    for values in (-src, src):
        want = oracle.convolution(cases.oracle_shape(case), values, w)
        for forward in (conv.forward, conv.forward_stepwise):
            forward(values, got)
            assert np.all(np.abs(got - want["dst"]) <= 1e-4 * np.abs(want["dst"]))
            assert np.array_equal(conv.forward_sums(), want["sums"])
            assert np.array_equal(conv.read(xb.SLOT_A, np.float32), want["a"])
            assert np.array_equal(conv.read(xb.SLOT_K, np.float32), want["k"])
    conv.close()


@pytest.mark.parametrize("mb", [2, 400])
def test_chain_into_padded_rows(oracle, mb):
    channels, side = (40, 290, 330, 24), 5
    x = src = synth.normal(3, mb * channels[0] * side * side)
    convs = []
    for i in range(3):
        d = (mb, channels[i + 1], channels[i], side, side, 3, 3, 1, 1, 1, 1)
        w = synth.normal(7 + i, d[1] * d[2] * 9, 0.05)
        convs.append(xb.Convolution(xb.ALGORITHM_BCAST, xb.NCHW, xb.OIHW, xb.NCHW, *d, w))
        want = oracle.convolution(Shape.make(*d, 0, 0, 0), x, w)
        x = want["dst"]
    got = np.full(x.size, np.nan, np.float32)
    for _ in range(2):
        xb.forward_chain(convs, src, got)
        assert np.array_equal(convs[2].forward_sums(), want["sums"])
        assert np.all(np.abs(got - x) <= 1e-4 * np.abs(x))
    for conv in convs:
        conv.close()
