"""Output rows of 241 to 256 pixels on the image-row kernel: such a tile has one accumulator instead
of two. One to three tiles per SM, both layouts, one and several filter blocks; sums, A and K bit for
bit against the oracle, floats to the parity contract's 1e-4."""
import numpy as np
import pytest

import cases
import xnor_nn_b200 as xb

pytestmark = pytest.mark.gpu

WIDE = [cases._c("one_row_each", 1, 24, 20, 3, 246, 3, 3, ph=1, pw=0),       # 244 pixels
        cases._c("241_pixels", 2, 24, 20, 30, 239, 3, 3, ph=2, pw=2),        # below two a SM
        cases._c("256_pixels", 4, 24, 20, 90, 252, 3, 3, ph=3, pw=3),
        cases._c("two_filter_blocks", 2, 200, 70, 90, 250, 3, 3, ph=2, pw=2),
        cases._c("channels_last", 4, 40, 300, 60, 254, 3, 3, ph=1, pw=1, fmt=(1, 1, 1))]


@pytest.mark.parametrize("case", WIDE, ids=[c[0] for c in WIDE])
def test_wide_rows(oracle, case):
    _, d, _, fmt = case
    src, w = cases.make_inputs(case)
    want = oracle.convolution(cases.oracle_shape(case), src, w)
    conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NHWC if fmt[0] else xb.NCHW,
                          xb.HWIO if fmt[1] else xb.OIHW, xb.NHWC if fmt[2] else xb.NCHW, d["mb"],
                          d["oc"], d["ic"], d["ih"], d["iw"], d["kh"], d["kw"], 1, 1, d["ph"],
                          d["pw"], w, kernel=xb.KERNEL_TCGEN05_I8_ROWS)
    assert conv.kernel == xb.KERNEL_TCGEN05_I8_ROWS and 241 <= conv.c.ow <= 256
    for call in (conv.forward, conv.forward_stepwise):
        dst = np.full(want["dst"].size, np.nan, np.float32)
        call(src, dst)
        assert np.array_equal(conv.forward_sums(), want["sums"])
        assert np.array_equal(conv.read(xb.SLOT_A, np.float32), want["a"])
        assert np.array_equal(conv.read(xb.SLOT_K, np.float32), want["k"])
        assert np.all(np.abs(dst - want["dst"]) <= 1e-4 * np.abs(want["dst"]))
    conv.close()
