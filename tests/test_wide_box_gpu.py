"""Box filters whose rows of A do not fit shared memory take one thread per output instead: 11 x 11
windows on rows of 1000 pixels, unit stride and stride 2, K bit for bit against the oracle."""
import numpy as np
import pytest

import cases
import xnor_nn_b200 as xb

pytestmark = pytest.mark.gpu

WIDE = [cases._c("wide_box", 1, 16, 1, 11, 1000, 11, 11),
        cases._c("wide_box_padded", 2, 16, 3, 13, 1000, 11, 11, ph=5, pw=5),
        cases._c("wide_box_stride_2", 2, 16, 1, 14, 1000, 11, 11, sh=2, sw=2, ph=3, pw=3)]


@pytest.mark.parametrize("case", WIDE, ids=[c[0] for c in WIDE])
def test_wide_box_filter(oracle, case):
    _, d, _, _ = case
    src, w = cases.make_inputs(case)
    want = oracle.convolution(cases.oracle_shape(case), src, w)
    conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NCHW, xb.OIHW, xb.NCHW, d["mb"], d["oc"], d["ic"],
                          d["ih"], d["iw"], d["kh"], d["kw"], d["sh"], d["sw"], d["ph"], d["pw"], w)
    for call in (conv.forward_stepwise, conv.forward):
        dst = np.full(want["dst"].size, np.nan, np.float32)
        call(src, dst)
        assert np.array_equal(conv.read(xb.SLOT_K, np.float32), want["k"])
        assert np.all(np.abs(dst - want["dst"]) <= 1e-4 * np.abs(want["dst"]))
    conv.close()
