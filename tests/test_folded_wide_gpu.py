"""Strided layers of fewer than eight channels on wide rows: the packer's blocks of 128 and of 256 threads
(few blocks with many loads each), one to three words a filter row, staged nibbles below and above the 48 KB
that need no opt-in and at the 192 KB that is its limit, both layouts. Sums, A and K bit for bit against the
oracle."""
import numpy as np
import pytest

import cases
import xnor_nn_b200 as xb

pytestmark = pytest.mark.gpu

WIDE = [cases._c("ic%d_%dx%d" % (ic, k, k), 1, 16, ic, 23, 2051, k, k, sh=s, sw=s, ph=k // 2, pw=k // 2)
        for ic, k, s in ((1, 11, 4), (2, 7, 4), (3, 11, 4), (4, 8, 4), (5, 11, 4), (7, 17, 5))] + [
    cases._c("many_blocks", 40, 16, 3, 121, 520, 11, 11, sh=4, sw=4),
    # 320 loads of a warp a block and more
    cases._c("320_loads", 1, 16, 4, 17, 635, 11, 11, sh=4, sw=4, ph=5, pw=5),
    cases._c("336_loads", 1, 16, 4, 17, 640, 11, 11, sh=4, sw=4, ph=5, pw=5),
    cases._c("over_48_kb", 2, 16, 7, 11, 1100, 11, 11, sh=11, sw=11, ph=400, pw=400),
    cases._c("192_kb", 1, 8, 7, 11, 1117, 11, 11, sh=11, sw=11, ph=1900, pw=1900),
    cases._c("channels_last", 2, 16, 3, 23, 2051, 11, 11, sh=4, sw=4, ph=5, pw=5, fmt=(1, 1, 1)),
    cases._c("channels_last_over_48_kb", 2, 16, 5, 22, 1110, 11, 11, sh=11, sw=11, ph=500, pw=500, fmt=(1, 1, 1)),
]


@pytest.mark.parametrize("case", WIDE, ids=[c[0] for c in WIDE])
def test_wide_folded_layer(oracle, case):
    _, d, _, fmt = case
    src, w = cases.make_inputs(case)
    want = oracle.convolution(cases.oracle_shape(case), src, w)
    conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NHWC if fmt[0] else xb.NCHW, xb.HWIO if fmt[1] else xb.OIHW,
                          xb.NHWC if fmt[2] else xb.NCHW, d["mb"], d["oc"], d["ic"], d["ih"], d["iw"],
                          d["kh"], d["kw"], d["sh"], d["sw"], d["ph"], d["pw"], w)
    assert conv.kernel == xb.KERNEL_TCGEN05_I8  # folded, not the popcount kernel
    for _ in range(2):
        dst = np.full(want["dst"].size, np.nan, np.float32)
        conv.forward(src, dst)
        assert np.array_equal(conv.forward_sums(), want["sums"])
        assert np.array_equal(conv.read(xb.SLOT_A, np.float32), want["a"])
        assert np.array_equal(conv.read(xb.SLOT_K, np.float32), want["k"])
        assert np.all(np.abs(dst - want["dst"]) <= 1e-4 * np.abs(want["dst"]))
    conv.close()
