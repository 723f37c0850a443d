"""The box filter behind K in its forms (binarize.cu): an output a thread with and without a compiled width,
by columns with one and two outputs a thread, on both sides of the rule (127 and 128 outputs an image) and
beyond shared memory. Odd numbers of output rows, rows of more outputs than a block has threads, staged rows
wider than a block, windows that leave the image on every side. K bit for bit against the oracle. (On the
popcount kernel, for which every pass runs the box filter on its own.)"""
import numpy as np
import pytest

import cases
import xnor_nn_b200 as xb

pytestmark = pytest.mark.gpu

# (width and height of the window, stride, image sides, padding)
FORMS = [
    (1, 2, (31, 33), 0), (2, 1, (20, 21), 1), (3, 1, (16, 18), 1), (3, 1, (5, 300), 1), (3, 3, (40, 41), 2),
    # by columns, one output: 128 outputs, 127, two passes over the columns of a staged row
    (5, 1, (16, 8), 2), (5, 1, (127, 1), 2), (5, 1, (9, 300), 2), (5, 2, (31, 33), 2), (5, 2, (13, 15), 2),
    (5, 4, (60, 61), 2),
    # two outputs: an even and an odd number of rows, few outputs, one row
    (7, 1, (16, 8), 3), (7, 1, (127, 1), 3), (7, 1, (23, 29), 3), (7, 1, (7, 300), 0), (7, 2, (33, 35), 3),
    (7, 2, (13, 15), 3), (7, 3, (50, 52), 3), (11, 4, (60, 63), 5), (11, 4, (30, 31), 0), (11, 5, (60, 60), 5),
    (8, 1, (20, 21), 4), (9, 2, (40, 43), 9), (9, 3, (60, 61), 8), (13, 1, (12, 40), 6), (13, 6, (90, 91), 0),
    (16, 8, (130, 131), 8), (9, 1, (40, 1100), 4),
]


@pytest.mark.parametrize("k, stride, sides, pad", FORMS)
def test_box_filter(oracle, k, stride, sides, pad):
    case = cases._c("box_%d_%d_%d_%d_%d" % (k, stride, *sides, pad), 3, 8, 3, *sides, k, k, sh=stride, sw=stride,
                    ph=pad, pw=pad)
    d = case[1]
    src, w = cases.make_inputs(case)
    want = oracle.convolution(cases.oracle_shape(case), src, w)
    conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NCHW, xb.OIHW, xb.NCHW, d["mb"], d["oc"], d["ic"], d["ih"],
                          d["iw"], d["kh"], d["kw"], d["sh"], d["sw"], d["ph"], d["pw"], w,
                          kernel=xb.KERNEL_POPC)
    dst = np.full(want["dst"].size, np.nan, np.float32)
    conv.forward(src, dst)
    assert np.array_equal(conv.read(xb.SLOT_A, np.float32), want["a"])
    assert np.array_equal(conv.read(xb.SLOT_K, np.float32), want["k"])
    conv.close()
