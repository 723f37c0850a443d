"""calculate_k of small layers in one launch (maps.cu): bands of one and of several rows, a last band that
is shorter or owns input rows no window sees, windows that leave the image on every side, strides, one to
sixteen tasks of 32 channels per pixel, both layouts with and without 16-byte loads; and the layers beyond
its limits, which take two launches. A and K bit for bit against the oracle."""
import numpy as np
import pytest

import cases
import xnor_nn_b200 as xb

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

CL = (1, 1, 1)
ONE_LAUNCH = [
    cases._c("one_pixel", 1, 8, 1, 1, 1, 1, 1),
    cases._c("ragged", 19, 101, 75, 31, 27, 3, 3, ph=1, pw=1),
    cases._c("bands_of_several_rows", 60, 16, 40, 11, 13, 3, 3, ph=1, pw=1),
    cases._c("five_by_five", 3, 16, 33, 14, 15, 5, 5, ph=2, pw=2),
    cases._c("eight_by_eight", 3, 16, 20, 14, 15, 8, 8, ph=3, pw=3),
    cases._c("stride_that_skips_rows", 2, 24, 70, 17, 15, 1, 1, sh=3, sw=3),
    cases._c("stride_2_rows_left_over", 5, 24, 40, 18, 15, 3, 3, sh=2, sw=2),
    cases._c("padding_as_large_as_the_filter", 2, 24, 20, 5, 6, 3, 3, ph=3, pw=3),
    cases._c("height_from_the_width_padding", 2, 24, 20, 9, 9, 3, 3, ph=0, pw=1),
    cases._c("512_channels", 3, 24, 512, 6, 7, 3, 3, ph=1, pw=1),
    cases._c("channels_last", 3, 44, 92, 10, 11, 3, 3, ph=1, pw=1, fmt=CL),
    cases._c("channels_last_odd", 3, 43, 91, 10, 11, 3, 3, ph=1, pw=1, fmt=CL),
]
# The height of the result follows from the padding of the width: blocks whose windows lie below the image
# altogether, which read nothing (test_map_bands_cpu.py walks what every block reads).
BELOW_THE_IMAGE = [
    cases._c("1x3_same", 8, 24, 64, 14, 14, 1, 3, ph=0, pw=1),
    cases._c("1x7_same", 8, 24, 64, 14, 14, 1, 7, ph=0, pw=3),
    cases._c("1x5_same", 4, 24, 64, 14, 14, 1, 5, ph=0, pw=2),
    cases._c("1x3_one_image_512_channels", 1, 24, 512, 56, 56, 1, 3, ph=0, pw=1),
    cases._c("3x3_no_rows_of_padding", 4, 24, 64, 9, 9, 3, 3, ph=0, pw=2),
    cases._c("1x1_padding_2", 2, 24, 64, 10, 10, 1, 1, ph=2, pw=2),
    cases._c("1x5_100x100", 1, 24, 64, 100, 100, 1, 5, ph=0, pw=2),
    cases._c("1x3_channels_last", 8, 24, 64, 14, 14, 1, 3, ph=0, pw=1, fmt=CL),
]
TWO_LAUNCHES = [
    cases._c("72_taps", 2, 16, 20, 14, 15, 9, 8, ph=4, pw=4),
    cases._c("over_16_megabytes", 65, 16, 64, 32, 32, 3, 3, ph=1, pw=1),
    cases._c("1025_channels_wide", 1, 16, 1025, 3, 64, 3, 3, ph=1, pw=1),
    # longer than two launches take: bands of 60 tasks, many blocks of few
    cases._c("long_bands", 19, 16, 464, 17, 17, 5, 5, ph=2, pw=2),
    cases._c("many_bands", 5, 16, 3, 161, 161, 5, 5, ph=2, pw=2),
]


def _run(oracle, case, launches):
    _, d, _, fmt = case
    src, w = cases.make_inputs(case)
    want = oracle.convolution(cases.oracle_shape(case), src, w)
    conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NHWC if fmt[0] else xb.NCHW,
                          xb.HWIO if fmt[1] else xb.OIHW, xb.NHWC if fmt[2] else xb.NCHW, d["mb"],
                          d["oc"], d["ic"], d["ih"], d["iw"], d["kh"], d["kw"], d["sh"], d["sw"],
                          d["ph"], d["pw"], w)
    dev = torch.from_numpy(np.ascontiguousarray(src)).cuda()
    torch.cuda.synchronize()
    before = xb.kernel_launches()
    assert conv.execute("calculate_k", src=dev) == xb.SUCCESS
    assert xb.kernel_launches() - before == launches
    assert np.array_equal(conv.read(xb.SLOT_A, np.float32), want["a"])
    assert np.array_equal(conv.read(xb.SLOT_K, np.float32), want["k"])
    conv.close()


@pytest.mark.parametrize("case", ONE_LAUNCH + BELOW_THE_IMAGE, ids=[c[0] for c in ONE_LAUNCH + BELOW_THE_IMAGE])
def test_one_launch(oracle, case):
    _run(oracle, case, 1)


@pytest.mark.parametrize("case", TWO_LAUNCHES, ids=[c[0] for c in TWO_LAUNCHES])
def test_beyond_its_limits(oracle, case):
    _run(oracle, case, 2)
