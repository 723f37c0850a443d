"""The position-tile kernel (conv_tcgen05.cu) on layers that Convolution.forward runs in one launch of another
kernel (conv_whole.cu): through the three executors, whose last one is always this kernel, with K from the
map. And on layers just beyond that kernel, with K box-filtered in the epilogue: one CTA a tile (a filter tile
that does not split into two) and pairs. Every form of the float stores, with filters of zeros. Sums, K, zeros
and signs bit for bit against the oracle, floats to the parity contract's 1e-4."""
import numpy as np
import pytest

import cases
import xnor_nn_b200 as xb

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

NHWC = (0, 0, 1)


def _layer(name, mb, oc, fmt=(0, 0, 0)):
    return cases._c(name, mb, oc, 40, 13, 13, 3, 3, ph=1, pw=1, fmt=fmt)


SMALL = [
    cases._c("nchw", 2, 48, 40, 9, 11, 3, 3, ph=1, pw=1),
    cases._c("nhwc", 2, 48, 40, 9, 11, 3, 3, ph=1, pw=1, fmt=NHWC),
    cases._c("nhwc_16_bytes", 2, 20, 40, 9, 11, 3, 3, ph=1, pw=1, fmt=NHWC),
    cases._c("nhwc_odd", 2, 13, 40, 9, 11, 3, 3, ph=1, pw=1, fmt=NHWC),
    cases._c("nhwc_oc20", 2, 20, 37, 6, 7, 3, 3, ph=1, pw=1, fmt=NHWC),
    cases._c("nhwc_oc13", 2, 13, 37, 6, 7, 3, 3, ph=1, pw=1, fmt=NHWC),
    cases._c("8_tiles_two_filter_tiles", 38, 512, 8, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("11_tiles_two_filter_tiles", 150, 384, 8, 2, 2, 3, 3, ph=1, pw=1),
    cases._c("conv4_one_image", 1, 256, 384, 13, 13, 3, 3, ph=1, pw=1),
    cases._c("conv4_30_images", 30, 256, 384, 13, 13, 3, 3, ph=1, pw=1),
    cases._c("conv4_channels_last", 20, 256, 384, 13, 13, 3, 3, ph=1, pw=1, fmt=(1, 1, 1)),
]
LARGE = [  # 245 tiles
    _layer("single_nchw", 160, 48), _layer("single_nchw_odd", 160, 45),
    _layer("single_nhwc", 160, 48, NHWC), _layer("single_nhwc_16_bytes", 160, 44, NHWC),
    _layer("single_nhwc_odd", 160, 13, NHWC), _layer("single_nhwc_two_tiles", 160, 270, NHWC),
    _layer("pairs_nhwc_16_bytes", 160, 20, NHWC), _layer("pairs_nhwc_odd", 160, 61, NHWC),
]


@pytest.mark.parametrize("case", SMALL + LARGE, ids=[c[0] for c in SMALL + LARGE])
def test_position_tiles(oracle, case):
    _, d, _, fmt = case
    src, w = cases.make_inputs(case)
    zero = [0, 5, d["oc"] - 1]
    if fmt[1]:
        w[..., zero] = 0.0
    else:
        w.reshape(d["oc"], -1)[zero] = 0.0
    want = oracle.convolution(cases.oracle_shape(case), src, w)
    zeros = want["dst"] == 0
    assert np.signbit(want["dst"][zeros]).any()
    conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NHWC if fmt[0] else xb.NCHW,
                          xb.HWIO if fmt[1] else xb.OIHW, xb.NHWC if fmt[2] else xb.NCHW, d["mb"],
                          d["oc"], d["ic"], d["ih"], d["iw"], d["kh"], d["kw"], d["sh"], d["sw"],
                          d["ph"], d["pw"], w, kernel=xb.KERNEL_TCGEN05_I8)
    src = torch.from_numpy(src).cuda()
    dst = torch.full((want["dst"].size,), float("nan"), device="cuda")
    torch.cuda.synchronize()
    before = xb.kernel_launches()
    if case in SMALL:
        conv.forward_stepwise(src, dst)
        assert xb.kernel_launches() - before == 3  # packer, maps, this kernel
    else:
        conv.forward(src, dst)
        assert xb.kernel_launches() - before == 2  # packer, this kernel
    conv.synchronize()
    dst = dst.cpu().numpy()
    assert np.all(np.abs(dst - want["dst"]) <= 1e-4 * np.abs(want["dst"]))
    assert np.array_equal(dst == 0, zeros)
    assert np.array_equal(np.signbit(dst), np.signbit(want["dst"]))
    assert np.array_equal(conv.forward_sums(), want["sums"])
    assert np.array_equal(conv.read(xb.SLOT_K, np.float32), want["k"])
    conv.close()
