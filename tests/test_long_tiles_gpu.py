"""Pairs whose tiles keep the tensor pipe busy for long have eight epilogue warps instead of sixteen
(conv_tcgen05.cu): every float store of theirs on tensors that live on the GPU, so that the whole minibatch is
one launch: NCHW, channels-last in 32-byte, 16-byte and single stores and on a result between two 16-byte
boundaries, accumulators that share columns and that do not, one and two filter tiles, filters of zeros (the
results' signs). test_tile_launch_cpu.py pins which layers take them. Sums and K bit for bit against the
oracle, floats to the parity contract's 1e-4."""
import numpy as np
import pytest

import cases
import xnor_nn_b200 as xb

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

NHWC = (0, 0, 1)
LONG_TILES = [
    cases._c("nchw_256_filters", 6400, 256, 320, 2, 2, 3, 3, ph=1, pw=1),
    cases._c("nchw_192_filters", 6400, 192, 384, 2, 2, 3, 3, ph=1, pw=1),
    cases._c("nchw_five_taps_odd_filters", 4000, 250, 96, 3, 2, 5, 5, ph=2, pw=2),
    cases._c("nchw_two_filter_tiles", 3250, 500, 320, 2, 2, 3, 3, ph=1, pw=1),
    cases._c("nhwc_256_filters", 6400, 256, 320, 2, 2, 3, 3, ph=1, pw=1, fmt=NHWC),
    cases._c("nhwc_252_filters", 6400, 252, 320, 2, 2, 3, 3, ph=1, pw=1, fmt=NHWC),
    cases._c("nhwc_251_filters", 6400, 251, 320, 2, 2, 3, 3, ph=1, pw=1, fmt=NHWC),
]


@pytest.mark.parametrize("case", LONG_TILES, ids=[c[0] for c in LONG_TILES])
def test_long_tiles_against_the_oracle(oracle, case):
    _, d, _, fmt = case
    src, w = cases.make_inputs(case)
    w.reshape(d["oc"], -1)[[0, 5, d["oc"] - 1]] = 0.0
    want = oracle.convolution(cases.oracle_shape(case), src, w)
    zeros = want["dst"] == 0
    assert np.signbit(want["dst"][zeros]).any()
    conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NCHW, xb.OIHW, xb.NHWC if fmt[2] else xb.NCHW, d["mb"],
                          d["oc"], d["ic"], d["ih"], d["iw"], d["kh"], d["kw"], d["sh"], d["sw"], d["ph"],
                          d["pw"], w)
    src = torch.from_numpy(src).cuda()
    n = want["dst"].size
    for shift in (0, 1) if fmt[2] else (0,):
        buffer = torch.full((n + 1,), float("nan"), device="cuda")
        torch.cuda.synchronize()
        before = xb.kernel_launches()
        conv.forward(src, buffer[shift:shift + n])
        assert xb.kernel_launches() - before == 2
        conv.synchronize()
        dst = buffer[shift:shift + n].cpu().numpy()
        assert np.all(np.abs(dst - want["dst"]) <= 1e-4 * np.abs(want["dst"]))
        assert np.array_equal(dst == 0, zeros)
        assert np.array_equal(np.signbit(dst), np.signbit(want["dst"]))
    assert np.array_equal(conv.forward_sums(), want["sums"])
    assert np.array_equal(conv.read(xb.SLOT_K, np.float32), want["k"])
    conv.close()
