"""Channels-last results that are stored float by float (a number of filters that is no multiple of four, or a result
between two 16-byte boundaries) from the forms of the position-tile kernel whose tiles serve all filter rows: these
leave the L1 as much room as the forms with a tile for each filter row.
test_scattered_results_cpu.py pins which layer takes which form. Sums and K bit for bit against the oracle, floats to
the parity contract's 1e-4."""
import numpy as np
import pytest

import cases
import xnor_nn_b200 as xb

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

LAST = (0, 0, 1)
LAYERS = [
    cases._c("resident_few_filters", 1600, 29, 384, 4, 4, 3, 3, ph=1, pw=1, fmt=LAST),
    cases._c("resident_three_accumulators", 1600, 118, 300, 4, 4, 3, 3, ph=1, pw=1, fmt=LAST),
    cases._c("resident_two_filter_tiles", 1600, 313, 250, 4, 4, 3, 3, ph=1, pw=1, fmt=LAST),
    cases._c("half_of_192", 1600, 187, 352, 4, 4, 3, 3, ph=1, pw=1, fmt=LAST),
    cases._c("whole_256", 1600, 253, 311, 4, 4, 3, 3, ph=1, pw=1, fmt=LAST),
    cases._c("streamed_224", 90, 210, 448, 14, 37, 3, 3, fmt=LAST),
    cases._c("streamed_256", 1600, 251, 576, 4, 4, 3, 3, ph=1, pw=1, fmt=LAST),
]


def _conv(case):
    _, d, _, fmt = case
    src, w = cases.make_inputs(case)
    conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NCHW, xb.OIHW, xb.NHWC if fmt[2] else xb.NCHW, d["mb"], d["oc"],
                          d["ic"], d["ih"], d["iw"], d["kh"], d["kw"], d["sh"], d["sw"], d["ph"], d["pw"], w)
    return conv, src, w


@pytest.mark.parametrize("case", LAYERS, ids=[c[0] for c in LAYERS])
def test_against_the_oracle(oracle, case):
    conv, src, w = _conv(case)
    want = oracle.convolution(cases.oracle_shape(case), src, w)
    src = torch.from_numpy(src).cuda()
    room = torch.empty(want["dst"].size + 1, device="cuda")
    for dst in (room[:-1], room[1:]):  # the second between two 16-byte boundaries
        dst.fill_(float("nan"))
        torch.cuda.synchronize()
        conv.forward(src, dst)
        conv.synchronize()
        assert np.all(np.abs(dst.cpu().numpy() - want["dst"]) <= 1e-4 * np.abs(want["dst"]))
        assert np.array_equal(conv.forward_sums(), want["sums"])
        assert np.array_equal(conv.read(xb.SLOT_K, np.float32), want["k"])
    conv.close()
