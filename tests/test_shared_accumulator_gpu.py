"""Several threads issue MMAs into one accumulator: four in the one-launch pass (conv_whole.cu), two in the
position-tile kernel. Sums of integers do not depend on the order, but none may be lost. Many passes of layers
with the fewest and many K chunks, narrow and 256-wide filter tiles, results bit for bit the same and the sums
those of the oracle."""
import numpy as np
import pytest

import cases
import xnor_nn_b200 as xb

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

LAYERS = [
    cases._c("whole_narrow_one_chunk", 1, 64, 64, 13, 13, 3, 3, ph=1, pw=1),
    cases._c("whole_narrow_two_chunks", 1, 256, 512, 13, 13, 3, 3, ph=1, pw=1),
    cases._c("whole_one_tap_three_chunks", 2, 256, 640, 13, 13, 1, 1),
    cases._c("whole_256_one_chunk", 40, 256, 60, 13, 13, 3, 3, ph=1, pw=1),
    cases._c("whole_256_two_chunks", 30, 256, 384, 13, 13, 3, 3, ph=1, pw=1),
    cases._c("pairs_columns", 75, 256, 96, 27, 27, 3, 3, ph=1, pw=1),
    cases._c("pairs_streamed", 120, 256, 384, 13, 13, 3, 3, ph=1, pw=1),
]


@pytest.mark.parametrize("case", LAYERS, ids=[c[0] for c in LAYERS])
def test_no_sum_is_lost(oracle, case):
    _, d, _, _ = case
    src, w = cases.make_inputs(case)
    want = oracle.convolution(cases.oracle_shape(case), src, w)
    conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NCHW, xb.OIHW, xb.NCHW, d["mb"], d["oc"], d["ic"], d["ih"],
                          d["iw"], d["kh"], d["kw"], d["sh"], d["sw"], d["ph"], d["pw"], w)
    src = torch.from_numpy(src).cuda()
    first = torch.empty(want["dst"].size, device="cuda")
    torch.cuda.synchronize()
    before = xb.kernel_launches()
    conv.forward(src, first)
    assert xb.kernel_launches() - before == (1 if case[0].startswith("whole") else 2)
    conv.synchronize()
    got = first.cpu().numpy()
    assert np.all(np.abs(got - want["dst"]) <= 1e-4 * np.abs(want["dst"]))
    assert np.array_equal(conv.forward_sums(), want["sums"])
    again = torch.empty_like(first)
    differ = torch.zeros((), dtype=torch.int64, device="cuda")
    conv.set_stream(torch.cuda.current_stream().cuda_stream or 1)  # 1: the legacy default stream
    for _ in range(300):
        again.fill_(float("nan"))
        conv.forward(src, again)
        differ += (again != first).sum()
    assert int(differ) == 0
    conv.close()
