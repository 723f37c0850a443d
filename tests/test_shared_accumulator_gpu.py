"""Several threads issue MMAs into one accumulator: four in the one-launch pass (conv_whole.cu), two in the
position-tile kernel, on single CTAs and on pairs, beside streamed filters (position tiles for one filter row and for
all of them), resident ones, columns, and in chained layers. Sums of integers do not depend on the order, but none
may be lost. Many passes of layers with the fewest and many K chunks, narrow and 256-wide filter tiles, results
bit for bit the same and the sums those of the oracle. test_tile_launch_cpu.py and test_chain_pairs_cpu.py pin
which form each layer takes: the one it is called after, but for pairs_streamed, whose filters are resident."""
import numpy as np
import pytest

import cases
import test_chain_pairs_gpu as chains
import xnor_nn_b200 as xb
from oracle.pyoracle import Shape
from xnor_nn_b200 import synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

LAYERS = [
    cases._c("whole_narrow_one_chunk", 1, 64, 64, 13, 13, 3, 3, ph=1, pw=1),
    cases._c("whole_narrow_two_chunks", 1, 256, 512, 13, 13, 3, 3, ph=1, pw=1),
    cases._c("whole_one_tap_three_chunks", 2, 256, 640, 13, 13, 1, 1),
    cases._c("whole_256_one_chunk", 40, 256, 60, 13, 13, 3, 3, ph=1, pw=1),
    cases._c("whole_256_two_chunks", 30, 256, 384, 13, 13, 3, 3, ph=1, pw=1),
    cases._c("pairs_columns", 75, 256, 96, 27, 27, 3, 3, ph=1, pw=1),
    cases._c("pairs_streamed", 120, 256, 384, 13, 13, 3, 3, ph=1, pw=1),  # resident: halves of its filter tiles fit
    cases._c("pairs_streamed_256_filters", 120, 256, 640, 13, 13, 3, 3, ph=1, pw=1),
    cases._c("pairs_streamed_192_filters", 120, 192, 640, 13, 13, 3, 3, ph=1, pw=1),
    cases._c("pairs_streamed_a_filter_row_at_a_time", 1200, 256, 300, 5, 5, 5, 5, ph=2, pw=2),
    cases._c("single_ctas", 120, 144, 300, 13, 13, 3, 3, ph=1, pw=1),
]
CHAINS = ["columns", "rows_of_all_filter_rows", "streamed", "streamed_192_filters", "ring"]


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


@pytest.mark.parametrize("name", CHAINS)
def test_no_sum_is_lost_in_chained_layers(oracle, name):
    """The first of two layers, which hands signs and means on: what the second one makes of them."""
    mb, ic, oc, ih, iw, kh, kw, ph, pw = chains.PAIRS[name]
    oh, ow = ih + 2 * ph - kh + 1, iw + 2 * pw - kw + 1
    layers = [(mb, oc, ic, ih, iw, kh, kw, 1, 1, ph, pw), (mb, 16, oc, oh, ow, 3, 3, 1, 1, 1, 1)]
    x = src = synth.normal(len(name), mb * ic * ih * iw)
    convs = []
    for i, d in enumerate(layers):
        w = synth.normal(5 + i, d[1] * d[2] * d[5] * d[6], 0.05)
        convs.append(xb.Convolution(xb.ALGORITHM_BCAST, xb.NCHW, xb.OIHW, xb.NCHW, *d, w))
        want = oracle.convolution(Shape.make(*d, 0, 0, 0), x, w)
        x = want["dst"]
    src = torch.from_numpy(src).cuda()
    first = torch.empty(x.size, device="cuda")
    again = torch.empty_like(first)
    differ = torch.zeros((), dtype=torch.int64, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream or 1  # 1: the legacy default stream
    for conv in convs:
        conv.set_stream(stream)
    xb.forward_chain(convs, src, first)
    torch.cuda.synchronize()
    assert np.all(np.abs(first.cpu().numpy() - x) <= 1e-4 * np.abs(x))
    assert np.array_equal(convs[1].forward_sums(), want["sums"])
    for _ in range(300):
        again.fill_(float("nan"))
        xb.forward_chain(convs, src, again)
        differ += (again != first).sum()
    assert int(differ) == 0
    for conv in convs:
        conv.close()
