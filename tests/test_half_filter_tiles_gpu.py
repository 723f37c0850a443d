"""Filter tiles of half a layer's width, whose filters stay in shared memory where the whole tile's would not
(conv_tcgen05.cu): a half that is part padding, operand rows that straddle
sectors and that do not, the last such number of tiles a pair, an odd number of position tiles, both orders of
the result; and the first layers beyond, which keep the whole width. test_half_filter_tiles_cpu.py pins which
layers take which. Sums and K bit for bit against the oracle, floats to the parity contract's 1e-4. A commit
that is lost makes a wait run out, and the next pass is right."""
import ctypes as C

import numpy as np
import pytest

import cases
import xnor_nn_b200 as xb

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

NHWC = (0, 0, 1)
HALVED = [
    cases._c("256_filters_odd_rows", 1700, 256, 288, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("part_padding", 1601, 250, 270, 4, 4, 3, 3, ph=1, pw=1, fmt=NHWC),
    cases._c("odd_rows_192_filters", 2400, 192, 350, 4, 3, 3, 3, ph=1, pw=1),
    cases._c("even_rows_192_filters", 1601, 192, 384, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("six_tiles_of_128", 700, 768, 290, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("even_rows_three_tiles_a_pair", 2200, 256, 512, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("odd_rows_four_tiles_a_pair", 3000, 256, 288, 4, 4, 3, 3, ph=1, pw=1),
]
WHOLE = [
    cases._c("128_filters", 3100, 128, 480, 4, 4, 4, 3, ph=1, pw=1),
    cases._c("even_rows_four_tiles_a_pair", 2400, 256, 320, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("even_rows_192_filters_four_tiles", 3200, 192, 384, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("two_filter_rows", 1601, 256, 608, 4, 4, 2, 3, ph=1, pw=1),
    cases._c("half_does_not_fit", 1200, 256, 544, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("a_round_more_for_one_tile_a_pair", 500, 768, 290, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("whole_fits", 1601, 256, 240, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("halves_that_do_not_split", 1601, 160, 480, 4, 4, 3, 3, ph=1, pw=1),
]


@pytest.mark.parametrize("case", HALVED + WHOLE, ids=[c[0] for c in HALVED + WHOLE])
def test_against_the_oracle(oracle, case):
    _, d, _, fmt = case
    src, w = cases.make_inputs(case)
    want = oracle.convolution(cases.oracle_shape(case), src, w)
    conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NCHW, xb.OIHW, xb.NHWC if fmt[2] else xb.NCHW, d["mb"],
                          d["oc"], d["ic"], d["ih"], d["iw"], d["kh"], d["kw"], d["sh"], d["sw"], d["ph"],
                          d["pw"], w)
    src = torch.from_numpy(src).cuda()
    dst = torch.full((want["dst"].size,), float("nan"), device="cuda")
    torch.cuda.synchronize()
    conv.forward(src, dst)
    conv.synchronize()
    assert np.all(np.abs(dst.cpu().numpy() - want["dst"]) <= 1e-4 * np.abs(want["dst"]))
    assert np.array_equal(conv.forward_sums(), want["sums"])
    assert np.array_equal(conv.read(xb.SLOT_K, np.float32), want["k"])
    conv.close()


@pytest.mark.parametrize("case", HALVED[:2], ids=[c[0] for c in HALVED[:2]])
def test_lost_commit_times_out_and_the_resources_stay_usable(case):
    _, d, _, _ = case
    src, w = cases.make_inputs(case)
    conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NCHW, xb.OIHW, xb.NCHW, d["mb"], d["oc"], d["ic"], d["ih"],
                          d["iw"], d["kh"], d["kw"], d["sh"], d["sw"], d["ph"], d["pw"], w)
    src = torch.from_numpy(src).cuda()
    good = torch.zeros(int(np.prod(conv.out_shape)), device="cuda")
    torch.cuda.synchronize()
    conv.forward(src, good)
    conv.synchronize()
    junk, again = torch.zeros_like(good), torch.zeros_like(good)
    torch.cuda.synchronize()
    conv._set(xb.SLOT_USER_DST, junk)
    st = xb.lib().xnor_nn_b200_selftest_lost_commit(C.byref(conv.c), conv.res, 5)
    assert st == xb.UNIMPLEMENTED
    assert "gave up waiting (site " in xb.last_error()
    conv.synchronize()  # the error word was consumed
    conv.forward(src, again)
    conv.synchronize()
    assert torch.equal(again, good)
    conv.close()
