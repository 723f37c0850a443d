"""Streamed filters beside position tiles that serve all filter rows (producer_halo and mma_role_halo in
conv_tcgen05.cu), whose two issuers take the taps of all rows in turn: an even and an odd number of taps, filter
rows of two taps and of nine, a box of 256 rows, five filter rows, one, three and four chunks, the last one full
and not, two filter tiles, accumulators that overlap, an odd number of position tiles; and the first layers
beyond, which have a tile for each filter row. test_streamed_blocks_cpu.py pins which layers take which. Sums and
K bit for bit against the oracle, floats to the parity contract's 1e-4. A commit that is lost makes a wait run out,
and the next pass is right."""
import ctypes as C

import numpy as np
import pytest

import cases
import xnor_nn_b200 as xb

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

BLOCKS = [
    cases._c("odd_taps", 1601, 256, 544, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("even_taps", 1601, 192, 1000, 4, 4, 2, 2),
    cases._c("four_rows_of_two", 1601, 256, 1024, 5, 4, 4, 2),
    cases._c("three_rows_of_nine", 300, 256, 256, 9, 12, 3, 9),
    cases._c("256_rows", 40, 512, 544, 9, 62, 3, 3, ph=1, pw=1),
    cases._c("five_rows_192_filters", 1200, 192, 300, 5, 5, 5, 5, ph=2, pw=2),
    cases._c("25_taps_odd_rows_160_filters", 1200, 160, 340, 5, 5, 5, 5, ph=2, pw=2),
    cases._c("two_filter_tiles", 1000, 384, 600, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("odd_filters", 1601, 251, 577, 4, 4, 3, 3, ph=1, pw=1),
]
ROWS = [
    cases._c("257_rows", 40, 512, 800, 9, 64, 3, 2),
    cases._c("five_rows_256_filters", 1200, 256, 300, 5, 5, 5, 5, ph=2, pw=2),
    cases._c("25_taps_odd_rows_192_filters", 1200, 192, 340, 5, 5, 5, 5, ph=2, pw=2),
    cases._c("one_filter_row", 1601, 512, 900, 4, 6, 1, 3),
]


@pytest.mark.parametrize("case", BLOCKS + ROWS, ids=[c[0] for c in BLOCKS + ROWS])
def test_against_the_oracle(oracle, case):
    _, d, _, _ = case
    src, w = cases.make_inputs(case)
    want = oracle.convolution(cases.oracle_shape(case), src, w)
    conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NCHW, xb.OIHW, xb.NCHW, d["mb"], d["oc"], d["ic"], d["ih"],
                          d["iw"], d["kh"], d["kw"], d["sh"], d["sw"], d["ph"], d["pw"], w)
    src = torch.from_numpy(src).cuda()
    for _ in range(2):
        dst = torch.full((want["dst"].size,), float("nan"), device="cuda")
        torch.cuda.synchronize()
        conv.forward(src, dst)
        conv.synchronize()
        assert np.all(np.abs(dst.cpu().numpy() - want["dst"]) <= 1e-4 * np.abs(want["dst"]))
        assert np.array_equal(conv.forward_sums(), want["sums"])
        assert np.array_equal(conv.read(xb.SLOT_K, np.float32), want["k"])
    conv.close()


@pytest.mark.parametrize("name", ["odd_taps", "five_rows_192_filters", "five_rows_256_filters"])
def test_lost_commit_times_out_and_the_resources_stay_usable(name):
    case = next(c for c in BLOCKS + ROWS if c[0] == name)
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
