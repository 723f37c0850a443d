"""Resident filters beside position tiles that serve all filter rows (producer_block and mma_role_block in
conv_tcgen05.cu), at the edges of what that takes: a box of 256 rows, two tiles in flight, eight filter rows'
and chunks' barriers, channel tails of the last chunk, an odd number of tiles, two and three filter tiles,
accumulators that overlap, folded layers; and the first layers beyond, which have a tile for each filter row.
test_position_blocks_cpu.py pins which layers take which. Sums, A and K bit for bit against the oracle, floats
to the parity contract's 1e-4. A commit that is lost makes a wait run out, and the next pass is right."""
import ctypes as C

import numpy as np
import pytest

import cases
import xnor_nn_b200 as xb

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

BLOCKS = [
    cases._c("256_rows", 41, 32, 130, 8, 64, 3, 1),
    cases._c("eight_groups", 1600, 32, 300, 4, 4, 4, 3, ph=1, pw=1),
    cases._c("two_tiles_in_flight", 90, 128, 480, 17, 29, 3, 3, ph=1, pw=1),
    cases._c("channel_tail_of_the_second_chunk", 1600, 64, 270, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("two_filter_tiles", 1600, 384, 256, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("three_filter_tiles", 900, 560, 250, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("overlapping_accumulators", 1601, 256, 130, 6, 4, 3, 1),
    cases._c("a_filter_row_as_one", 1100, 96, 60, 4, 4, 2, 3, ph=1, pw=1),
    cases._c("folded", 450, 96, 3, 27, 29, 11, 11, sh=4, sw=4, ph=2, pw=2),
]
ROWS = [
    cases._c("257_rows", 41, 32, 240, 8, 64, 3, 2),
    cases._c("nine_groups", 1600, 32, 520, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("one_filter_row", 1600, 32, 300, 4, 6, 1, 3),
    cases._c("rows_of_64_bytes", 2400, 64, 90, 4, 4, 2, 1),
]


def _conv(case):
    _, d, _, _ = case
    src, w = cases.make_inputs(case)
    conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NCHW, xb.OIHW, xb.NCHW, d["mb"], d["oc"], d["ic"], d["ih"],
                          d["iw"], d["kh"], d["kw"], d["sh"], d["sw"], d["ph"], d["pw"], w)
    return conv, src, w


@pytest.mark.parametrize("case", BLOCKS + ROWS, ids=[c[0] for c in BLOCKS + ROWS])
def test_against_the_oracle(oracle, case):
    conv, src, w = _conv(case)
    want = oracle.convolution(cases.oracle_shape(case), src, w)
    src = torch.from_numpy(src).cuda()
    for _ in range(2):
        dst = torch.full((want["dst"].size,), float("nan"), device="cuda")
        torch.cuda.synchronize()
        conv.forward(src, dst)
        conv.synchronize()
        assert np.all(np.abs(dst.cpu().numpy() - want["dst"]) <= 1e-4 * np.abs(want["dst"]))
        assert np.array_equal(conv.forward_sums(), want["sums"])
        assert np.array_equal(conv.read(xb.SLOT_A, np.float32), want["a"])
        assert np.array_equal(conv.read(xb.SLOT_K, np.float32), want["k"])
    conv.close()


@pytest.mark.parametrize("case", BLOCKS[:2], ids=[c[0] for c in BLOCKS[:2]])
def test_lost_commit_times_out_and_the_resources_stay_usable(case):
    conv, src, _ = _conv(case)
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
