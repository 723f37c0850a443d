"""Layers whose position tiles are loaded once, as 16-byte channel columns, beside filters that stay in
shared memory: one to seven columns a position (odd numbers take the next position's first one with
them), tiles of exactly 256 positions, even and odd numbers of tiles, one and two filter tiles, fewer
groups of operands than filter barriers, as many and more, filter rows of one instruction, two position
tiles in flight and eight. Beside them layers on the other side of the rule (few tiles a pair, one or two
filter rows, 257 positions, folded layers), whose tiles have rows of 128 bytes. test_tile_launch_cpu.py
pins which form each takes. Sums and K bit for bit against the oracle, floats to the parity contract's
1e-4."""
import numpy as np
import pytest

import cases
import xnor_nn_b200 as xb

pytestmark = pytest.mark.gpu

# (name, mb, oc, ic, ih, iw, kh, kw): more than 148 tiles of 128 positions, so pairs take several
COLUMNS = [
    cases._c("one_column", 1300, 32, 20, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("one_column_seven_taps", 700, 32, 9, 5, 5, 7, 7, ph=3, pw=3),
    cases._c("one_column_rows_of_one_instruction", 2000, 32, 32, 4, 5, 3, 2),
    cases._c("two_columns_96_filters", 1600, 96, 64, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("two_columns_eight_groups", 1000, 64, 64, 7, 4, 8, 3, ph=1, pw=1),
    cases._c("three_columns_ten_groups", 1000, 96, 75, 5, 4, 5, 5, ph=2, pw=2),
    cases._c("three_columns_256_filters", 850, 256, 96, 5, 5, 5, 5, ph=2, pw=2),
    cases._c("three_columns_two_filter_tiles", 1600, 290, 70, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("five_columns_three_tiles", 1600, 64, 131, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("seven_columns_three_rows_no_border", 2000, 96, 224, 5, 4, 3, 3),
    cases._c("256_positions_three_tiles", 160, 96, 40, 3, 61, 3, 5, ph=1, pw=1),
    cases._c("two_tiles_in_flight", 160, 256, 224, 3, 61, 3, 3, ph=1, pw=1),
]
ROWS = [
    cases._c("two_columns", 1300, 64, 64, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("three_columns_five_taps", 800, 96, 75, 5, 4, 5, 5, ph=2, pw=2),
    cases._c("three_columns_wide_tiles", 760, 256, 96, 5, 5, 5, 5, ph=2, pw=2),
    cases._c("five_columns", 1300, 64, 131, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("seven_columns_no_border", 1300, 96, 224, 4, 4, 2, 3),
    cases._c("one_row_of_taps", 1300, 32, 70, 4, 5, 1, 3),
    cases._c("one_group", 1300, 32, 32, 4, 5, 1, 3),
    cases._c("one_group_of_one_instruction", 2000, 32, 20, 3, 5, 1, 2),
    cases._c("256_positions", 80, 32, 40, 3, 61, 3, 5, ph=1, pw=1),
    cases._c("257_positions", 80, 32, 40, 3, 62, 3, 4, ph=1, pw=1),
    cases._c("257_positions_three_tiles", 160, 96, 40, 3, 62, 3, 4, ph=1, pw=1),
    cases._c("folded_two_rows", 700, 64, 40, 10, 11, 3, 3, sh=2, sw=2, ph=1, pw=1),
    cases._c("folded_few_channels", 300, 96, 3, 27, 29, 11, 11, sh=4, sw=4, ph=2, pw=2),
]


@pytest.mark.parametrize("case", COLUMNS + ROWS, ids=[c[0] for c in COLUMNS + ROWS])
def test_position_columns_against_the_oracle(oracle, case):
    _, d, _, _ = case
    src, w = cases.make_inputs(case)
    want = oracle.convolution(cases.oracle_shape(case), src, w)
    conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NCHW, xb.OIHW, xb.NCHW, d["mb"], d["oc"], d["ic"],
                          d["ih"], d["iw"], d["kh"], d["kw"], d["sh"], d["sw"], d["ph"], d["pw"], w)
    dst = np.full(want["dst"].size, np.nan, np.float32)
    conv.forward(src, dst)
    assert np.array_equal(conv.forward_sums(), want["sums"])
    assert np.array_equal(conv.read(xb.SLOT_K, np.float32), want["k"])
    assert np.all(np.abs(dst - want["dst"]) <= 1e-4 * np.abs(want["dst"]))
    conv.close()
