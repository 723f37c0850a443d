"""Layers whose position tiles are loaded once, as 16-byte channel columns, beside filters that stay in
shared memory: one to seven columns a position (odd numbers take the next position's first one with
them), rows of taps and folded layers, tiles of exactly 256 positions and of one more (which take the
other form), an odd number of tiles, one group of operands and more groups than filter barriers. Sums
and K bit for bit against the oracle, floats to the parity contract's 1e-4."""
import numpy as np
import pytest

import cases
import xnor_nn_b200 as xb

pytestmark = pytest.mark.gpu

# (name, mb, oc, ic, ih, iw, kh, kw): more than 148 tiles of 128 positions, so pairs take several
COLUMNS = [
    cases._c("one_column", 1300, 32, 20, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("one_column_seven_taps", 700, 32, 9, 5, 5, 7, 7, ph=3, pw=3),
    cases._c("two_columns", 1300, 64, 64, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("three_columns_five_taps", 800, 96, 75, 5, 4, 5, 5, ph=2, pw=2),
    cases._c("three_columns_wide_tiles", 760, 256, 96, 5, 5, 5, 5, ph=2, pw=2),
    cases._c("five_columns", 1300, 64, 131, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("seven_columns_no_border", 1300, 96, 224, 4, 4, 2, 3),
    cases._c("one_row_of_taps", 1300, 32, 70, 4, 5, 1, 3),
    cases._c("256_positions", 80, 32, 40, 3, 61, 3, 5, ph=1, pw=1),
    cases._c("257_positions", 80, 32, 40, 3, 62, 3, 4, ph=1, pw=1),
    cases._c("folded_two_rows", 700, 64, 40, 10, 11, 3, 3, sh=2, sw=2, ph=1, pw=1),
    cases._c("folded_few_channels", 300, 96, 3, 27, 29, 11, 11, sh=4, sw=4, ph=2, pw=2),
]


@pytest.mark.parametrize("case", COLUMNS, ids=[c[0] for c in COLUMNS])
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
