"""Layers whose filters stay in shared memory while a pair of SMs walks its position tiles: several
rounds of tiles, one and several filter tiles, odd and even numbers of operand groups, accumulators
that overlap, and a last round that only some pairs take part in. With position tiles of 128-, 64- and
32-byte rows: one tap and three per filter row, folded layers, filter rows as one operand. And as
16-byte columns (test_tile_launch_cpu.py pins which layer takes which form). Sums and K bit for bit
against the oracle, floats to the parity contract's 1e-4."""
import numpy as np
import pytest

import cases
import xnor_nn_b200 as xb

pytestmark = pytest.mark.gpu

# (name, mb, oc, ic, ih, iw, kh, kw): more than 148 tiles of 128 positions, or several filter tiles
COLUMNS = [
    cases._c("row_of_taps_as_one_even_groups", 1200, 32, 60, 4, 4, 5, 5, ph=2, pw=2),
    cases._c("overlapping_accumulators", 1600, 250, 33, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("two_filter_tiles", 1600, 290, 33, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("three_filter_tiles", 900, 560, 20, 5, 5, 3, 3, ph=1, pw=1),
]
ROWS = [
    cases._c("row_of_taps_as_one_odd_groups", 1600, 32, 40, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("three_taps_a_row", 1600, 32, 250, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("three_taps_a_row_two_chunks", 1600, 32, 300, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("two_rows", 2400, 64, 130, 4, 4, 2, 1),
    cases._c("single_tap", 2400, 64, 130, 4, 4, 1, 1),
    cases._c("single_tap_overlapping_accumulators", 2400, 250, 130, 4, 4, 1, 1),
    cases._c("three_rows_overlapping_accumulators", 1600, 256, 130, 6, 4, 3, 1),
    cases._c("three_taps_overlapping_accumulators", 1600, 250, 250, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("single_tap_two_filter_tiles", 2400, 290, 130, 4, 4, 1, 1),
    cases._c("three_taps_two_filter_tiles", 1600, 290, 250, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("three_taps_three_filter_tiles", 800, 560, 250, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("rows_of_32_bytes_single_tap", 2400, 64, 60, 4, 4, 1, 1),
    cases._c("rows_of_64_bytes_single_tap", 2400, 64, 90, 4, 4, 1, 1),
    cases._c("rows_of_32_bytes_wide_image", 40, 32, 20, 12, 90, 3, 2, ph=1, pw=1),
    cases._c("rows_of_64_bytes_wide_image", 40, 32, 20, 12, 90, 3, 3, ph=1, pw=1),
    cases._c("folded_overlapping_accumulators", 700, 256, 40, 10, 11, 3, 3, sh=2, sw=2, ph=1, pw=1),
    cases._c("folded_few_channels", 450, 96, 3, 27, 29, 11, 11, sh=4, sw=4, ph=2, pw=2),
]
RESIDENT = COLUMNS + ROWS


@pytest.mark.parametrize("case", RESIDENT, ids=[c[0] for c in RESIDENT])
def test_resident_filters_against_the_oracle(oracle, case):
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
