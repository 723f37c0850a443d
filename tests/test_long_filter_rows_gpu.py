"""Position columns with filter rows of 1 KB and more: 32 instructions a row, of which a lane knows the
start of one each, and more, whose starts are worked out chunk by chunk. Two to seven columns a position,
chunks that are not full, up to 22 of them. test_tile_launch_cpu.py pins that they take columns. Sums and K
bit for bit against the oracle, floats to the parity contract's 1e-4."""
import numpy as np
import pytest

import cases
import xnor_nn_b200 as xb

pytestmark = pytest.mark.gpu

LONG_ROWS = [
    cases._c("32_instructions", 700, 32, 112, 2, 20, 3, 16, ph=1, pw=1),
    cases._c("36_instructions_two_columns", 290, 96, 39, 2, 38, 3, 33, ph=2, pw=2),
    cases._c("36_instructions_five_columns", 900, 64, 150, 2, 16, 3, 14, ph=1, pw=1),
    cases._c("40_instructions", 600, 32, 112, 2, 24, 3, 19, ph=1, pw=1),
    cases._c("88_instructions_seven_columns", 520, 32, 214, 2, 26, 3, 25, ph=1, pw=1),
]


@pytest.mark.parametrize("case", LONG_ROWS, ids=[c[0] for c in LONG_ROWS])
def test_long_filter_rows_against_the_oracle(oracle, case):
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
