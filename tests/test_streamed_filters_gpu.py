"""Pairs of SMs whose filters do not fit shared memory: filter tiles stream through a ring while one
position tile with a halo serves a filter row, and two issuers take alternate filter tiles. An odd
number of them per position tile makes the issuers swap who starts the next one, and filter rows
split unevenly between them. More than two rounds of tiles; every sum and result against the popcount
kernel, the first and last images against the oracle as well."""
import numpy as np
import pytest

import cases
import xnor_nn_b200 as xb

pytestmark = pytest.mark.gpu

# 36 (5x5 filters) or 25 frame positions an image, more than 296 position tiles
STREAMED = [
    cases._c("25_steps_overlapping_accumulators", 1080, 256, 240, 4, 4, 5, 5, ph=2, pw=2),
    cases._c("25_steps_three_accumulators", 1080, 150, 240, 4, 4, 5, 5, ph=2, pw=2),
    cases._c("27_steps_channel_tail", 1560, 256, 520, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("27_steps_two_filter_tiles", 1560, 320, 530, 4, 4, 3, 3, ph=1, pw=1),
]


@pytest.mark.parametrize("case", STREAMED, ids=[c[0] for c in STREAMED])
def test_streamed_filters(oracle, case):
    _, d, _, _ = case
    src, w = cases.make_inputs(case)
    got = {}
    for kernel in (xb.KERNEL_TCGEN05_I8, xb.KERNEL_POPC):
        conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NCHW, xb.OIHW, xb.NCHW, d["mb"], d["oc"],
                              d["ic"], d["ih"], d["iw"], d["kh"], d["kw"], 1, 1, d["ph"], d["pw"],
                              w, kernel=kernel)
        assert conv.kernel == kernel
        dst = np.full(int(np.prod(conv.out_shape)), np.nan, np.float32)
        conv.forward(src, dst)
        got[kernel] = conv.forward_sums(), dst
        conv.close()
    for a, b in zip(got[xb.KERNEL_TCGEN05_I8], got[xb.KERNEL_POPC]):
        assert np.array_equal(a, b)
    sums, dst = got[xb.KERNEL_TCGEN05_I8]
    for first, n in ((0, 2), (d["mb"] - 1, 1)):
        shape = cases.oracle_shape((case[0], dict(d, mb=n), case[2], case[3]))
        want = oracle.convolution(shape, np.ascontiguousarray(src[first:first + n]), w)
        per = want["dst"].size // n
        assert np.array_equal(sums[first * per:(first + n) * per], want["sums"])
        assert np.array_equal(dst[first * per:(first + n) * per], want["dst"])
