"""The tensor-core kernels add +-1 products in fp32, which is exact as long as no sum leaves the range
in which every integer is a float: 2^24 operands at most (larger layers run on the popcount kernel,
test_plan_routes_cpu.py). One output pixel with hundreds of thousands of operands, and with all 2^24
of them: sums near the ends of that range and near zero, alpha and the results against the oracle."""
import numpy as np
import pytest

import xnor_nn_b200 as xb
from oracle.pyoracle import Shape

pytestmark = pytest.mark.gpu


def _check(oracle, ic, k, oc, src, w, kernel):
    want = oracle.convolution(Shape.make(1, oc, ic, k, k, k, k), src, w)
    conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NCHW, xb.OIHW, xb.NCHW, 1, oc, ic, k, k, k, k, 1, 1,
                          0, 0, w, kernel=kernel)
    assert conv.kernel == kernel
    dst = np.full(oc, np.nan, np.float32)
    conv.forward(src, dst)
    assert np.array_equal(conv.forward_sums(), want["sums"])
    assert np.array_equal(conv.read(xb.SLOT_ALPHA, np.float32), want["alpha"])
    assert np.all(np.abs(dst - want["dst"]) <= 1e-4 * np.abs(want["dst"]))
    conv.close()
    return want["sums"]


@pytest.mark.parametrize("kernel", [xb.KERNEL_TCGEN05_I8, xb.KERNEL_TCGEN05_I8_ROWS],
                         ids=["tiles", "rows"])
def test_odd_number_of_operands(oracle, kernel):
    """4095 channels, 9 x 9: 331695 operands, an odd number, so every sum is odd."""
    ic, k, oc = 4095, 9, 20
    rng = np.random.default_rng(3)
    src = np.where(rng.random((1, ic, k, k)) < 0.5, 1.0, -1.0).astype(np.float32)
    w = np.empty((oc, ic, k, k), np.float32)
    for f in range(oc):  # filter f agrees with the source in a share of f / (oc - 1) of the places
        w[f] = np.where(rng.random((ic, k, k)) < f / (oc - 1), src[0], -src[0])
    sums = _check(oracle, ic, k, oc, src, w, kernel)
    assert sums[0] == -ic * k * k and sums[-1] == ic * k * k


def test_as_many_operands_as_the_tensor_cores_take(oracle):
    """16384 channels, 32 x 32 = 2^24 operands: all agree, all but seven, and half of them in a row
    (the running sum goes half way up and back)."""
    ic, k = 16384, 32
    src = np.ones((1, ic, k, k), np.float32)
    w = np.ones((1, ic, k, k), np.float32)
    assert _check(oracle, ic, k, 1, src, w, xb.KERNEL_TCGEN05_I8)[0] == 2 ** 24
    flat = w.reshape(-1)
    flat[[0, 1, 77, 4096, 100001, 9999999, 2 ** 24 - 1]] = -1.0
    assert _check(oracle, ic, k, 1, src, w, xb.KERNEL_TCGEN05_I8)[0] == 2 ** 24 - 14
    flat[:] = 1.0
    flat.reshape(ic, k, k)[:, k // 2:] = -1.0
    assert _check(oracle, ic, k, 1, src, w, xb.KERNEL_TCGEN05_I8)[0] == 0
