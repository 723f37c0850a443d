"""Which kernel a layer is planned on, at the lines where the rules change. Host code only."""
import ctypes as C

import pytest

import xnor_nn_b200 as xb


def _kernel(mb, oc, ic, ih, iw, kh, kw, sh=1, sw=1, ph=0, pw=0, kernel=xb.KERNEL_AUTO):
    c = xb.ConvolutionDesc()
    st = xb.lib().xnor_nn_b200_init_convolution(
        C.byref(c), xb.ALGORITHM_BCAST, xb.NCHW, xb.OIHW, xb.NCHW, mb, oc, ic, ih, iw, kh, kw, sh,
        sw, ph, pw, kernel)
    assert st == xb.SUCCESS
    k = xb.lib().xnor_nn_b200_kernel_of(C.byref(c))
    xb.lib().xnor_nn_destroy_convolution(C.byref(c))
    return k


@pytest.fixture(autouse=True)
def _no_override(monkeypatch):
    monkeypatch.delenv("XNOR_NN_B200_KERNEL", raising=False)


def test_sums_that_fp32_cannot_hold_run_on_popc():
    assert _kernel(1, 1, 16384, 32, 32, 32, 32) == xb.KERNEL_TCGEN05_I8      # 2^24 operands
    assert _kernel(1, 1, 16385, 32, 32, 32, 32) == xb.KERNEL_POPC
    assert _kernel(1, 1, 16384, 32, 32, 32, 32, kernel=xb.KERNEL_TCGEN05_I8_ROWS) == \
        xb.KERNEL_TCGEN05_I8_ROWS
    for kernel in (xb.KERNEL_TCGEN05_I8, xb.KERNEL_TCGEN05_I8_ROWS):
        assert _kernel(1, 1, 16385, 32, 32, 32, 32, kernel=kernel) == xb.KERNEL_POPC
    # the same limit on a strided layer
    assert _kernel(1, 1, 16384, 32, 33, 32, 32, sh=1, sw=2) == xb.KERNEL_TCGEN05_I8
    assert _kernel(1, 1, 16385, 32, 33, 32, 32, sh=1, sw=2) == xb.KERNEL_POPC


@pytest.mark.parametrize("ow", [16, 240, 241, 250, 256])
def test_rows_that_only_the_image_row_kernel_serves(ow):
    """Paddings as large as the filter: output rows of up to 256 pixels stay on the tensor cores,
    whether the kernel is chosen or asked for."""
    for kernel in (xb.KERNEL_AUTO, xb.KERNEL_TCGEN05_I8_ROWS):
        assert _kernel(2, 24, 20, 9, ow - 4, 3, 3, ph=3, pw=3, kernel=kernel) == \
            xb.KERNEL_TCGEN05_I8_ROWS
        assert _kernel(2, 24, 20, 9, ow, 3, 3, ph=0, pw=1, kernel=kernel) == \
            xb.KERNEL_TCGEN05_I8_ROWS
    assert _kernel(2, 24, 20, 9, ow, 3, 3, ph=1, pw=1, kernel=xb.KERNEL_TCGEN05_I8_ROWS) == \
        xb.KERNEL_TCGEN05_I8_ROWS


def test_rows_beyond_an_accumulator_run_on_popc():
    assert _kernel(2, 24, 20, 9, 253, 3, 3, ph=3, pw=3) == xb.KERNEL_POPC
    assert _kernel(2, 24, 20, 9, 257, 3, 3, ph=1, pw=1) == xb.KERNEL_TCGEN05_I8


def test_strided_layers_of_few_channels_fold_while_their_bits_fit():
    """The packer stages half a byte per value, in 192 KB (the rule counts a bit, in 48). Borders count in a
    row's pitch even where a wide stride skips most of them."""
    assert _kernel(1, 8, 7, 16, 1000, 8, 8, sh=8, sw=8) == xb.KERNEL_TCGEN05_I8
    assert _kernel(1, 8, 7, 11, 1117, 11, 11, sh=11, sw=11, ph=1900, pw=1900) == xb.KERNEL_TCGEN05_I8
    assert _kernel(1, 8, 7, 11, 1117, 11, 11, sh=11, sw=11, ph=2000, pw=2000) == xb.KERNEL_POPC
    # one output column: it reads 11 columns, 4000 columns of border in front of it
    assert _kernel(1, 8, 7, 11, 1100, 11, 11, sh=11, sw=9400, ph=4, pw=4100) == xb.KERNEL_POPC
