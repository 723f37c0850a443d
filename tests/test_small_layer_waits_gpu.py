"""Bounded waits of the one-launch pass (conv_whole.cu) and of calculate_k in one launch (maps.cu) that run
out, in the form that leaves the GPU healthy: the test hook shortens the limit and loses a commit, an arrival of the packed operand or the
hand-over of running sums. Every role winds down, loads and MMAs in flight are waited for, the host turns
the error word into a status, and the next pass on the same resources is right, bit for bit."""
import ctypes as C

import numpy as np
import pytest

import xnor_nn_b200 as xb
from xnor_nn_b200 import synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

COMMIT, OPERAND, TURN, TURN_OF_K = 0, 1, 2, 3


def _layer(layer, mb):
    L = synth.layer_shape(layer, mb=mb)
    src, w = synth.make_inputs(layer, mb=mb)
    conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NCHW, xb.OIHW, xb.NCHW, L.mb, L.oc, L.ic, L.ih, L.iw,
                          L.kh, L.kw, L.sh, L.sw, L.ph, L.pw, w)
    return conv, torch.from_numpy(src).cuda(), torch.zeros(int(np.prod(conv.out_shape)), device="cuda")


# One image: narrow filter tiles, all of them in shared memory (the producer is through before anyone gives
# up). 30 images: a ring that comes round, so the producer gives up with loads in flight.
@pytest.mark.parametrize("mb", [1, 30])
@pytest.mark.parametrize("lost, sites", [(COMMIT, (4,)), (OPERAND, (9, 4, 1)), (TURN, (21, 9, 4, 1))],
                         ids=["commit", "operand", "turn"])
def test_gives_up_and_the_resources_stay_usable(lost, sites, mb):
    conv, src, good = _layer("A", mb)
    torch.cuda.synchronize()
    before = xb.kernel_launches()
    conv.forward(src, good)
    assert xb.kernel_launches() - before == 1  # the kernel this is about
    conv.synchronize()
    junk = torch.zeros_like(good)
    torch.cuda.synchronize()
    conv._set(xb.SLOT_USER_SRC, src)
    conv._set(xb.SLOT_USER_DST, junk)
    st = xb.lib().xnor_nn_b200_selftest_small_layer(C.byref(conv.c), conv.res, 5, lost)
    assert st == xb.UNIMPLEMENTED
    err = xb.last_error()
    # waits that start within microseconds of one another: the first to run out is recorded; the producer
    # waits (1) only for a ring that comes round
    allowed = sites if mb == 30 else [s for s in sites if s != 1]
    assert any("gave up waiting (site %d)" % s in err for s in allowed), err
    conv.synchronize()  # the error word was consumed
    again = torch.zeros_like(good)
    torch.cuda.synchronize()
    conv.forward(src, again)
    conv.synchronize()
    assert torch.equal(again, good)
    conv.close()


@pytest.mark.parametrize("mb", [1, 19])
def test_calculate_k_gives_up_and_the_resources_stay_usable(mb):
    conv, src, dst = _layer("A", mb)
    torch.cuda.synchronize()
    before = xb.kernel_launches()
    assert conv.execute("calculate_k", src=src) == xb.SUCCESS
    assert xb.kernel_launches() - before == 1  # the kernel this is about
    want = conv.read(xb.SLOT_A, np.float32), conv.read(xb.SLOT_K, np.float32)
    conv._set(xb.SLOT_USER_SRC, src)
    conv._set(xb.SLOT_USER_DST, dst)
    st = xb.lib().xnor_nn_b200_selftest_small_layer(C.byref(conv.c), conv.res, 5, TURN_OF_K)
    assert st == xb.UNIMPLEMENTED
    assert "gave up waiting (site 21)" in xb.last_error()
    conv.synchronize()
    assert conv.execute("calculate_k", src=src) == xb.SUCCESS
    conv.synchronize()
    assert np.array_equal(conv.read(xb.SLOT_A, np.float32), want[0])
    assert np.array_equal(conv.read(xb.SLOT_K, np.float32), want[1])
    conv.close()


def test_hook_refuses_what_it_cannot_run():
    hook = xb.lib().xnor_nn_b200_selftest_small_layer
    conv, src, dst = _layer("A", 256)  # more tiles than SMs
    host = np.zeros(dst.numel(), np.float32)
    conv._set(xb.SLOT_USER_SRC, src)
    conv._set(xb.SLOT_USER_DST, dst)
    assert hook(C.byref(conv.c), conv.res, 5, COMMIT) == xb.ERROR_INVALID_INPUT
    conv.close()
    conv, src, dst = _layer("A", 1)
    conv._set(xb.SLOT_USER_SRC, src)
    conv._set(xb.SLOT_USER_DST, host)
    assert hook(C.byref(conv.c), conv.res, 5, COMMIT) == xb.ERROR_INVALID_INPUT
    conv._set(xb.SLOT_USER_DST, dst)
    assert hook(C.byref(conv.c), conv.res, 0, COMMIT) == xb.ERROR_INVALID_INPUT
    assert hook(C.byref(conv.c), conv.res, 5, 7) == xb.ERROR_INVALID_INPUT
    conv.close()
    conv, src, dst = _layer("D", 64)  # over 16 MB
    conv._set(xb.SLOT_USER_SRC, src)
    conv._set(xb.SLOT_USER_DST, dst)
    assert hook(C.byref(conv.c), conv.res, 5, TURN_OF_K) == xb.ERROR_INVALID_INPUT
    conv.close()
