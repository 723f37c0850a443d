"""Resident filters beside position tiles that serve all filter rows, with three accumulators, which two epilogue teams
share in turn (mma_role_block in conv_tcgen05.cu); test_tile_launch_cpu.py pins that these layers have three. Sums
and K bit for bit against the oracle, floats to the parity contract's 1e-4. A commit that is lost makes a wait run
out, and the next pass is right: a team must not take another team's later commit for the one that was lost."""
import ctypes as C

import numpy as np
import pytest

import cases
import xnor_nn_b200 as xb

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

LAYERS = [
    cases._c("one_issuer", 3100, 160, 250, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("two_issuers", 3100, 128, 300, 4, 4, 3, 3, ph=1, pw=1),
    cases._c("two_filter_tiles", 1601, 313, 250, 4, 4, 3, 3, ph=1, pw=1),
]


def _conv(case):
    _, d, _, _ = case
    src, w = cases.make_inputs(case)
    conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NCHW, xb.OIHW, xb.NCHW, d["mb"], d["oc"], d["ic"], d["ih"],
                          d["iw"], d["kh"], d["kw"], d["sh"], d["sw"], d["ph"], d["pw"], w)
    return conv, src, w


@pytest.mark.parametrize("case", LAYERS, ids=[c[0] for c in LAYERS])
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
        assert np.array_equal(conv.read(xb.SLOT_K, np.float32), want["k"])
    conv.close()


@pytest.mark.parametrize("case", LAYERS, ids=[c[0] for c in LAYERS])
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
