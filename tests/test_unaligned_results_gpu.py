"""Results that start between two 16-byte boundaries, such as a view that begins a float into a buffer: every
kernel with wide stores (16 and 32 bytes a store on channels-last results, bulk copies of rows) writes what
it writes to an aligned buffer, bit for bit, and nothing beside it."""
import pytest

import cases
import xnor_nn_b200 as xb

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

CL, C_ = (1, 1, 1), cases._c
LAYERS = [
    (C_("whole_oc44", 3, 44, 92, 10, 11, 3, 3, ph=1, pw=1, fmt=CL), xb.KERNEL_AUTO),
    (C_("whole_oc64", 3, 64, 64, 10, 11, 3, 3, ph=1, pw=1, fmt=CL), xb.KERNEL_AUTO),
    (C_("whole_nchw", 3, 44, 92, 10, 11, 3, 3, ph=1, pw=1), xb.KERNEL_AUTO),
    # more position tiles than SMs: single CTAs (a filter tile of 48 does not split into two), then pairs
    (C_("tiles_oc36", 160, 36, 40, 13, 13, 3, 3, ph=1, pw=1, fmt=CL), xb.KERNEL_AUTO),
    (C_("tiles_oc48", 160, 48, 40, 13, 13, 3, 3, ph=1, pw=1, fmt=CL), xb.KERNEL_AUTO),
    (C_("pairs_oc60", 160, 60, 40, 13, 13, 3, 3, ph=1, pw=1, fmt=CL), xb.KERNEL_AUTO),
    (C_("pairs_oc64", 160, 64, 40, 13, 13, 3, 3, ph=1, pw=1, fmt=CL), xb.KERNEL_AUTO),
    (C_("pairs_nchw", 160, 64, 40, 13, 13, 3, 3, ph=1, pw=1), xb.KERNEL_AUTO),
    (C_("folded_oc20", 3, 20, 3, 37, 41, 7, 7, sh=2, sw=2, ph=3, pw=3, fmt=CL), xb.KERNEL_AUTO),
    (C_("rows_oc44", 3, 44, 92, 10, 11, 3, 3, ph=1, pw=1, fmt=CL), xb.KERNEL_TCGEN05_I8_ROWS),
    (C_("rows_nchw", 3, 44, 92, 10, 11, 3, 3, ph=1, pw=1), xb.KERNEL_TCGEN05_I8_ROWS),
    (C_("popc_oc44", 3, 44, 92, 10, 11, 3, 3, ph=1, pw=1, fmt=CL), xb.KERNEL_POPC),
]


@pytest.mark.parametrize("layer", LAYERS, ids=[c[0][0] for c in LAYERS])
def test_result_at_any_float(layer):
    case, kernel = layer
    _, d, _, fmt = case
    src, w = cases.make_inputs(case)
    conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NHWC if fmt[0] else xb.NCHW,
                          xb.HWIO if fmt[1] else xb.OIHW, xb.NHWC if fmt[2] else xb.NCHW, d["mb"],
                          d["oc"], d["ic"], d["ih"], d["iw"], d["kh"], d["kw"], d["sh"], d["sw"],
                          d["ph"], d["pw"], w, kernel=kernel)
    src = torch.from_numpy(src).cuda()
    want = torch.empty(conv.out_shape, device="cuda")
    conv.forward(src, want)
    conv.synchronize()
    n = want.numel()
    assert want.data_ptr() % 32 == 0
    for shift in (1, 2, 3, 4):  # 4: on 16 bytes, not on 32
        for stepwise in (False, True):
            buffer = torch.full((n + 16,), 7.0, device="cuda")
            torch.cuda.synchronize()
            (conv.forward_stepwise if stepwise else conv.forward)(src, buffer[shift:shift + n])
            conv.synchronize()
            assert torch.equal(buffer[shift:shift + n].view_as(want), want)
            assert bool((buffer[:shift] == 7.0).all()) and bool((buffer[shift + n:] == 7.0).all())
    conv.close()
