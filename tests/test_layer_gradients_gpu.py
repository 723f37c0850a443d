"""The gradients of the torch layer, which come from one library call where both are asked for and the input is
contiguous, and from one each otherwise: every combination against the two library functions by themselves."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("contiguous", [True, False])
@pytest.mark.parametrize("wanted", [(True, True), (True, False), (False, True)],
                         ids=["both", "of_the_input", "of_the_weights"])
def test_gradients(wanted, contiguous):
    from torch.nn import grad as library

    from xnor_nn_b200.torch_layer import XnorConv2d
    torch.manual_seed(4)
    layer = XnorConv2d(24, 17, 3, padding=1).cuda()
    layer.weight.requires_grad_(wanted[1])
    x = torch.randn(5, 24, 9, 8, device="cuda")
    if not contiguous:
        x = x.to(memory_format=torch.channels_last)
    x.requires_grad_(wanted[0])
    y = layer(x)
    g = torch.randn_like(y)
    # not through x.grad, which takes on the strides of x
    got = iter(torch.autograd.grad(y, [t for t, asked in ((x, wanted[0]), (layer.weight, wanted[1])) if asked], g))
    w = layer.weight.detach()
    signs = torch.where(w < 0, -1.0, 1.0) * w.mean()
    # sums of at most 153 (filters x taps) and 360 (images x positions) products in TF32 at worst
    if wanted[0]:
        have, want = next(got), library.conv2d_input(x.shape, signs, g, padding=1)
        assert have.is_contiguous() and have.shape == want.shape
        assert (have - want).abs().max() <= 153 * 2.0 ** -10 * signs.abs().max() * g.abs().max()
    if wanted[1]:
        have, want = next(got), library.conv2d_weight(x.detach().contiguous(), w.shape, g, padding=1)
        assert have.shape == want.shape
        assert (have - want).abs().max() <= 360 * 2.0 ** -10 * x.abs().max() * g.abs().max()
