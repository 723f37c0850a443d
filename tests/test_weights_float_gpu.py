"""binarize_weights_float on the device, at the sizes where its scratch changes: up to 511 weights, and in
place, the block sums have memory of their own; from 512 weights on the result holds them until the end.
Both ways add in the same fixed shape, so they agree bit for bit. Against 64 bits the mean is off by less
than a rounding (2^-24 of the mean |w|) for each of the additions a value goes through: elems / 65536 + 1 in
a thread, eight in each of two trees, one product."""
import numpy as np
import pytest

import xnor_nn_b200 as xb

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("elems", [1, 255, 256, 511, 512, 513, 767, 65537, 330 * 257])
def test_scratch_in_the_result(elems):
    conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NCHW, xb.OIHW, xb.NCHW, 1, elems, 1, 1, 1, 1, 1, 1, 1,
                          0, 0)
    w = torch.randn(elems, generator=torch.Generator().manual_seed(elems), dtype=torch.float32) * 0.05
    w[0] = 0.0
    dev = w.cuda()
    stream = torch.cuda.current_stream().cuda_stream
    out = torch.full((elems + 1,), float("nan"), device="cuda")[:elems]
    for _ in range(2):
        conv.binarize_weights_float(dev, out, stream=stream)
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    assert np.array_equal(dev.cpu().numpy(), w.numpy())  # the source is left alone
    conv.binarize_weights_float(dev, dev, stream=stream)
    torch.cuda.synchronize()
    assert np.array_equal(got, dev.cpu().numpy())
    sign = np.where(w.numpy() >= 0, 1.0, -1.0)
    mean = w.double().mean().item()
    bound = (elems / 65536 + 1 + 8 + 8 + 1) * 2.0 ** -24 * w.abs().double().mean().item()
    assert np.all(np.abs(got - sign * mean) <= bound + 1e-30)
    conv.close()
