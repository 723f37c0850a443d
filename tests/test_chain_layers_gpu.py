"""Chains over layers that the position-tile kernel cannot serve (paddings that differ or are as
large as the filter: the image-row kernel's), and the order in which a chained layer sums |result|.
Reference: the oracle, layer by layer."""
import numpy as np
import pytest

import xnor_nn_b200 as xb
from oracle.pyoracle import Shape
from xnor_nn_b200 import synth

pytestmark = pytest.mark.gpu

REL_TOL = 1e-4      # the float tolerance of the parity contract
A_REL_TOL = 1e-5    # mean-|x| map: a reordered sum of a few hundred non-negative terms


def _layer(mb, ic, oc, ih, iw, k, ph, pw, src=xb.NCHW, dst=xb.NCHW, kernel=None):
    return dict(mb=mb, ic=ic, oc=oc, ih=ih, iw=iw, k=k, ph=ph, pw=pw, src=src, dst=dst, kernel=kernel)


def _build(layers, seed):
    convs, weights, shapes = [], [], []
    for i, d in enumerate(layers):
        w = synth.normal(seed + 17 * i, d["oc"] * d["ic"] * d["k"] ** 2, 0.05)
        convs.append(xb.Convolution(xb.ALGORITHM_BCAST, d["src"], xb.OIHW, d["dst"], d["mb"],
                                    d["oc"], d["ic"], d["ih"], d["iw"], d["k"], d["k"], 1, 1,
                                    d["ph"], d["pw"], w, kernel=d["kernel"]))
        weights.append(w)
        shapes.append(Shape.make(d["mb"], d["oc"], d["ic"], d["ih"], d["iw"], d["k"], d["k"], 1, 1,
                                 d["ph"], d["pw"], 0, 0, 0))
    return convs, weights, shapes


CHAINS = {
    "last_uneven": [_layer(2, 20, 40, 9, 9, 3, 1, 1), _layer(2, 40, 24, 9, 9, 3, 0, 1)],
    "first_uneven": [_layer(2, 20, 40, 9, 9, 3, 0, 1), _layer(2, 40, 24, 9, 9, 3, 1, 1)],
    "last_padded_as_the_filter": [_layer(2, 40, 33, 4, 5, 3, 1, 1), _layer(2, 33, 16, 4, 5, 3, 3, 3)],
    "first_padded_as_the_filter": [_layer(2, 40, 33, 4, 5, 3, 3, 3), _layer(2, 33, 16, 8, 9, 3, 1, 1)],
    "middle_1x1_padded": [_layer(2, 24, 48, 5, 6, 3, 1, 1), _layer(2, 48, 40, 5, 6, 1, 1, 1),
                          _layer(2, 40, 16, 7, 8, 3, 1, 1)],
    "all_uneven": [_layer(2, 20, 40, 9, 9, 3, 0, 1), _layer(2, 40, 260, 9, 9, 3, 0, 1),
                   _layer(2, 260, 24, 9, 9, 3, 0, 1)],
    # a last layer asked onto the image-row kernel runs on position tiles in a chain: more tiles than
    # SMs, rows of 32 and of 64 bytes
    "last_asked_onto_rows_32": [_layer(2140, 24, 40, 2, 2, 3, 1, 1),
                                _layer(2140, 40, 32, 2, 2, 3, 1, 1, kernel=xb.KERNEL_TCGEN05_I8_ROWS)],
    "last_asked_onto_rows_64": [_layer(2140, 24, 100, 2, 2, 3, 1, 1),
                                _layer(2140, 100, 32, 2, 2, 3, 1, 1, kernel=xb.KERNEL_TCGEN05_I8_ROWS)],
    # what a layer between two others was declared to store or to read does not matter in a chain
    "layouts_differ": [_layer(2, 20, 40, 9, 9, 3, 0, 1, dst=xb.NHWC),
                       _layer(2, 40, 48, 9, 9, 3, 0, 1, dst=xb.NCHW),
                       _layer(2, 48, 24, 9, 9, 3, 1, 1, src=xb.NHWC)],
}


@pytest.mark.parametrize("name", list(CHAINS))
def test_chain_over_image_row_layers(oracle, name):
    layers = CHAINS[name]
    torch = pytest.importorskip("torch")
    convs, weights, shapes = _build(layers, 2000 + len(name))
    d0 = layers[0]
    src = synth.normal(79 + len(name), d0["mb"] * d0["ic"] * d0["ih"] * d0["iw"])
    x = src
    for shape, w in zip(shapes, weights):
        want = oracle.convolution(shape, x, w)
        x = want["dst"]
    ddst = torch.full((want["dst"].size,), float("nan"), device="cuda")
    torch.cuda.synchronize()
    xb.forward_chain(convs, src, ddst)  # the source comes from the host: the call has waited
    got = ddst.cpu().numpy()
    assert np.array_equal(convs[-1].forward_sums(), want["sums"])
    a = convs[-1].read(xb.SLOT_A, np.float32)
    assert np.all(np.abs(a - want["a"]) <= A_REL_TOL * np.abs(want["a"]))
    assert np.all(np.abs(got - want["dst"]) <= REL_TOL * np.abs(want["dst"]))
    for cv in convs:
        cv.close()

def test_same_image_gives_the_same_bits_anywhere_in_a_batch():
    """256 filters (accumulators that overlap), three rounds of tiles per thread block: an image's
    A, K and results do not depend on which round its positions fall into."""
    torch = pytest.importorskip("torch")
    mb = 256
    layers = [_layer(mb, 64, 256, 13, 13, 3, 1, 1), _layer(mb, 256, 32, 13, 13, 3, 1, 1)]
    convs, _, _ = _build(layers, 4000)
    src = torch.from_numpy(synth.normal(5, 64 * 169)).cuda().repeat(mb)
    dst = torch.empty(mb * 32 * 169, device="cuda")
    torch.cuda.synchronize()
    xb.forward_chain(convs, src, dst)
    convs[0].synchronize()
    for what in (convs[1].read(xb.SLOT_A, np.float32), convs[1].read(xb.SLOT_K, np.float32),
                 dst.cpu().numpy()):
        bits = what.view(np.uint32).reshape(mb, -1)
        assert np.array_equal(bits, np.broadcast_to(bits[0], bits.shape))
    for cv in convs:
        cv.close()
