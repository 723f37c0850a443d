"""The work a user of this library has it do, as cases whose cost can be measured.

A case is a dict of plain values; `entry` names the public call it goes through:

  forward  Convolution.forward on tensors that live on the GPU: the three stages in one call
  steps    the upstream sequence binarize_data, calculate_k, forward through the executor pointers
  host     Convolution.forward on host buffers (what a program linked against upstream passes):
           upload, stages and download belong to the call
  chain    forward_chain over consecutive layers (`oc` lists their filter counts)
  train    XnorConv2d forward and backward; the weights count as changed after every pass, so
           each pass packs them again, as it does between two optimiser steps

`nhwc` = channels-last source, HWIO weights and channels-last result. Layers have square filters
(`k`), strides and paddings. Activations are standard normal, as after a batch normalisation,
weights normal with a small deviation; both come from the seed alone.
"""
import random

import torch

import xnor_nn_b200 as xb
from xnor_nn_b200.torch_layer import XnorConv2d


def _case(name, entry, mb, ic, ih, iw, oc, k, stride=1, pad=0, nhwc=False, pinned=True):
    c = dict(name=name, entry=entry, mb=mb, ic=ic, ih=ih, iw=iw, oc=str(oc), k=k, stride=stride,
             pad=pad, nhwc=nhwc)
    if entry == "host":
        c["pinned"] = pinned
    return c


def listed():
    return [
        # one image through AlexNet conv4: interactive inference, latency and launches
        _case("conv4_mb1", "forward", 1, 384, 13, 13, 256, 3, pad=1),
        # an eighth of the full minibatch: a small server batch, or a GPU's share of eight
        _case("conv4_mb32", "forward", 32, 384, 13, 13, 256, 3, pad=1),
        # the benchmark layers at their full minibatch: throughput inference
        _case("conv4_mb256", "forward", 256, 384, 13, 13, 256, 3, pad=1),
        _case("conv3_mb256", "forward", 256, 256, 13, 13, 384, 3, pad=1),
        _case("conv2_mb128", "forward", 128, 96, 27, 27, 256, 5, pad=2),
        _case("vgg512_mb64", "forward", 64, 512, 28, 28, 512, 3, pad=1),
        # AlexNet conv1: three channels, 11 x 11 filters, stride 4
        _case("conv1_mb64", "forward", 64, 3, 227, 227, 96, 11, stride=4),
        # sizes that divide nothing, through upstream's own three calls
        _case("ragged_mb19", "steps", 19, 75, 31, 27, 101, 3, pad=1),
        # channels-last tensors, the layout other frameworks keep them in
        _case("conv4_nhwc_mb64", "forward", 64, 384, 13, 13, 256, 3, pad=1, nhwc=True),
        # AlexNet conv3 -> conv4 -> conv5 with no float tensor between the layers
        _case("chain345_mb128", "chain", 128, 256, 13, 13, "384,256,256", 3, pad=1),
        # a training step of one layer: forward, both gradients, weights packed again
        _case("train_conv3_mb64", "train", 64, 256, 13, 13, 384, 3, pad=1),
        # a CPU program's tensors: pinned host memory in, pinned host memory out
        _case("conv4_host_mb256", "host", 256, 384, 13, 13, 256, 3, pad=1),
    ]


def _widths(case):
    return [int(v) for v in case["oc"].split(",")]


def _out(case, size):
    return (size + 2 * case["pad"] - case["k"]) // case["stride"] + 1


def _layers(case):
    """(ic, ih, iw, oc, oh, ow) of every layer the case runs."""
    ic, ih, iw = case["ic"], case["ih"], case["iw"]
    rows = []
    for oc in _widths(case):
        oh, ow = _out(case, ih), _out(case, iw)
        rows.append((ic, ih, iw, oc, oh, ow))
        ic, ih, iw = oc, oh, ow
    return rows


def _binary_ops(case):
    return sum(2.0 * case["mb"] * oc * oh * ow * ic * case["k"] ** 2
               for ic, _, _, oc, oh, ow in _layers(case))


def _elements(case):
    """Source elements, weights, result elements."""
    rows = _layers(case)
    ic, ih, iw = rows[0][:3]
    oc, oh, ow = rows[-1][3:]
    weights = sum(r[0] * r[3] for r in rows) * case["k"] ** 2
    return case["mb"] * ic * ih * iw, weights, case["mb"] * oc * oh * ow


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng: random.Random):
    """Another layer of the ranges above: 1 to 256 images, 3 to 512 channels, up to 512 filters,
    images from 6 to 227 pixels wide, filters from 1 x 1 to 11 x 11, strides 1, 2 and 4."""
    while True:
        entry = rng.choice(["forward"] * 6 + ["steps", "host", "chain", "train"])
        first = entry in ("forward", "steps", "host") and rng.random() < 0.15
        if first:  # the first layer of a network: few channels, a large image, maybe a stride
            ic, ih = rng.choice([1, 3, 3, 4]), _log_int(rng, 28, 227)
            k, stride = rng.choice([(3, 1), (5, 1), (7, 2), (11, 4)])
            pad = rng.choice([0, k // 2])
            oc = _log_int(rng, 16, 96)
        else:
            ic, ih = _log_int(rng, 16, 512), _log_int(rng, 6, 56)
            k = rng.choice([1, 3, 3, 3, 5])
            stride = 2 if entry in ("forward", "steps") and rng.random() < 0.1 else 1
            pad = k // 2 if rng.random() < 0.8 else 0
            oc = _log_int(rng, 16, 512)
        iw = ih if rng.random() < 0.7 else max(6, ih + rng.randint(-4, 4))
        if rng.random() < 0.5:  # channel counts of real networks are mostly round
            ic = ic if first else max(16, ic // 16 * 16)
            oc = max(16, oc // 16 * 16)
        if entry == "chain":
            pad = k // 2
            more = [max(16, _log_int(rng, 16, 512) // 16 * 16) for _ in range(rng.randint(1, 2))]
            oc = ",".join(str(v) for v in [oc] + more)
        nhwc = entry in ("forward", "steps", "host") and rng.random() < 0.25
        case = _case("", entry, _log_int(rng, 1, 256), ic, ih, iw, oc, k, stride, pad, nhwc,
                     pinned=rng.random() < 0.7)
        del case["name"]
        src, weights, dst = _elements(case)
        ops = _binary_ops(case)
        if min(r[4] for r in _layers(case)) < 1 or min(r[5] for r in _layers(case)) < 1:
            continue
        # no costlier than the largest listed ones: the layers with a stride or next to no
        # channels against conv1, host buffers against the pinned minibatch, the rest against VGG
        words = dst * k * k * -(-ic // 32)
        if (stride > 1 or first) and words > 64 * 96 * 55 * 55 * 121:
            continue
        if entry == "host" and (src + dst) * (1 if case["pinned"] else 5) > 27_000_000:
            continue
        if entry == "train" and (ops > 20e9 or src + dst > 8_000_000):
            continue
        if 4 * (src + weights + dst) > 200e6 or ops > 230e9:
            continue
        return case


def _normal(gen, shape, std=1.0):
    return torch.randn(shape, generator=gen, device="cuda", dtype=torch.float32) * std


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    mb, k, s, p = case["mb"], case["k"], case["stride"], case["pad"]
    nhwc = case["nhwc"]
    ic, ih, iw = case["ic"], case["ih"], case["iw"]
    src = _normal(gen, (mb, ih, iw, ic) if nhwc else (mb, ic, ih, iw))
    if case["entry"] == "train":
        oc = _widths(case)[0]
        layer = XnorConv2d(ic, oc, k, stride=s, padding=p).cuda()
        with torch.no_grad():
            layer.weight.copy_(_normal(gen, layer.weight.shape, 0.05))
        grad = _normal(gen, (mb, oc, _out(case, ih), _out(case, iw)))
        return dict(entry="train", layer=layer, src=src.requires_grad_(), grad=grad)
    convs = []
    fmt = (xb.NHWC, xb.HWIO, xb.NHWC) if nhwc else (xb.NCHW, xb.OIHW, xb.NCHW)
    for c_in, h, w, c_out, _, _ in _layers(case):
        weights = _normal(gen, (k, k, c_in, c_out) if nhwc else (c_out, c_in, k, k), 0.05)
        convs.append(xb.Convolution(xb.ALGORITHM_BCAST, *fmt, mb, c_out, c_in, h, w, k, k, s, s,
                                    p, p, weights))
    dst = torch.empty(convs[-1].out_shape, device="cuda", dtype=torch.float32)
    if case["entry"] == "host":
        src, dst = src.cpu(), torch.empty(dst.shape, dtype=torch.float32)
        if case["pinned"]:
            src, dst = src.pin_memory(), dst.pin_memory()
    return dict(entry=case["entry"], convs=convs, src=src, dst=dst)


def run(state):
    entry, src = state["entry"], state["src"]
    if entry == "train":
        layer = state["layer"]
        src.grad = layer.weight.grad = None
        y = layer(src)
        y.backward(state["grad"])
        return y, src.grad, layer.weight.grad
    dst = state["dst"]
    if entry == "chain":
        xb.forward_chain(state["convs"], src, dst)
    elif entry == "steps":
        state["convs"][0].forward_stepwise(src, dst)
    else:
        state["convs"][0].forward(src, dst)
    return dst


def work(case):
    """One pass: the float source and weights in, the float result out. A training pass also
    takes the result's gradient in, puts both other gradients out and does the two float
    convolutions of the backward pass."""
    src, weights, dst = _elements(case)
    ops = _binary_ops(case)
    if case["entry"] == "train":
        return dict(bytes=4 * (2 * src + 2 * weights + 2 * dst), flops=3 * ops)
    # weights are packed before the call: a bit each is what a pass has to read
    return dict(bytes=4 * (src + dst) + weights / 8, flops=ops)


def tolerance(case):
    # The integer sums are exact; what may differ is the rounding of the 32-bit sums behind the
    # scale factors. The float gradients are computed in TF32 (11-bit significands).
    return {"rel": 1e-3} if case["entry"] == "train" else {"rel": 1e-5}
