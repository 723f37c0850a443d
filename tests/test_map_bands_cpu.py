"""calculate_k in one launch reads pixels of its source and no others (cpp/map_bands.cpp walks what every lane of
every block reads): filters of 1 x 1 to 7 x 7, equal and unequal paddings, some beyond the filter, strides, one
image and several. The height of the result follows from the padding of the width, so that with unequal paddings
the windows of whole blocks can lie below the image."""
import json
import os
import subprocess

import pytest

import cases
import test_maps_gpu as gpu
from xnor_nn_b200 import build


@pytest.fixture(scope="module")
def walk(tmp_path_factory):
    build.build()
    exe = str(tmp_path_factory.mktemp("map_bands") / "map_bands")
    objs = [os.path.join(build.OBJ, n + ".o") for n in ("conv_tcgen05.cu", "plan.cpp", "tensormap.cpp")]
    subprocess.check_call(
        ["g++", "-std=c++17", "-O2", "-I", os.path.join(build.ROOT, "include"), "-I", build.CSRC, "-I",
         "/usr/local/cuda/include", os.path.join(os.path.dirname(__file__), "cpp", "map_bands.cpp")] +
        objs + ["-o", exe])
    env = {k: v for k, v in os.environ.items() if k != "XNOR_NN_B200_KERNEL"}

    def run(layers):
        out = subprocess.check_output([exe] + [",".join(map(str, d)) for d in layers], text=True, env=env)
        return [json.loads(line) for line in out.splitlines()]
    return run


def check(layers, got):
    for d, g in zip(layers, got):
        if g["served"]:
            assert 0 <= g["least"] and g["most"] < g["pixels"] and g["last"] <= g["pixels"], (d, g)
            assert g["rows_not_left_once"] == 0, (d, g)
            assert g["groups"] <= 32 and g["tasks"] <= 64, (d, g)


def test_every_pixel_is_one_of_the_source(walk):
    layers = [(mb, 16, ic, ih, iw, kh, kw, s, s, ph, pw)
              for mb, ic, ih, iw in [(1, 64, 13, 13), (1, 5, 40, 33), (8, 64, 14, 14), (19, 33, 7, 9), (2, 64, 1, 5)]
              for kh in range(1, 8) for kw in range(1, 8) for s in (1, 2)
              for ph, pw in [(0, 0), (kh // 2, kw // 2), (0, kw // 2), (kh // 2, 0), (0, kw - 1), (kh + 2, 1),
                             (1, kw + 2), (kw + 3, kw + 3)]
              if ih + 2 * pw >= kh and iw + 2 * pw >= kw]
    got = walk(layers)
    check(layers, got)
    assert sum(g["served"] for g in got) > 2000 and sum(g["served"] and g["empty"] > 0 for g in got) > 100


def test_layers_whose_last_windows_lie_below_the_image(walk):
    keys = ("mb", "oc", "ic", "ih", "iw", "kh", "kw", "sh", "sw", "ph", "pw")
    layers = [tuple(c[1][k] for k in keys) for c in gpu.BELOW_THE_IMAGE]
    got = walk(layers)
    check(layers, got)
    assert all(g["served"] and g["empty"] for g in got), got
