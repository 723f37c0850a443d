"""Which layers have filter tiles of half their width, from what the launcher hands the driver
(cpp/tile_launch.cpp): either side of each line of that rule."""
import json
import os
import subprocess

import pytest

import cases
import test_half_filter_tiles_gpu as gpu
from xnor_nn_b200 import build

LAYERS = gpu.HALVED + gpu.WHOLE + [
    cases._c("alexnet_conv4", 256, 256, 384, 13, 13, 3, 3, ph=1, pw=1),
    cases._c("alexnet_conv3", 256, 384, 256, 13, 13, 3, 3, ph=1, pw=1),
    cases._c("vgg", 64, 512, 512, 28, 28, 3, 3, ph=1, pw=1)]


@pytest.fixture(scope="module")
def launch(tmp_path_factory):
    build.build()
    exe = str(tmp_path_factory.mktemp("tile_launch") / "tile_launch")
    objs = [os.path.join(build.OBJ, n + ".o") for n in ("conv_tcgen05.cu", "plan.cpp", "tensormap.cpp")]
    subprocess.check_call(
        ["g++", "-std=c++17", "-O1", "-I", os.path.join(build.ROOT, "include"), "-I", build.CSRC, "-I",
         "/usr/local/cuda/include", os.path.join(os.path.dirname(__file__), "cpp", "tile_launch.cpp")] +
        objs + ["-o", exe])
    keys = ("mb", "oc", "ic", "ih", "iw", "kh", "kw", "sh", "sw", "ph", "pw")
    env = {k: v for k, v in os.environ.items() if k != "XNOR_NN_B200_KERNEL"}

    def run(**more):
        out = subprocess.check_output([exe] + [",".join(str(c[1][k]) for k in keys) for c in LAYERS], text=True,
                                      env={**env, **more}).splitlines()
        return dict(zip([c[0] for c in LAYERS], [json.loads(line) for line in out]))
    return run


@pytest.fixture(scope="module")
def launches(launch):
    return launch()


def test_which_layers_have_half_the_width(launches):
    tiles = {name: got["n_tiles"] for name, got in launches.items()}
    assert [tiles[c[0]] for c in gpu.HALVED] == [2, 2, 2, 2, 6, 2, 2]
    assert [tiles[c[0]] for c in gpu.WHOLE] == [1, 1, 1, 1, 1, 3, 1, 1]
    assert (tiles["alexnet_conv4"], tiles["alexnet_conv3"], tiles["vgg"]) == (2, 2, 2)
    halved = [launches[c[0]] for c in gpu.HALVED] + [launches["alexnet_conv4"]]
    # resident, with a tile for all filter rows and a barrier for each filter row's and chunk's filters
    assert all(g["pair"] and g["resident"] and g["halo"] > 136 and g["stages"] == g["groups"] for g in halved)
    assert {g["m_tiles"] % 2 for g in halved} == {0, 1} and not any(g["shared_cols"] for g in halved)
    whole = [launches[c[0]] for c in gpu.WHOLE if c[0] != "whole_fits"] + [launches["vgg"]]
    assert all(g["pair"] and not g["resident"] for g in whole) and launches["whole_fits"]["resident"]


def test_halves_are_resident_on_fewer_pairs(launch):
    """Where fewer pairs than half the SMs can be resident, a layer is halved only if each of those that run keeps to
    one filter tile: a halved layer that streams its filters would read its positions twice for nothing."""
    names = [c[0] for c in gpu.HALVED] + ["alexnet_conv4"]
    halved = whole = 0
    for pairs in range(1, 75):
        got = launch(PAIRS=str(pairs))
        for name in names:
            g = got[name]
            assert g["served"] and g["pair"] and g["grid"] <= 2 * pairs
            # these have filter tiles of 192 or 256, halved 96 or 128, and 2, 2, 2, 2, 6, 2, 2 and 2 of the latter
            if g["n_tiles"] == (6 if name == "six_tiles_of_128" else 2):
                assert g["resident"], (pairs, name, g)
                halved += 1
            else:
                whole += 1
    assert halved > 200 and whole > 100, (halved, whole)  # the line of three tiles a pair moves too
