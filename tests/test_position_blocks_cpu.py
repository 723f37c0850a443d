"""Which layers with resident filters have position tiles that serve all filter rows, from what the launcher
hands the driver (cpp/tile_launch.cpp): either side of each line of that rule."""
import json
import os
import subprocess

import pytest

import cases
import test_position_blocks_gpu as gpu
from xnor_nn_b200 import build

LAYERS = gpu.BLOCKS + gpu.ROWS + [
    cases._c("alexnet_conv3", 256, 384, 256, 13, 13, 3, 3, ph=1, pw=1),
    cases._c("alexnet_conv1", 64, 96, 3, 227, 227, 11, 11, sh=4, sw=4)]


@pytest.fixture(scope="module")
def launches(tmp_path_factory):
    build.build()
    exe = str(tmp_path_factory.mktemp("tile_launch") / "tile_launch")
    objs = [os.path.join(build.OBJ, n + ".o") for n in ("conv_tcgen05.cu", "plan.cpp", "tensormap.cpp")]
    subprocess.check_call(
        ["g++", "-std=c++17", "-O1", "-I", os.path.join(build.ROOT, "include"), "-I", build.CSRC, "-I",
         "/usr/local/cuda/include", os.path.join(os.path.dirname(__file__), "cpp", "tile_launch.cpp")] +
        objs + ["-o", exe])
    keys = ("mb", "oc", "ic", "ih", "iw", "kh", "kw", "sh", "sw", "ph", "pw")
    env = {k: v for k, v in os.environ.items() if k != "XNOR_NN_B200_KERNEL"}
    out = subprocess.check_output([exe] + [",".join(str(c[1][k]) for k in keys) for c in LAYERS], text=True,
                                  env=env).splitlines()
    return dict(zip([c[0] for c in LAYERS], [json.loads(line) for line in out]))


def test_which_layers_have_blocks(launches):
    for name, got in launches.items():
        assert got["resident"] and got["pair"] and not got["planes"], name
        boxes = [m["box"] for m in got["maps"] if m["ptr"] == got["activations"]]
        assert [b[1] for b in boxes] == [got["halo"]], name
        # positions of all taps, and a barrier for the filters of each filter row and chunk; or 128 positions,
        # with a halo of eight where a filter row has several taps
        _, d, _, _ = next(c for c in LAYERS if c[0] == name)
        kh, wp = d["kh"], d["iw"] + d["pw"]
        if d["sh"] > 1:
            kh, wp = -(-kh // d["sh"]), (d["iw"] + 2 * d["pw"] - d["kw"]) // d["sw"] + 1
        if name in [c[0] for c in gpu.ROWS]:
            assert (got["halo"], got["stages"]) == (136 if got["tap_kw"] > 1 else 128, 2), name
        else:
            assert (got["halo"], got["stages"]) == (128 + (kh - 1) * wp + got["tap_kw"] - 1, got["groups"]), name
    blocks = [launches[c[0]] for c in gpu.BLOCKS]
    assert {g["halo"] for g in blocks} >= {256} and {g["a_slots"] for g in blocks} >= {2, 8}
    assert {g["groups"] for g in blocks} >= {2, 8} and {g["shared_cols"] for g in blocks} == {0, 1}
    assert {g["n_tiles"] for g in blocks} == {1, 2, 3} and {g["m_tiles"] % 2 for g in blocks} == {0, 1}
    # one issuer where the taps of a filter row keep the tensor pipe for more than 800 cycles, else two
    assert {n: g["issuers"] for n, g in launches.items() if n in [c[0] for c in gpu.BLOCKS] + ["alexnet_conv3"]} == {
        "256_rows": 2, "eight_groups": 2, "two_tiles_in_flight": 2, "channel_tail_of_the_second_chunk": 2,
        "two_filter_tiles": 1, "three_filter_tiles": 1, "overlapping_accumulators": 2, "a_filter_row_as_one": 2,
        "folded": 2, "alexnet_conv3": 1}
    rows = [launches[c[0]] for c in gpu.ROWS]
    assert {g["kchunk"] for g in rows} == {64, 128} and 9 in {g["groups"] for g in rows}
