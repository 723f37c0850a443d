"""Which layers with streamed filters have position tiles that serve all filter rows, from what the launcher hands
the driver (cpp/tile_launch.cpp): either side of each line of that rule."""
import json
import os
import subprocess

import cases
import test_streamed_blocks_gpu as gpu
from xnor_nn_b200 import build

LAYERS = gpu.BLOCKS + gpu.ROWS + [cases._c("vgg", 64, 512, 512, 28, 28, 3, 3, ph=1, pw=1)]


def test_which_layers_have_blocks(tmp_path):
    build.build()
    exe = str(tmp_path / "tile_launch")
    objs = [os.path.join(build.OBJ, n + ".o") for n in ("conv_tcgen05.cu", "plan.cpp", "tensormap.cpp")]
    subprocess.check_call(
        ["g++", "-std=c++17", "-O1", "-I", os.path.join(build.ROOT, "include"), "-I", build.CSRC, "-I",
         "/usr/local/cuda/include", os.path.join(os.path.dirname(__file__), "cpp", "tile_launch.cpp")] +
        objs + ["-o", exe])
    keys = ("mb", "oc", "ic", "ih", "iw", "kh", "kw", "sh", "sw", "ph", "pw")
    env = {k: v for k, v in os.environ.items() if k != "XNOR_NN_B200_KERNEL"}
    out = subprocess.check_output([exe] + [",".join(str(c[1][k]) for k in keys) for c in LAYERS], text=True,
                                  env=env).splitlines()
    got = dict(zip([c[0] for c in LAYERS], [json.loads(line) for line in out]))
    for name, d, _, _ in LAYERS:
        g = got[name]
        assert g["pair"] and g["halo"] and not g["resident"] and g["issuers"] == 2, (name, g)
        rows = 128 + (d["kh"] - 1) * (d["iw"] + d["pw"]) + d["kw"] - 1
        assert g["halo"] == (136 if name in [c[0] for c in gpu.ROWS] else rows), (name, g)
    blocks = [got[c[0]] for c in gpu.BLOCKS]
    assert {g["halo"] for g in blocks} >= {256} and {g["m_tiles"] % 2 for g in blocks} == {0, 1}
    assert {g["shared_cols"] for g in blocks} == {0, 1} and {g["n_tiles"] for g in blocks} == {1, 2}
    assert {g["tap_kw"] for g in blocks} == {2, 3, 5, 9}
