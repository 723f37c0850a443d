"""What the launcher leaves the L1 in layers whose channels-last results are stored float by float
(cpp/tile_launch.cpp)."""
import json
import os
import subprocess

import test_scattered_results_gpu as gpu
from xnor_nn_b200 import build

NEAR = 195 * 1024  # with the system's 1 KB a block 196 KB, which leaves 60 KB


def test_the_l1_keeps_60_kilobytes(tmp_path):
    build.build()
    exe = str(tmp_path / "tile_launch")
    objs = [os.path.join(build.OBJ, n + ".o") for n in ("conv_tcgen05.cu", "plan.cpp", "tensormap.cpp")]
    subprocess.check_call(
        ["g++", "-std=c++17", "-O1", "-I", os.path.join(build.ROOT, "include"), "-I", build.CSRC, "-I",
         "/usr/local/cuda/include", os.path.join(os.path.dirname(__file__), "cpp", "tile_launch.cpp")] +
        objs + ["-o", exe])
    keys = ("mb", "oc", "ic", "ih", "iw", "kh", "kw", "sh", "sw", "ph", "pw")
    env = {k: v for k, v in os.environ.items() if k != "XNOR_NN_B200_KERNEL"}

    def run(layers):
        out = subprocess.check_output([exe] + [",".join(map(str, d)) for d in layers], text=True, env=env)
        return [json.loads(line) for line in out.splitlines()]

    sizes = [tuple(c[1][k] for k in keys) for c in gpu.LAYERS]
    got = dict(zip([c[0] for c in gpu.LAYERS], run([d + (1,) for d in sizes])))
    first = dict(zip(got, run(sizes)))
    for name, g in got.items():
        assert g["served"] and g["pair"] and g["halo"] > 136, (name, g)
        assert g["resident"] == (not name.startswith(("streamed", "whole"))), (name, g)
        assert g["smem"] <= NEAR and (g["a_slots"] >= 2 if g["resident"] else g["stages"] >= 4), (name, g)
    # a tile of 256 is not halved, one of 192 is; results in whole sectors take the room
    assert got["whole_256"]["n_tiles"] == 1 and first["whole_256"]["n_tiles"] == 2
    assert got["half_of_192"]["n_tiles"] == first["half_of_192"]["n_tiles"] == 2
    assert sum(g["smem"] > NEAR for g in first.values()) >= 5
    # a layer whose filters leave no room for two tiles beside them keeps them, whatever the L1 has left
    tight = run([(40, 251, 256, 30, 34, 3, 3, 1, 1, 1, 1, 1)])[0]
    assert tight["resident"] and tight["a_slots"] >= 2 and tight["smem"] > NEAR, tight
