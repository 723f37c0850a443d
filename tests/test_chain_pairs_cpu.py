"""Which chained layers run on CTA pairs, and in which form of the kernel (cpp/chain_launch.cpp)."""
import json
import os
import subprocess

import test_chain_pairs_gpu as gpu
import test_shared_accumulator_gpu
from xnor_nn_b200 import build

# Where a pair's longer hand-shakes cost more than its lighter loads save, either side of each line of the rule:
# the same layer on more images or with more filters
LINES = {  # name: (layer alone, layer on pairs)
    "narrow_odd_rows_more_tiles": ((400, 96, 192, 7, 7, 5, 5, 2, 2), (400, 96, 224, 7, 7, 5, 5, 2, 2)),
    "narrow_odd_rows_fewer_tiles": ((22, 160, 224, 18, 18, 5, 5, 2, 2), (22, 160, 256, 18, 18, 5, 5, 2, 2)),
    "narrow_odd_rows_tiles": ((28, 96, 384, 23, 23, 5, 5, 2, 2), (60, 96, 384, 23, 23, 5, 5, 2, 2)),
    "narrow_part_chunk_tiles": ((50, 100, 512, 18, 18, 3, 3, 1, 1), (100, 100, 1024, 18, 18, 3, 3, 1, 1)),
    "wide_odd_rows_fewer_tiles": ((21, 416, 160, 22, 22, 3, 3, 1, 1), (21, 416, 192, 22, 22, 3, 3, 1, 1)),
    "wide_part_chunk_more_tiles": ((200, 320, 192, 13, 13, 3, 3, 1, 1), (200, 320, 256, 13, 13, 3, 3, 1, 1)),
    "wide_part_chunk_fewer_tiles": ((64, 384, 256, 13, 13, 3, 3, 1, 1), (64, 384, 320, 13, 13, 3, 3, 1, 1)),
    "wide_part_chunk_few_tiles": ((20, 384, 192, 13, 13, 3, 3, 1, 1), (20, 384, 256, 13, 13, 3, 3, 1, 1)),
}
MORE = {"conv3": (128, 256, 384, 13, 13, 3, 3, 1, 1), "conv4": (128, 384, 256, 13, 13, 3, 3, 1, 1)}


def test_which_chained_layers_run_on_pairs(tmp_path):
    build.build()
    exe = str(tmp_path / "chain_launch")
    here = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cpp")
    objs = [os.path.join(build.OBJ, n + ".o") for n in ("conv_tcgen05.cu", "plan.cpp", "tensormap.cpp")]
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-I", os.path.join(build.ROOT, "include"), "-I",
                           build.CSRC, "-I", "/usr/local/cuda/include", os.path.join(here, "chain_launch.cpp")] +
                          objs + ["-o", exe])
    lines = {(name, on): d for name, both in LINES.items() for on, d in zip((False, True), both)}
    layers = {**gpu.PAIRS, **gpu.SINGLE, **MORE, **lines}
    order = (0, 2, 1, 3, 4, 5, 6, 7, 8)  # filters before channels
    out = subprocess.check_output([exe] + [",".join(str(d[i]) for i in order) for d in layers.values()],
                                  text=True).splitlines()
    got = dict(zip(layers, [json.loads(line) for line in out]))
    assert all(g["served"] and g["epilogue_warps"] == 16 for g in got.values())
    assert {key for key in lines if got.pop(key)["pair"] != key[1]} == set()
    pairs = {name: g for name, g in got.items() if g["pair"]}
    assert set(pairs) == set(gpu.PAIRS) | {"conv4"}
    form = {name: "columns" if g["planes"] else "resident" if g["resident"] else "halo" if g["halo"] else "ring"
            for name, g in pairs.items()}
    assert form == {"columns": "columns", "rows_of_all_filter_rows": "resident",
                    "rows_of_a_filter_row": "resident", "streamed": "halo", "streamed_two_filter_tiles": "halo",
                    "streamed_four_tiles_odd_filters": "halo", "streamed_192_filters": "halo",
                    "ring": "ring", "fewer_tiles_than_sms": "halo",
                    "part_chunk_fewer_tiles_than_sms": "halo", "conv4": "halo"}, form
    assert pairs["rows_of_all_filter_rows"]["halo"] > 136 >= pairs["rows_of_a_filter_row"]["halo"]
    assert {g["n_tiles"] for g in pairs.values()} == {1, 2, 4}
    assert {g["shared_cols"] for g in pairs.values()} == {0, 1}
    assert {g["m_tiles"] % 2 for g in pairs.values()} == {0, 1}
    # one position tile a pair at a time, all of its filter tiles in a row
    assert all(g["grid"] == 2 * min(74, (g["m_tiles"] + 1) // 2) for g in pairs.values())
    # the test of two issuers on one accumulator repeats each form
    assert all(pairs[name]["issuers"] == 2 for name in test_shared_accumulator_gpu.CHAINS)
    assert {form[name] for name in test_shared_accumulator_gpu.CHAINS} == set(form.values())
