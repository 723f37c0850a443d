"""What the position-tile launcher asks of the driver (tests/cpp/tile_launch.cpp): addresses, extents,
strides and boxes of every tensor map keep to what cuTensorMapEncodeTiled documents, each stride
building on the one before it, and no box reaches past the frame. (Rows may overlap: filter rows that
are one operand row run on into the next positions.) Which layers load their position tiles as 16-byte
columns, at the lines where that was measured to stop paying. And that the layers of the GPU tests take
the forms of the kernel that they are there for. Host code only."""
import json
import os
import subprocess

import pytest

import cases
import test_folded_gpu
import test_long_filter_rows_gpu
import test_long_tiles_gpu
import test_position_columns_gpu
import test_resident_filters_gpu
import test_shared_accumulator_gpu
import test_streamed_filters_gpu
import test_three_accumulators_gpu
from xnor_nn_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))
# (name, mb, oc, ic, ih, iw, kh, kw): either side of each line of the rule
FASTER_AS_COLUMNS = [
    cases._c("conv2", 128, 256, 96, 27, 27, 5, 5, ph=2, pw=2),
    cases._c("three_tiles_a_pair", 75, 256, 96, 27, 27, 3, 3, ph=1, pw=1),
    cases._c("two_tiles_a_pair_32_channels", 71, 192, 32, 17, 17, 5, 5, ph=2, pw=2),
    cases._c("33_channels_96_filters", 266, 96, 33, 14, 14, 3, 3, ph=1, pw=1),
    cases._c("33_channels_64_filters_four_rows", 160, 64, 33, 17, 17, 4, 4, ph=2, pw=2),
    cases._c("two_tiles_in_flight", 40, 256, 224, 56, 56, 3, 3, ph=1, pw=1),
]
FASTER_AS_ROWS = [
    cases._c("two_filter_rows", 71, 384, 128, 28, 28, 2, 2, ph=1, pw=1),
    cases._c("one_filter_row", 306, 384, 160, 14, 14, 1, 3),
    cases._c("two_tiles_a_pair", 45, 256, 96, 27, 27, 3, 3, ph=1, pw=1),
    cases._c("two_tiles_a_pair_33_channels", 90, 192, 33, 17, 17, 3, 3, ph=1, pw=1),
    cases._c("33_channels_64_filters", 266, 64, 33, 14, 14, 3, 3, ph=1, pw=1),
    cases._c("filters_not_resident_beside_rows", 1129, 192, 127, 8, 8, 5, 5, ph=2, pw=2),
    cases._c("257_rows", 80, 256, 96, 3, 62, 3, 4, ph=1, pw=1),
]
GPU_COLUMNS = test_position_columns_gpu.COLUMNS + test_resident_filters_gpu.COLUMNS
# either side of the lines of the rule for eight epilogue warps
EIGHT_WARPS = test_long_tiles_gpu.LONG_TILES + [
    cases._c("conv2_eight_warps", 128, 256, 96, 27, 27, 5, 5, ph=2, pw=2),
    cases._c("vgg_eight_warps", 64, 512, 512, 28, 28, 3, 3, ph=1, pw=1),
]
SIXTEEN_WARPS = [
    cases._c("three_long_tiles_a_pair", 256, 256, 384, 13, 13, 3, 3, ph=1, pw=1),
    cases._c("4608_cycles", 180, 256, 256, 28, 28, 3, 3, ph=1, pw=1),
    cases._c("4224_cycles", 180, 256, 224, 28, 28, 3, 3, ph=1, pw=1),
]
LOST_COMMIT = cases._c("lost_commit", 64, 256, 96, 27, 27, 5, 5, ph=2, pw=2)
SHARED_ACCUMULATOR = [c for c in test_shared_accumulator_gpu.LAYERS if not c[0].startswith("whole")]
LAYERS = (FASTER_AS_COLUMNS + FASTER_AS_ROWS + GPU_COLUMNS + test_position_columns_gpu.ROWS +
          test_resident_filters_gpu.ROWS + [LOST_COMMIT] + test_streamed_filters_gpu.STREAMED +
          test_folded_gpu.FOLDED + test_long_filter_rows_gpu.LONG_ROWS + EIGHT_WARPS + SIXTEEN_WARPS +
          SHARED_ACCUMULATOR + test_three_accumulators_gpu.LAYERS + cases.SHAPE_CASES + [
              cases._c("alexnet_conv3_mb256", 256, 384, 256, 13, 13, 3, 3, ph=1, pw=1),
              cases._c("alexnet_conv4_mb256", 256, 256, 384, 13, 13, 3, 3, ph=1, pw=1)])


@pytest.fixture(scope="module")
def launches(tmp_path_factory):
    """What the launcher did with each of LAYERS, in order."""
    build.build()
    exe = str(tmp_path_factory.mktemp("tile_launch") / "tile_launch")
    objs = [os.path.join(build.OBJ, n + ".o") for n in ("conv_tcgen05.cu", "plan.cpp", "tensormap.cpp")]
    subprocess.check_call(
        ["g++", "-std=c++17", "-O1", "-I", os.path.join(build.ROOT, "include"), "-I", build.CSRC, "-I",
         "/usr/local/cuda/include", os.path.join(HERE, "cpp", "tile_launch.cpp")] + objs + ["-o", exe])
    keys = ("mb", "oc", "ic", "ih", "iw", "kh", "kw", "sh", "sw", "ph", "pw")
    env = {k: v for k, v in os.environ.items() if k != "XNOR_NN_B200_KERNEL"}
    out = subprocess.check_output(
        [exe] + [",".join(str(c[1][k]) for k in keys) for c in LAYERS], text=True, env=env).splitlines()
    assert len(out) == len(LAYERS)
    return [json.loads(line) for line in out]


def _of(launches, layers):
    """The launches of consecutive layers of LAYERS."""
    at = LAYERS.index(layers[0])
    assert LAYERS[at:at + len(layers)] == layers
    return launches[at:at + len(layers)]


@pytest.mark.parametrize("i", range(len(LAYERS)), ids=[c[0] for c in LAYERS])
def test_tensor_maps_keep_to_the_documented_rules(launches, i):
    got = launches[i]
    for m in got.get("maps", ()):
        assert m["ptr"] % 16 == 0
        assert all(0 < d <= 1 << 32 for d in m["dim"])
        assert all(0 < b <= 256 for b in m["box"])
        assert m["box"][0] % 16 == 0 and m["box"][0] <= (16, 32, 64, 128)[m["swizzle"]]
        assert all(s % 16 == 0 and s < 1 << 40 for s in m["stride"])
        for near, far in zip(m["stride"], m["stride"][1:]):
            assert far % near == 0, m
        if m["ptr"] == got["activations"]:
            last = m["dim"][0] + sum((d - 1) * s for d, s in zip(m["dim"][1:], m["stride"]))
            assert last <= got["rows"] * got["icp"], m


@pytest.mark.parametrize("i", range(len(FASTER_AS_COLUMNS + FASTER_AS_ROWS)),
                         ids=[c[0] for c in FASTER_AS_COLUMNS + FASTER_AS_ROWS])
def test_columns_where_they_are_faster(launches, i):
    got = launches[i]
    boxes = [m["box"][0] for m in got["maps"] if m["ptr"] == got["activations"]]
    assert (boxes == [16]) == (i < len(FASTER_AS_COLUMNS)), boxes


def test_gpu_tests_of_position_columns_reach_them(launches):
    got = _of(launches, GPU_COLUMNS)
    assert all(g["planes"] and g["resident"] and g["issuers"] == 2 for g in got + _of(launches, [LOST_COMMIT]))
    assert {g["icp"] // 16 for g in got} >= {1, 2, 3, 5, 7}
    assert {g["a_slots"] for g in got} >= {2, 8} and 256 in {g["plane_rows"] for g in got}
    assert {g["kchunk"] for g in got} == {32, 64, 128}
    assert {g["m_tiles"] % 2 for g in got} == {0, 1} and {g["n_tiles"] for g in got} == {1, 2, 3}
    assert min(g["groups"] for g in got) < 8 < max(g["groups"] for g in got)
    assert 8 in {g["groups"] for g in got} and 1 in {g["shared_cols"] for g in got}
    assert not any(g["planes"] for g in _of(launches, test_position_columns_gpu.ROWS))


def test_eight_epilogue_warps_on_long_tiles(launches):
    assert [g["epilogue_warps"] for g in _of(launches, EIGHT_WARPS)] == [8] * len(EIGHT_WARPS)
    assert [g["epilogue_warps"] for g in _of(launches, SIXTEEN_WARPS)] == [16] * len(SIXTEEN_WARPS)
    got = _of(launches, test_long_tiles_gpu.LONG_TILES)
    assert {g["shared_cols"] for g in got} == {0, 1} and {g["n_tiles"] for g in got} == {1, 2}


def test_gpu_tests_of_long_filter_rows_reach_columns(launches):
    layers = test_long_filter_rows_gpu.LONG_ROWS
    got = _of(launches, layers)
    assert all(g["planes"] and g["resident"] and g["issuers"] == 2 for g in got)
    starts = [g["groups"] // c[1]["kh"] * g["kchunk"] // 32 for g, c in zip(got, layers)]
    assert starts == [32, 36, 36, 40, 88]


def test_gpu_tests_of_resident_rows_reach_them(launches):
    got = _of(launches, test_resident_filters_gpu.ROWS)
    assert all(g["resident"] and not g["planes"] and g["pair"] for g in got)
    seen = {(g["tap_kw"], g["n_tiles"], g["shared_cols"]) for g in got}
    assert seen >= {(t, n, c) for t in (1, 3) for n, c in ((1, 0), (1, 1), (2, 0))} | {(3, 3, 0)}
    assert {g["kchunk"] for g in got} == {32, 64, 128} and {g["groups"] % 2 for g in got} == {0, 1}


def test_gpu_tests_of_streamed_filters_reach_them(launches):
    got = _of(launches, test_streamed_filters_gpu.STREAMED)
    assert all(g["halo"] and not g["resident"] and g["issuers"] == 2 for g in got)


def test_gpu_tests_of_shared_accumulators_reach_each_form_with_two_issuers(launches):
    got = dict(zip([c[0] for c in SHARED_ACCUMULATOR], _of(launches, SHARED_ACCUMULATOR)))
    assert all(g["issuers"] == 2 for g in got.values())
    form = {name: ("pair " if g["pair"] else "single ") +
                  ("columns" if g["planes"] else "resident" if g["resident"] else "streamed" if g["halo"] else "ring")
            for name, g in got.items()}
    assert form == {"pairs_columns": "pair columns", "pairs_streamed": "pair resident",
                    "pairs_streamed_256_filters": "pair streamed", "pairs_streamed_192_filters": "pair streamed",
                    "pairs_streamed_a_filter_row_at_a_time": "pair streamed", "single_ctas": "single ring"}
    # a position tile for all filter rows, but where the name says otherwise
    assert {name for name, g in got.items() if g["halo"] > 136} == {
        "pairs_streamed", "pairs_streamed_256_filters", "pairs_streamed_192_filters"}
    assert (got["pairs_streamed_256_filters"]["shared_cols"], got["pairs_streamed_192_filters"]["shared_cols"]) == (1, 0)


def test_gpu_tests_of_three_accumulators_reach_them(launches):
    got = _of(launches, test_three_accumulators_gpu.LAYERS)
    assert all(g["pair"] and g["resident"] and g["halo"] > 136 and g["accumulators"] == 3 for g in got)
    assert [(g["issuers"], g["n_tiles"]) for g in got] == [(1, 1), (2, 1), (1, 2)]
    assert all(g["m_tiles"] * g["n_tiles"] > 3 * g["grid"] for g in got)  # a fourth tile has the first one's
