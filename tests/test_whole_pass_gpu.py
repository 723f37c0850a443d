"""Forward passes of small layers in one launch (conv_whole.cu), at the edges of what that takes: one and
148 tiles, tiles of many images and of part of a row, positions of one to sixteen 16-byte columns (odd
numbers, channel tails, several K chunks), filters split into narrow tiles, both layouts with and without
16-byte loads, and the first layers beyond each limit, which take two launches. Sums (from the packed
frame the pass leaves), A and K bit for bit against the oracle, floats to the parity contract's 1e-4."""
import numpy as np
import pytest

import cases
import xnor_nn_b200 as xb

pytestmark = pytest.mark.gpu

CL = (1, 1, 1)
ONE_LAUNCH = [
    cases._c("one_tile_one_channel", 1, 16, 1, 5, 5, 3, 3, ph=1, pw=1),
    cases._c("many_images_a_tile", 140, 24, 20, 2, 2, 3, 3, ph=1, pw=1),
    cases._c("part_of_a_row_16_groups", 2, 40, 70, 5, 180, 3, 3, ph=1, pw=1),
    cases._c("148_tiles", 148, 33, 40, 8, 16, 1, 1),
    cases._c("147_tiles_two_filter_tiles", 73, 300, 16, 8, 16, 1, 1),
    cases._c("odd_columns_a_row_as_one", 3, 50, 90, 11, 9, 3, 3, ph=1, pw=1),
    cases._c("five_taps_a_row_as_one", 2, 70, 33, 14, 15, 5, 5, ph=2, pw=2),
    cases._c("swizzled_one_chunk_tail", 2, 96, 230, 9, 10, 3, 3, ph=1, pw=1),
    cases._c("swizzled_two_chunks_tail", 2, 250, 300, 9, 10, 3, 3, ph=1, pw=1),
    cases._c("swizzled_sixteen_columns", 3, 48, 512, 7, 9, 3, 3, ph=1, pw=1),
    cases._c("one_tap_rows_of_32_bytes", 3, 20, 50, 9, 9, 1, 1),
    cases._c("one_tap_rows_of_64_bytes", 3, 20, 100, 9, 9, 1, 1),
    cases._c("column_of_taps", 3, 20, 100, 9, 9, 3, 1),
    cases._c("no_padding", 3, 20, 260, 9, 9, 3, 3),
    cases._c("three_filter_tiles", 1, 520, 64, 13, 13, 3, 3, ph=1, pw=1),
    cases._c("ring_comes_round", 30, 256, 384, 13, 13, 3, 3, ph=1, pw=1),
    cases._c("channels_last_16_byte_loads", 3, 44, 92, 10, 11, 3, 3, ph=1, pw=1, fmt=CL),
    cases._c("channels_last_odd", 3, 43, 91, 10, 11, 3, 3, ph=1, pw=1, fmt=CL),
    cases._c("channels_last_whole_sectors", 20, 256, 384, 13, 13, 3, 3, ph=1, pw=1, fmt=CL),
    cases._c("channels_last_source_only", 3, 44, 92, 10, 11, 3, 3, ph=1, pw=1, fmt=(1, 0, 0)),
    cases._c("packed_twice_less_work", 10, 300, 256, 14, 14, 3, 3, ph=1, pw=1),
    cases._c("filter_of_zeros_and_ties", 2, 16, 6, 6, 7, 2, 2, ph=1, pw=1, fill="affine"),
]
TWO_LAUNCHES = [
    cases._c("149_tiles", 149, 33, 40, 8, 16, 1, 1),
    cases._c("513_rows", 1, 20, 33, 5, 191, 3, 4, ph=1, pw=1),
    cases._c("81_tasks", 1, 20, 860, 9, 9, 1, 1),
    # as long as the general path's work, half of it repeated; with a quarter of it one launch again
    cases._c("packed_twice", 40, 300, 256, 14, 14, 3, 3, ph=1, pw=1),
    cases._c("wide_halos", 16, 31, 229, 27, 27, 5, 5, ph=2, pw=2),
]


def _run(oracle, case, launches):
    _, d, _, fmt = case
    src, w = cases.make_inputs(case)
    want = oracle.convolution(cases.oracle_shape(case), src, w)
    conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NHWC if fmt[0] else xb.NCHW,
                          xb.HWIO if fmt[1] else xb.OIHW, xb.NHWC if fmt[2] else xb.NCHW, d["mb"],
                          d["oc"], d["ic"], d["ih"], d["iw"], d["kh"], d["kw"], d["sh"], d["sw"],
                          d["ph"], d["pw"], w)
    for _ in range(2):  # the second pass finds the frame that the first one left
        dst = np.full(want["dst"].size, np.nan, np.float32)
        before = xb.kernel_launches()
        conv.forward(src, dst)
        assert xb.kernel_launches() - before == launches
        assert np.array_equal(conv.forward_sums(), want["sums"])
        assert np.array_equal(conv.read(xb.SLOT_A, np.float32), want["a"])
        assert np.array_equal(conv.read(xb.SLOT_K, np.float32), want["k"])
        assert np.all(np.abs(dst - want["dst"]) <= 1e-4 * np.abs(want["dst"]))
    conv.close()


@pytest.mark.parametrize("case", ONE_LAUNCH, ids=[c[0] for c in ONE_LAUNCH])
def test_one_launch(oracle, case):
    _run(oracle, case, 1)


@pytest.mark.parametrize("case", TWO_LAUNCHES, ids=[c[0] for c in TWO_LAUNCHES])
def test_beyond_its_limits(oracle, case):
    _run(oracle, case, 2)


def test_result_over_the_source():
    """A pass whose result overlaps its source packs all of it before it stores anything: two launches."""
    torch = pytest.importorskip("torch")
    gen = torch.Generator(device="cuda").manual_seed(5)
    x = torch.randn(12, 64, 14, 14, generator=gen, device="cuda")
    w = torch.randn(64, 64, 3, 3, generator=gen, device="cuda")
    conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NCHW, xb.OIHW, xb.NCHW, 12, 64, 64, 14, 14, 3, 3, 1, 1, 1,
                          1, w)
    want = torch.empty_like(x)
    counts = []
    shifted = torch.empty(x.numel() + 5, device="cuda")
    torch.cuda.synchronize()
    for src, dst in ((x, want), (x.clone(), None), (shifted[:-5].view_as(x), shifted[5:].view_as(x))):
        if dst is None:
            dst = src
        elif dst is not want:
            src.copy_(x)
        torch.cuda.synchronize()
        before = xb.kernel_launches()
        conv.forward(src, dst)
        counts.append(xb.kernel_launches() - before)
        conv.synchronize()
        assert torch.equal(dst, want)
    assert counts == [1, 2, 2]
    conv.close()


@pytest.mark.parametrize("between", [False, True], ids=["pass", "calculate_k_and_pass"])
def test_new_weights_before_every_pass(between):
    """Filters packed anew and the pass that reads them follow each other on the stream with nothing waited for in
    between, alone and with a kernel that lets its successor start early: every pass has its own filters."""
    torch = pytest.importorskip("torch")
    gen = torch.Generator(device="cuda").manual_seed(9)
    conv = xb.Convolution(xb.ALGORITHM_BCAST, xb.NCHW, xb.OIHW, xb.NCHW, 2, 64, 96, 9, 9, 3, 3, 1, 1, 1, 1)
    x = torch.randn(2, 96, 9, 9, generator=gen, device="cuda")
    weights = [torch.randn(64, 96, 3, 3, generator=gen, device="cuda") for _ in range(2)]
    conv.set_stream(torch.cuda.current_stream().cuda_stream or 1)  # 1: the legacy default stream
    want = [torch.empty(conv.out_shape, device="cuda") for _ in weights]
    for w, y in zip(weights, want):
        conv.change_weights(w)
        torch.cuda.synchronize()
        conv.forward(x, y)
        torch.cuda.synchronize()
    assert not torch.equal(*want)
    got = torch.empty((200, *conv.out_shape), device="cuda")
    before = xb.kernel_launches()
    for i in range(200):
        conv.change_weights(weights[i % 2])
        if between:
            assert conv.execute("calculate_k", src=x) == xb.SUCCESS
        conv.forward(x, got[i])
    assert xb.kernel_launches() - before == 200 * (3 if between else 2)
    assert all(torch.equal(got[i], want[i % 2]) for i in range(200))
    conv.close()
