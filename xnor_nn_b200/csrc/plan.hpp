// Host-side description of one binary convolution on the device: geometry, the kernel family
// chosen for it, and the layout of every internal buffer. One Plan hangs off
// xnor_nn_convolution_t::state (the role upstream's Implementation object plays,
// src/implementation.hpp:11-25); it is immutable after xnor_nn_init_convolution.
#pragma once

#include <cstddef>
#include <cstdint>

#include "xnor_nn.h"

namespace xb200 {

// Which convolution kernel consumes the packed operands. The packed layouts differ per family,
// so the choice is fixed at init and every executor of the descriptor follows it.
enum Family : int {
    kPopc = 0,          // bits, LOP3 + POPC on the integer pipe; any stride, padding and format
    kTcgen05 = 2,       // +-1 as 4-bit floats, tcgen05.mma kind::mxf4 into tensor memory; stride 1
    kTcgen05Rows = 3,   // request only: the same family, forced onto its image-row kernel
    kAuto = -1,
};

// Accumulator columns of the image-row kernel: two of them and 32 columns of block scales fill
// the 512 columns of tensor memory. Rows of more pixels, up to kImgWideColumns, have a single
// accumulator, which the next tile waits for.
constexpr int kImgColumns = 240;
constexpr int kImgWideColumns = 256;

struct Plan {
    // geometry (copied from the descriptor so kernels never chase the caller's struct)
    int mb, ic, ih, iw, oc, oh, ow, kh, kw, sh, sw, ph, pw;
    bool src_nhwc, w_hwio, dst_nhwc;
    bool formats_ok;  // false: an unknown tensor format was requested -> xnor_nn_unimplemented

    Family family;

    // scalars rounded on the host exactly as upstream computes them
    float inv_ic;   // 1.f / IC                     (src/bcast_calculate_k.cpp:42)
    float inv_khw;  // 1.f / KH / KW                (src/bcast_calculate_k.cpp:43)
    float inv_chw;  // 1.f / (IC*KH*KW)             (src/bcast_binarize_weights.cpp:95)

    // ---- bit layout (kPopc) -------------------------------------------------------------
    // activations: uint32 [mb][ih][iw][icw]; channel c is bit (31 - c%32) of word c/32; bits
    //              past the last channel are 0.
    // weights:     uint32 [kh][kw][icw][ocp]; same bit order, bits past the last channel 0,
    //              so absent channels xor to 0 on both sides.
    int icw;  // 32-bit words per pixel
    int ocp;  // output channels rounded up to the kernel's channel tile

    // ---- 4-bit layout (kTcgen05) -----------------------------------------------------------
    // A value is a 4-bit float (e2m1): +1 = 0x2, -1 = 0xA, 0 = 0x0, channel c in the low (c even)
    // or high nibble of byte c/2. Activations are +-1 on a zero frame so that a filter tap is a
    // constant row shift: rows of (iw + pw) positions (the pw zeros after a row double as the left
    // border of the next one), (ih + ph) rows per image (same sharing between images), lead rows
    // of zeros in front. Position q of image n, row h, column w sits at row
    //   lead + (n*(ih+ph) + h)*(iw+pw) + w
    // of a [rows][icp] byte matrix, and tap (kh,kw) of the output at q reads row
    //   q + (kh-ph)*(iw+pw) + (kw-pw).
    int icp;        // bytes from a position to the next: row_bytes, rounded up to 64 where that pays
    int row_bytes;  // bytes of a position: two channels each, rounded up to 16
    int tap_pitch;  // bytes from a packed filter's row to the next filter's
    int kchunk;     // bytes of K per pipeline stage: 128, 64 or 32 (= the swizzle span)
    int wp, hp;     // iw + pw, ih + ph
    int lead;       // zero rows in front of the first image
    long rows;      // rows allocated (frame + tail slack so every tile load is in range)
    long q_total;   // positions the kernel computes (mb*hp*wp), a multiple of nothing
    int ocp16;      // output channels rounded up to 16 (UMMA N granularity)
    int n_tile;     // UMMA N per accumulator (<= 256, multiple of 16)

    // Layers of few channels: the kw taps of a filter row read neighbouring positions, and
    // positions are contiguous, so the operand row of position q can simply run on into the next
    // kw - 1 positions: one tap per filter row, kw*icp bytes deep, from the same activations (a
    // tensor map whose rows overlap). Weights are then [kh][ocp16][tap_pitch]. The copy engine moves
    // full 128-byte rows instead of kw short ones, and 64-channel slices are not cut off at every tap.
    bool cat;

    // ---- folded layers (kTcgen05, strides) -------------------------------------------------
    // A strided layer becomes a unit-stride one for the same kernel: a position of the frame is an
    // output column ow and a block hb of sh input rows, and its channels are the values
    //   x[c][hb*sh - ph + i][ow*sw - pw + j],  i < fold_rows = min(kh, sh), j < kw, c < ic,
    // in the order (i, j, c) with the channels rounded up to eight or, with fewer than eight
    // channels, (c, i, j) with the columns rounded up to eight (fold_field; else 0): fold_ic in
    // all. Output row oh then reads the fold_taps = ceil(kh/sh) blocks oh, oh+1, ...: a
    // fold_taps x 1 filter whose rows past kh are zero weights. The frame has no border (what lies
    // outside the image is stored as zeros): wp = ow, hp = oh + fold_taps - 1, lead = 0, and icp,
    // kchunk describe fold_ic channels.
    bool fold;
    int fold_rows, fold_taps, fold_ic, fold_field;
    int fold_span;      // input columns an output row reads: (ow-1)*sw + kw
    int fold_channels;  // channels the packer stages at a time (all of them, or a multiple of 8)

    // ---- tiling of the image-row kernel (kTcgen05, conv_tcgen05_img.cu) ---------------------
    // That kernel puts 128 filters on the UMMA M side and, on the N side, `img_rows` whole output
    // rows of one image (img_rows * ow <= 240 positions, or one row of up to 256, rounded up to 16
    // for the instruction).
    // Tiles are dealt round-robin to one CTA per SM; the tiles of a last, partly filled round are
    // cut in two row halves so that they spread over twice as many SMs.
    bool frame_walk;     // the position-tile kernel can serve the shape
    bool img;            // the forward pass launches the image-row kernel (else the position-tile one)
    bool img_forced;     // asked for by name, or the position-tile kernel cannot serve the shape
    int img_rows;        // output rows per tile
    int img_n;           // UMMA N of a whole tile
    int img_row_blocks;  // tiles per image column = ceil(oh / img_rows)
    int img_m_blocks;    // ceil(oc / 128)
    int img_tiles;       // mb * img_row_blocks * img_m_blocks
    int img_whole;       // tiles [0, img_whole) run whole, the rest as two halves each
    int img_half_rows;   // rows of the first half (0: nothing is split)
    int img_n_half;      // UMMA N of a half tile
    int img_grid;        // CTAs launched
    int img_stages;      // operand pipeline depth
    int img_staging;     // result staging buffers shared by the four epilogue warps (1, 2 or 4)

    size_t bytes[xnor_nn_resource_number];
};

// The layer the tensor-core kernel is launched on: the plan itself, or the unit-stride layer a
// strided one was folded into. (The box filter K is the original layer's and computed apart.)
Plan conv_view(const Plan &p);
// The row of signs that the packer of a folded layer with fewer than eight channels stages, in units of 32
// columns (four words of nibbles): all columns of the image with the border in front, and all that is
// read of them.
int fold_bit_pitch(const Plan &p);
// Rows behind the last position that tile loads may reach.
long frame_slack(const Plan &p);

int div_up_i(int a, int b);

// SMs of the current device (148 on B200); the same figure when no device can be asked, so that
// plans made on a machine without a GPU come out as they would on the target.
int sm_count();

// Fills a Plan from the descriptor fields and the requested family (kAuto: pick by shape).
// Never fails: unknown formats are remembered and reported by the executors.
void make_plan(Plan *p, const xnor_nn_convolution_t *c, Family requested);

// (Re)derives the image-row tiling from the plan's geometry and minibatch; called by make_plan and
// for every minibatch slice of a plan. Leaves p->img false when the shape does not suit.
void plan_image_rows(Plan *p);
// Result staging of the image-row kernel: words per filter row when every filter's run is staged
// on its own (room for a shift of up to three words; an odd multiple of 4, so that the rows of 32
// filters spread over the shared-memory banks as well as a multiple of 4 can), and
// bytes of one staging buffer (32 rows, or a dense 32 x OH*OW block for whole-image tiles).
int img_staging_row_words(const Plan &p);
size_t img_staging_bytes(const Plan &p);

const char *family_name(Family f);

}  // namespace xb200
