// Launch parameters of the position-tile kernel (conv_tcgen05.cu), in a header of their own so that
// host code can read what the launcher decided.
#pragma once

#include <cstdint>

#include "kernels.cuh"

namespace xb200 {

struct TcArgs {
    const float *alpha;
    const float *kmap;   // K per output pixel, or null: box-filter it from amap in the epilogue
    const float *amap;   // mean |x| per input pixel (used when kmap is null)
    float *kmap_out;     // where the epilogue records the K it computed (may be null)
    float inv_khw;
    int ih, iw, kh;
    float *dst;
    int32_t *sums;
    int *error;
    long q_total;
    int m_tiles, n_tiles, n_tile;
    FastDiv by_frame, by_wp;  // position -> image, row (q_total < 2^30)
    int kchunk, chunks_per_tap, kw, ph, pw;
    int taps, tap_kw;  // filter taps as the operands see them, columns among them (see Plan::cat)
    int wp, hp, lead, oh, ow, oc, ocp16;
    uint32_t idesc;
    uint32_t desc_hi;  // upper 32 bits of the shared-memory matrix descriptors
    uint32_t a_bytes, stage_bytes, tx_bytes;
    int dst_nhwc;
    // chained layers: instead of floats the epilogue writes the next layer's packed input
    uint8_t *emit_bin;    // next layer's +-1 nibble frame, or null
    float *emit_a;        // next layer's mean-|x| map
    int e_wp, e_hp, e_lead, e_icp;  // the next layer's frame geometry
    float e_inv_ic;       // 1.f / (next layer's channels = this layer's filters)
    int n_inner;          // 1: a CTA works through all filter tiles of a pixel tile in a row
    unsigned long long wait_ns;  // bound of every mbarrier wait
    int drop_commit;      // self-test: CTA 0 leaves out the commit that publishes its first tile
    int issuers;          // threads that issue MMAs: 1, or 2 taking alternate pipeline stages
    int n_stages;         // ring buffers in use
    // Halo mode (pairs, filters at least two taps wide): the position tile of a
    // filter row is loaded once, with the kw - 1 positions that follow it, and serves all kw taps
    // of the row (a tap is a row offset into the tile), or, with `block`, those of all filter rows; the ring
    // then holds filter tiles only.
    int halo;             // 0, or rows of a position tile: 128 + 8 (128 with a single tap per row), up to 256 with block
    int n_a_slots;        // halo tiles in flight
    uint32_t a_slot_bytes, b_ring_off, b_slot_bytes, b_bytes;
    // Resident filters (pairs whose tiles all have the same filter tile, if its operands of all
    // taps fit shared memory beside three position tiles of 128-byte rows): filter tiles are loaded
    // once and stay. Position tiles as in halo mode or as columns:
    int resident;
    // A position tile of `halo` rows serves all filter rows: beside resident filters (producer_block, which loads a
    // chunk's filters behind the first tile's positions of that chunk) and streamed ones (producer_halo).
    int block;
    // Resident filters with position tiles of 16-byte channel columns (producer_planes): columns of a
    // tile, positions of it and positions from one column to the next (a multiple of 8), bytes per
    // position and the upper half of its matrix descriptors. 0: not so.
    int planes, plane_rows, plane_pitch, pos_bytes;
    uint32_t plane_desc_hi;
    int kk_last;          // MMAs of a tap's last channel chunk: its 64-channel slices that hold
                          // channels at all (the chunk is padded with zeros to kchunk bytes)
    uint32_t acc_step;    // columns from the first accumulator to the second
    int n_acc;            // accumulators in tensor memory
    int teams;            // epilogue teams that take the tiles in turn: 1, 2 or 4
    FastDiv by_acc;       // tile -> round of the accumulators
    int shared_cols;      // the accumulators overlap (n_tile > kAccStep)
};

}  // namespace xb200
