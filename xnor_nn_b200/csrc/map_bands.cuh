// The bands of calculate_k in one launch (maps.cu): which layers it takes, how their output rows are dealt to
// blocks and which pixels of the source a block reads. Host code too, so that a test can walk the addresses.
#pragma once

#include "kernels.cuh"

namespace xb200 {
namespace bands {

constexpr int kWarps = 8, kThreads = 32 * kWarps;
constexpr int kMaxGroups = 32, kMaxTasks = 8 * kWarps, kTileFloats = 8 * 1024;
// More source than this keeps the GPU busy for longer than a launch takes the host, and bands read what
// their windows share more than once.
constexpr long kMaxBytes = 16L << 20;

struct MapArgs {
    const float *src;
    float *a, *k;
    int *error;
    unsigned long long wait_ns;
    int turn_step;             // 1, 0 in a self-test (ConvSelfTest)
    float inv_ic, inv_khw;
    int ic, hw, ih, iw, vec;
    int oh, ow, kh, kw, sh, sw, ph, pw;
    int rows, bands;           // output rows of a block, blocks of an image
    int lines, span, columns;  // rows and columns of A that a block's windows see; tasks of a group
    FastDiv by_hw, by_iw, by_ow;
};

// What block `block` does: output rows from oy0 of image n, whose windows start at input row y0; the rows of A that
// it leaves in the map; and the pixels first .. last that it adds up, in groups of 32. Rows above and below the
// image are none of them: a band whose windows lie there altogether, as unequal paddings or ones beyond the
// filter make them, has no tasks, and last - 1 is a pixel of image n in any case.
struct Band {
    int n, oy0, y0, own0, own1, first, last, groups, tasks;
};
__host__ __device__ inline Band band_of(const MapArgs &g, int block) {
    Band b;
    b.n = block / g.bands;
    const int band = block - b.n * g.bands;
    b.oy0 = band * g.rows;
    b.y0 = b.oy0 * g.sh - g.ph;
    b.own0 = b.oy0 * g.sh;
    b.own1 = band + 1 < g.bands ? b.own0 + g.rows * g.sh : g.ih;
    const int lo = b.y0 < 0 ? 0 : b.y0 < g.ih ? b.y0 : g.ih;
    const int seen = b.y0 + g.lines > b.own1 ? b.y0 + g.lines : b.own1;
    const int hi = seen > g.ih ? g.ih : seen > lo ? seen : lo;
    b.first = b.n * g.hw + lo * g.iw;
    b.last = b.n * g.hw + hi * g.iw;
    b.groups = (b.last - b.first + 31) >> 5;
    b.tasks = b.groups * g.columns;
    return b;
}

// What the launch takes, to a sixth (fitted to 78 layers of more than 5.9 us): a block's warps walk its tasks
// one after the other, and all blocks share the SMs. Two launches take a host 5.7 us, most of which passes on
// several streams hide. Over 285 layers (drawn from 1 to 256 images, 1 to 512 channels, 6 to 227 pixels, up to
// 16 MB), the three upstream calls with two launches here over those with one: 1.02 on one stream and 1.14
// among others if all take one, 1.035 and 1.14 with this rule; the 48 that it takes out 0.90 and 1.005 (19
// images of 464 channels, 17 x 17, filters of 5 x 5: 44.6 and 60.6 us on one stream, calculate_k alone 7.0 and
// 18.8). That was with counters for the hand-overs of running sums. With barriers 70 layers just beyond the line (8.5
// to 12 us by this formula) would take one launch 0.93 and 1.14 times as fast as two, 0.72 to 1.13 and 0.93 to 1.69.
inline double launch_us(long blocks, long tasks, long outputs, int taps) {
    return 3.6 + 0.58 * (double)(blocks * tasks) / (8.0 * sm_count()) + 0.74 * (double)((tasks + 7) / 8) +
           0.58 * (double)((outputs + kThreads - 1) / kThreads) * taps / 25;
}

// Bands: as tall as leaves a block per SM, and at least so tall that most of what a band reads is its own.
inline bool maps_shape(const Plan &p, MapArgs *g) {
    if (p.mb < 1 || p.oh < 1 || p.ow < 1 || p.ic < 1 || p.ih < 1 || p.iw < 1) return false;
    if (4L * p.mb * p.ic * p.ih * p.iw > kMaxBytes) return false;
    if (p.sh < 1 || p.sw < 1 || p.ph < 0 || p.pw < 0 || p.kh < 1 || p.kw < 1) return false;
    if ((long)p.kh * p.kw > 64 || (long)p.oh * p.ow > 1 << 20) return false;
    g->columns = div_up_i(p.ic, 32);
    const long span = (long)(p.ow - 1) * p.sw + p.kw;
    int rows = (int)((long)p.mb * p.oh / sm_count());
    if (rows < p.kh - 1) rows = p.kh - 1;
    if (rows < 1) rows = 1;
    if (rows > p.oh) rows = p.oh;
    for (;; rows--) {
        const long lines = (long)(rows - 1) * p.sh + p.kh;
        // input rows of a band, the rows below the last window with the last band
        const int bands = div_up_i(p.oh, rows);
        const long tail = p.ih - (long)(bands - 1) * rows * p.sh + p.ph;
        const long reach = (long)rows * p.sh + p.ph;
        long most = lines > reach ? lines : reach;
        if (tail > most) most = tail;
        if (most > p.ih) most = p.ih;
        const long groups = (most * p.iw + 31) / 32;
        if (groups <= kMaxGroups && groups * g->columns <= kMaxTasks && lines * span <= kTileFloats) {
            g->rows = rows;
            g->bands = bands;
            g->lines = (int)lines;
            g->span = (int)span;
            return (long)p.mb * bands < 1L << 30 &&
                   launch_us((long)p.mb * bands, groups * g->columns, (long)rows * p.ow, p.kh * p.kw) <= 8.5;
        }
        if (rows == 1) return false;
    }
}

}  // namespace bands
}  // namespace xb200
