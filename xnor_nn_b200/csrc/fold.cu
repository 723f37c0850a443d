// Activation packer of folded layers (strided convolutions, plan.hpp): one pass over the fp32
// source that leaves, for every output column and block of sh input rows, the +-1 nibbles of all
// the values the filter's columns see there, and, when asked for, the per-pixel mean |x| map.
// Takes the place of upstream src/bcast_binarize_data.cpp:43-73 and the first loop of
// src/bcast_calculate_k.cpp:49-66 for these layers.
//
// A block owns one row block of one image. It reads the sh rows of a group of channels (with an
// NCHW source they are one contiguous run per channel), each value once: |x|/IC goes into the
// pixel's running sum, channels ascending as upstream adds them, and the sign to its place in
// shared memory, where borders and rows outside the image are zeros. Then every thread assembles
// 32-bit words (eight nibbles) of the packed rows, found through a table that is the same for all
// columns; a block's words are one contiguous run. Input rows that no output row reads still get
// their mean |x|, from blocks that pack nothing.
//
// Fewer than eight channels (fold_few_kernel): the eight nibbles of a word are neighbouring
// columns. Both halves are bound by instruction issue, so a warp reads 32 neighbouring columns, a
// vote turns their signs into one word of bits, and a thread, which keeps its place in the column,
// takes eight bits from two words and spreads them to nibbles. AlexNet conv1 on 64 images (40 MB
// in, 20 MB out): 22 us; 32 without the channels and the pair of words compiled in, 37-39 with a byte staged per value and a table lookup per word
// (28 M warp instructions), 55 with every nibble fetched on its own.
// Otherwise (fold_kernel) they are neighbouring channels of a pixel, put together once per pixel
// and copied.
#include "kernels.cuh"

#include <atomic>

namespace xb200 {

namespace {

constexpr int kThreads = 256;
constexpr int kTasks = 4;   // few channels: warp loads per channel before the first is used

struct FoldArgs {
    const float *src;
    uint32_t *out;
    float *a;
    int ic, ih, iw, hw;
    int rows, sh, sw, ph, pw, kw;  // rows = Plan::fold_rows
    int hb, ow, span, words;       // packed row blocks and columns; words = 32-bit words per column
    int pitch;                     // staged row: words (few channels: of 32 columns' bits)
    int group;                     // channels staged at a time
    int row_blocks;                // blocks of sh rows that cover the image
    int nw;                        // words of a column per group of channels
    long img_stride, c_stride, px_stride;
    float inv_ic;
    int stage_off, table_off;      // bytes into dynamic shared memory
    int chunks;                    // few channels: words of bits that hold a row's columns
    FastDiv by_iw, by_nw, by_chunks;
};

// Eight bits to the low bits of eight nibbles.
__device__ __forceinline__ uint32_t spread(uint32_t b) {
    b = (b | (b << 12)) & 0x000F000Fu;
    b = (b | (b << 6)) & 0x03030303u;
    return (b | (b << 3)) & 0x11111111u;
}

// IC channels (0: up to seven, four at a time); TWO: a row of a filter is two words of a column,
// which are put together and stored as one.
template <bool WITH_A, int IC, bool TWO>
__global__ void __launch_bounds__(kThreads) fold_few_kernel(const FoldArgs g) {
    extern __shared__ __align__(16) uint8_t smem[];
    uint32_t *bits = reinterpret_cast<uint32_t *>(smem);  // [channel][row][pitch], 1 = negative

    const int n = blockIdx.x / g.row_blocks, hb = blockIdx.x - n * g.row_blocks;
    const int h0 = hb * g.sh - g.ph;  // input row of the block's first line
    const int lines = min(g.sh, g.ih - h0), first = h0 < 0 ? -h0 : 0;
    const bool packs = hb < g.hb;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    dependency_release();
    dependency_wait();

    // a task is 32 neighbouring columns (borders included) of a line
    const float *img = g.src + n * g.img_stride + (long)h0 * g.iw * g.px_stride;
    float *a = g.a + (long)n * g.hw + (long)h0 * g.iw;
    const int tasks = lines * g.chunks;
    for (int t0 = first * g.chunks + warp; t0 < tasks; t0 += kTasks * kThreads / 32) {
        float acc[kTasks] = {};
        int px[kTasks];  // pixel of this lane, or -1
#pragma unroll
        for (int k = 0; k < kTasks; k++) {
            const int t = t0 + k * kThreads / 32;
            const int line = (int)g.by_chunks((uint32_t)t);
            const int ix = 32 * (t - line * g.chunks) + lane - g.pw;
            px[k] = t < tasks && ix >= 0 && ix < g.iw ? line * g.iw + ix : -1;
        }
        constexpr int NC = IC > 0 ? IC : 4;
        const int ic = IC > 0 ? IC : g.ic;
        for (int c = 0; c < ic; c += NC) {
            float v[kTasks][NC];
#pragma unroll
            for (int k = 0; k < kTasks; k++) {
                const float *s = img + px[k] * (int)g.px_stride + c * g.c_stride;
#pragma unroll
                for (int i = 0; i < NC; i++)
                    v[k][i] = px[k] >= 0 && c + i < ic ? __ldg(s + i * g.c_stride) : 0.f;
            }
#pragma unroll
            for (int k = 0; k < kTasks; k++) {
                const int t = t0 + k * kThreads / 32;
                const int line = (int)g.by_chunks((uint32_t)t);
                const bool keep = packs && t < tasks && line < g.rows;  // the same in all lanes
                uint32_t *to = bits + (c * g.rows + line) * g.pitch + (t - line * g.chunks);
#pragma unroll
                for (int i = 0; i < NC; i++) {
                    if (c + i >= ic) break;
                    if (WITH_A) acc[k] = __fadd_rn(acc[k], __fmul_rn(fabsf(v[k][i]), g.inv_ic));
                    if (keep) {
                        const uint32_t b = __ballot_sync(0xffffffffu, __float_as_int(v[k][i]) < 0);
                        if (lane == 0) to[i * g.rows * g.pitch] = b;
                    }
                }
            }
        }
        if (WITH_A) {
#pragma unroll
            for (int k = 0; k < kTasks; k++)
                if (px[k] >= 0) a[px[k]] = acc[k];
        }
    }
    if (!packs) return;
    __syncthreads();

    // Item w of a column: a word, i.e. eight columns q of row i of channel c, or both of a row's two.
    // Threads are dealt whole columns' worth of items, so that a thread keeps its w.
    constexpr int SPAN = TWO ? 16 : 8;
    const int per = TWO ? 1 : (g.kw + 7) / 8;
    const int groups = g.nw < kThreads ? (int)g.by_nw(kThreads) : 1;
    const int group = g.nw < kThreads ? (int)g.by_nw(threadIdx.x) : 0;
    if (group >= groups) return;
    uint32_t *out = g.out + ((long)n * g.hb + hb) * g.ow * g.words;
    for (int w = threadIdx.x - group * g.nw; w < g.nw; w += kThreads) {
        const int f = w / per, q = w - f * per, i = f % g.rows;
        const bool row_in = h0 + i >= 0 && h0 + i < g.ih;
        const int left = row_in ? g.kw - 8 * q : 0;
        const uint32_t exist0 = first_nibbles(0xFFFFFFFFu, left);
        const uint32_t exist1 = TWO ? first_nibbles(0xFFFFFFFFu, left - 8) : 0u;
        const uint32_t *row = bits + f * g.pitch;
        for (int col = group; col < g.ow; col += groups) {
            const int x = col * g.sw + 8 * q;  // border columns in front included
            uint32_t b = 0, mask0 = exist0, mask1 = exist1;
            if (row_in) b = __funnelshift_r(row[x >> 5], row[(x >> 5) + 1], x & 31);
            if (x < g.pw || x + SPAN > g.pw + g.iw) {  // columns outside the image
                const int before = g.pw - x, inside = g.pw + g.iw - x;
                mask0 = first_nibbles(mask0, inside) & ~first_nibbles(0xFFFFFFFFu, before);
                if (TWO)
                    mask1 = first_nibbles(mask1, inside - 8) & ~first_nibbles(0xFFFFFFFFu, before - 8);
            }
            const uint32_t w0 = ((spread(b & 0xFFu) << 3) | 0x22222222u) & mask0;
            if (TWO) {
                const uint32_t w1 = ((spread((b >> 8) & 0xFFu) << 3) | 0x22222222u) & mask1;
                *reinterpret_cast<uint2 *>(out + col * g.words + 2 * w) = make_uint2(w0, w1);
            } else {
                out[col * g.words + w] = w0;
            }
        }
    }
}

template <bool WITH_A>
__global__ void __launch_bounds__(kThreads) fold_kernel(const FoldArgs g) {
    extern __shared__ __align__(16) uint8_t smem[];
    float *sums = reinterpret_cast<float *>(smem);
    uint32_t *words = reinterpret_cast<uint32_t *>(smem + g.stage_off);
    uint32_t *from = reinterpret_cast<uint32_t *>(smem + g.table_off);  // staged place of a word
    uint32_t *to = from + g.nw;  // its place in the column

    const int n = blockIdx.x / g.row_blocks, hb = blockIdx.x - n * g.row_blocks;
    const int h0 = hb * g.sh - g.ph;  // input row of the block's first line
    const int lines = min(g.sh, g.ih - h0), first = h0 < 0 ? -h0 : 0;
    const bool packs = hb < g.hb;
    const int n_px = lines > 0 ? lines * g.iw : 0;
    dependency_release();
    const float *img = g.src + n * g.img_stride + (long)h0 * g.iw * g.px_stride;

    if (packs) {
        for (int i = threadIdx.x; i < (g.table_off - g.stage_off) / 4; i += kThreads) words[i] = 0u;
        for (int w = threadIdx.x; w < g.nw; w += kThreads) {
            // channels 8 c8 ... of row i, column j
            const int n8 = (g.group + 7) / 8, t = w / n8, c8 = w - t * n8;
            const int i = t / g.kw, j = t - i * g.kw;
            from[w] = (uint32_t)((c8 * g.rows + i) * g.pitch + j);
            to[w] = (uint32_t)(t * ((g.ic + 7) / 8) + c8);
        }
    }
    __syncthreads();
    dependency_wait();
    for (int c0 = 0; c0 < g.ic; c0 += g.group) {
        const int nc = min(g.group, g.ic - c0);
        for (int p = first * g.iw + threadIdx.x; p < n_px; p += kThreads) {
            const int line = (int)g.by_iw((uint32_t)p), x = p - line * g.iw + g.pw;
            const bool keep = packs && line < g.rows && x < g.span;
            uint32_t *slot = words + line * g.pitch + x;
            const float *s = img + p * g.px_stride + c0 * g.c_stride;
            float acc = !WITH_A || c0 == 0 ? 0.f : sums[p];
            for (int c = 0; c < nc; c += 16) {
                float v[16];
#pragma unroll
                for (int i = 0; i < 16; i++)
                    v[i] = c + i < nc ? __ldg(s + (c + i) * g.c_stride) : 0.f;
                if (WITH_A) {
#pragma unroll
                    for (int i = 0; i < 16; i++)
                        if (c + i < nc) acc = __fadd_rn(acc, __fmul_rn(fabsf(v[i]), g.inv_ic));
                }
#pragma unroll
                for (int h = 0; h < 16; h += 8)
                    if (keep && c + h < nc)
                        slot[(c + h) / 8 * g.rows * g.pitch] = first_nibbles(
                            sign_nibbles(reinterpret_cast<const uint32_t *>(v) + h), nc - c - h);
            }
            if (WITH_A) {
                if (c0 + nc < g.ic) sums[p] = acc;
                else g.a[(long)n * g.hw + (long)h0 * g.iw + p] = acc;
            }
        }
        if (!packs) continue;
        __syncthreads();
        uint32_t *out = g.out + ((long)n * g.hb + hb) * g.ow * g.words + c0 / 8;
        // the last group of channels may be smaller than the table's
        const int c8_end = ((g.ic + 7) / 8) - c0 / 8;
        int col = (int)g.by_nw(threadIdx.x), w = threadIdx.x - col * g.nw;
        const int dcol = (int)g.by_nw(kThreads), dw = kThreads - dcol * g.nw;
        while (col < g.ow) {
            const uint32_t at = from[w], dst = to[w];
            if (g.group >= g.ic || (int)(dst % ((g.ic + 7) / 8)) < c8_end) {
                out[(long)col * g.words + dst] = words[at + (uint32_t)(col * g.sw)];
            }
            col += dcol;
            w += dw;
            if (w >= g.nw) { w -= g.nw; col++; }
        }
        __syncthreads();
    }
}

using FoldFn = void (*)(FoldArgs);
template <bool WITH_A, bool TWO>
FoldFn few_kernel_of(int ic) {
    switch (ic) {
        case 1: return fold_few_kernel<WITH_A, 1, TWO>;
        case 2: return fold_few_kernel<WITH_A, 2, TWO>;
        case 3: return fold_few_kernel<WITH_A, 3, TWO>;
        case 4: return fold_few_kernel<WITH_A, 4, TWO>;
        default: return fold_few_kernel<WITH_A, 0, TWO>;
    }
}
FoldFn few_kernel(bool with_a, bool two, int ic) {
    return with_a ? (two ? few_kernel_of<true, true>(ic) : few_kernel_of<true, false>(ic))
                  : (two ? few_kernel_of<false, true>(ic) : few_kernel_of<false, false>(ic));
}

}  // namespace

cudaError_t launch_fold(const Plan &p, const float *src, void *bin_src, float *a, cudaStream_t s) {
    FoldArgs g;
    g.src = src; g.out = (uint32_t *)bin_src; g.a = a;
    g.ic = p.ic; g.ih = p.ih; g.iw = p.iw; g.hw = p.ih * p.iw;
    g.rows = p.fold_rows; g.sh = p.sh; g.sw = p.sw; g.ph = p.ph; g.pw = p.pw; g.kw = p.kw;
    g.hb = p.hp; g.ow = p.ow; g.span = p.fold_span; g.words = p.icp / 4;
    const bool few = p.fold_field > 0;
    g.group = p.fold_channels;
    g.row_blocks = div_up_i(p.ih + p.ph, p.sh);
    if (g.row_blocks < g.hb) g.row_blocks = g.hb;
    g.img_stride = (long)p.ic * p.ih * p.iw;
    g.c_stride = p.src_nhwc ? 1 : (long)p.ih * p.iw;
    g.px_stride = p.src_nhwc ? p.ic : 1;
    g.inv_ic = p.inv_ic;
    g.by_iw = FastDiv((uint32_t)p.iw);
    g.chunks = div_up_i(p.iw + p.pw, 32);
    g.by_chunks = FastDiv((uint32_t)g.chunks);
    const bool two = few && p.fold_field == 16;
    g.pitch = few ? fold_bit_pitch(p) : p.fold_span;
    const int n8 = div_up_i(p.fold_channels, 8);
    g.nw = few ? p.ic * p.fold_rows * (two ? 1 : p.fold_field / 8) : p.fold_rows * p.kw * n8;
    g.by_nw = FastDiv((uint32_t)g.nw);
    g.stage_off = a && p.fold_channels < p.ic ? div_up_i(4 * p.sh * p.iw, 16) * 16 : 0;
    const int staged = 4 * (few ? p.ic : n8) * p.fold_rows * g.pitch;
    g.table_off = g.stage_off + div_up_i(staged, 16) * 16;
    const size_t smem = g.table_off + (few ? 0 : 8 * (size_t)g.nw);
    void (*kernel)(FoldArgs) = few ? few_kernel(a != nullptr, two, p.ic)
                               : a ? fold_kernel<true> : fold_kernel<false>;
    static std::atomic<bool> opted_in[64][2];
    int dev = 0;
    cudaGetDevice(&dev);
    std::atomic<bool> &done = opted_in[dev & 63][a ? 1 : 0];
    // few channels: the bits fit the 48 KB that need no opt-in (fold_ok)
    if (!few && !done.load(std::memory_order_acquire)) {
        const cudaError_t e =
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
        if (e != cudaSuccess) return e;
        done.store(true, std::memory_order_release);
    }
    note_launch();
    return launch_overlapped(kernel, dim3((unsigned)(p.mb * g.row_blocks)), dim3(kThreads), smem, s,
                             1, g);
}

}  // namespace xb200
