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
// FEW (fewer than eight channels): the eight nibbles of a word are neighbouring columns. A value
// is staged as a byte; a word is three aligned 32-bit loads, two funnel shifts and five
// instructions that squeeze eight bytes into eight nibbles. Otherwise they are neighbouring
// channels of a pixel, put together once per pixel and copied. (The first version fetched every
// nibble of every word on its own: 55 us for AlexNet conv1 on 64 images, which is 40 MB in and
// 20 MB out.)
#include "kernels.cuh"

#include <atomic>

namespace xb200 {

namespace {

constexpr int kThreads = 256;
constexpr int kPixels = 4;  // FEW: pixels x channels loaded before the first is used

struct FoldArgs {
    const float *src;
    uint32_t *out;
    float *a;
    int ic, ih, iw, hw;
    int rows, sh, sw, ph, pw, kw;  // rows = Plan::fold_rows
    int hb, ow, span, words;       // packed row blocks and columns; words = 32-bit words per column
    int pitch;                     // staged row: bytes (FEW) or words
    int group;                     // channels staged at a time
    int row_blocks;                // blocks of sh rows that cover the image
    int nw;                        // words of a column per group of channels
    long img_stride, c_stride, px_stride;
    float inv_ic;
    int stage_off, table_off;      // bytes into dynamic shared memory
    FastDiv by_iw, by_nw;
};

template <bool WITH_A, bool FEW>
__global__ void __launch_bounds__(kThreads) fold_kernel(const FoldArgs g) {
    extern __shared__ __align__(16) uint8_t smem[];
    float *sums = reinterpret_cast<float *>(smem);
    uint8_t *stage = smem + g.stage_off;
    uint32_t *words = reinterpret_cast<uint32_t *>(stage);
    uint32_t *from = reinterpret_cast<uint32_t *>(smem + g.table_off);  // staged place of a word
    uint32_t *to = from + g.nw;  // FEW: nibbles of it that exist; else its place in the column

    const int n = blockIdx.x / g.row_blocks, hb = blockIdx.x - n * g.row_blocks;
    const int h0 = hb * g.sh - g.ph;  // input row of the block's first line
    const int lines = min(g.sh, g.ih - h0), first = h0 < 0 ? -h0 : 0;
    const bool packs = hb < g.hb;
    const int n_px = lines > 0 ? lines * g.iw : 0;
    const float *img = g.src + n * g.img_stride + (long)h0 * g.iw * g.px_stride;

    if (packs) {
        for (int i = threadIdx.x; i < (g.table_off - g.stage_off) / 4; i += kThreads) words[i] = 0u;
        for (int w = threadIdx.x; w < g.nw; w += kThreads) {
            if (FEW) {  // word q of the columns of row i of channel c
                const int per = (g.kw + 7) / 8, f = w / per, q = w - f * per;
                from[w] = (uint32_t)(f * g.pitch + 8 * q);
                to[w] = (uint32_t)(g.kw - 8 * q);
            } else {    // channels 8 c8 ... of row i, column j
                const int n8 = (g.group + 7) / 8, t = w / n8, c8 = w - t * n8;
                const int i = t / g.kw, j = t - i * g.kw;
                from[w] = (uint32_t)((c8 * g.rows + i) * g.pitch + j);
                to[w] = (uint32_t)(t * ((g.ic + 7) / 8) + c8);
            }
        }
    }
    __syncthreads();
    for (int c0 = 0; c0 < g.ic; c0 += g.group) {
        if (FEW) {
            for (int p0 = first * g.iw + threadIdx.x; p0 < n_px; p0 += kPixels * kThreads) {
                float acc[kPixels] = {};
                for (int c = 0; c < g.ic; c += 4) {
                    float v[kPixels][4];
#pragma unroll
                    for (int k = 0; k < kPixels; k++)
#pragma unroll
                        for (int i = 0; i < 4; i++)
                            if (c + i < g.ic && p0 + k * kThreads < n_px)
                                v[k][i] = __ldg(img + (p0 + k * kThreads) * g.px_stride +
                                                (c + i) * g.c_stride);
#pragma unroll
                    for (int k = 0; k < kPixels; k++) {
                        const int p = p0 + k * kThreads;
                        if (p >= n_px) break;
                        const int line = (int)g.by_iw((uint32_t)p), x = p - line * g.iw + g.pw;
                        const bool keep = packs && line < g.rows && x < g.span;
#pragma unroll
                        for (int i = 0; i < 4; i++)
                            if (c + i < g.ic) {
                                if (WITH_A)
                                    acc[k] = __fadd_rn(acc[k], __fmul_rn(fabsf(v[k][i]), g.inv_ic));
                                if (keep)
                                    stage[((c + i) * g.rows + line) * g.pitch + x] =
                                        (uint8_t)(0x2u | ((__float_as_uint(v[k][i]) >> 28) & 0x8u));
                            }
                    }
                }
                if (WITH_A) {
#pragma unroll
                    for (int k = 0; k < kPixels; k++)
                        if (p0 + k * kThreads < n_px)
                            g.a[(long)n * g.hw + (long)h0 * g.iw + p0 + k * kThreads] = acc[k];
                }
            }
        } else {
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
            if (FEW) {
                const uint32_t byte = at + (uint32_t)(col * g.sw);
                const uint32_t *s = words + (byte >> 2);
                const uint32_t w0 = s[0], w1 = s[1], w2 = s[2];
                uint32_t lo = __funnelshift_r(w0, w1, 8 * (byte & 3));
                uint32_t hi = __funnelshift_r(w1, w2, 8 * (byte & 3));
                lo |= lo >> 4;
                hi |= hi >> 4;
                out[(long)col * g.words + w] = first_nibbles(prmt(lo, hi, 0x6420u), (int)dst);
            } else if (g.group >= g.ic || (int)(dst % ((g.ic + 7) / 8)) < c8_end) {
                out[(long)col * g.words + dst] = words[at + (uint32_t)(col * g.sw)];
            }
            col += dcol;
            w += dw;
            if (w >= g.nw) { w -= g.nw; col++; }
        }
        __syncthreads();
    }
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
    // FEW: a word may be read up to twelve bytes past a row's last value
    g.pitch = few ? div_up_i(p.fold_span + 12, 4) * 4 : p.fold_span;
    const int n8 = div_up_i(p.fold_channels, 8);
    g.nw = few ? p.ic * p.fold_rows * (p.fold_field / 8) : p.fold_rows * p.kw * n8;
    g.by_nw = FastDiv((uint32_t)g.nw);
    g.stage_off = a && p.fold_channels < p.ic ? div_up_i(4 * p.sh * p.iw, 16) * 16 : 0;
    const int staged = few ? p.ic * p.fold_rows * g.pitch : 4 * n8 * p.fold_rows * g.pitch;
    g.table_off = g.stage_off + div_up_i(staged, 16) * 16;
    const size_t smem = g.table_off + 8 * (size_t)g.nw;
    auto kernel = few ? (a ? fold_kernel<true, true> : fold_kernel<false, true>)
                      : (a ? fold_kernel<true, false> : fold_kernel<false, false>);
    static std::atomic<bool> opted_in[64][4];
    int dev = 0;
    cudaGetDevice(&dev);
    std::atomic<bool> &done = opted_in[dev & 63][(a ? 1 : 0) + (few ? 2 : 0)];
    if (!done.load(std::memory_order_acquire)) {
        const cudaError_t e =
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
        if (e != cudaSuccess) return e;
        done.store(true, std::memory_order_release);
    }
    kernel<<<(unsigned)(p.mb * g.row_blocks), kThreads, smem, s>>>(g);
    note_launch();
    return cudaGetLastError();
}

}  // namespace xb200
