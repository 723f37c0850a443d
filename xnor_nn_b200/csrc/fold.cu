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
// columns. Bound by instruction issue, then by the loads in flight. A warp reads 32 neighbouring columns of
// eight lines or column groups at once; a lane's eight signs are one word of nibbles, and a transposition
// among eight lanes (three exchanges) makes it the word of eight neighbouring columns, zero where there is
// no image. The second half then only shifts and masks pairs of words. AlexNet conv1 on 64 images (40 MB
// in, 20 MB out), launched alone: 26.7 us and 21.3 M warp instructions with a vote per 32 signs, bits
// spread to nibbles for every column that reads them; 20.8 us and 11.2 M now (a pass among others 55.0 ->
// 50.6). Before that: 37-39 us with a byte staged per value and a table lookup per word, 55 with every nibble
// fetched on its own.
// Otherwise (fold_kernel) they are neighbouring channels of a pixel, put together once per pixel
// and copied.
#include "kernels.cuh"

#include <atomic>

namespace xb200 {

namespace {

constexpr int kThreads = 256;
constexpr int kTasks = 8;   // few channels: warp loads per channel before the first is used

struct FoldArgs {
    const float *src;
    uint32_t *out;
    float *a;
    int ic, ih, iw, hw;
    int rows, sh, sw, ph, pw, kw;  // rows = Plan::fold_rows
    int hb, ow, span, words;       // packed row blocks and columns; words = 32-bit words per column
    int pitch;                     // staged row: words (few channels: of eight columns)
    int group;                     // channels staged at a time
    int row_blocks;                // blocks of sh rows that cover the image
    int nw;                        // words of a column per group of channels
    long img_stride, c_stride, px_stride;
    float inv_ic;
    int stage_off, table_off;      // bytes into dynamic shared memory
    int chunks;                    // few channels: 32 columns each, of a row
    FastDiv by_iw, by_nw, by_chunks;
};

// Eight lanes (numbered by `sub`) hold a word of eight nibbles each: nibble i of lane j becomes nibble j
// of lane i. Three exchanges: halves, bytes, nibbles.
struct NibbleTranspose {
    uint32_t halves, bytes, keep;
    int turn;
    __device__ __forceinline__ explicit NibbleTranspose(int sub)
        : halves(sub & 4 ? 0x3276u : 0x5410u), bytes(sub & 2 ? 0x3715u : 0x6240u),
          keep(sub & 1 ? 0xF0F0F0F0u : 0x0F0F0F0Fu), turn(sub & 1 ? 28 : 4) {}
    __device__ __forceinline__ uint32_t operator()(uint32_t w) const {
        w = prmt(w, __shfl_xor_sync(0xffffffffu, w, 4), halves);
        w = prmt(w, __shfl_xor_sync(0xffffffffu, w, 2), bytes);
        const uint32_t other = __shfl_xor_sync(0xffffffffu, w, 1);
        return (w & keep) | (__funnelshift_l(other, other, turn) & ~keep);
    }
};

// IC channels (0: up to seven, four at a time); TWO: a row of a filter is two words of a column,
// which are put together and stored as one.
template <bool WITH_A, int IC, bool TWO, int THREADS>
__global__ void __launch_bounds__(THREADS) fold_few_kernel(const FoldArgs g) {
    extern __shared__ __align__(16) uint8_t smem[];
    uint32_t *nibbles = reinterpret_cast<uint32_t *>(smem);  // [channel][row][pitch], eight columns a word
    constexpr int kWarps = THREADS / 32;

    const int n = blockIdx.x / g.row_blocks, hb = blockIdx.x - n * g.row_blocks;
    const int h0 = hb * g.sh - g.ph;  // input row of the block's first line
    const int lines = min(g.sh, g.ih - h0), first = h0 < 0 ? -h0 : 0;
    const bool packs = hb < g.hb;
    // warp-uniform, and known to be: what depends on a task alone is computed once per warp
    const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    dependency_release();
    // rows outside the image and what a column reaches past it are zeros
    if (packs)
        for (int i = threadIdx.x; i < g.ic * g.rows * g.pitch; i += THREADS) nibbles[i] = 0u;
    __syncthreads();
    dependency_wait();

    // A task is 32 neighbouring columns (borders included) of a line; a warp has eight in flight. Their
    // signs of a channel are a lane's eight nibbles, which transposed among eight lanes are the words of
    // eight columns that are wanted: lane l gets columns 8 (l / 8) ... of task l % 8.
    const float *img = g.src + n * g.img_stride + (long)h0 * g.iw * g.px_stride;
    float *a = g.a + (long)n * g.hw + (long)h0 * g.iw;
    const int tasks = lines * g.chunks;
    const NibbleTranspose transpose(lane & 7);
    for (int t0 = first * g.chunks + warp; t0 < tasks; t0 += kTasks * kWarps) {
        float acc[kTasks] = {};
        unsigned px[kTasks];  // pixel of this lane, from the line h0 on
        uint32_t exist = 0;   // nibble k: the lane's column of task k is in the image
#pragma unroll
        for (int k = 0; k < kTasks; k++) {
            const int t = t0 + k * kWarps;
            const int line = (int)g.by_chunks((uint32_t)t);
            const int ix = 32 * (t - line * g.chunks) + lane - g.pw;
            px[k] = (unsigned)(line * g.iw + ix);
            if (t < tasks && (unsigned)ix < (unsigned)g.iw) exist |= 0xFu << (4 * k);
        }
        // the task whose words this lane stores
        const int mine = t0 + (lane & 7) * kWarps, my_line = (int)g.by_chunks((uint32_t)mine);
        const bool keep = packs && mine < tasks && my_line < g.rows;
        uint32_t *to = nibbles + my_line * g.pitch + 4 * (mine - my_line * g.chunks) + (lane >> 3);
        constexpr int NC = IC > 0 ? IC : 4;
        const int ic = IC > 0 ? IC : g.ic;
        for (int c = 0; c < ic; c += NC) {
            float v[NC][kTasks];
#pragma unroll
            for (int i = 0; i < NC; i++) {
                // a warp-uniform channel plane and a lane's 32-bit offset into the row block
                const char *plane = reinterpret_cast<const char *>(img + (c + i) * g.c_stride);
                const unsigned size = 4u * (unsigned)g.px_stride;
#pragma unroll
                for (int k = 0; k < kTasks; k++)
                    v[i][k] = (exist >> (4 * k) & 1u) && c + i < ic
                                  ? __ldg(reinterpret_cast<const float *>(plane + px[k] * size))
                                  : 0.f;
            }
#pragma unroll
            for (int i = 0; i < NC; i++) {
                if (c + i >= ic) break;
                const uint32_t w =
                    transpose(sign_nibbles(reinterpret_cast<const uint32_t *>(v[i])) & exist);
                if (keep) to[(c + i) * g.rows * g.pitch] = w;
                if (WITH_A) {
#pragma unroll
                    for (int k = 0; k < kTasks; k++)
                        acc[k] = __fadd_rn(acc[k], __fmul_rn(fabsf(v[i][k]), g.inv_ic));
                }
            }
        }
        if (WITH_A) {
#pragma unroll
            for (int k = 0; k < kTasks; k++)
                if (exist >> (4 * k) & 1u) a[px[k]] = acc[k];
        }
    }
    if (!packs) return;
    __syncthreads();

    // Item w of a column: a word, i.e. eight columns q of row i of channel c, or both of a row's two.
    // Threads are dealt whole columns' worth of items, so that a thread keeps its w.
    const int per = TWO ? 1 : (g.kw + 7) / 8;
    const int groups = g.nw < THREADS ? (int)g.by_nw(THREADS) : 1;
    const int group = g.nw < THREADS ? (int)g.by_nw(threadIdx.x) : 0;
    if (group >= groups) return;
    uint32_t *out = g.out + ((long)n * g.hb + hb) * g.ow * g.words;
    for (int w = threadIdx.x - group * g.nw; w < g.nw; w += THREADS) {
        const int f = w / per, q = w - f * per;
        const uint32_t mask0 = first_nibbles(0xFFFFFFFFu, g.kw - 8 * q);
        const uint32_t mask1 = TWO ? first_nibbles(0xFFFFFFFFu, g.kw - 8) : 0u;
        const uint32_t *row = nibbles + f * g.pitch;
        uint32_t *o = out + group * g.words + (TWO ? 2 * w : w);
        int x = group * g.sw + 8 * q;  // border columns in front included
        for (int col = group; col < g.ow; col += groups, x += groups * g.sw, o += groups * g.words) {
            const uint32_t *at = row + (x >> 3);
            const uint32_t b0 = at[0], b1 = at[1];
            const uint32_t w0 = __funnelshift_r(b0, b1, 4 * (x & 7)) & mask0;
            if (TWO) {
                const uint32_t w1 = __funnelshift_r(b1, at[2], 4 * (x & 7)) & mask1;
                *reinterpret_cast<uint2 *>(o) = make_uint2(w0, w1);
            } else {
                *o = w0;
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
template <bool WITH_A, bool TWO, int THREADS>
FoldFn few_kernel_of(int ic) {
    switch (ic) {
        case 1: return fold_few_kernel<WITH_A, 1, TWO, THREADS>;
        case 2: return fold_few_kernel<WITH_A, 2, TWO, THREADS>;
        case 3: return fold_few_kernel<WITH_A, 3, TWO, THREADS>;
        case 4: return fold_few_kernel<WITH_A, 4, TWO, THREADS>;
        default: return fold_few_kernel<WITH_A, 0, TWO, THREADS>;
    }
}
template <int THREADS>
FoldFn few_kernel(bool with_a, bool two, int ic) {
    return with_a ? (two ? few_kernel_of<true, true, THREADS>(ic) : few_kernel_of<true, false, THREADS>(ic))
                  : (two ? few_kernel_of<false, true, THREADS>(ic) : few_kernel_of<false, false, THREADS>(ic));
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
    g.pitch = few ? 4 * fold_bit_pitch(p) : p.fold_span;
    const int n8 = div_up_i(p.fold_channels, 8);
    g.nw = few ? p.ic * p.fold_rows * (two ? 1 : p.fold_field / 8) : p.fold_rows * p.kw * n8;
    g.by_nw = FastDiv((uint32_t)g.nw);
    g.stage_off = a && p.fold_channels < p.ic ? div_up_i(4 * p.sh * p.iw, 16) * 16 : 0;
    const int staged = 4 * (few ? p.ic : n8) * p.fold_rows * g.pitch;
    g.table_off = g.stage_off + div_up_i(staged, 16) * 16;
    const size_t smem = g.table_off + (few ? 0 : 8 * (size_t)g.nw);
    const long blocks = (long)p.mb * g.row_blocks;
    // Blocks of 256 threads where those of 128 would leave SMs with room for more of them (eight fit, four with
    // five to seven channels) and each has more loads than a round or two. Packer alone, 128 -> 256 threads,
    // us: 2048 columns of 3 channels, 406 blocks of 780 loads 27.6 -> 16.1, 805 of 390 18.4 -> 14.3; 1024
    // columns, 812 blocks of 396 17.1 -> 13.1; 7 channels, 348 blocks of 924 28.2 -> 16.9. Slower: two images of
    // 2048 columns, 116 blocks of 780, 9.4 -> 11.2 (one image 8.5 -> 6.3, four 18.3 -> 12.0).
    const bool wide = few && blocks < (p.ic < 5 ? 8 : 4) * sm_count() && p.ic * p.sh * g.chunks > 320;
    const FoldFn kernel = wide   ? few_kernel<256>(a != nullptr, two, p.ic)
                          : few  ? few_kernel<128>(a != nullptr, two, p.ic)
                          : a    ? fold_kernel<true>
                                 : fold_kernel<false>;
    // per device and kernel, once; few channels: fold_ok counts a bit a value, four of which take 192 KB at
    // most
    static std::atomic<bool> opted_in[64][2][2][2][6];
    int dev = 0;
    cudaGetDevice(&dev);
    std::atomic<bool> &done = opted_in[dev & 63][wide ? 1 : 0][a ? 1 : 0][two ? 1 : 0][few ? (p.ic < 5 ? p.ic : 0) : 5];
    if (smem > 48 * 1024 && !done.load(std::memory_order_acquire)) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (few ? 200 : 160) * 1024);
        if (e != cudaSuccess) return e;
        done.store(true, std::memory_order_release);
    }
    note_launch();
    return launch_overlapped(kernel, dim3((unsigned)blocks), dim3(few && !wide ? 128 : kThreads), smem, s, 1, g);
}

}  // namespace xb200
