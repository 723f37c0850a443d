// Weight-side kernels: sign packing, alpha = mean |w| per output channel, and the per-pixel
// count of contributing operands, in one launch. A training step runs it once per pass.
//
// alpha is summed in upstream's (ic, kh, kw) order (src/bcast_binarize_weights.cpp:99-114) and
// therefore rounds identically: a serial chain of IC*KH*KW additions per filter, four cycles each,
// which is what bounds the launch (3456 additions: 7.3 us). So every filter gets a chain of its
// own (OIHW: one warp per filter; HWIO: one lane, because 32 neighbouring filters share a line),
// the loads of the next stretch are in flight while the current one is added up, and packing and
// counting run in other blocks of the same launch meanwhile.
#include "kernels.cuh"

namespace xb200 {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kStretch = 256;  // OIHW: elements a warp stages at a time
constexpr int kSlab = 64;      // HWIO: elements of 32 filters a block stages at a time

struct WArgs {
    const float *w;
    int oc, ic, kh, kw;
    float *alpha;
    float inv_chw;
    uint32_t *out;
    int rows;   // filters per tap in the packed matrix (padded with zero filters)
    int words;  // 32-bit words per packed row
    int nibbles;  // 1: [tap][row][word of 8 channels]; 0: bits, [tap][word of 32 channels][row]
    int fold_rows, fold_field;  // folded layers (plan.hpp): a tap is sh filter rows
    int taps;
    int cat_words;  // rows that hold all columns of a filter row (Plan::cat): words per column, or 0
    int32_t *op_c;
    int ih, iw, oh, ow, sh, sw, ph, pw;
    int alpha_blocks, pack_blocks;  // roles by block index: alpha, packing, then counting
};

template <bool HWIO>
__device__ __forceinline__ long w_index(const WArgs &g, int oc, int c, int tap) {
    return HWIO ? ((long)tap * g.ic + c) * g.oc + oc : ((long)oc * g.ic + c) * (g.kh * g.kw) + tap;
}

__device__ __forceinline__ unsigned sign_clear(float x) { return (~__float_as_uint(x)) >> 31; }

// alpha, OIHW: a warp walks its filter's contiguous run, lane 0 adds.
__device__ __forceinline__ void alpha_oihw(const WArgs &g, float (*stage)[kStretch]) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int oc = blockIdx.x * kWarps + warp;
    if (oc >= g.oc) return;
    const int n = g.ic * g.kh * g.kw;
    const float *p = g.w + (long)oc * n;
    float *t = stage[warp];
    float acc = 0.f, v[kStretch / 32];
#pragma unroll
    for (int i = 0; i < kStretch / 32; i++) {
        const int e = i * 32 + lane;
        v[i] = e < n ? __ldg(p + e) : 0.f;
    }
    for (int e0 = 0; e0 < n; e0 += kStretch) {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < kStretch / 32; i++) t[i * 32 + lane] = __fmul_rn(fabsf(v[i]), g.inv_chw);
        __syncwarp();
#pragma unroll
        for (int i = 0; i < kStretch / 32; i++) {
            const int e = e0 + kStretch + i * 32 + lane;
            v[i] = e < n ? __ldg(p + e) : 0.f;
        }
        if (lane == 0) {
            const int m = min(kStretch, n - e0);
            int e = 0;
            for (; e + 32 <= m; e += 32) {
                float4 q[8];
#pragma unroll
                for (int j = 0; j < 8; j++) q[j] = *reinterpret_cast<const float4 *>(t + e + 4 * j);
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    acc = __fadd_rn(acc, q[j].x);
                    acc = __fadd_rn(acc, q[j].y);
                    acc = __fadd_rn(acc, q[j].z);
                    acc = __fadd_rn(acc, q[j].w);
                }
            }
            for (; e < m; e++) acc = __fadd_rn(acc, t[e]);
        }
    }
    if (lane == 0) g.alpha[oc] = acc;
}

// alpha, HWIO: 32 neighbouring filters are one line of every (tap, channel); the block stages
// kSlab elements of them, warp 0 adds, one lane per filter.
__device__ __forceinline__ void alpha_hwio(const WArgs &g, float (*stage)[kSlab][32]) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int oc = blockIdx.x * 32 + lane;
    const int khw = g.kh * g.kw, n = g.ic * khw;
    float acc = 0.f, v[kSlab / kWarps];
    auto fetch = [&](int e0) {
#pragma unroll
        for (int i = 0; i < kSlab / kWarps; i++) {
            const int e = e0 + i * kWarps + warp;  // position in upstream's (ic, kh, kw) walk
            const int c = e / khw, tap = e - c * khw;
            v[i] = e < n && oc < g.oc ? __ldg(g.w + w_index<true>(g, oc, c, tap)) : 0.f;
        }
    };
    fetch(0);
    int b = 0;
    for (int e0 = 0; e0 < n; e0 += kSlab, b ^= 1) {
#pragma unroll
        for (int i = 0; i < kSlab / kWarps; i++)
            stage[b][i * kWarps + warp][lane] = __fmul_rn(fabsf(v[i]), g.inv_chw);
        __syncthreads();  // slab b is complete; the other one has been added up
        fetch(e0 + kSlab);
        if (warp == 0) {
            const int m = min(kSlab, n - e0);
            if (m == kSlab) {
#pragma unroll
                for (int e = 0; e < kSlab; e++) acc = __fadd_rn(acc, stage[b][e][lane]);
            } else {
                for (int e = 0; e < m; e++) acc = __fadd_rn(acc, stage[b][e][lane]);
            }
        }
    }
    if (warp == 0 && oc < g.oc) g.alpha[oc] = acc;
}

// One 32-bit word of the packed matrix per thread; channels and filters that do not exist are 0.
// OIHW: the items of a filter are neighbours, so that its run stays in the L1 while its taps are
// read with a stride; HWIO: neighbouring threads take neighbouring filters.
template <bool HWIO>
__device__ __forceinline__ void pack(const WArgs &g) {
    const int taps = g.taps, span = g.nibbles ? 8 : 32;
    const long total = (long)taps * g.rows * g.words;
    const long i = (long)(blockIdx.x - g.alpha_blocks) * kThreads + threadIdx.x;
    if (i >= total) return;
    int f, tap, word;
    if (HWIO) {
        f = (int)(i % g.rows);
        word = (int)(i / g.rows % g.words);
        tap = (int)(i / ((long)g.rows * g.words));
    } else {
        word = (int)(i % g.words);
        tap = (int)(i / g.words % taps);
        f = (int)(i / ((long)g.words * taps));
    }
    uint32_t v = 0;
    if (f < g.oc) {
        int c0 = word * span, from = tap;
        if (g.cat_words) {
            const int j = word / g.cat_words;
            c0 = j < g.kw ? c0 - j * g.cat_words * span : g.ic;  // past the last column nothing
            from = tap * g.kw + j;
        }
        if (g.fold_rows) {
            const int ic8 = (g.ic + 7) / 8 * 8;
            for (int b = 0; b < 8; b++) {
                int c, i, j;
                if (g.fold_field) {
                    j = (c0 + b) % g.fold_field;
                    i = (c0 + b) / g.fold_field % g.fold_rows;
                    c = (c0 + b) / (g.fold_field * g.fold_rows);
                } else {
                    c = (c0 + b) % ic8;
                    j = (c0 + b) / ic8 % g.kw;
                    i = (c0 + b) / (ic8 * g.kw);
                }
                const int kh = tap * g.sh + i;
                if (c < g.ic && i < g.fold_rows && j < g.kw && kh < g.kh)
                    v |= (sign_clear(__ldg(g.w + w_index<HWIO>(g, f, c, kh * g.kw + j))) ? 0x2u : 0xAu)
                         << (4 * b);
            }
        } else if (g.nibbles) {
            const int n = min(span, g.ic - c0);
#pragma unroll
            for (int b = 0; b < 8; b++)
                if (b < n)
                    v |= (sign_clear(__ldg(g.w + w_index<HWIO>(g, f, c0 + b, from))) ? 0x2u : 0xAu)
                         << (4 * b);
        } else {
            const int n = min(span, g.ic - c0);
            for (int b = 0; b < n; b++)
                v |= sign_clear(__ldg(g.w + w_index<HWIO>(g, f, c0 + b, tap))) << (31 - b);
        }
    }
    g.out[g.nibbles ? ((long)tap * g.rows + f) * g.words + word
                    : ((long)tap * g.words + word) * g.rows + f] = v;
}

__device__ __forceinline__ void count_operands(const WArgs &g) {
    const int o = (int)(blockIdx.x - g.alpha_blocks - g.pack_blocks) * kThreads + threadIdx.x;
    if (o >= g.oh * g.ow) return;
    const int y = o / g.ow, x = o - y * g.ow;
    int rows = 0, cols = 0;
    for (int i = 0; i < g.kh; i++) {
        const int h = y * g.sh - g.ph + i;
        rows += h >= 0 && h < g.ih;
    }
    for (int j = 0; j < g.kw; j++) {
        const int w = x * g.sw - g.pw + j;
        cols += w >= 0 && w < g.iw;
    }
    g.op_c[o] = rows * cols * g.ic;
}

template <bool HWIO>
__global__ void __launch_bounds__(kThreads) weights_kernel(const WArgs g) {
    __shared__ __align__(16) float stage[HWIO ? 2 * kSlab * 32 : kWarps * kStretch];
    if ((int)blockIdx.x < g.alpha_blocks) {
        if (HWIO) alpha_hwio(g, reinterpret_cast<float (*)[kSlab][32]>(stage));
        else alpha_oihw(g, reinterpret_cast<float (*)[kStretch]>(stage));
    } else if ((int)blockIdx.x < g.alpha_blocks + g.pack_blocks) {
        pack<HWIO>(g);
    } else {
        count_operands(g);
    }
}

}  // namespace

cudaError_t launch_binarize_weights(const Plan &p, const float *w, void *bin_w, float *alpha,
                                    int32_t *op_c, cudaStream_t s) {
    WArgs g;
    g.w = w; g.oc = p.oc; g.ic = p.ic; g.kh = p.kh; g.kw = p.kw;
    g.alpha = alpha; g.inv_chw = p.inv_chw;
    g.out = (uint32_t *)bin_w;
    g.nibbles = p.family == kTcgen05;
    g.rows = g.nibbles ? p.ocp16 : p.ocp;
    g.words = g.nibbles ? p.tap_pitch / 4 : p.icw;
    g.cat_words = p.cat ? p.icp / 4 : 0;
    g.fold_rows = p.fold ? p.fold_rows : 0;
    g.fold_field = p.fold_field;
    g.taps = p.fold ? p.fold_taps : p.cat ? p.kh : p.kh * p.kw;
    g.op_c = op_c;
    g.ih = p.ih; g.iw = p.iw; g.oh = p.oh; g.ow = p.ow;
    g.sh = p.sh; g.sw = p.sw; g.ph = p.ph; g.pw = p.pw;
    const int per_block = p.w_hwio ? 32 : kWarps;  // filters an alpha block sums
    g.alpha_blocks = (p.oc + per_block - 1) / per_block;
    g.pack_blocks = (int)(((long)g.taps * g.rows * g.words + kThreads - 1) / kThreads);
    const int count_blocks = (p.oh * p.ow + kThreads - 1) / kThreads;
    const unsigned grid = (unsigned)(g.alpha_blocks + g.pack_blocks + count_blocks);
    if (p.w_hwio) weights_kernel<true><<<grid, kThreads, 0, s>>>(g);
    else weights_kernel<false><<<grid, kThreads, 0, s>>>(g);
    note_launch();
    return cudaGetLastError();
}

// ---- float binarisation for the training backward pass ----------------------------------------
// to = sign(from) * mean(from) over the whole filter bank (upstream
// src/binarize_weights_float.cpp:3-25; the mean is of the signed values, as upstream has it).
// Upstream accumulates the sum in an OpenMP loop without a reduction clause, so its result depends
// on the thread schedule; here the sum has one fixed shape: thread t of block b adds elements
// b*256 + t, + 65536, + 131072, ... in ascending order, a block folds its 256 running sums with
// a fixed binary tree, and every block of the second kernel folds the 256 block sums with the
// same tree. The result is therefore reproducible and within rounding of the one-thread sum.
namespace {
constexpr int kWfBlocks = 256, kWfThreads = 256;

__device__ __forceinline__ float fold256(float v, float *sh) {
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int w = kWfThreads / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) sh[threadIdx.x] = __fadd_rn(sh[threadIdx.x], sh[threadIdx.x + w]);
        __syncthreads();
    }
    return sh[0];
}

__global__ void __launch_bounds__(kWfThreads) wf_partial_kernel(const float *from, long elems,
                                                                float *partial) {
    __shared__ float sh[kWfThreads];
    float acc = 0.f;
    for (long i = (long)blockIdx.x * kWfThreads + threadIdx.x; i < elems;
         i += (long)kWfBlocks * kWfThreads)
        acc = __fadd_rn(acc, from[i]);
    const float total = fold256(acc, sh);
    if (threadIdx.x == 0) partial[blockIdx.x] = total;
}

// Elements begin .. elems.
__global__ void __launch_bounds__(kWfThreads) wf_scale_kernel(const float *from, float *to, long begin,
                                                              long elems, const float *partial,
                                                              float inv_elems) {
    __shared__ float sh[kWfThreads];
    const float mean = __fmul_rn(fold256(partial[threadIdx.x], sh), inv_elems);
    for (long i = begin + (long)blockIdx.x * kWfThreads + threadIdx.x; i < elems;
         i += (long)gridDim.x * kWfThreads)
        to[i] = __fmul_rn(from[i] >= .0f ? 1.f : -1.f, mean);
}
}  // namespace

// The block sums need 1 KB of scratch. The result itself serves, where it has that much and is not also
// the source: its first 256 elements hold the sums until everything behind them is written, then a block
// that has read them overwrites them. Stream-ordered scratch, which the other cases take, costs the host
// 20 us a call (a training step of one layer 258 -> 238 us), and where the stream is waited for between
// calls, so that its memory goes back each time, 500 and more.
cudaError_t launch_binarize_weights_float(long elems, const float *from, float *to,
                                          cudaStream_t s) {
    const bool in_result = elems >= 2 * kWfBlocks && (to + elems <= from || from + elems <= to);
    float *partial = to;
    if (!in_result) {
        const cudaError_t e = cudaMallocAsync(&partial, kWfBlocks * sizeof(float), s);
        if (e != cudaSuccess) return e;
    }
    wf_partial_kernel<<<kWfBlocks, kWfThreads, 0, s>>>(from, elems, partial);
    note_launch();
    const long begin = in_result ? kWfBlocks : 0;
    const float inv = 1.f / (float)elems;
    long blocks = (elems - begin + kWfThreads - 1) / kWfThreads;
    if (blocks > 1184) blocks = 1184;
    if (blocks < 1) blocks = 1;
    wf_scale_kernel<<<(unsigned)blocks, kWfThreads, 0, s>>>(from, to, begin, elems, partial, inv);
    note_launch();
    if (in_result) {
        static_assert(kWfBlocks == kWfThreads, "one block reads all sums before it writes");
        wf_scale_kernel<<<1, kWfThreads, 0, s>>>(from, to, 0, begin, partial, inv);
        note_launch();
    }
    const cudaError_t e = cudaGetLastError();
    const cudaError_t f = in_result ? cudaSuccess : cudaFreeAsync(partial, s);
    return e != cudaSuccess ? e : f;
}

}  // namespace xb200
