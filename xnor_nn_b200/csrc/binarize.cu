// Activation-side kernels: sign packing with the fused mean-|x| map, and the K box filter.
//
// All three are bound by HBM bandwidth: the fp32 source (4 B per element) is read exactly once
// and 1/32 (bits) or 1/8 (4-bit values) of that is written. One thread owns one pixel and walks its
// channels in ascending order, so the mean-|x| sum is accumulated in the very order upstream
// uses (src/bcast_calculate_k.cpp:55-65) and rounds identically; with an NCHW source the 32
// lanes of a warp read 32 neighbouring pixels of one channel plane, a full 128-byte line.
#include "kernels.cuh"

#include <atomic>

namespace xb200 {

namespace {
// Source floats are read exactly once: keep them out of the L1 so that the loads in flight are
// not limited by its size (conv4 step 61.0 -> 57.0 us together with the carve-out below).
__device__ __forceinline__ float ld_stream(const float *p) {
    float v;
    asm("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}


enum OutKind { kBitsDense = 0, kNibblesFramed = 2 };

struct BinArgs {
    const float *src;
    void *out;
    float *a;
    long n_px;        // mb*ih*iw
    int ic, hw, iw;   // hw = ih*iw
    long img_stride;  // elements between images in src
    long c_stride;    // elements between channels of one pixel
    long px_stride;   // elements between pixels of one image
    float inv_ic;
    int words;        // 32-bit words per packed row (icw, or icp/4 for nibbles)
    int wp, hp, lead, ih;
};

__device__ __forceinline__ unsigned sign_clear(float x) { return (~__float_as_uint(x)) >> 31; }

// Row of the packed matrix that pixel (n, h, w) owns.
template <int KIND>
__device__ __forceinline__ long packed_row(const BinArgs &g, long px) {
    if (KIND == kBitsDense) return px;
    const int n = (int)(px / g.hw);
    const int r = (int)(px - (long)n * g.hw);
    const int h = r / g.iw, w = r - h * g.iw;
    return g.lead + ((long)n * g.hp + h) * g.wp + w;
}

template <int KIND, bool WITH_A, bool WITH_PACK>
__global__ void __launch_bounds__(128) binarize_kernel(const BinArgs g) {
    const long px = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (px >= g.n_px) return;
    const int n = (int)(px / g.hw);
    const int r = (int)(px - (long)n * g.hw);
    const float *p = g.src + n * g.img_stride + r * g.px_stride;
    uint32_t *row = WITH_PACK ? (uint32_t *)g.out + packed_row<KIND>(g, px) * g.words : nullptr;

    float acc = 0.f;
    const int full = g.ic & ~31;
    int c = 0;
    for (; c < full; c += 32) {
        float v[32];
#pragma unroll
        for (int i = 0; i < 32; i++) v[i] = __ldg(p + (long)(c + i) * g.c_stride);
        if (WITH_A) {
#pragma unroll
            for (int i = 0; i < 32; i++) acc = __fadd_rn(acc, __fmul_rn(fabsf(v[i]), g.inv_ic));
        }
        if (WITH_PACK) {
            if (KIND == kNibblesFramed) {
#pragma unroll
                for (int j = 0; j < 4; j++)
                    row[c / 8 + j] = sign_nibbles(reinterpret_cast<const uint32_t *>(v) + 8 * j);
            } else {
                uint32_t w = 0;
#pragma unroll
                for (int i = 0; i < 32; i++) w = (w << 1) | sign_clear(v[i]);
                row[c / 32] = w;
            }
        }
    }
    if (c < g.ic) {  // channel tail: absent channels pack as zero
        uint32_t wbits = 0;
        uint32_t wnib[4] = {0, 0, 0, 0};
        for (int i = 0; i < 32; i++) {
            unsigned bit = 0;
            if (c + i < g.ic) {
                const float x = __ldg(p + (long)(c + i) * g.c_stride);
                if (WITH_A) acc = __fadd_rn(acc, __fmul_rn(fabsf(x), g.inv_ic));
                bit = sign_clear(x);
                wnib[i / 8] |= (bit ? 0x2u : 0xAu) << (4 * (i % 8));
            }
            wbits = (wbits << 1) | bit;
        }
        if (WITH_PACK) {
            if (KIND == kNibblesFramed) {
#pragma unroll
                for (int j = 0; j < 4; j++) row[c / 8 + j] = wnib[j];
            } else {
                row[c / 32] = wbits;
            }
        }
    }
    if (WITH_A) g.a[px] = acc;
}

// ---- +-1 nibbles on the frame: the layout the tensor-core convolution reads -------------------
//
// A block of four warps owns 32 neighbouring pixels and walks the channels in chunks of TCC. All
// warps load, one chunk ahead, so that a chunk's loads are in flight while the previous one is
// consumed. |x|/IC goes to a float tile and the sign nibbles to a second tile in shared memory,
// both pixel-major. Warp 0 then adds the float tile up channel by channel, one lane per pixel,
// which keeps upstream's summation order, while the other warps copy the nibbles out, 8 bytes per
// lane. Five blocks are resident per SM (nine of the 96-channel kind): the shared-memory
// carve-out is sized for that, see launch_bin().
//
// NCHW: lane = pixel, warp w takes the w-th quarter of a chunk's channels, so a load instruction
// reads one 128-byte line of a channel plane. NHWC: a pixel's channels are contiguous, TCC / 4
// lanes read them with 16-byte loads and a warp's loads cover whole pixels; one thread per pixel
// instead, which the first version had, reads with a stride of IC floats and took 42 us for
// AlexNet conv4 on 64 images.
//
// The kernel is as much bound by instruction issue as by memory. Hence: the sign nibbles of eight
// floats come from six byte permutes and two logic operations; both tiles are written and read
// with wide shared-memory accesses, their rows padded so that these stay (nearly) free of bank
// conflicts; pixel coordinates are 32-bit (the host sends anything larger to the generic kernel).
//
// TCC = 4 TPER channels per chunk: 128; 96 for channel counts that are a multiple of 96 but not
// of 128 (AlexNet conv2), where a 128-channel chunk would leave a quarter of the threads without
// work; 64 and 32 for layers that have no more channels than that.
// Bytes past the last channel of a packed row are zero from allocation, and only zeros are
// ever written there.
constexpr int TPX = 32;    // pixels per block
constexpr int TWARPS = 4;

// Element i of a column of floats whose rows are `pitch` bytes apart. The plain expression on
// 64-bit element offsets compiled to seven integer instructions per load; 32-bit byte offsets to
// about five; WIDE states the address as the one 32 x 32 + 64-bit multiply-add it is. Measured
// on the pass with the mean-|x| map: 128-channel chunks 16.7-17.0 -> 15.5 us on conv4 (whole step
// 50.6 -> 49.5 us), 21.7 -> 21.2 on the VGG layer; 96-channel chunks 9.3 -> 9.6 us on conv2, so
// that kernel keeps the plain form.
template <bool WIDE>
__device__ __forceinline__ const float *row_ptr(const float *p, unsigned i, unsigned pitch) {
    if (WIDE) {
        unsigned long long d;
        asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(d) : "r"(i), "r"(pitch), "l"(p));
        return reinterpret_cast<const float *>(d);
    }
    return reinterpret_cast<const float *>(reinterpret_cast<const char *>(p) + (size_t)(i * pitch));
}

__device__ __forceinline__ float4 ld_stream4(const float *p) {
    float4 v;
    asm("ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];"
        : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
        : "l"(p));
    return v;
}

template <bool WITH_A, bool WITH_PACK, bool NHWC, int TPER>
__global__ void __launch_bounds__(TWARPS * 32) binarize_nibbles_kernel(const BinArgs g) {
    constexpr int TCC = TPER * TWARPS;  // channels per chunk
    constexpr int FLD = TCC + 4;        // floats per pixel of the float tile
    constexpr int TLD = TCC / 2 + (TPER == 32 ? 16 : 8);  // bytes per pixel of the nibble tile
    constexpr int LPP = TCC / 4;        // NHWC: lanes per pixel,
    constexpr int PPI = 32 / LPP;       // pixels per load instruction of a warp,
    constexpr int LOADS = TPX / TWARPS / PPI;  // and 16-byte loads per thread and chunk
    static_assert(!NHWC || 4 * LOADS == TPER, "a thread stages as many floats either way");
    __shared__ __align__(16) float f_s[WITH_A ? TPX * FLD : 4];
    __shared__ __align__(16) uint8_t b_s[WITH_PACK ? TPX * TLD : 8];
    __shared__ long row_s[TPX];  // a pixel's packed row, as an offset in units of 8 bytes

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // The dependent grid (the convolution) may be launched once every block of this grid has
    // got this far, i.e. when none is waiting for an SM any more; its CTAs then move in as SMs
    // drain and set themselves up under this grid's tail (conv4 step 56.6 -> 55.5 us against
    // triggering at the end of the block). They wait for this grid's results themselves.
    dependency_release();
    dependency_wait();  // nothing of an earlier kernel is read or overwritten before this
    const unsigned px = blockIdx.x * TPX + lane;
    const bool live = px < (unsigned)g.n_px;
    const int n_live = (int)min((unsigned)TPX, (unsigned)g.n_px - blockIdx.x * TPX);  // pixels of this block
    const unsigned n = live ? px / (unsigned)g.hw : 0u;
    const unsigned r = live ? px - n * (unsigned)g.hw : 0u;
    if (warp == 0) {
        const unsigned h = r / (unsigned)g.iw, w = r - h * (unsigned)g.iw;
        const long row = g.lead + ((long)n * g.hp + h) * g.wp + w;
        row_s[lane] = live ? row * (g.words >> 1) : -1;
    }

    const int c_end = g.ic;
    float acc = 0.f;
    float v[TPER];
    // NCHW: warp w owns the TPER consecutive channels [TPER w, TPER (w + 1)) of every chunk.
    // NHWC: load j of this thread is four channels of pixel p0 + j * PPI.
    const int cw = NHWC ? 4 * (lane % LPP) : TPER * warp;
    const int p0 = NHWC ? warp * (TPX / TWARPS) + lane / LPP : 0;
    const float *pw = NHWC ? g.src + (long)(blockIdx.x * TPX + p0) * g.ic + cw
                           : g.src + (long)n * g.img_stride + r + (long)cw * g.hw;
    const unsigned pitch = (unsigned)g.hw * 4u;  // bytes between channels; the host checks the range
    const bool vec = NHWC && (g.ic & 3) == 0 && (reinterpret_cast<uintptr_t>(g.src) & 15) == 0;
    auto fetch = [&](int c0) {
        if (NHWC) {
            const float *p = pw + c0;
#pragma unroll
            for (int j = 0; j < LOADS; j++, p += (long)PPI * g.ic) {
                const bool in = p0 + j * PPI < n_live;
                if (vec) {
                    const float4 t = in && c0 + cw < g.ic ? ld_stream4(p) : make_float4(0.f, 0.f, 0.f, 0.f);
                    v[4 * j] = t.x; v[4 * j + 1] = t.y; v[4 * j + 2] = t.z; v[4 * j + 3] = t.w;
                } else {
#pragma unroll
                    for (int i = 0; i < 4; i++)
                        v[4 * j + i] = in && c0 + cw + i < g.ic ? __ldg(p + i) : 0.f;
                }
            }
        } else {
            const float *pn = pw + (long)c0 * g.hw;
            if (live && c0 + TCC <= g.ic) {
#pragma unroll
                for (int i = 0; i < TPER; i++) v[i] = ld_stream(row_ptr<TPER == 32>(pn, i, pitch));
            } else {
#pragma unroll
                for (int i = 0; i < TPER; i++)
                    v[i] = (live && c0 + cw + i < g.ic) ? ld_stream(row_ptr<TPER == 32>(pn, i, pitch)) : 0.f;
            }
        }
    };
    fetch(0);
    for (int c0 = 0; c0 < c_end; c0 += TCC) {
        const int left = g.ic - (c0 + cw);  // channels from this thread's first one on
        if (WITH_A) {
#pragma unroll
            for (int j = 0; j < TPER / 4; j++) {
                float4 *f4 = reinterpret_cast<float4 *>(
                    NHWC ? f_s + (p0 + j * PPI) * FLD + cw : f_s + lane * FLD + cw + 4 * j);
                *f4 = make_float4(__fmul_rn(fabsf(v[4 * j]), g.inv_ic),
                                  __fmul_rn(fabsf(v[4 * j + 1]), g.inv_ic),
                                  __fmul_rn(fabsf(v[4 * j + 2]), g.inv_ic),
                                  __fmul_rn(fabsf(v[4 * j + 3]), g.inv_ic));
            }
        }
        if (WITH_PACK) {
            const uint32_t *u = reinterpret_cast<const uint32_t *>(v);
            if (NHWC) {
#pragma unroll
                for (int j = 0; j < LOADS; j++) {
                    uint32_t w = ((u[4 * j] >> 28) & 0x8u) | ((u[4 * j + 1] >> 24) & 0x80u) |
                                 ((u[4 * j + 2] >> 20) & 0x800u) | ((u[4 * j + 3] >> 16) & 0x8000u) |
                                 0x2222u;
                    w = first_nibbles(w, left >= 4 ? 8 : left);
                    *reinterpret_cast<uint16_t *>(b_s + (p0 + j * PPI) * TLD + cw / 2) = (uint16_t)w;
                }
            } else {
                uint32_t w[TPER / 8];
#pragma unroll
                for (int j = 0; j < TPER / 8; j++)  // channels past the last one are zero
                    w[j] = first_nibbles(sign_nibbles(u + 8 * j), left - 8 * j);
                uint8_t *b = b_s + lane * TLD + cw / 2;
                if (TPER == 32) {
                    *reinterpret_cast<uint4 *>(b) = make_uint4(w[0], w[1], w[TPER / 8 - 2], w[TPER / 8 - 1]);
                } else if (TPER == 16) {
                    *reinterpret_cast<uint2 *>(b) = make_uint2(w[0], w[TPER / 8 - 1]);
                } else {
#pragma unroll
                    for (int j = 0; j < TPER / 8; j++) reinterpret_cast<uint32_t *>(b)[j] = w[j];
                }
            }
        }
        __syncthreads();
        if (c0 + TCC < c_end) fetch(c0 + TCC);  // fly while this chunk is consumed
        if (WITH_A && warp == 0) {
            const int nc = min(TCC, g.ic - c0);
            const float *fr = f_s + lane * FLD;
            if (nc == TCC) {
#pragma unroll
                for (int j0 = 0; j0 < TCC; j0 += 16) {
                    float4 t[4];
#pragma unroll
                    for (int j = 0; j < 4; j++) t[j] = *reinterpret_cast<const float4 *>(fr + j0 + 4 * j);
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        acc = __fadd_rn(acc, t[j].x);
                        acc = __fadd_rn(acc, t[j].y);
                        acc = __fadd_rn(acc, t[j].z);
                        acc = __fadd_rn(acc, t[j].w);
                    }
                }
            } else {  // channel tail: same order
                int j = 0;
                for (; j + 4 <= nc; j += 4) {
                    const float4 t = *reinterpret_cast<const float4 *>(fr + j);
                    acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, t.x), t.y), t.z), t.w);
                }
                for (; j < nc; j++) acc = __fadd_rn(acc, fr[j]);
            }
        } else if (WITH_PACK) {
            // TCC / 16 lanes write a pixel's chunk, 8 bytes each
            const int first = WITH_A ? warp - 1 : warp, step = WITH_A ? TWARPS - 1 : TWARPS;
            const int n8 = (min(TCC, g.ic - c0) + 15) / 16;
            constexpr int LPW = TCC / 16;  // lanes per pixel and chunk
            constexpr int PPW = 32 / LPW;  // pixels a warp writes per pass
            const int sub = lane / LPW, wl = lane % LPW;
            if (sub < PPW && wl < n8) {
                uint2 *out = reinterpret_cast<uint2 *>(g.out) + (c0 >> 4) + wl;
                const uint8_t *tile = b_s + 8 * wl;
                for (int pi = PPW * first + sub; pi < n_live; pi += PPW * step)
                    out[row_s[pi]] = *reinterpret_cast<const uint2 *>(tile + pi * TLD);
            }
        }
        __syncthreads();
    }
    if (WITH_A && warp == 0 && live) g.a[px] = acc;
}

// ---- K: box filter of A ------------------------------------------------------------------------
// A block takes a few output rows of one image: what they read of A goes to shared memory, already
// multiplied by 1/(KH*KW) (each term of upstream's sum is that product) and with zeros where the
// window leaves the image (adding +0 to a sum of non-negative terms changes nothing), and a thread
// adds up an output's terms in upstream's order. A staged row has its columns sorted by their
// remainder modulo the stride, so that neighbouring outputs read neighbouring words.
struct BoxArgs {
    const float *a;
    float *k;
    int ih, iw, oh, ow, kh, kw, sh, sw, ph, pw;
    float inv_khw;
    int rows, row_blocks;  // output rows per block, blocks per image
    int span, phase;       // columns of A an output row reads; words per remainder
    int lines;             // rows of A staged
    int cols, line_step;   // box_filter_columns_kernel: threads on a staged row; rows staged at a time
    FastDiv by_cols, by_sw, by_ow;
};
// Apart from the others' arguments: with the table among them those kernels, which do not read it, took up
// to 3 % longer.
struct BoxTapArgs {
    BoxArgs box;
    FastDiv by_span;
    int tap[11];  // word of tap j, from the output's first
};

constexpr int kBoxThreads = 256, kBoxAhead = 8;
constexpr int kBoxSmem = 40 * 1024;

// An output a thread. Tap j is a fixed distance from the output's first word: three instructions per term
// for the filter widths that are compiled in (KW). AlexNet conv1 on 64 images, 121 taps: 18.8 us with the
// terms read from global memory one after the other, 16.4 like this.
template <int KW>
__global__ void __launch_bounds__(kBoxThreads) box_filter_kernel(const BoxTapArgs t) {
    const BoxArgs &g = t.box;
    extern __shared__ __align__(16) float tile[];
    dependency_release();
    dependency_wait();
    const int n = blockIdx.x / g.row_blocks;
    const int oy0 = (blockIdx.x - n * g.row_blocks) * g.rows;
    const int n_out = min(g.rows, g.oh - oy0) * g.ow;
    const int y0 = oy0 * g.sh - g.ph, pitch = g.phase * g.sw;
    const float *img = g.a + (long)n * g.ih * g.iw;
#pragma unroll 4
    for (int i = threadIdx.x; i < g.lines * g.span; i += kBoxThreads) {
        const int line = (int)t.by_span((uint32_t)i), xx = i - line * g.span;
        const int y = y0 + line, x = xx - g.pw, xs = (int)g.by_sw((uint32_t)xx);
        float v = 0.f;
        if (y >= 0 && y < g.ih && x >= 0 && x < g.iw)
            v = __fmul_rn(__ldg(img + y * g.iw + x), g.inv_khw);
        tile[line * pitch + (xx - xs * g.sw) * g.phase + xs] = v;
    }
    __syncthreads();
    for (int o = threadIdx.x; o < n_out; o += kBoxThreads) {
        const int r = (int)g.by_ow((uint32_t)o), x = o - r * g.ow;
        const float *row = tile + r * g.sh * pitch + x;
        float acc = 0.f;
        for (int i = 0; i < g.kh; i++, row += pitch) {
            if (KW > 0) {
#pragma unroll
                for (int j = 0; j < KW; j++) acc = __fadd_rn(acc, row[t.tap[j]]);
            } else {
                for (int j = 0, at = 0, rem = 0; j < g.kw; j++) {
                    acc = __fadd_rn(acc, row[rem * g.phase + at]);
                    if (++rem == g.sw) { rem = 0; at++; }
                }
            }
        }
        g.k[((long)n * g.oh + oy0 + r) * g.ow + x] = acc;
    }
}

// A line of the window of the thread's upper output (FIRST), of its lower one (SECOND), or of both.
template <int KW, int SW, bool FIRST, bool SECOND>
__device__ __forceinline__ void add_line(const BoxArgs &g, const float *row, float &first, float &second) {
    if (KW > 0) {
#pragma unroll
        for (int j = 0; j < KW; j++) {
            const float v = row[j % SW * g.phase + j / SW];
            if (FIRST) first = __fadd_rn(first, v);
            if (SECOND) second = __fadd_rn(second, v);
        }
    } else {
        for (int j = 0, at = 0, rem = 0; j < g.kw; j++) {
            const float v = row[rem * g.phase + at];
            if (FIRST) first = __fadd_rn(first, v);
            if (SECOND) second = __fadd_rn(second, v);
            if (++rem == g.sw) { rem = 0; at++; }
        }
    }
}

// A thread keeps its column while it stages, eight lines at a time, and all its loads go out before the
// first is used; tap j is word j / SW of remainder j % SW, known to the compiler. TWO: it adds up two
// outputs, one below the other, and reads what their windows share once. AlexNet conv1 on 64 images,
// launched alone: 16.4 us with the kernel above (8.8 M warp instructions), 13.8 like this (5.5 M).
template <int KW, int SW, bool TWO>
__global__ void __launch_bounds__(kBoxThreads) box_filter_columns_kernel(const BoxArgs g) {
    extern __shared__ __align__(16) float tile[];
    dependency_release();
    dependency_wait();
    const int n = blockIdx.x / g.row_blocks;
    const int oy0 = (blockIdx.x - n * g.row_blocks) * g.rows;
    const int y0 = oy0 * g.sh - g.ph, pitch = g.phase * g.sw;
    const float *img = g.a + (long)n * g.ih * g.iw;
    const int first = (int)g.by_cols(threadIdx.x);
    // staged lines that the image has
    const int lo = min(max(0, -y0), g.lines), hi = min(g.lines, g.ih - y0);
    for (int c = threadIdx.x - first * g.cols; c < g.span && first < g.line_step; c += g.cols) {
        const int xs = (int)g.by_sw((uint32_t)c), x = c - g.pw;
        const bool in = x >= 0 && x < g.iw;
        float *to = tile + (c - xs * g.sw) * g.phase + xs;
        // every load is of an address that exists, so that none waits behind a branch of another
        const float *from = img + y0 * g.iw + min(max(x, 0), g.iw - 1);
        int line = lo + first;
        if (hi - lo > 2 * g.line_step) {
            for (; line < hi; line += kBoxAhead * g.line_step) {
                float v[kBoxAhead];
#pragma unroll
                for (int i = 0; i < kBoxAhead; i++)
                    v[i] = __ldg(from + min(line + i * g.line_step, hi - 1) * g.iw);
#pragma unroll
                for (int i = 0; i < kBoxAhead; i++)
                    if (line + i * g.line_step < hi)
                        to[(line + i * g.line_step) * pitch] = in ? __fmul_rn(v[i], g.inv_khw) : 0.f;
            }
        } else if (line < hi) {  // one line a thread, or two
            const int other = min(line + g.line_step, hi - 1);
            const float u = __ldg(from + line * g.iw), v = __ldg(from + other * g.iw);
            to[line * pitch] = in ? __fmul_rn(u, g.inv_khw) : 0.f;
            if (line + g.line_step < hi) to[other * pitch] = in ? __fmul_rn(v, g.inv_khw) : 0.f;
        }
        for (int line = first; line < lo; line += g.line_step) to[line * pitch] = 0.f;
        for (int line = max(hi, 0) + first; line < g.lines; line += g.line_step) to[line * pitch] = 0.f;
    }
    __syncthreads();
    const int n_out = (TWO ? g.rows >> 1 : g.rows) * g.ow;
    for (int o = threadIdx.x; o < n_out; o += kBoxThreads) {
        const int q = (int)g.by_ow((uint32_t)o), x = o - q * g.ow, r = TWO ? 2 * q : q;
        const float *row = tile + r * g.sh * pitch + x;
        float upper = 0.f, lower = 0.f;
        int i = 0;
        if (TWO) {
            for (; i < g.sh; i++, row += pitch) add_line<KW, SW, true, false>(g, row, upper, lower);
            for (; i < g.kh; i++, row += pitch) add_line<KW, SW, true, true>(g, row, upper, lower);
            for (; i < g.sh + g.kh; i++, row += pitch) add_line<KW, SW, false, true>(g, row, upper, lower);
        } else {
            for (; i < g.kh; i++, row += pitch) add_line<KW, SW, true, false>(g, row, upper, lower);
        }
        float *to = g.k + ((long)n * g.oh + oy0 + r) * g.ow + x;
        if (oy0 + r < g.oh) to[0] = upper;
        if (TWO && oy0 + r + 1 < g.oh) to[g.ow] = lower;
    }
}

// Windows that do not fit shared memory: one thread per output, straight from A.
__global__ void __launch_bounds__(kBoxThreads) box_filter_wide_kernel(const BoxArgs g) {
    dependency_release();
    dependency_wait();
    const long o = (long)blockIdx.x * kBoxThreads + threadIdx.x;
    const long plane = (long)g.oh * g.ow;
    const long n = o / plane;
    const int r = (int)(o - n * plane), y = r / g.ow, x = r - y * g.ow;
    if (y >= g.oh || n >= g.row_blocks) return;  // row_blocks: images here
    const float *img = g.a + n * g.ih * g.iw;
    float acc = 0.f;
    for (int i = 0; i < g.kh; i++) {
        const int h = y * g.sh - g.ph + i;
        if (h < 0 || h >= g.ih) continue;
        for (int j = 0; j < g.kw; j++) {
            const int w = x * g.sw - g.pw + j;
            if (w < 0 || w >= g.iw) continue;
            acc = __fadd_rn(acc, __fmul_rn(__ldg(img + h * g.iw + w), g.inv_khw));
        }
    }
    g.k[o] = acc;
}

using BoxTapFn = void (*)(BoxTapArgs);
BoxTapFn box_kernel(int kw) {
    return kw == 1    ? box_filter_kernel<1>
           : kw == 3  ? box_filter_kernel<3>
           : kw == 5  ? box_filter_kernel<5>
           : kw == 7  ? box_filter_kernel<7>
           : kw == 11 ? box_filter_kernel<11>
                      : box_filter_kernel<0>;
}
// The same by columns; null where the other kernel is the better one.
using BoxFn = void (*)(BoxArgs);
BoxFn box_columns_kernel(int kw, int sw, bool two) {
    if (!two)
        return kw == 5 && sw == 1   ? box_filter_columns_kernel<5, 1, false>
               : kw == 5 && sw == 2 ? box_filter_columns_kernel<5, 2, false>
                                    : nullptr;
    if (kw == 7 && sw == 1) return box_filter_columns_kernel<7, 1, true>;
    if (kw == 7 && sw == 2) return box_filter_columns_kernel<7, 2, true>;
    if (kw == 11 && sw == 4) return box_filter_columns_kernel<11, 4, true>;
    return kw == 1 || kw == 3 || kw == 5 || kw == 7 || kw == 11 ? nullptr
                                                                : box_filter_columns_kernel<0, 1, true>;
}

BinArgs bin_args(const Plan &p, const float *src, void *out, float *a) {
    BinArgs g;
    g.src = src; g.out = out; g.a = a;
    g.n_px = (long)p.mb * p.ih * p.iw;
    g.ic = p.ic; g.hw = p.ih * p.iw; g.iw = p.iw; g.ih = p.ih;
    g.img_stride = (long)p.ic * p.ih * p.iw;
    g.c_stride = p.src_nhwc ? 1 : (long)p.ih * p.iw;
    g.px_stride = p.src_nhwc ? p.ic : 1;
    g.inv_ic = p.inv_ic;
    g.words = p.family == kTcgen05 ? p.icp / 4 : p.icw;
    g.wp = p.wp; g.hp = p.hp; g.lead = p.lead;
    return g;
}

// tiled kernels: blocks per SM the carve-out is sized for (chunks of 128 and of 96 channels)
constexpr int kResidentBlocks = 5, kResidentBlocks96 = 9;

template <bool WITH_A, bool WITH_PACK, bool NHWC, int TPER>
cudaError_t launch_tiled(const BinArgs &g, cudaStream_t s) {
    // Shared-memory carve-out sized for a fixed number of blocks per SM, once per device. Left
    // to itself the driver sizes it for as many blocks as the thread count allows, which
    // leaves the L1 too small: the loads in flight occupy it although they do not allocate
    // lines to keep, and a kernel that streams with 32 loads per thread outstanding does not
    // need that many warps. Measured on conv4, minibatch 256, pass with the mean-|x| map:
    // eight blocks (an L1 of 32 KB) 20.4 us, seven or six (64 KB) 16.9-17.3, five (96 KB)
    // 17.0-17.1 with the whole step 0.5 us shorter, four or three (128 KB) 18.1. The
    // 96-channel kernel on conv2: nine of its blocks (the same 64 KB of L1) 9.3 us, seven
    // (96 KB) 9.7, five 11.2.
    auto kernel = binarize_nibbles_kernel<WITH_A, WITH_PACK, NHWC, TPER>;
    static std::atomic<bool> tuned[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (!tuned[dev & 63].exchange(true, std::memory_order_acq_rel)) {
        int smem_sm = 0;
        cudaFuncAttributes fa;
        cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
        if (smem_sm > 0 && cudaFuncGetAttributes(&fa, kernel) == cudaSuccess) {
            const int resident = TPER == 32 ? kResidentBlocks : kResidentBlocks96;
            long pct = (100L * resident * ((long)fa.sharedSizeBytes + 1024) + smem_sm - 1) / smem_sm;
            if (pct > 100) pct = 100;
            cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, (int)pct);
        }
        (void)cudaGetLastError();
    }
    note_launch();
    // Launched with programmatic stream serialisation like the convolution: behind one of
    // this library's kernels (which trigger early) the blocks become resident while it
    // drains and wait in dependency_wait(); behind anything else nothing changes.
    return launch_overlapped(kernel, dim3((unsigned)((g.n_px + TPX - 1) / TPX)),
                             dim3(TWARPS * 32), 0, s, 1, g);
}

template <bool WITH_A, bool WITH_PACK>
cudaError_t launch_bin(const Plan &p, const BinArgs &g, cudaStream_t s) {
    const int threads = 128;
    const unsigned blocks = (unsigned)((g.n_px + threads - 1) / threads);
    if (blocks == 0) return cudaSuccess;
    if ((p.family == kTcgen05 || !WITH_PACK) && g.n_px < (1L << 31) - TPX &&
        (long)p.ih * p.iw < (1L << 24)) {
        if (p.src_nhwc) {
            if (g.ic <= 32) return launch_tiled<WITH_A, WITH_PACK, true, 8>(g, s);
            if (g.ic <= 64) return launch_tiled<WITH_A, WITH_PACK, true, 16>(g, s);
            return launch_tiled<WITH_A, WITH_PACK, true, 32>(g, s);
        }
        if (g.ic <= 32) return launch_tiled<WITH_A, WITH_PACK, false, 8>(g, s);
        if (g.ic <= 64) return launch_tiled<WITH_A, WITH_PACK, false, 16>(g, s);
        if (g.ic % 96 == 0 && g.ic % 128 != 0)
            return launch_tiled<WITH_A, WITH_PACK, false, 24>(g, s);
        return launch_tiled<WITH_A, WITH_PACK, false, 32>(g, s);
    }
    switch (p.family) {
        case kPopc: binarize_kernel<kBitsDense, WITH_A, WITH_PACK><<<blocks, threads, 0, s>>>(g); break;
        default: binarize_kernel<kNibblesFramed, WITH_A, WITH_PACK><<<blocks, threads, 0, s>>>(g); break;
    }
    note_launch();
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_binarize_data(const Plan &p, const float *src, void *bin_src, float *a,
                                 cudaStream_t s) {
    if (p.fold) return launch_fold(p, src, bin_src, a, s);
    const BinArgs g = bin_args(p, src, bin_src, a);
    return a ? launch_bin<true, true>(p, g, s) : launch_bin<false, true>(p, g, s);
}

cudaError_t launch_mean_abs(const Plan &p, const float *src, float *a, cudaStream_t s) {
    const BinArgs g = bin_args(p, src, nullptr, a);
    return launch_bin<true, false>(p, g, s);
}

cudaError_t launch_box_filter(const Plan &p, const float *a, float *k, cudaStream_t s) {
    BoxArgs g;
    g.a = a; g.k = k;
    g.ih = p.ih; g.iw = p.iw; g.oh = p.oh; g.ow = p.ow; g.kh = p.kh; g.kw = p.kw;
    g.sh = p.sh; g.sw = p.sw; g.ph = p.ph; g.pw = p.pw;
    g.inv_khw = p.inv_khw;
    if (p.mb < 1 || p.oh < 1 || p.ow < 1) return cudaSuccess;
    g.span = (p.ow - 1) * p.sw + p.kw;
    g.phase = div_up_i(g.span, p.sw);
    g.by_sw = FastDiv((uint32_t)p.sw); g.by_ow = FastDiv((uint32_t)p.ow);
    auto lines = [&](int rows) { return (long)(rows - 1) * p.sh + p.kh; };
    auto bytes = [&](int rows) { return 4L * lines(rows) * g.phase * p.sw; };
    // By columns where an image's outputs are enough for half a block's threads; two outputs a thread where
    // their windows are large and share half of their lines at least. calculate_k on 18 MB of one channel
    // (150 us of it the mean |x|), an output a thread -> this: 5 x 5 on 56 x 56 198.6 -> 190.3 us, 7 x 7
    // 209 -> 186, 9 x 9 295 -> 240, 9 x 9 with stride 2 191.5 -> 179, 13 x 13 412 -> 306; on 256 x 256
    // 7 x 7 247 -> 202, 11 x 11 with stride 4 168.3 -> 167.9. Images of 49 outputs (14 x 14, stride 2)
    // 174.8 -> 184.8 with 5 x 5, 178.8 -> 191.6 with 7 x 7; 7 x 7 images 232 to 266 -> 288 to 374.
    // Widths that only the other kernel has compiled in: 3 x 3 178 -> 187 on 28 x 28, 203 -> 215 on 256 x
    // 256, 11 x 11 246 -> 273 on 56 x 56, with stride 2 181 -> 191.
    const bool two = p.kh >= 2 * p.sh && p.kh * p.kw >= 49 && p.oh > 1 && bytes(2) <= kBoxSmem;
    const BoxFn by_columns = (long)p.oh * p.ow >= kBoxThreads / 2 ? box_columns_kernel(p.kw, p.sw, two) : nullptr;
    const int up = by_columns && two ? 2 : 1;
    // about one thread for each, if the rows that takes fit shared memory
    g.rows = up * (kBoxThreads / p.ow);
    if (g.rows > div_up_i(p.oh, up) * up) g.rows = div_up_i(p.oh, up) * up;
    if (g.rows < up) g.rows = up;
    while (g.rows > up && bytes(g.rows) > kBoxSmem) g.rows -= up;
    note_launch();
    if (bytes(g.rows) > kBoxSmem) {
        g.row_blocks = p.mb;
        const long n_out = (long)p.mb * p.oh * p.ow;
        return launch_overlapped(box_filter_wide_kernel,
                                 dim3((unsigned)((n_out + kBoxThreads - 1) / kBoxThreads)),
                                 dim3(kBoxThreads), 0, s, 1, g);
    }
    g.row_blocks = div_up_i(p.oh, g.rows);
    g.lines = (int)lines(g.rows);
    const unsigned blocks = (unsigned)(p.mb * g.row_blocks);
    // Launched under the tail of the packer, as the convolution is under its own: conv1 mb64 63.7 ->
    // 60.7 us a pass, the three upstream calls of an odd layer 20.6 -> 19.4.
    if (by_columns) {
        const int cols = div_up_i(g.span, 32) * 32;
        g.cols = cols < kBoxThreads ? cols : kBoxThreads;
        g.line_step = kBoxThreads / g.cols;
        g.by_cols = FastDiv((uint32_t)g.cols);
        return launch_overlapped(by_columns, dim3(blocks), dim3(kBoxThreads), (size_t)bytes(g.rows), s, 1, g);
    }
    BoxTapArgs t;
    t.box = g;
    t.by_span = FastDiv((uint32_t)g.span);
    for (int j = 0; j < 11; j++) t.tap[j] = j % p.sw * g.phase + j / p.sw;
    return launch_overlapped(box_kernel(p.kw), dim3(blocks), dim3(kBoxThreads), (size_t)bytes(g.rows), s, 1, t);
}

}  // namespace xb200
