// Packing the source by tasks of 32 neighbouring pixels x 32 channels, a task a warp (conv_whole.cu,
// maps.cu): loads, and the sum of |x| over the channels in upstream's order, which tasks of the same pixels
// hand on from warp to warp.
#pragma once

#include "kernels.cuh"

namespace xb200 {
namespace tasks {

// The pixel that lane `lane` reads of group `group` of a tile's pixels first .. last, channels-first: a lane behind
// the last pixel reads that one, which has to be a pixel of the source (the first one serves a tile of none
// in front of all).
__host__ __device__ inline int lane_pixel(int first, int last, int group, int lane) {
    const int px = first + 32 * group + lane < last ? first + 32 * group + lane : last - 1;
    return px < 0 ? 0 : px;
}

#ifdef __CUDACC__
// 32 channels of 32 pixels, channels-last: eight lanes read a pixel's channels, four each (with 16-byte
// loads where they are aligned) and four pixels at a time, and an 8 x 8 transposition of those quadruples
// leaves a lane with all channels of pixel 4 (lane % 8) + lane / 8.
__device__ __forceinline__ void transpose8(float *v, int sub) {
#pragma unroll
    for (int d = 4; d > 0; d >>= 1) {
        const bool up = sub & d;
#pragma unroll
        for (int j = 0; j < 8; j++) {
            if (j & d) continue;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                // the quadruple that goes to the partner: j + d from the lower lane, j from the upper
                const float send = up ? v[4 * j + i] : v[4 * (j + d) + i];
                const float got = __shfl_xor_sync(0xffffffffu, send, d);
                if (up) v[4 * j + i] = got;
                else v[4 * (j + d) + i] = got;
            }
        }
    }
}

__device__ __forceinline__ void mul2(float &a, float &b, float by) {
    asm("{\n\t.reg .b64 x, y;\n\t"
        "mov.b64 x, {%0, %1};\n\t"
        "mov.b64 y, {%2, %2};\n\t"
        "mul.rn.f32x2 x, x, y;\n\t"
        "mov.b64 {%0, %1}, x;\n\t}"
        : "+f"(a), "+f"(b)
        : "f"(by));
}

// `tile`: its pixels first .. last, in groups of 32; `g`: the source. Lane l has pixel l of the group,
// channels-last after transpose8 pixel 4 (l % 8) + l / 8.
template <bool NHWC, class Args, class Tile>
__device__ __forceinline__ void load_task(const Args &g, const Tile &tile, int t, int lane, float *v) {
    const int col = t / tile.groups, gr = t - col * tile.groups;
    const int c0 = 32 * col, nc = min(32, g.ic - c0);
    if (NHWC) {  // transpose8 puts it in order
        const int sub = lane & 7, px = tile.first + 32 * gr + (lane >> 3);
        const float *p = g.src + (long)px * g.ic + c0 + 4 * sub;
#pragma unroll
        for (int j = 0; j < 8; j++, p += (long)4 * g.ic) {
            const bool in = px + 4 * j < tile.last;
            if (g.vec) {
                float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
                if (in && 4 * sub < nc) x = __ldg(reinterpret_cast<const float4 *>(p));
                v[4 * j] = x.x; v[4 * j + 1] = x.y; v[4 * j + 2] = x.z; v[4 * j + 3] = x.w;
            } else {
#pragma unroll
                for (int i = 0; i < 4; i++) v[4 * j + i] = in && 4 * sub + i < nc ? __ldg(p + i) : 0.f;
            }
        }
        return;
    }
    // What becomes of a lane without a pixel is not used. With a path of their own such lanes took their warp
    // through the loads twice: with one path, and no masks on full columns, passes of AlexNet conv4 in one launch
    // (conv_whole.cu) on one image 11.1 -> 10.0 us on one stream, on 32 images 16.4 -> 15.6 and among others
    // 5.97 -> 5.62.
    const unsigned px = (unsigned)lane_pixel(tile.first, tile.last, gr, lane);
    // an address is a warp-uniform channel plane and a lane's 32-bit offset into it (the host checks
    // the range)
    const unsigned n = g.by_hw(px), r = px - n * g.hw;
    const unsigned at = 4u * (n * (unsigned)(g.ic * g.hw) + r);
    const char *plane = reinterpret_cast<const char *>(g.src) + (size_t)c0 * g.hw * 4;
    const size_t pitch = (size_t)g.hw * 4;
    if (nc == 32) {
#pragma unroll
        for (int i = 0; i < 32; i++) v[i] = __ldg(reinterpret_cast<const float *>(plane + i * pitch + at));
    } else {
#pragma unroll
        for (int i = 0; i < 32; i++)
            v[i] = i < nc ? __ldg(reinterpret_cast<const float *>(plane + i * pitch + at)) : 0.f;
    }
}

// |x| / IC = |x / IC|: two products an instruction, the sign goes with the addition.
__device__ __forceinline__ void scale_task(float *v, float inv_ic) {
#pragma unroll
    for (int i = 0; i < 32; i += 2) mul2(v[i], v[i + 1], inv_ic);
}
__device__ __forceinline__ float sum_task(const float *v, int nc, float acc) {
    if (nc == 32) {
#pragma unroll
        for (int i = 0; i < 32; i++) acc = __fadd_rn(acc, fabsf(v[i]));
    } else {
#pragma unroll
        for (int i = 0; i < 32; i++)
            if (i < nc) acc = __fadd_rn(acc, fabsf(v[i]));
    }
    return acc;
}
#endif

}  // namespace tasks
}  // namespace xb200
