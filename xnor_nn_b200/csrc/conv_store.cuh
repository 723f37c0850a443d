// Float stores of the one-launch pass (conv_whole.cu): a warp's 32 positions (one per lane) times its share
// of a tile's filters, from tensor memory to the result. epilogue_role in conv_tcgen05.cu, which also has
// sums and chained layers to serve, keeps these forms inline: through these functions chained layers
// (AlexNet conv3 to conv5, 128 images) took 46.2 instead of 43.6 us.
#pragma once

#include "kernels.cuh"
#include "tc_ptx.cuh"

namespace xb200 {
namespace tc {

// The pixel and the filters that a lane stores.
struct StoreAt {
    float *dst;
    int oc, oc0, n_valid;  // filters; the tile's first one, and how many of the tile exist
    int n, r;              // image, pixel in it
    long pix, ohw;         // n * ohw + r
    float kk;
    bool valid;            // the lane's position is a pixel
};

// NCHW: for one filter the 32 lanes hold 32 neighbouring pixels, so a store instruction writes one
// contiguous run. `al` = alpha from the tile's first filter on, in shared memory.
__device__ __forceinline__ void store_nchw(const StoreAt &s, const float *al, int n_tile, uint32_t taddr,
                                           int cgroup, int cgroups) {
    float *out = s.dst + ((long)s.n * s.oc + s.oc0) * s.ohw + s.r;
    for (int c0 = 32 * cgroup; c0 < n_tile; c0 += 32 * cgroups) {
        uint32_t v[32];
        if (c0 + 32 <= n_tile) {
            ld32(taddr + (uint32_t)c0, v);
        } else {  // N is a multiple of 16, not always of 32
            ld16(taddr + (uint32_t)c0, v);
        }
        wait_ld();
        if (s.valid) {
            const int lim = s.n_valid - c0;
            float *o = out + (long)c0 * s.ohw;
            if (lim >= 32) {
                // full group: alpha by 16-byte shared loads, one running pointer
                const float4 *a4 = reinterpret_cast<const float4 *>(al + c0);
#pragma unroll
                for (int j = 0; j < 32; j += 4) {
                    const float4 a = a4[j >> 2];
                    // streaming stores: the result is not read again by this library,
                    // and lines that leave L2 while this kernel runs (which needs little
                    // of HBM) do not have to leave it under the next, bandwidth-bound pass
                    __stcs(o, scaled(v[j], a.x, s.kk));
                    __stcs(o + s.ohw, scaled(v[j + 1], a.y, s.kk));
                    __stcs(o + 2 * s.ohw, scaled(v[j + 2], a.z, s.kk));
                    __stcs(o + 3 * s.ohw, scaled(v[j + 3], a.w, s.kk));
                    o += 4 * s.ohw;
                }
            } else {
#pragma unroll
                for (int j = 0; j < 32; j++)
                    if (j < lim) __stcs(o + (long)j * s.ohw, scaled(v[j], al[c0 + j], s.kk));
            }
        }
    }
}

// NHWC, a number of filters that is a multiple of four and a result that starts on 16 bytes: a thread
// owns one pixel and 16 neighbouring filters at a time, which are contiguous in the result.
__device__ __forceinline__ void store_nhwc(const StoreAt &s, const float *al, int n_tile, uint32_t taddr,
                                           int cgroup, int cgroups) {
    float *out = s.dst + s.pix * s.oc + s.oc0;
    // 256-bit stores need 32-byte alignment: rows and tiles that are multiples of 8
    // floats on a result buffer aligned likewise
    const bool wide = (s.oc & 7) == 0 && (s.oc0 & 7) == 0 && ((uintptr_t)s.dst & 31) == 0;
    for (int c0 = 16 * cgroup; c0 < n_tile; c0 += 16 * cgroups) {
        uint32_t v[16];
        ld16(taddr + (uint32_t)c0, v);
        wait_ld();
        if (s.valid && wide && c0 + 16 <= s.n_valid) {
            // 16 results = two whole 32-byte sectors, one 256-bit store each
            float x[16];
#pragma unroll
            for (int j = 0; j < 16; j++)
                x[j] = scaled(v[j], al[c0 + j], s.kk);
#pragma unroll
            for (int h = 0; h < 16; h += 8)
                asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                             ::"l"(out + c0 + h), "f"(x[h]), "f"(x[h + 1]), "f"(x[h + 2]),
                               "f"(x[h + 3]), "f"(x[h + 4]), "f"(x[h + 5]), "f"(x[h + 6]),
                               "f"(x[h + 7])
                             : "memory");
        } else if (s.valid) {
#pragma unroll
            for (int j = 0; j < 16; j += 4) {
                if (c0 + j >= s.n_valid) break;  // oc and n_valid are multiples of 4
                float4 x;
                x.x = scaled(v[j], al[c0 + j], s.kk);
                x.y = scaled(v[j + 1], al[c0 + j + 1], s.kk);
                x.z = scaled(v[j + 2], al[c0 + j + 2], s.kk);
                x.w = scaled(v[j + 3], al[c0 + j + 3], s.kk);
                *reinterpret_cast<float4 *>(out + c0 + j) = x;
            }
        }
    }
}

// NHWC, any number of filters and any start of the result.
__device__ __forceinline__ void store_nhwc_odd(const StoreAt &s, const float *al, int n_tile,
                                               uint32_t taddr, int cgroup, int cgroups) {
    float *out = s.dst + s.pix * s.oc + s.oc0;
    for (int c0 = 16 * cgroup; c0 < n_tile; c0 += 16 * cgroups) {
        uint32_t v[16];
        ld16(taddr + (uint32_t)c0, v);
        wait_ld();
        if (s.valid) {
#pragma unroll
            for (int j = 0; j < 16; j++)
                if (c0 + j < s.n_valid) out[c0 + j] = scaled(v[j], al[c0 + j], s.kk);
        }
    }
}

}  // namespace tc
}  // namespace xb200
