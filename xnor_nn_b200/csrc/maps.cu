// calculate_k of small layers in one launch: mean |x| and its box filter (upstream
// src/bcast_calculate_k.cpp:13-88), where the general path launches one kernel for each (binarize.cu). A
// block takes a band of output rows of one image and adds up the pixels its windows see, by tasks
// (pixel_tasks.cuh), into shared memory; rows that two bands see are added by both, in the same order, and
// left in the map by the one that owns them. Then a thread adds up an output's terms in upstream's order.
// Bound by the latency of its few rounds of loads; what it is for is the launch it saves, 2 us of the host's:
// the three upstream calls on 19 images of 75 channels, 31 x 27, take 9.6 instead of 12.8 us a pass among
// others, a microsecond of it less work in the caller, and 16.5 instead of 17.0 on one stream; 15 images of 304
// channels, 9 x 9, filters of 5 x 5, 9.9 instead of 13.0 among others, 24.6 and 24.4 on one stream.
#include "kernels.cuh"
#include "map_bands.cuh"
#include "pixel_tasks.cuh"
#include "tc_ptx.cuh"

namespace xb200 {

namespace {

using namespace bands;
using namespace tasks;

template <bool NHWC>
__global__ void __launch_bounds__(kThreads) maps_kernel(const MapArgs g) {
    __shared__ float tile[kTileFloats];  // mean |x| / (KH*KW), zeros outside the image
    __shared__ float sum[kMaxGroups][32];
    // The channels before a task's have been added up: a barrier a task, used once. As counters that are polled (the
    // three calls on one stream): 512 channels of 14 x 14, eight images 18.4 us instead of 17.7; 384 of 13 x 13,
    // four 17.5 and 17.1; 128 of 14 x 14, 40 images 12.9 and 12.7.
    __shared__ unsigned long long turn[kMaxTasks];
    __shared__ int abort_flag;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const Band b = band_of(g, (int)blockIdx.x);
    for (int i = threadIdx.x; i < g.lines * g.span; i += kThreads) tile[i] = 0.f;
    if (threadIdx.x < kMaxTasks) tc::mbar_init(tc::smem_u32(&turn[threadIdx.x]), 1);
    if (threadIdx.x == 0) abort_flag = 0;
    dependency_release();
    __syncthreads();
    dependency_wait();
    for (int t = warp; t < b.tasks; t += kWarps) {
        const int col = t / b.groups, gr = t - col * b.groups;
        const int nc = min(32, g.ic - 32 * col);
        float v[32];
        load_task<NHWC>(g, b, t, lane, v);
        if (NHWC) transpose8(v, lane & 7);
        scale_task(v, g.inv_ic);
        float acc = 0.f;
        if (col > 0) {
            if (!tc::warp_wait(tc::smem_u32(&turn[t]), 0, &abort_flag, g.error, 21, g.wait_ns)) break;
            acc = *(const volatile float *)&sum[gr][lane];
        }
        acc = sum_task(v, nc, acc);
        const int px = b.first + 32 * gr + (NHWC ? 4 * (lane & 7) + (lane >> 3) : lane);
        if (col + 1 < g.columns) {
            sum[gr][lane] = acc;
            __syncwarp();
            if (lane == 0 && g.turn_step) tc::mbar_arrive(tc::smem_u32(&turn[t + b.groups]));
        } else if (px < b.last) {
            const int r = px - b.n * g.hw, y = (int)g.by_iw((uint32_t)r), x = r - y * g.iw;
            if (y >= b.own0 && y < b.own1) g.a[px] = acc;
            if (y - b.y0 < g.lines && x + g.pw < g.span)
                tile[(y - b.y0) * g.span + x + g.pw] = __fmul_rn(acc, g.inv_khw);
        }
    }
    __syncthreads();
    if (abort_flag) return;
    const int n_out = min(g.rows, g.oh - b.oy0) * g.ow;
    for (int o = threadIdx.x; o < n_out; o += kThreads) {
        const int r = (int)g.by_ow((uint32_t)o), x = o - r * g.ow;
        const float *row = tile + r * g.sh * g.span + x * g.sw;
        float acc = 0.f;
        for (int i = 0; i < g.kh; i++, row += g.span)
            for (int j = 0; j < g.kw; j++) acc = __fadd_rn(acc, row[j]);
        g.k[((long)b.n * g.oh + b.oy0 + r) * g.ow + x] = acc;
    }
}

}  // namespace

bool maps_ok(const Plan &p) {
    MapArgs g;
    return maps_shape(p, &g);
}

cudaError_t launch_maps(const Plan &p, const float *src, float *a, float *k, int *error_word,
                        cudaStream_t s, const ConvSelfTest *test) {
    MapArgs g;
    if (!maps_shape(p, &g)) return cudaErrorNotSupported;
    g.src = src; g.a = a; g.k = k; g.error = error_word;
    g.wait_ns = test && test->wait_ns ? test->wait_ns : 2000000000ull;
    g.turn_step = test && test->drop_turn ? 0 : 1;
    g.inv_ic = p.inv_ic; g.inv_khw = p.inv_khw;
    g.ic = p.ic; g.hw = p.ih * p.iw; g.ih = p.ih; g.iw = p.iw;
    g.vec = p.src_nhwc && p.ic % 4 == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0;
    g.oh = p.oh; g.ow = p.ow; g.kh = p.kh; g.kw = p.kw; g.sh = p.sh; g.sw = p.sw; g.ph = p.ph; g.pw = p.pw;
    g.by_hw = FastDiv((uint32_t)g.hw); g.by_iw = FastDiv((uint32_t)p.iw); g.by_ow = FastDiv((uint32_t)p.ow);
    note_launch();
    auto kernel = p.src_nhwc ? maps_kernel<true> : maps_kernel<false>;
    return launch_overlapped(kernel, dim3((unsigned)(p.mb * g.bands)), dim3(kThreads), 0, s, 1, g);
}

}  // namespace xb200
