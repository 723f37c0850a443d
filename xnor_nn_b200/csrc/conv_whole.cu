// A whole forward pass in one launch, for layers of at most one tile of 128 positions x N filters per
// SM: small minibatches, where the two launches of the general path (packer, convolution) and the
// hand-over between them cost more than the work.
//
// A CTA packs what its tile reads by itself, from the float source straight into the operand layout in
// shared memory, and multiplies it there; nothing passes between CTAs. Pixels in the tiles' halos are
// read by each of them, and a layer of several filter tiles is packed once for each: SMs that would
// idle do that. The packed frame, the mean-|x| map and K are left in their buffers as the general path
// leaves them, by the CTA whose tile a pixel's position belongs to (its first filter tile).
//
//   warps 1-20  workers: a task is 32 neighbouring pixels x 32 channels, a warp load per channel. The
//               sign nibbles of a lane's pixel are one 16-byte column of the operand, the products
//               |x|/IC stay in registers until the channels before them have been added up (upstream's
//               order: tasks of the same pixels hand their running sums on). Tasks are dealt by columns
//               first, so the operand's first K chunk is complete while later ones are being packed.
//               Then the same warps are the epilogue: K from the mean |x| of the tile's pixels, which
//               is in shared memory, scaling and stores.
//   warp 0      TMA: filter tiles (K chunk by K chunk, all taps of each) into a ring
//   warps 21-24 MMA issuers on every fourth filter tile. The accumulator is zeroed before, so that none of
//               their instructions overwrites it, and sums of integers do not depend on the order. That no
//               instruction's sum is lost when two of different issuers follow one another on the same
//               columns is an assumption about the tensor pipe (it executes a CTA's instructions one
//               after the other, whoever issued them), not a documented guarantee, which names one
//               issuing thread. test_shared_accumulator_gpu.py watches it. Accumulators of their own would
//               not need it, but four fit for filter tiles of up to 112 filters only.
//
// The operand is, per K chunk of 128 bytes, rows of positions in the 128-byte swizzle, in which a tap is
// a row offset (conv_tcgen05.cu, halo tiles); where filter rows are one operand row (Plan::cat) or a
// position has no 128 bytes, it is [column][position][16 bytes], the unswizzled form that position
// columns have there (producer_planes), in which a tap is a start address.
//
// What bounds it, in cycles of a tile of AlexNet conv4 (136 pixels of 384 channels, 384 KB of filters per
// 256, 1.9 GHz) in a pass that is waited for, on one image, on 32, and on 64 channels-last: 1700 to 1900 until the
// kernel before has been waited for; 8800, 10300 and 13300 of packing (three tasks a worker; an SM takes floats in at
// 20 to 25 bytes a cycle, and 12, 16 or 24 workers, or loads a task ahead, do not change that), which the filter loads
// share the way with; 3100, 9000 and 8000 until the last MMA is done (one image has narrow filter tiles, all of which
// are in shared memory by then; 256 filters come through the ring meanwhile); 1000, 5200 and 6200 of stores. One
// issuer needs about 500 cycles a filter tile, mostly the chain of scalar instructions around its MMAs, hence four
// (MMAs of one image, with the packing of then: 6700 -> 5300). Times in us, two launches -> one: a pass among others on three streams, back to back on one
// stream, waited for: conv4 on one image 7.2 -> 3.9, 12.8 -> 9.6, 23.6 -> 21.0; on 32 images 8.2 -> 5.3,
// 16.4 -> 14.8, 25.0 -> 26.2; on 64 images channels-last 11.4 to 12.2 -> 11.4, 20.9 -> 18.0, 29.9 -> 29.9 (the
// last two as measured before the next paragraph's changes); 16 channels of 31 x 31, five images 8.7 -> 5.3,
// 7.5 -> 5.5, 20.0 -> 18.2 (the same). The first is bound by the host, for which a launch is 2.0 us.
//
// What made the packing shorter (12000 cycles before), on one stream in us, one image and 32: one path
// through a task's loads, whichever lanes have a pixel, 11.1 -> 10.0 and 16.4 -> 15.6; a barrier for each
// hand-over of a running sum instead of counters that are polled, 10.1 -> 9.7 and 15.6 -> 15.1; the accumulator
// cleared by the issuers, which have nothing to issue yet, instead of by packing warps, 9.7 -> 9.5 and 15.1 ->
// 14.8.
#include <cuda.h>

#include <atomic>

#include "conv_store.cuh"
#include "kernels.cuh"
#include "pixel_tasks.cuh"
#include "tc_ptx.cuh"

namespace xb200 {

namespace {

using namespace tc;
using namespace tasks;

constexpr int BM = 128;
constexpr int kWorkers = 20;
constexpr int kIssuers = 4;
constexpr int kFirstIssuer = 1 + kWorkers;  // warps: TMA, workers, issuers
static_assert(kIssuers == 4, "four neighbouring warps, a quadrant of tensor memory each");
constexpr int kThreads = 32 * (1 + kWorkers + kIssuers);
// Four tasks a worker. 7 x 402 channels of 29 x 29 (78 tasks): 7.1 -> 5.6 us among others, 16.3 -> 14.2 on
// one stream, 27.0 -> 26.6 alone; 492 channels of 51 x 51 (128 tasks): 6.7 -> 7.1, 13.3 -> 20.2, 24.2 -> 32.
constexpr int kMaxTasks = 4 * kWorkers;
constexpr int kMaxStages = 36, kMaxParts = 8, kMaxGroups = 16, kMaxRows = 32 * kMaxGroups;

struct WholeArgs {
    const float *src, *alpha;
    uint8_t *bin;     // packed frame
    float *a, *k;     // mean |x| and K maps
    float *dst;
    int *error;
    float inv_ic, inv_khw;
    int ic, hw, ih, iw, n_px, vec;
    int wp, hp, lead, q_total, icp;
    int kh, kw, oh, ow, oc, dst_nhwc;
    int n_tile, n_tiles, ocp16;
    int tap_kw, taps, chunks, kchunk, kk_last;  // filter taps and K chunks of a tap as the filters have them
    int swizzled, columns, planes, pitch, rows, odd;  // operand: 16-byte columns of a position, of the tile; positions
    int part_columns, parts;  // columns of a K chunk; K chunks of the operand
    int n_stages;
    uint32_t b_bytes, stage_bytes, b_off;
    uint32_t idesc, a_desc_hi, b_desc_hi, tmem_cols;
    unsigned long long wait_ns;
    int turn_step;                      // 1; these three are otherwise in self-tests only (ConvSelfTest)
    int more_commits, more_operand;     // arrivals that CTA 0 waits for in vain
    FastDiv by_frame, by_wp, by_hw, by_iw;
};

struct __align__(16) Control {
    unsigned long long full[kMaxStages], empty[kMaxStages];
    unsigned long long packed[kMaxParts];    // a K chunk's columns are in place
    unsigned long long acc_full, cleared, drain[kIssuers];
    uint32_t tmem_base;
    int abort_flag;
    alignas(16) float alpha[256];
    // The channels before a task's have been added up. A barrier a task, used once: as counters in shared memory,
    // polled with acquire loads and passed on with release stores, turns cost a pass of AlexNet conv4 on 32 images
    // 15.6 us instead of 15.1 on one stream, one image 10.1 instead of 9.7.
    unsigned long long turn[kMaxTasks];
    float sum[kMaxGroups][32];
    float a[kMaxRows];                       // mean |x| on the tile's rows of the frame
};
constexpr int kControlBytes = (sizeof(Control) + 1023) / 1024 * 1024;

// Pixels in front of frame position q.
__device__ __forceinline__ int pixels_before(const WholeArgs &g, int q) {
    if (q <= 0) return 0;
    const int n = (int)g.by_frame((uint32_t)q), rem = q - n * (g.hp * g.wp);
    const int h = (int)g.by_wp((uint32_t)rem), w = rem - h * g.wp;
    const int in = h >= g.ih ? g.hw : h * g.iw + min(w, g.iw);
    return min(n * g.hw + in, g.n_px);
}

// The pixels of a tile, in groups of 32, and where they come from. A task is a group and 32 channels.
struct Tile {
    int mt, q0, first, last, groups, tasks;
    __device__ __forceinline__ Tile(const WholeArgs &g, int mt_) : mt(mt_), q0(mt_ * BM - g.lead) {
        first = pixels_before(g, q0);
        last = pixels_before(g, q0 + g.rows);
        groups = max(1, (last - first + 31) >> 5);
        tasks = groups * g.columns;
    }
};

// Signs to the operand and, from the pixel's own tile, to the packed frame; then |x| to the sum.
template <bool NHWC>
__device__ __forceinline__ bool finish_task(const WholeArgs &g, Control *ctl, uint8_t *operand,
                                            const Tile &tile, bool owner, int t, int lane, float *v) {
    const int col = t / tile.groups, gr = t - col * tile.groups;
    const int nc = min(32, g.ic - 32 * col);
    if (NHWC) transpose8(v, lane & 7);
    const int px = tile.first + 32 * gr + (NHWC ? 4 * (lane & 7) + (lane >> 3) : lane);
    const bool live = px < tile.last;
    const int n = live ? (int)g.by_hw((uint32_t)px) : 0, r = live ? px - n * g.hw : 0;
    const int h = (int)g.by_iw((uint32_t)r), w = r - h * g.iw;
    const int q = (n * g.hp + h) * g.wp + w, row = q - tile.q0;
    const uint32_t *u = reinterpret_cast<const uint32_t *>(v);
    uint4 s;
    s = make_uint4(sign_nibbles(u), sign_nibbles(u + 8), sign_nibbles(u + 16), sign_nibbles(u + 24));
    if (nc < 32) {
        s.x = first_nibbles(s.x, nc);
        s.y = first_nibbles(s.y, nc - 8);
        s.z = first_nibbles(s.z, nc - 16);
        s.w = first_nibbles(s.w, nc - 24);
    }
    if (live) {
        const int o = g.swizzled ? (((col >> 3) * g.pitch + row) << 7) + (((col ^ row) & 7) << 4)
                                 : (col * g.pitch + row) << 4;
        *reinterpret_cast<uint4 *>(operand + o) = s;
        if (g.odd && col == 0 && row > 0)  // the column after a position's last one
            *reinterpret_cast<uint4 *>(operand + (g.columns * g.pitch + row - 1) * 16) = s;
    }
    fence_async_smem();
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&ctl->packed[col / g.part_columns]));
    const bool mine = owner && live && q >> 7 == tile.mt;
    if (mine) *reinterpret_cast<uint4 *>(g.bin + (long)(g.lead + q) * g.icp + 16 * col) = s;
    scale_task(v, g.inv_ic);
    float acc = 0.f;
    if (col > 0) {
        if (!warp_wait(smem_u32(&ctl->turn[t]), 0, &ctl->abort_flag, g.error, 21, g.wait_ns)) return false;
        acc = *(const volatile float *)&ctl->sum[gr][lane];
    }
    acc = sum_task(v, nc, acc);
    if (col + 1 < g.columns) {
        ctl->sum[gr][lane] = acc;
        __syncwarp();
        if (lane == 0 && g.turn_step) mbar_arrive(smem_u32(&ctl->turn[t + tile.groups]));
    } else if (live) {
        ctl->a[row] = acc;
        if (mine) g.a[px] = acc;
    }
    return true;
}

template <int WHO>
__device__ __forceinline__ void issue(const WholeArgs &g, Control *ctl, const uint8_t *operand, uint32_t b0,
                                      uint32_t tmem_base, uint32_t scales) {
    volatile int *abort_flag = &ctl->abort_flag;
    const int steps = g.taps * g.chunks;
    const bool leader = elect_one();
    const uint64_t a_hi = (uint64_t)g.a_desc_hi << 32, b_hi = (uint64_t)g.b_desc_hi << 32;
    const uint32_t lbo = (uint32_t)g.pitch, row_units = g.swizzled ? 8u : 1u;
    const uint32_t a_lo0 = ((smem_u32(operand) >> 4) & 0x3FFF) | ((g.swizzled ? 1u : lbo) << 16);
    const uint32_t b_lo0 = ((b0 >> 4) & 0x3FFF) | (1u << 16), b_units = g.stage_bytes >> 4;
    int stage = WHO % g.n_stages, tap = WHO, done = WHO;
    uint32_t phase = 0;
    {
        // Block scales and an accumulator of zeros, a quadrant of tensor memory each: the issuers have nothing to do
        // yet, while every column of a pixel group waits for the one before (with four of the workers on it conv4
        // on 32 images took 15.1 us instead of 14.8 on one stream).
        const uint32_t quadrant = (uint32_t)(((kFirstIssuer + WHO) & 3) * 32) << 16;
        fill_scales(scales + quadrant, 16);
        fill_columns(tmem_base + quadrant, g.n_tile, 0u);
        fence_before();
        __syncwarp();
        if (leader) mbar_arrive(smem_u32(&ctl->cleared));
    }
    bool ok = warp_wait(smem_u32(&ctl->cleared), 0, abort_flag, g.error, 2, g.wait_ns);
    fence_after();
    for (int chunk = 0; ok && chunk < g.chunks; chunk++, tap -= g.taps) {
        // where the K chunk's instructions start, from the tap's first position and column
        uint32_t start[4];
        if (g.swizzled) {
#pragma unroll
            for (int k = 0; k < 4; k++) start[k] = (uint32_t)(chunk * g.pitch * 8 + 2 * k);
        } else {
            const int byte = chunk * g.kchunk;
            int pos = byte / g.icp, c = (byte - pos * g.icp) >> 4;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                start[k] = (uint32_t)c * lbo + (uint32_t)pos;
                c += 2;
                if (c >= g.columns) { c -= g.columns; pos++; }
                if (c >= g.columns) { c -= g.columns; pos++; }
            }
        }
        const int kk = chunk == g.chunks - 1 ? g.kk_last : g.kchunk >> 5;
        if (chunk < g.parts)
            ok = warp_wait(smem_u32(&ctl->packed[chunk]), 0, abort_flag, g.error, 9, g.wait_ns);
        int row = tap / g.tap_kw, kw = tap - row * g.tap_kw;
        for (; ok && tap < g.taps; tap += kIssuers, done += kIssuers) {
            ok = warp_wait(smem_u32(&ctl->full[stage]), phase, abort_flag, g.error, 3, g.wait_ns);
            if (!ok) break;
            if (leader) {
                const uint32_t at = a_lo0 + (uint32_t)(row * g.wp + kw) * row_units;
                const uint64_t bdesc = b_hi | (uint64_t)(b_lo0 + (uint32_t)stage * b_units);
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (k < kk)
                        mma_mxf4<false>(tmem_base, a_hi | (uint64_t)(at + start[k]),
                                        bdesc + (uint64_t)(2 * k), g.idesc, scales, 1u);
                // only a buffer that is loaded again has to be handed back
                if (done + g.n_stages < steps) commit(smem_u32(&ctl->empty[stage]));
            }
            __syncwarp();
            kw += kIssuers;
            while (kw >= g.tap_kw) { kw -= g.tap_kw; row++; }
            stage += kIssuers;
            if (stage >= g.n_stages) { stage -= g.n_stages; phase ^= 1u; }
        }
    }
    if (leader) {
        if (ok) commit(smem_u32(&ctl->acc_full));
        commit(smem_u32(&ctl->drain[WHO]));
    }
    // MMAs already issued finish before tensor memory is released: the epilogue's wait says so, unless
    // some role gave up, be it after this one is through
    mbar_wait_quiet(smem_u32(&ctl->drain[WHO]), 0, g.wait_ns);
    __syncwarp();
}

template <bool NHWC>
__global__ void __launch_bounds__(kThreads, 1)
conv_whole_kernel(const __grid_constant__ CUtensorMap map_b, const WholeArgs g) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *base = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    Control *ctl = (Control *)base;
    uint8_t *operand = base + kControlBytes;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int mt = (int)blockIdx.x / g.n_tiles, nt = (int)blockIdx.x - mt * g.n_tiles;
    volatile int *abort_flag = &ctl->abort_flag;

    const Tile tile(g, mt);
    if (threadIdx.x == 0) {
        for (int s = 0; s < g.n_stages; s++) {
            mbar_init(smem_u32(&ctl->full[s]), 1);
            mbar_init(smem_u32(&ctl->empty[s]), 1);
        }
        for (int i = 0; i < g.parts; i++)
            mbar_init(smem_u32(&ctl->packed[i]),
                      (uint32_t)(tile.groups * min(g.part_columns, g.columns - i * g.part_columns) +
                                 (blockIdx.x == 0 ? g.more_operand : 0)));
        mbar_init(smem_u32(&ctl->acc_full), (uint32_t)(kIssuers + (blockIdx.x == 0 ? g.more_commits : 0)));
        mbar_init(smem_u32(&ctl->cleared), 4);
        for (int i = 0; i < kIssuers; i++) mbar_init(smem_u32(&ctl->drain[i]), 1);
        ctl->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_b) : "memory");
    }
    if (warp == kFirstIssuer)
        for (int i = lane; i < kMaxTasks; i += 32) mbar_init(smem_u32(&ctl->turn[i]), 1);
    if (warp == 0) tmem_alloc(smem_u32(&ctl->tmem_base), g.tmem_cols);
    const int worker = warp - 1;
    const bool works = worker >= 0 && worker < kWorkers;
    float v[32];
    if (works) {
        // borders, absent channels and what a K chunk reaches past them are zero
        for (int i = (int)threadIdx.x - 32; i < g.planes * g.pitch; i += 32 * kWorkers)
            reinterpret_cast<uint4 *>(operand)[i] = make_uint4(0, 0, 0, 0);
        for (int i = (int)threadIdx.x - 32; i < g.rows; i += 32 * kWorkers) ctl->a[i] = 0.f;
        fence_async_smem();
        // the first loads fly while barriers and tensor memory are set up
        dependency_wait();
        if (worker < tile.tasks) load_task<NHWC>(g, tile, worker, lane, v);
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem_base = ctl->tmem_base, scales = tmem_base + g.tmem_cols - 16;
    dependency_release();

    const uint32_t b0 = smem_u32(base) + g.b_off;
    const int steps = g.taps * g.chunks;
    if (warp == 0) {
        // ---- filter tiles ---- (the kernel before may have written them; the workers waited for it before the
        // barrier above, so this returns at once)
        const bool leader = elect_one();
        dependency_wait();
        int stage = 0, sent = 0, tap = 0, chunk = 0;
        uint32_t phase = 0;
        bool ok = true;
        for (; sent < steps; sent++) {
            ok = warp_wait(smem_u32(&ctl->empty[stage]), phase ^ 1, abort_flag, g.error, 1, g.wait_ns);
            if (!ok) break;
            if (leader) {
                const uint32_t bar = smem_u32(&ctl->full[stage]);
                mbar_expect_tx(bar, g.b_bytes);
                tma_load_2d(b0 + (uint32_t)stage * g.stage_bytes, &map_b, chunk * g.kchunk,
                            tap * g.ocp16 + nt * g.n_tile, bar);
            }
            __syncwarp();
            if (++stage == g.n_stages) { stage = 0; phase ^= 1; }
            if (++tap == g.taps) { tap = 0; chunk++; }
        }
        // Loads in flight land in this CTA's shared memory, which it may not leave before, whoever gave up
        // and when.
        for (int i = max(0, sent - g.n_stages); i < sent; i++)
            mbar_wait_quiet(smem_u32(&ctl->full[i % g.n_stages]), (uint32_t)(i / g.n_stages) & 1u, g.wait_ns);
    } else if (warp == kFirstIssuer) {
        issue<0>(g, ctl, operand, b0, tmem_base, scales);
    } else if (warp == kFirstIssuer + 1) {
        issue<1>(g, ctl, operand, b0, tmem_base, scales);
    } else if (warp == kFirstIssuer + 2) {
        issue<2>(g, ctl, operand, b0, tmem_base, scales);
    } else if (warp == kFirstIssuer + 3) {
        issue<3>(g, ctl, operand, b0, tmem_base, scales);
    } else {
        // ---- workers: pack, then drain the accumulator ----
        const int oc0 = nt * g.n_tile;
        for (int i = (int)threadIdx.x - 32; i < g.n_tile; i += 32 * kWorkers)
            ctl->alpha[i] = oc0 + i < g.oc ? __ldg(g.alpha + oc0 + i) : 0.f;
        bool ok = true;
        for (int t = worker; ok && t < tile.tasks; t += kWorkers) {
            if (t != worker) load_task<NHWC>(g, tile, t, lane, v);
            ok = finish_task<NHWC>(g, ctl, operand, tile, nt == 0, t, lane, v);
        }
        bar_sync(1, 32 * kWorkers);  // every mean |x| is in place
        const int quad = warp & 3, cgroup = worker >> 2, cgroups = kWorkers / 4;
        const int at = quad * 32 + lane;
        const uint32_t q = (uint32_t)(mt * BM + at);
        const int n = (int)g.by_frame(q), rem = (int)q - n * (g.hp * g.wp);
        const int oh = (int)g.by_wp((uint32_t)rem), ow = rem - oh * g.wp;
        const bool valid = q < (uint32_t)g.q_total && oh < g.oh && ow < g.ow;
        const long ohw = (long)g.oh * g.ow;
        const int r = oh * g.ow + ow;
        const long pix = (long)n * ohw + r;
        // K = box filter of the mean |x|, each term scaled by 1/(KH*KW), added in upstream's tap order
        // (src/bcast_calculate_k.cpp:69-85); borders are zeros, and adding +0 to a sum of terms that
        // are not negative changes nothing
        float kk = 0.f;
        for (int i = 0; i < g.kh; i++)
            for (int j = 0; j < g.kw; j++)
                kk = __fadd_rn(kk, __fmul_rn(ctl->a[at + i * g.wp + j], g.inv_khw));
        if (valid && cgroup == 0 && nt == 0) g.k[pix] = kk;
        ok = ok && mbar_wait(smem_u32(&ctl->acc_full), 0, abort_flag, g.error, 4, g.wait_ns);
        ok = __all_sync(0xffffffffu, ok);
        if (ok) {
            fence_after();
            const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16);
            const StoreAt to = {g.dst, g.oc, oc0, min(g.n_tile, g.oc - oc0), n, r, pix, ohw, kk, valid};
            if (!g.dst_nhwc)
                store_nchw(to, ctl->alpha, g.n_tile, taddr, cgroup, cgroups);
            else if ((g.oc & 3) == 0 && ((uintptr_t)g.dst & 15) == 0)
                store_nhwc(to, ctl->alpha, g.n_tile, taddr, cgroup, cgroups);
            else
                store_nhwc_odd(to, ctl->alpha, g.n_tile, taddr, cgroup, cgroups);
        }
    }
    fence_before();
    __syncthreads();
    if (warp == 0) {
        fence_after();
        tmem_free(tmem_base, g.tmem_cols);
    }
}

// Operand geometry and shared memory of a layer's tiles; false if the layer is not one for this kernel.
bool whole_shape(const Plan &p, WholeArgs *g, size_t *smem) {
    if (p.family != kTcgen05 || p.img || p.fold || !p.frame_walk || p.mb < 1 || p.q_total < 1) return false;
    const long m_tiles = (p.q_total + BM - 1) / BM;
    // Filter tiles as wide as they can be, so that a layer is packed once where that will do: conv4 on 32
    // images takes 5.8 us a pass among others in 49 tiles of 256 filters, 8.9 in 98 of 128 (alone 28.1 and
    // 25.3). Narrower while the tiles fill no more than a third of the SMs: filters and results of a tile
    // take less time then and nothing else wants the SMs (one image, 2 tiles of 256 -> 16 of 32: 12.0 ->
    // 11.7 us on one stream).
    g->n_tile = div_up_i(div_up_i(p.oc, div_up_i(p.oc, 256)), 16) * 16;
    while (g->n_tile / 2 >= 32 && m_tiles * div_up_i(p.oc, (g->n_tile / 2 + 15) / 16 * 16) <= sm_count() / 3)
        g->n_tile = (g->n_tile / 2 + 15) / 16 * 16;
    g->n_tiles = div_up_i(p.oc, g->n_tile);
    if (m_tiles * g->n_tiles > sm_count() || 4L * p.mb * p.ic * p.ih * p.iw >= 1L << 32) return false;
    g->rows = BM + (p.kh - 1) * p.wp + p.kw - 1;
    g->columns = p.row_bytes / 16;
    g->odd = p.cat && (g->columns & 1);
    g->planes = g->columns + (g->columns & 1);
    if (!p.cat && p.kchunk == 128) g->planes = (g->columns + 7) & ~7;
    g->pitch = (g->rows + 7 + 8) & ~7;
    g->swizzled = !p.cat && p.kchunk == 128;
    const int tap_bytes = p.cat ? p.kw * p.icp : p.row_bytes;
    g->tap_kw = p.cat ? 1 : p.kw;
    g->taps = p.kh * g->tap_kw;
    g->kchunk = p.kchunk;
    g->chunks = div_up_i(tap_bytes, p.kchunk);
    const int values = p.cat ? 2 * (p.kw - 1) * p.icp + p.ic : p.ic;
    g->kk_last = (values - (g->chunks - 1) * 2 * p.kchunk + 63) / 64;
    g->part_columns = p.cat ? g->columns : p.kchunk / 16;
    g->parts = div_up_i(g->columns, g->part_columns);
    if (g->rows > kMaxRows || g->parts > kMaxParts || g->pitch >= 1 << 14) return false;
    g->b_bytes = (uint32_t)(g->n_tile * p.kchunk);
    g->stage_bytes = (g->b_bytes + 1023u) & ~1023u;
    // a group of pixels is 32, or fewer if borders are in between
    const int tasks = div_up_i(g->rows, 32) * g->columns;
    if (tasks > kMaxTasks) return false;
    // Not where pixels are packed more than 1.6 times (by neighbouring tiles, in halos, and by each filter tile)
    // and the tiles, dealt to all SMs, come to more than 5.5 us: the general path does that
    // work once, and with passes on several streams hides its second launch under it. The time of two launches
    // over that of one, geometric means: of 275 layers that ran here before (drawn from 1 to 256 images, 16 to
    // 512 channels and filters, 6 to 56 pixels) among others 1.33, on one stream 1.22, waited for 1.04; of the
    // eleven that this rule takes out 0.90, 1.06 and 0.95; 384 filters on 256 channels of 13 x 13, 48 images,
    // 0.75, 1.03 and 0.93. What stays slower alone is few tiles of many filters, which leave most SMs idle:
    // conv4 on 16 to 48 images 1.2 to 1.4 among others, 0.82 to 0.99 on one stream, 0.87 to 0.95 waited for.
    // The formula still gives a tile of conv4 what it takes (14900 cycles on one image, 26400 on 32; measured 14600
    // and 26200), but those means are from before the packing got shorter, and the line is behind that: of 60 layers
    // just beyond it (up to 14000 instead of 10450) one launch would now be 1.17 times as fast as two on one stream
    // (0.84 to 1.49), 1.05 among others (0.81 to 1.36).
    const long mma_cycles = (long)g->taps * ((g->chunks - 1) * (p.kchunk / 32) + g->kk_last) * g->n_tile / 2;
    const long tile_cycles = 1200 + 4000 * div_up_i(tasks, kWorkers) + mma_cycles * 11 / 10 + 22 * g->n_tile;
    const bool repeats = 10L * g->n_tiles * g->rows > 16L * BM;
    if (repeats && m_tiles * g->n_tiles * tile_cycles > 10450L * sm_count()) return false;  // at 1.9 GHz
    const size_t operand = (size_t)g->planes * g->pitch * 16;
    g->b_off = (uint32_t)((kControlBytes + operand + 1023) & ~(size_t)1023);
    const size_t room = 227 * 1024 - 1024, want = 128 * 1024;
    if (g->b_off + (size_t)g->stage_bytes > room) return false;
    // The floats that are being loaded pass through the L1, which is what shared memory leaves of it.
    int stages = g->b_off < want ? (int)((want - g->b_off) / g->stage_bytes) : 0;
    if (stages < 4) stages = 4;
    const int all = g->taps * g->chunks;
    if (stages > kMaxStages) stages = kMaxStages;
    if (stages > all) stages = all;
    while (g->b_off + (size_t)stages * g->stage_bytes > room) stages--;
    // A buffer that comes round has to come to the same issuer: to one that skips a phase of its barrier,
    // a buffer whose previous load has not landed looks full.
    if (stages < all) stages &= ~(kIssuers - 1);
    if (stages < 1) return false;
    g->n_stages = stages;
    *smem = 1024 + g->b_off + (size_t)g->n_stages * g->stage_bytes;
    return true;
}

}  // namespace

bool whole_ok(const Plan &p) {
    WholeArgs g;
    size_t smem;
    return whole_shape(p, &g, &smem);
}

cudaError_t launch_conv_whole(const Plan &p, const float *src, void *bin_src, const void *bin_w,
                              const float *alpha, float *a, float *k, float *dst, int *error_word,
                              cudaStream_t s, const ConvSelfTest *test) {
    WholeArgs g;
    size_t smem;
    if (!whole_shape(p, &g, &smem)) return cudaErrorNotSupported;
    g.src = src; g.alpha = alpha; g.bin = (uint8_t *)bin_src; g.a = a; g.k = k; g.dst = dst;
    g.error = error_word;
    g.inv_ic = p.inv_ic; g.inv_khw = p.inv_khw;
    g.ic = p.ic; g.hw = p.ih * p.iw; g.ih = p.ih; g.iw = p.iw; g.n_px = p.mb * p.ih * p.iw;
    g.vec = p.src_nhwc && p.ic % 4 == 0 && (reinterpret_cast<uintptr_t>(src) & 15) == 0;
    g.wp = p.wp; g.hp = p.hp; g.lead = p.lead; g.q_total = (int)p.q_total; g.icp = p.icp;
    g.kh = p.kh; g.kw = p.kw; g.oh = p.oh; g.ow = p.ow; g.oc = p.oc; g.dst_nhwc = p.dst_nhwc;
    g.ocp16 = p.ocp16;
    g.idesc = mxf4_idesc(BM, (uint32_t)g.n_tile);
    const uint32_t layout = p.kchunk == 128 ? 2u : p.kchunk == 64 ? 4u : 6u;
    g.b_desc_hi = ((uint32_t)(8 * p.kchunk) >> 4) | (1u << 14) | (layout << 29);
    // columns: 128 bytes from eight positions to the next, no swizzle
    g.a_desc_hi = g.swizzled ? g.b_desc_hi : 8u | (1u << 14);
    g.tmem_cols = 32;
    while (g.tmem_cols < (uint32_t)g.n_tile + 16) g.tmem_cols *= 2;
    g.wait_ns = test && test->wait_ns ? test->wait_ns : 2000000000ull;
    g.turn_step = test && test->drop_turn ? 0 : 1;
    g.more_commits = test ? test->drop_commit : 0;
    g.more_operand = test ? test->drop_operand : 0;
    g.by_frame = FastDiv((uint32_t)(p.hp * p.wp)); g.by_wp = FastDiv((uint32_t)p.wp);
    g.by_hw = FastDiv((uint32_t)g.hw); g.by_iw = FastDiv((uint32_t)p.iw);
    CUtensorMap map_b;
    const int tap_bytes = p.cat ? p.kw * p.icp : p.row_bytes;
    if (!encode_bytes_2d(&map_b, bin_w, (uint64_t)g.taps * p.ocp16, (uint64_t)tap_bytes,
                         (uint64_t)p.tap_pitch, (uint32_t)p.kchunk, (uint32_t)g.n_tile))
        return cudaErrorNotSupported;
    int dev = 0;
    cudaGetDevice(&dev);
    static std::atomic<bool> opted_in[64][2];
    auto kernel = p.src_nhwc ? conv_whole_kernel<true> : conv_whole_kernel<false>;
    std::atomic<bool> &done = opted_in[dev & 63][p.src_nhwc];
    if (!done.load(std::memory_order_acquire)) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 58);
        if (e != cudaSuccess) return e;
        done.store(true, std::memory_order_release);
    }
    note_launch();
    const int m_tiles = (int)((p.q_total + BM - 1) / BM);
    return launch_overlapped(kernel, dim3(m_tiles * g.n_tiles), dim3(kThreads), smem, s, 1,
                             map_b, g);
}

}  // namespace xb200
