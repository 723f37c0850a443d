// Binary convolution as an implicit GEMM on the 5th-generation tensor cores.
//
// Operands are 4-bit floats, +-1 (0 where a channel, a filter or an image border does not exist),
// and sums of them are exact in fp32 below 2^24 (plan.cpp sees to that), so the accumulator is the
// signed agreement count S of upstream's kernel
// (src/default/bcast_convolution_default.cpp:60-103) exactly: products of absent operands are 0,
// which is upstream's "skip the tap" (:71-72) and its op_c correction (:102) in one. Against the
// 8-bit integer kind the tensor pipe does twice the work per cycle on half the operand bytes.
//
//   D[position][filter] += A[position + shift(tap)][channel] * B[tap][filter][channel]
//
// The activations live on a zero frame (plan.hpp) on which every filter tap is a constant row
// shift, so the A tile of a tap is a plain 2-D TMA box at a shifted row; no im2col buffer exists.
// Positions on the frame border are computed and dropped by the epilogue.
//
// One CTA per SM, persistent over (position tile, filter tile) pairs:
//   warp 0      an elected lane issues TMA loads (cp.async.bulk.tensor.2d, each CTA fetching its own
//               tiles) into a ring of shared-memory buffers; completion is counted on an
//               mbarrier per buffer
//   warp 1      allocates tensor memory; an elected lane issues tcgen05.mma.kind::mxf4 (M=128,
//               N<=256, K=64 per instruction) into one of two to four accumulators in tensor
//               memory, and tcgen05.commit hands buffers back / accumulators on
//   warp 18     a second MMA issuer; the two take alternate ring buffers
//   warps 2-17  epilogue: tcgen05.ld the accumulator (a warp owns 32 TMEM lanes = 32 positions and a
//               share of the columns), scale by alpha[filter] * K[position] in upstream's order
//               and store; runs under the next tiles' MMAs thanks to the other accumulators.
//               (In pairs with long tiles 2-9, and the second issuer 10.)
//
// Layers of more than one round of tiles run as clusters of two CTAs on tcgen05 cta_group::2:
// the pair shares a tile of 256 positions x N filters, each CTA loads its own 128 positions and
// half of the filter tile, the leader issues M = 256 instructions for both, and each CTA's
// epilogue drains its own tensor memory. A pair loads a position tile only once per filter row and
// channel chunk, with a halo of the positions that follow it, and the taps of the row read that
// tile at row offsets (producer_halo / mma_role_halo); filters that fit are loaded once and stay
// (mma_role_resident), in layers of few channels beside position tiles that serve all taps of the
// filter (mma_role_planes). Where the positions of all filter rows are one box, a position tile is
// loaded once a chunk for all of them, beside resident filters (mma_role_block) and streamed ones (producer_halo
// with g.block). What bounds a tile is the tensor pipe (128 cycles per MMA of 256 filters)
// or, when its loads share the way to L2 with the stores of the tile before it, those: AlexNet conv4
// on 256 images, with 256 streamed filters a tile, took 8200 cycles a tile without the other's stores and 10500
// with them (pipe: 6900); it has 128 resident ones now.
//
// The epilogue has three forms: floats in NCHW (a warp store is one contiguous run of a filter
// plane), floats in NHWC (a thread owns whole 32-byte sectors and writes them with 256-bit
// stores), and, for chained layers, no floats at all: the sign of every result goes into the next
// layer's frame and sum |result| into its mean-|x| map (ChainTarget in kernels.cuh).
//
// Every wait on an mbarrier is bounded in time: when the bound is hit the kernel records where
// in *error, every role winds down, copies in flight are waited for (again bounded), tensor
// memory is released and the kernel returns.
#include <cuda.h>

#include <atomic>
#include <cstddef>
#include <cstdlib>

#include "conv_tile_args.cuh"
#include "kernels.cuh"
#include "tc_ptx.cuh"

namespace xb200 {

namespace {

using namespace tc;

constexpr int BM = 128;            // positions per tile = UMMA M = TMEM lanes
constexpr int kMaxStages = 8;       // ring buffers: as many as fit, at most this
constexpr int kEpiWarps = 16;       // epilogue warps: 4 TMEM lane quadrants x column groups;
constexpr int kFewEpiWarps = 8;     // in pairs whose tiles are long (launch_conv_tcgen05)
// Tensor memory: two to four accumulators of n_tile columns and, in the last 16 columns, the block
// scales. 2 x 256 + 16 is more than the 512 there are, so accumulators of 256 columns share 16 of them
// (the last of the first = the first of the second): the epilogue empties those before anything
// else and says so (Control::shared_free), and the next tile's first MMA waits for it.
constexpr uint32_t kTmemCols = 512;
constexpr uint32_t kScaleCol = 496;
constexpr int kAccStep = 240;        // columns between the accumulators' starts, at most
constexpr int kMaxAcc = 4;
constexpr int kMaxASlots = 8;        // halo tiles in flight

// The second MMA issuer is a warp of its own, behind the epilogue's.
constexpr int threads_of(int epi_warps) { return 64 + 32 * epi_warps + 32; }

// ---- the kernel --------------------------------------------------------------------------------

constexpr int kAlphaSmem = 2048;  // filters whose alpha is staged in shared memory


struct __align__(16) Control {
    unsigned long long full[kMaxStages];
    unsigned long long empty[kMaxStages];
    unsigned long long acc_full[kMaxAcc];
    unsigned long long acc_empty[kMaxAcc];
    unsigned long long a_full[kMaxASlots];  // halo mode: a halo tile has landed / has been used up
    unsigned long long a_empty[kMaxASlots];
    unsigned long long started[kMaxAcc];  // two issuers: the tile's first MMAs (one overwrites) are done
    unsigned long long drain[2];
    unsigned long long shared_free;  // the columns both accumulators use have been read
    uint32_t tmem_base;
    int abort_flag;
    alignas(16) float alpha[kAlphaSmem];  // read with 16-byte loads
    float fold[2][4][kEpiWarps / 4][32];  // chained layers: per-warp partial sums of |y|
};
constexpr int kControlBytes = (sizeof(Control) + 1023) / 1024 * 1024;
static_assert(offsetof(Control, alpha) % 16 == 0, "alpha is read as float4");

// Which tile a CTA (PAIR: a pair of CTAs) works on in its it-th round. Default: tiles are dealt
// round-robin with the filter tile as the fast index. n_inner: pixel tiles are dealt round-robin
// and a CTA walks all filter tiles of its pixel tile back to back (so that per-pixel state can be
// carried across them in registers). A pair's tile is two neighbouring pixel tiles, one per CTA.
template <bool PAIR>
struct Deal {
    int unit, units, m_units;
    __device__ __forceinline__ Deal(const TcArgs &g)
        : unit(PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x),
          units(PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x),
          m_units(PAIR ? (g.m_tiles + 1) >> 1 : g.m_tiles) {}
    __device__ __forceinline__ int rounds(const TcArgs &g) const {
        if (g.n_inner) {
            const int mine = (m_units - unit + units - 1) / units;
            return mine > 0 ? mine * g.n_tiles : 0;
        }
        return (m_units * g.n_tiles - unit + units - 1) / units;
    }
    // mt = pixel tile of this CTA
    __device__ __forceinline__ void at(const TcArgs &g, int it, int &mt, int &nt) const {
        int mu;
        if (g.n_inner) {
            const int r = it / g.n_tiles;
            nt = it - r * g.n_tiles;
            mu = unit + r * units;
        } else {
            const int tile = unit + it * units;
            mu = tile / g.n_tiles;
            nt = tile - mu * g.n_tiles;
        }
        mt = PAIR ? 2 * mu + (int)(blockIdx.x & 1) : mu;
    }
};

// ---- epilogue role ---------------------------------------------------------------------------------
// Warp w may touch TMEM lanes [32*(w%4), 32*(w%4)+32); several warps share a quadrant and split
// its columns between them.
// EMITS: chained layers' results, and no others, on pairs. (On single CTAs both kinds have one kernel: the layers
// of a chain then find its instructions in the caches. Two kernels: three layers on 64 images 23.0 -> 24.0 us.)
template <bool PAIR, int EPI, bool EMITS>
__device__ __forceinline__ void epilogue_role(const TcArgs &g, Control *ctl, uint32_t tmem_base,
                                              int warp, int lane, bool alpha_in_smem) {
    volatile int *abort_flag = &ctl->abort_flag;
    const Deal<PAIR> deal(g);
    const int rounds = deal.rounds(g);
    // a pair's accumulators are handed back on the leader's barriers
    const uint32_t acc_empty0 =
        PAIR ? mapa(smem_u32(&ctl->acc_empty[0]), 0) : smem_u32(&ctl->acc_empty[0]);
    const uint32_t shared_free0 =
        PAIR ? mapa(smem_u32(&ctl->shared_free), 0) : smem_u32(&ctl->shared_free);
    // Several warps share a quadrant and split its columns between them. The warps form
    // one, two or four teams that take the tiles in turn: what a tile costs an epilogue warp is
    // mostly latency (its pixel's K, the accumulator's barrier, the loads from tensor memory, the
    // stores going out), and tiles of different teams overlap it.
    const int quad = warp & 3;
    const int cgroups = EPI / 4 / g.teams, team = (warp - 2) / (4 * cgroups);
    const int cgroup = ((warp - 2) >> 2) - team * cgroups;
    const int frame = g.hp * g.wp;
    const long ohw = (long)g.oh * g.ow;
    const bool emits = EMITS || (!PAIR && g.emit_bin);
    bool ok = true;   // false once a wait ran out somewhere in the CTA
    float run = 0.f;  // chained layers: running sum of |y| over the filter tiles of a pixel
    for (int it = team; it < rounds; it += g.teams) {
        int mt, nt;
        deal.at(g, it, mt, nt);
        const int use = (int)g.by_acc((uint32_t)it), b = it - use * g.n_acc;
        const uint32_t acc_phase = use & 1;
        const uint32_t q = (uint32_t)mt * BM + quad * 32 + lane;
        const int n = (int)g.by_frame(q);
        const uint32_t rem = q - (uint32_t)n * (uint32_t)frame;
        const int oh = (int)g.by_wp(rem), ow = (int)rem - oh * g.wp;
        const bool valid = q < (uint32_t)g.q_total && oh < g.oh && ow < g.ow;
        const int r = oh * g.ow + ow;
        const long pix = (long)n * ohw + r;
        float kk = 0.f;
        // chained layers: K scales a pixel's mean |x|, which one column group writes after the last filter tile
        if (valid && !g.sums && (!emits || (cgroup == 0 && nt == g.n_tiles - 1))) {
            if (g.kmap) {
                kk = __ldg(g.kmap + pix);
            } else {
                // K = box filter of A over the taps inside the image, each term scaled by
                // 1/(KH*KW), added in upstream's tap order (src/bcast_calculate_k.cpp:69-85)
                const float *img = g.amap + (long)n * g.ih * g.iw;
                for (int i = 0; i < g.kh; i++) {
                    const int y = oh - g.ph + i;
                    if (y < 0 || y >= g.ih) continue;
                    for (int j = 0; j < g.kw; j++) {
                        const int x = ow - g.pw + j;
                        if (x < 0 || x >= g.iw) continue;
                        kk = __fadd_rn(kk, __fmul_rn(__ldg(img + y * g.iw + x), g.inv_khw));
                    }
                }
                if (g.kmap_out && cgroup == 0 && (emits || nt == 0)) g.kmap_out[pix] = kk;
            }
        }
        const int oc0 = nt * g.n_tile;
        const int n_valid = min(g.n_tile, g.oc - oc0);  // real filters in this tile
        if (ok)
            ok = mbar_wait(smem_u32(&ctl->acc_full[b]), acc_phase, abort_flag, g.error, 4,
                           g.wait_ns);
        ok = __all_sync(0xffffffffu, ok);  // tcgen05.ld below needs the whole warp
        if (!ok) {
            // Given up: touch nothing any more. The chained epilogue's warps of a quadrant meet
            // on a named barrier once per tile; a warp that has given up keeps that appointment
            // so that one that has not (yet) cannot be left waiting there.
            if (emits) {
                bar_sync(1 + quad, 32 * (EPI / 4));
                continue;
            }
            break;
        }
        fence_after();
        const uint32_t taddr = tmem_base + ((uint32_t)(quad * 32) << 16) + (uint32_t)b * g.acc_step;
        // the warp that owns the columns shared with the other accumulator reads them first
        const bool shared = g.shared_cols && cgroup == (b ? 0 : cgroups - 1);
        const bool reverse = shared && b == 0;
        auto columns_read = [&](int step) {
            if (!shared || step != 0) return;
            fence_before();
            __syncwarp();
            if (lane == 0) {
                if (PAIR) mbar_arrive_cluster(shared_free0);
                else mbar_arrive(shared_free0);
            }
        };
        if (emits) {
            // Chained layers: y = (S * alpha) * K is not stored. alpha and K are never negative,
            // so the sign bit of y is the sign bit of S: it goes straight into the next layer's
            // frame (filters past the last one 0). |y| summed over the filters and divided by
            // their number is that layer's mean-|x| map; K is common to a pixel, so the sum runs
            // over |S| * alpha and is scaled once at the end. A thread owns one pixel and 32
            // neighbouring filters = 16 contiguous bytes of the frame.
            const float *al = alpha_in_smem ? ctl->alpha + oc0 : g.alpha + oc0;
            uint8_t *row = g.emit_bin +
                           ((long)g.e_lead + ((long)n * g.e_hp + oh) * g.e_wp + ow) * g.e_icp +
                           oc0 / 2;
            const int room = g.e_icp - oc0 / 2;  // bytes of the row from here on
            float part = 0.f;
            // The partial sum is added up in ascending order whichever accumulator the tile is in:
            // shared columns at the end (the last 16 of 256) are fetched first and kept.
            uint32_t kept[16];
            if (reverse) {
                ld16(taddr + (uint32_t)g.n_tile - 16u, kept);
                wait_ld();
                columns_read(0);
            }
            for (int c0 = 32 * cgroup; c0 < g.n_tile; c0 += 32 * cgroups) {
                uint32_t v[32];
                const int width = g.n_tile - c0 >= 32 ? 32 : 16;
                if (reverse && c0 + 32 == g.n_tile) {
                    ld16(taddr + (uint32_t)c0, v);
#pragma unroll
                    for (int j = 0; j < 16; j++) v[16 + j] = kept[j];
                } else if (width == 32) {
                    ld32(taddr + (uint32_t)c0, v);
                } else {
#pragma unroll
                    for (int j = 16; j < 32; j++) v[j] = 0;
                    ld16(taddr + (uint32_t)c0, v);
                }
                wait_ld();
                if (!reverse) columns_read(c0 == 32 * cgroup ? 0 : 1);
                if (valid) {
                    const int lim = min(n_valid - c0, width);
                    uint32_t w[4];
                    // a sum of zero counts as positive, whatever sign the adder gave it
#pragma unroll
                    for (int j = 0; j < 32; j++)
                        v[j] = __float_as_uint(__fadd_rn(__uint_as_float(v[j]), 0.f));
#pragma unroll
                    for (int j = 0; j < 4; j++)
                        w[j] = first_nibbles(sign_nibbles(v + 8 * j), lim - 8 * j);
                    if (alpha_in_smem && lim >= 32) {
                        const float4 *a4 = reinterpret_cast<const float4 *>(al + c0);
#pragma unroll
                        for (int j = 0; j < 32; j += 4) {
                            const float4 a = a4[j >> 2];
                            part = fmaf(fabsf(__uint_as_float(v[j])), a.x, part);
                            part = fmaf(fabsf(__uint_as_float(v[j + 1])), a.y, part);
                            part = fmaf(fabsf(__uint_as_float(v[j + 2])), a.z, part);
                            part = fmaf(fabsf(__uint_as_float(v[j + 3])), a.w, part);
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; j++)
                            if (j < lim) part = fmaf(fabsf(__uint_as_float(v[j])), al[c0 + j], part);
                    }
                    // n_tile is a multiple of 16: a thread's bytes start on 8, often on 16
                    uint8_t *o = row + c0 / 2;
                    if (width == 32 && c0 / 2 + 16 <= room && (oc0 & 31) == 0) {
                        *reinterpret_cast<uint4 *>(o) = make_uint4(w[0], w[1], w[2], w[3]);
                    } else {
                        if (c0 / 2 + 8 <= room) *reinterpret_cast<uint2 *>(o) = make_uint2(w[0], w[1]);
                        if (width == 32 && c0 / 2 + 16 <= room)
                            *reinterpret_cast<uint2 *>(o + 8) = make_uint2(w[2], w[3]);
                    }
                }
            }
            // Fold the column groups' partial sums in a fixed order (group 0, 1, 2, 3, then the
            // next filter tile), so the map is reproducible; the four warps of a lane quadrant
            // meet on a named barrier of their own.
            ctl->fold[it & 1][quad][cgroup][lane] = part;
            bar_sync(1 + quad, 32 * (EPI / 4));
            if (cgroup == 0) {
                if (nt == 0) run = 0.f;
#pragma unroll
                for (int c = 0; c < EPI / 4; c++)
                    run = __fadd_rn(run, ctl->fold[it & 1][quad][c][lane]);
                if (nt == g.n_tiles - 1 && valid)
                    g.emit_a[pix] = __fmul_rn(__fmul_rn(run, kk), g.e_inv_ic);
            }
        } else if (!g.sums && !g.dst_nhwc) {
            // NCHW floats: for one filter the 32 lanes hold 32 neighbouring pixels, so a
            // store instruction writes one contiguous run.
            float *out = g.dst + ((long)n * g.oc + oc0) * ohw + r;
            const float *al = alpha_in_smem ? ctl->alpha + oc0 : g.alpha + oc0;
            const int steps = (g.n_tile - 32 * cgroup + 32 * cgroups - 1) / (32 * cgroups);
            for (int i = 0; i < steps; i++) {
                const int c0 = 32 * (cgroup + cgroups * (reverse ? steps - 1 - i : i));
                uint32_t v[32];
                if (c0 + 32 <= g.n_tile) {
                    ld32(taddr + (uint32_t)c0, v);
                } else {  // N is a multiple of 16, not always of 32
                    ld16(taddr + (uint32_t)c0, v);
                }
                wait_ld();
                columns_read(i);
                if (valid) {
                    const int lim = n_valid - c0;
                    float *o = out + (long)c0 * ohw;
                    if (alpha_in_smem && lim >= 32) {
                        // full group: alpha by 16-byte shared loads, one running pointer
                        const float4 *a4 = reinterpret_cast<const float4 *>(al + c0);
#pragma unroll
                        for (int j = 0; j < 32; j += 4) {
                            const float4 a = a4[j >> 2];
                            // streaming stores: the result is not read again by this library,
                            // and lines that leave L2 while this kernel runs (which needs little
                            // of HBM) do not have to leave it under the next, bandwidth-bound pass
                            __stcs(o, scaled(v[j], a.x, kk));
                            __stcs(o + ohw, scaled(v[j + 1], a.y, kk));
                            __stcs(o + 2 * ohw, scaled(v[j + 2], a.z, kk));
                            __stcs(o + 3 * ohw, scaled(v[j + 3], a.w, kk));
                            o += 4 * ohw;
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; j++)
                            if (j < lim) __stcs(o + (long)j * ohw, scaled(v[j], al[c0 + j], kk));
                    }
                }
            }
        } else if (!g.sums && g.dst_nhwc && (g.oc & 3) == 0 && ((uintptr_t)g.dst & 15) == 0) {
            // NHWC floats: a thread owns one pixel and 16 neighbouring filters at a time, which
            // are contiguous in the result: four 16-byte stores. (A result that starts between two
            // 16-byte boundaries, such as a view into a buffer, is stored float by float below.)
            float *out = g.dst + pix * g.oc + oc0;
            const float *al = alpha_in_smem ? ctl->alpha + oc0 : g.alpha + oc0;
            // 256-bit stores need 32-byte alignment: rows and tiles that are multiples of 8
            // floats on a result buffer aligned likewise
            const bool wide = (g.oc & 7) == 0 && (oc0 & 7) == 0 && ((uintptr_t)g.dst & 31) == 0;
            const int steps = (g.n_tile - 16 * cgroup + 16 * cgroups - 1) / (16 * cgroups);
            for (int i = 0; i < steps; i++) {
                const int c0 = 16 * (cgroup + cgroups * (reverse ? steps - 1 - i : i));
                uint32_t v[16];
                ld16(taddr + (uint32_t)c0, v);
                wait_ld();
                columns_read(i);
                if (valid && wide && c0 + 16 <= n_valid) {
                    // 16 results = two whole 32-byte sectors, one 256-bit store each
                    float x[16];
#pragma unroll
                    for (int j = 0; j < 16; j++)
                        x[j] = scaled(v[j], al[c0 + j], kk);
#pragma unroll
                    for (int h = 0; h < 16; h += 8)
                        asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                                     ::"l"(out + c0 + h), "f"(x[h]), "f"(x[h + 1]), "f"(x[h + 2]),
                                       "f"(x[h + 3]), "f"(x[h + 4]), "f"(x[h + 5]), "f"(x[h + 6]),
                                       "f"(x[h + 7])
                                     : "memory");
                } else if (valid) {
#pragma unroll
                    for (int j = 0; j < 16; j += 4) {
                        if (c0 + j >= n_valid) break;  // oc and n_valid are multiples of 4
                        float4 x;
                        x.x = scaled(v[j], al[c0 + j], kk);
                        x.y = scaled(v[j + 1], al[c0 + j + 1], kk);
                        x.z = scaled(v[j + 2], al[c0 + j + 2], kk);
                        x.w = scaled(v[j + 3], al[c0 + j + 3], kk);
                        *reinterpret_cast<float4 *>(out + c0 + j) = x;
                    }
                }
            }
        } else {
            const int steps = (g.n_tile - 16 * cgroup + 16 * cgroups - 1) / (16 * cgroups);
            for (int i = 0; i < steps; i++) {
                const int c0 = 16 * (cgroup + cgroups * (reverse ? steps - 1 - i : i));
                uint32_t v[16];
                ld16(taddr + (uint32_t)c0, v);
                wait_ld();
                columns_read(i);
                if (valid) {
#pragma unroll
                    for (int j = 0; j < 16; j++) {
                        const int oc = oc0 + c0 + j;
                        if (oc >= g.oc) continue;
                        if (g.sums) {
                            g.sums[((long)n * g.oc + oc) * ohw + r] = (int)__uint_as_float(v[j]);
                        } else {
                            const float x = scaled(v[j], __ldg(g.alpha + oc), kk);
                            if (g.dst_nhwc) g.dst[pix * g.oc + oc] = x;
                            else g.dst[((long)n * g.oc + oc) * ohw + r] = x;
                        }
                    }
                }
            }
        }
        fence_before();
        if (PAIR) {
            // one arrival per warp: tcgen05.wait::ld is warp-wide, so every lane's reads are done
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(acc_empty0 + 8u * (uint32_t)b);
        } else {
            mbar_arrive(acc_empty0 + 8u * (uint32_t)b);
        }
    }
}

// ---- TMA producer role: position and filter tiles of a step in one ring buffer ---------------------
template <bool PAIR>
__device__ __forceinline__ void producer_ring(const TcArgs &g, Control *ctl,
                                              const CUtensorMap *map_a, const CUtensorMap *map_b,
                                              uint32_t stage0, uint32_t rank) {
    volatile int *abort_flag = &ctl->abort_flag;
    const bool leader = elect_one();
    const Deal<PAIR> deal(g);
    const int rounds = deal.rounds(g), ksteps = g.taps * g.chunks_per_tap;
    int stage = 0;
    uint32_t phase = 0;
    uint32_t armed = 0;  // bit s: stage s holds a load nobody is known to have consumed
    uint32_t armed_parity = 0;
    bool ok = true;
    // a pair counts both CTAs' bytes on the leader's barrier
    const uint32_t full_local = smem_u32(&ctl->full[0]);
    const uint32_t full0 = PAIR && rank != 0 ? mapa(full_local, 0) : full_local;
    const int b_rows = PAIR ? g.n_tile >> 1 : g.n_tile;  // filter rows this CTA loads
    for (int it = 0; ok && it < rounds; it++) {
        int mt, nt;
        deal.at(g, it, mt, nt);
        int row = g.lead + mt * BM - g.ph * g.wp - g.pw;  // tap (0,0)
        int brow = nt * g.n_tile + (int)rank * b_rows;
        int kw = 0, chunk = 0;
        for (int ks = 0; ks < ksteps; ks++) {
            const uint32_t ebar = smem_u32(&ctl->empty[stage]);
            ok = warp_wait(ebar, phase ^ 1, abort_flag, g.error, 1, g.wait_ns);
            if (!ok) break;
            armed &= ~(1u << stage);
            const uint32_t bar = full0 + 8u * (uint32_t)stage;
            const uint32_t sa = stage0 + (uint32_t)stage * g.stage_bytes;
            if (leader && PAIR) {
                if (rank == 0) mbar_expect_tx(bar, 2u * g.tx_bytes);  // bar is local here
                tma_load_2d_pair(sa, map_a, chunk * g.kchunk, row, bar);
                tma_load_2d_pair(sa + g.a_bytes, map_b, chunk * g.kchunk, brow, bar);
            } else if (leader) {
                mbar_expect_tx(bar, g.tx_bytes);
                tma_load_2d(sa, map_a, chunk * g.kchunk, row, bar);
                tma_load_2d(sa + g.a_bytes, map_b, chunk * g.kchunk, brow, bar);
            }
            armed |= 1u << stage;
            armed_parity = (armed_parity & ~(1u << stage)) | (phase << stage);
            if (++stage == g.n_stages) { stage = 0; phase ^= 1; }
            if (++chunk == g.chunks_per_tap) {  // next filter tap
                chunk = 0;
                brow += g.ocp16;
                if (++kw == g.tap_kw) { kw = 0; row += g.wp - (g.tap_kw - 1); }
                else row += 1;
            }
        }
    }
    if (rank == 0) {
        // Loads already issued land in this CTA's shared memory: wait for them (bounded) before
        // the CTA may exit. Whoever consumes them waits for them too, unless something gives up,
        // be it after this role is through. (The partner of a pair cannot wait on the leader's
        // barrier; it stays until the leader has got through this and both have met at the
        // cluster barrier at the end.)
        for (int s = 0; s < g.n_stages; s++)
            if (armed & (1u << s)) {
                mbar_wait_quiet(smem_u32(&ctl->full[s]), (armed_parity >> s) & 1u,
                                g.wait_ns);
            }
    }
}

// ---- MMA issuer role -----------------------------------------------------------------------------
// One lane feeds the tensor pipe; the instructions of a pipeline stage (KK tcgen05.mma and the
// tcgen05.commit that hands the stage back) cost that thread more cycles than the pipe needs for
// them unless N is 256. With two issuers the stages are dealt alternately (issuer i takes stages
// i, i+2, ... of the running stage sequence, which continues across tiles), each commits its own
// stages, and both commit to the accumulator's barrier (count 2) after their last stage of a
// tile: a commit covers the MMAs of the committing thread only. The sum is over integers, so the
// order in which the two threads' MMAs reach the pipe does not matter (that none of their sums is
// lost is an assumption about the pipe, which executes them one after the other, and not documented
// for several issuing threads; test_shared_accumulator_gpu.py watches it), except for the tile's
// first instruction, which overwrites the accumulator: its issuer waits for the epilogue to have
// drained the accumulator, and the other issuer waits until it has been executed (started[], a
// commit: nothing orders the MMAs of two threads that have only been issued). The ring has an even
// number of buffers then, so that a buffer always has the same issuer, which sees every phase of
// its barrier: to one that skips a phase, a buffer whose previous load has not landed looks full.
template <int KK, bool PAIR>
__device__ __forceinline__ void mma_role(const TcArgs &g, Control *ctl, uint32_t tmem_base,
                                         uint32_t stage0, int who) {
    volatile int *abort_flag = &ctl->abort_flag;
    const bool leader = elect_one();
    const int rounds = Deal<PAIR>(g).rounds(g);
    if (rounds == 0) return;
    const int ksteps = g.taps * g.chunks_per_tap;  // >= g.issuers (the launcher sees to it)
    const int n_iss = g.issuers;
    const uint64_t hi = (uint64_t)g.desc_hi << 32;
    const uint32_t a_lo0 = ((stage0 >> 4) & 0x3FFF) | (1u << 16);
    const uint32_t b_lo0 = (((stage0 + g.a_bytes) >> 4) & 0x3FFF) | (1u << 16);
    const uint32_t stage_units = g.stage_bytes >> 4;
    const uint32_t full0 = smem_u32(&ctl->full[0]), empty0 = smem_u32(&ctl->empty[0]);
    const int n_stages = g.n_stages;  // >= g.issuers
    int it = 0, ks = who, stage = who;
    // position of this thread's current stage among the chunks of its tap
    int chunk = who % g.chunks_per_tap;
    const int chunk_step = n_iss % g.chunks_per_tap;
    uint32_t phase = 0;
    bool ok = true, entered = false;
    int b = 0;  // the tile's accumulator and how often it has come round
    uint32_t acc_phase = 0;
    for (;;) {
        if (!entered) {
            if (ks == 0)
                ok = warp_wait(smem_u32(&ctl->acc_empty[b]), acc_phase ^ 1, abort_flag, g.error, 2,
                               g.wait_ns);
            else if (n_iss > 1)
                ok = warp_wait(smem_u32(&ctl->started[b]), acc_phase, abort_flag, g.error, 6,
                               g.wait_ns);
            if (ok && ks == 0 && g.shared_cols && it > 0)
                ok = warp_wait(smem_u32(&ctl->shared_free), (uint32_t)(it - 1) & 1u, abort_flag,
                               g.error, 7, g.wait_ns);
            if (!ok) break;
            fence_after();
            entered = true;
        }
        const uint32_t fbar = full0 + 8u * (uint32_t)stage;
        ok = warp_wait(fbar, phase, abort_flag, g.error, 3, g.wait_ns);
        if (!ok) break;
        const uint32_t d_tmem = tmem_base + (uint32_t)b * g.acc_step;
        const uint32_t desc_off = (uint32_t)stage * stage_units;
        const uint64_t adesc = hi | (uint64_t)(a_lo0 + desc_off);
        const uint64_t bdesc = hi | (uint64_t)(b_lo0 + desc_off);
        // slices of zero padding behind the last channel are not multiplied
        const int kk = chunk == g.chunks_per_tap - 1 ? g.kk_last : KK;
        if (leader) {
#pragma unroll
            for (int k = 0; k < KK; k++) {
                if (k < kk) {
                    mma_mxf4<PAIR>(d_tmem, adesc + (uint64_t)(2 * k), bdesc + (uint64_t)(2 * k),
                                   g.idesc, tmem_base + kScaleCol, (k == 0 && ks == 0) ? 0u : 1u);
                }
            }
            if (PAIR) commit_pair(empty0 + 8u * (uint32_t)stage);  // frees the stage in both CTAs
            else commit(empty0 + 8u * (uint32_t)stage);
            if (n_iss > 1 && ks == 0) {
                if (PAIR) commit_pair(smem_u32(&ctl->started[b]));
                else commit(smem_u32(&ctl->started[b]));
            }
        }
        __syncwarp();
        stage += n_iss;
        if (stage >= n_stages) { stage -= n_stages; phase ^= 1u; }
        chunk += chunk_step;
        if (chunk >= g.chunks_per_tap) chunk -= g.chunks_per_tap;
        ks += n_iss;
        if (ks >= ksteps) {  // this thread's share of the tile is issued
            ks -= ksteps;
            if (leader && !(g.drop_commit && it == 0 && blockIdx.x == 0)) {
                if (PAIR) commit_pair(smem_u32(&ctl->acc_full[b]));
                else commit(smem_u32(&ctl->acc_full[b]));
            }
            entered = false;
            if (++it >= rounds) break;
            if (++b == g.n_acc) { b = 0; acc_phase ^= 1u; }
        }
    }
    // Every MMA this thread has issued finishes before tensor memory is released. (The epilogue waits
    // for that as well, unless something gives up, be it after this role is through.)
    if (leader) {
        if (PAIR) commit_pair_here(smem_u32(&ctl->drain[who]));
        else commit(smem_u32(&ctl->drain[who]));
    }
    mbar_wait_quiet(smem_u32(&ctl->drain[who]), 0, g.wait_ns);
}

// ---- halo mode (pairs only): producer and MMA issuers ----------------------------------------------
// Step order inside a tile: filter row kh, channel chunk, filter column kw (the sums are integers:
// any order gives the same result). A group = the kw steps of one (kh, chunk): one halo tile of
// g.halo positions in slot G % n_a_slots (G counts groups across tiles), kw filter tiles in
// consecutive slots of the filter ring. With g.block a group is all kh kw steps of one chunk, whose
// halo tile holds the positions of all of them, so that the positions are loaded once a tile instead of
// once a filter row: the loads of a tile of conv3-sized layers go from 3 x 17 KB and 9 x 12 to 20 KB and
// 9 x 12 a chunk. A descriptor that starts r rows into a 128-byte-swizzled
// tile reads rows r .. r + 127 of it (the swizzle is a function of the shared-memory address), so
// tap kw of the group is the halo tile's descriptor advanced by kw rows.
__device__ __forceinline__ void producer_halo(const TcArgs &g, Control *ctl,
                                              const CUtensorMap *map_a, const CUtensorMap *map_b,
                                              uint32_t stage0, uint32_t rank) {
    volatile int *abort_flag = &ctl->abort_flag;
    const bool leader = elect_one();
    const Deal<true> deal(g);
    const int rounds = deal.rounds(g);
    const uint32_t full_l = smem_u32(&ctl->full[0]), afull_l = smem_u32(&ctl->a_full[0]);
    // a pair counts both CTAs' bytes on the leader's barriers
    const uint32_t full0 = rank != 0 ? mapa(full_l, 0) : full_l;
    const uint32_t afull0 = rank != 0 ? mapa(afull_l, 0) : afull_l;
    const uint32_t empty0 = smem_u32(&ctl->empty[0]), aempty0 = smem_u32(&ctl->a_empty[0]);
    const int b_rows = g.n_tile >> 1;
    const int kh_groups = g.block ? 1 : g.kh, group_taps = g.block ? g.taps : g.tap_kw;
    const uint32_t a_bytes = (uint32_t)g.halo * (uint32_t)g.kchunk;
    int sb = 0, sa = 0;
    uint32_t pb = 0, pa = 0;
    uint32_t armed_b = 0, parity_b = 0, armed_a = 0, parity_a = 0;
    bool ok = true;
    for (int it = 0; ok && it < rounds; it++) {
        int mt, nt;
        deal.at(g, it, mt, nt);
        const int row0 = g.lead + mt * BM - g.ph * g.wp - g.pw;  // tap (0,0)
        const int brow0 = nt * g.n_tile + (int)rank * b_rows;
        for (int kh = 0; ok && kh < kh_groups; kh++) {
            for (int chunk = 0; ok && chunk < g.chunks_per_tap; chunk++) {
                const uint32_t aebar = aempty0 + 8u * (uint32_t)sa;
                ok = warp_wait(aebar, pa ^ 1, abort_flag, g.error, 8, g.wait_ns);
                if (!ok) break;
                const uint32_t abar = afull0 + 8u * (uint32_t)sa;
                const uint32_t adst = stage0 + (uint32_t)sa * g.a_slot_bytes;
                // resident filters travel with the first round's position tiles
                const bool with_b = g.resident && it == 0;
                const uint32_t bytes =
                    2u * (a_bytes + (with_b ? (uint32_t)g.tap_kw * g.b_bytes : 0u));
                if (leader) {
                    if (rank == 0) mbar_expect_tx(abar, bytes);  // abar is local here
                    tma_load_2d_pair(adst, map_a, chunk * g.kchunk, row0 + kh * g.wp, abar);
                }
                armed_a |= 1u << sa;
                parity_a = (parity_a & ~(1u << sa)) | (pa << sa);
                if (++sa == g.n_a_slots) { sa = 0; pa ^= 1; }
                int brow = brow0 + kh * g.tap_kw * g.ocp16;
                if (g.resident) {
                    if (with_b && leader) {
                        uint32_t bdst = stage0 + g.b_ring_off +
                                        (uint32_t)((kh * g.chunks_per_tap + chunk) * g.tap_kw) *
                                            g.b_slot_bytes;
                        for (int kw = 0; kw < g.tap_kw; kw++) {
                            tma_load_2d_pair(bdst, map_b, chunk * g.kchunk, brow, abar);
                            brow += g.ocp16;
                            bdst += g.b_slot_bytes;
                        }
                    }
                    __syncwarp();
                    continue;
                }
                for (int tap = 0; tap < group_taps; tap++, brow += g.ocp16) {
                    const uint32_t ebar = empty0 + 8u * (uint32_t)sb;
                    ok = warp_wait(ebar, pb ^ 1, abort_flag, g.error, 1, g.wait_ns);
                    if (!ok) break;
                    const uint32_t bar = full0 + 8u * (uint32_t)sb;
                    const uint32_t bdst = stage0 + g.b_ring_off + (uint32_t)sb * g.b_slot_bytes;
                    if (leader) {
                        if (rank == 0) mbar_expect_tx(bar, 2u * g.b_bytes);
                        tma_load_2d_pair(bdst, map_b, chunk * g.kchunk, brow, bar);
                    }
                    armed_b |= 1u << sb;
                    parity_b = (parity_b & ~(1u << sb)) | (pb << sb);
                    if (++sb == g.n_stages) { sb = 0; pb ^= 1; }
                }
            }
        }
    }
    if (rank == 0) {
        // as in producer_ring: loads already issued land before the CTA may exit
        for (int s = 0; s < g.n_stages; s++)
            if (armed_b & (1u << s))
                mbar_wait_quiet(full_l + 8u * (uint32_t)s, (parity_b >> s) & 1u, g.wait_ns);
        for (int s = 0; s < g.n_a_slots; s++)
            if (armed_a & (1u << s))
                mbar_wait_quiet(afull_l + 8u * (uint32_t)s, (parity_a >> s) & 1u, g.wait_ns);
    }
}

template <int KK>
__device__ __forceinline__ void mma_role_halo(const TcArgs &g, Control *ctl, uint32_t tmem_base,
                                              uint32_t stage0, int who) {
    volatile int *abort_flag = &ctl->abort_flag;
    const bool leader = elect_one();
    const int rounds = Deal<true>(g).rounds(g);
    if (rounds == 0) return;
    const int ksteps = g.taps * g.chunks_per_tap;  // >= g.issuers; a multiple of g.tap_kw
    const int n_iss = g.issuers, kwn = g.block ? g.taps : g.tap_kw;
    const uint64_t hi = (uint64_t)g.desc_hi << 32;
    const uint32_t a_lo0 = ((stage0 >> 4) & 0x3FFF) | (1u << 16);
    const uint32_t b_lo0 = (((stage0 + g.b_ring_off) >> 4) & 0x3FFF) | (1u << 16);
    const uint32_t a_units = g.a_slot_bytes >> 4, b_units = g.b_slot_bytes >> 4;
    const uint32_t row_units = (uint32_t)g.kchunk >> 4;  // one position further
    const uint32_t full0 = smem_u32(&ctl->full[0]), empty0 = smem_u32(&ctl->empty[0]);
    const uint32_t afull0 = smem_u32(&ctl->a_full[0]), aempty0 = smem_u32(&ctl->a_empty[0]);
    int it = 0, ks = who;
    int sb = who % g.n_stages;
    uint32_t pb = 0;
    // the group of this thread's current step: its column kw, its halo slot
    int kw = who % kwn, sa = (who / kwn) % g.n_a_slots;
    uint32_t pa = ((who / kwn) / g.n_a_slots) & 1u;
    int chunk = (who / kwn) % g.chunks_per_tap;  // groups walk the chunks, then the filter rows
    // the step's tap as a row of its position tile, and the filter columns left in its filter row
    const int skip = g.wp - g.tap_kw;
    int row = kw + kw / g.tap_kw * skip, to_go = g.tap_kw - kw % g.tap_kw;
    bool ok = true, entered = false, a_seen = false;
    int b = 0;  // the tile's accumulator and how often it has come round
    uint32_t acc_phase = 0;
    for (;;) {
        if (!entered) {
            if (ks == 0)
                ok = warp_wait(smem_u32(&ctl->acc_empty[b]), acc_phase ^ 1, abort_flag, g.error, 2,
                               g.wait_ns);
            else if (n_iss > 1)
                ok = warp_wait(smem_u32(&ctl->started[b]), acc_phase, abort_flag, g.error, 6,
                               g.wait_ns);
            if (ok && ks == 0 && g.shared_cols && it > 0)
                ok = warp_wait(smem_u32(&ctl->shared_free), (uint32_t)(it - 1) & 1u, abort_flag,
                               g.error, 7, g.wait_ns);
            if (!ok) break;
            fence_after();
            entered = true;
        }
        if (!a_seen) {  // first step of this thread in the group: the halo tile must have landed
            const uint32_t abar = afull0 + 8u * (uint32_t)sa;
            ok = warp_wait(abar, pa, abort_flag, g.error, 9, g.wait_ns);
            if (!ok) break;
            a_seen = true;
        }
        const uint32_t fbar = full0 + 8u * (uint32_t)sb;
        ok = warp_wait(fbar, pb, abort_flag, g.error, 3, g.wait_ns);
        if (!ok) break;
        fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)b * g.acc_step;
        const uint64_t adesc =
            hi | (uint64_t)(a_lo0 + (uint32_t)sa * a_units + (uint32_t)row * row_units);
        const uint64_t bdesc = hi | (uint64_t)(b_lo0 + (uint32_t)sb * b_units);
        const int kk = chunk == g.chunks_per_tap - 1 ? g.kk_last : KK;
        if (leader) {
#pragma unroll
            for (int k = 0; k < KK; k++) {
                if (k < kk) {
                    mma_mxf4<true>(d_tmem, adesc + (uint64_t)(2 * k), bdesc + (uint64_t)(2 * k),
                                   g.idesc, tmem_base + kScaleCol, (k == 0 && ks == 0) ? 0u : 1u);
                }
            }
            commit_pair(empty0 + 8u * (uint32_t)sb);
            if (n_iss > 1 && ks == 0) {
                commit_pair(smem_u32(&ctl->started[b]));
            }
        }
        __syncwarp();
        sb += n_iss;
        if (sb >= g.n_stages) { sb -= g.n_stages; pb ^= 1u; }
        kw += n_iss;
        row += n_iss;
        to_go -= n_iss;
        if (to_go <= 0) { to_go += g.tap_kw; row += skip; }
        if (kw >= kwn) {
            // this thread's last step of the group is issued: its reads of the halo tile are
            // covered by this commit (both issuers commit: the barrier counts them)
            if (leader) {
                commit_pair(aempty0 + 8u * (uint32_t)sa);
            }
            do {
                kw -= kwn;
                if (++sa == g.n_a_slots) { sa = 0; pa ^= 1u; }
                if (++chunk == g.chunks_per_tap) chunk = 0;
            } while (kw >= kwn);
            row = kw;
            to_go = g.tap_kw - kw;
            a_seen = false;
        }
        ks += n_iss;
        if (ks >= ksteps) {  // this thread's share of the tile is issued
            ks -= ksteps;
            if (leader && !(g.drop_commit && it == 0 && blockIdx.x == 0)) {
                commit_pair(smem_u32(&ctl->acc_full[b]));
            }
            entered = false;
            if (++it >= rounds) break;
            if (++b == g.n_acc) { b = 0; acc_phase ^= 1u; }
        }
    }
    if (leader) commit_pair_here(smem_u32(&ctl->drain[who]));
    mbar_wait_quiet(smem_u32(&ctl->drain[who]), 0, g.wait_ns);
}

// Resident filters beside position tiles of rows, a tile for each filter row: rows of fewer than 128 bytes, a single
// filter row, and what mma_role_block has no room or barriers for. The only thing that arrives is position
// tiles, so a group (the taps of a filter row on one channel chunk) is one wait, kw * KK MMAs and one
// commit, from one issuer: about 500 cycles a group and 30 an instruction (layers of 64 filters that
// differ in nothing else), where the tensor pipe needs N / 2 an instruction. Wide tiles with several
// taps a group hide that, narrow ones are bound by it. With the filters streamed a pair moved 320 KB
// per CTA and tile of AlexNet conv2 (on rows then) through L2, which took 11400 cycles under the
// result stores of another tile (tensor pipe: 5100).
template <int KK>
__device__ __forceinline__ void mma_role_resident(const TcArgs &g, Control *ctl, uint32_t tmem_base,
                                                  uint32_t stage0) {
    volatile int *abort_flag = &ctl->abort_flag;
    const bool leader = elect_one();
    const int rounds = Deal<true>(g).rounds(g);
    if (rounds == 0) return;
    const int groups = g.kh * g.chunks_per_tap;
    const uint64_t hi = (uint64_t)g.desc_hi << 32;
    const uint32_t a_lo0 = ((stage0 >> 4) & 0x3FFF) | (1u << 16);
    const uint32_t b_lo0 = (((stage0 + g.b_ring_off) >> 4) & 0x3FFF) | (1u << 16);
    const uint32_t a_units = g.a_slot_bytes >> 4, b_units = g.b_slot_bytes >> 4;
    const uint32_t row_units = (uint32_t)g.kchunk >> 4;  // one position further
    const uint32_t afull0 = smem_u32(&ctl->a_full[0]), aempty0 = smem_u32(&ctl->a_empty[0]);
    int sa = 0, b = 0;
    uint32_t pa = 0, acc_phase = 0;
    bool ok = true;
    for (int it = 0; it < rounds; it++) {
        const uint32_t d_tmem = tmem_base + (uint32_t)b * g.acc_step;
        ok = warp_wait(smem_u32(&ctl->acc_empty[b]), acc_phase ^ 1, abort_flag, g.error, 2, g.wait_ns);
        if (ok && g.shared_cols && it > 0)
            ok = warp_wait(smem_u32(&ctl->shared_free), (uint32_t)(it - 1) & 1u, abort_flag, g.error,
                           7, g.wait_ns);
        if (!ok) break;
        for (int gr = 0, chunk = 0; gr < groups; gr++) {
            ok = warp_wait(afull0 + 8u * (uint32_t)sa, pa, abort_flag, g.error, 9, g.wait_ns);
            if (!ok) break;
            fence_after();
            const int kk = chunk == g.chunks_per_tap - 1 ? g.kk_last : KK;
            if (leader) {
                uint64_t adesc = hi | (uint64_t)(a_lo0 + (uint32_t)sa * a_units);
                uint64_t bdesc = hi | (uint64_t)(b_lo0 + (uint32_t)(gr * g.tap_kw) * b_units);
                for (int kw = 0; kw < g.tap_kw; kw++, adesc += row_units, bdesc += b_units) {
#pragma unroll
                    for (int k = 0; k < KK; k++) {
                        if (k < kk) {
                            mma_mxf4<true>(d_tmem, adesc + (uint64_t)(2 * k),
                                           bdesc + (uint64_t)(2 * k), g.idesc,
                                           tmem_base + kScaleCol, (gr | kw | k) == 0 ? 0u : 1u);
                        }
                    }
                }
                commit_pair(aempty0 + 8u * (uint32_t)sa);
            }
            __syncwarp();
            if (++sa == g.n_a_slots) { sa = 0; pa ^= 1u; }
            if (++chunk == g.chunks_per_tap) chunk = 0;
        }
        if (!ok) break;
        if (leader && !(g.drop_commit && it == 0 && blockIdx.x == 0)) {
            commit_pair(smem_u32(&ctl->acc_full[b]));
        }
        __syncwarp();
        if (++b == g.n_acc) { b = 0; acc_phase ^= 1u; }
    }
    if (leader) commit_pair_here(smem_u32(&ctl->drain[0]));
    mbar_wait_quiet(smem_u32(&ctl->drain[0]), 0, g.wait_ns);
}

// Resident filters beside position tiles that serve all filter rows: a tile is the 128-byte rows of one K chunk
// for every position that any tap reads, 128 + (kh-1) wp + kw-1 of them, and a tap is a row offset. Loaded once per
// K chunk it is 20 KB for AlexNet conv3, where tiles for each filter row are 51 KB, beside which the results leave
// the SM; and an issuer waits and commits once per chunk. (The launcher says where two issuers
// share a tile's filter rows.) One issuer, kernel alone, tiles for each filter row -> these: conv3 on
// 256 images 22.9 -> 22.4 us, conv1 on 64 23.8 -> 21.4, and 1.00 to 1.11 times as fast, median 1.034, over 30
// layers drawn from 16 to 256 images, 3 to 512 channels and filters, 6 to 56 pixels (first layers 60 to 227).
__device__ __forceinline__ void producer_block(const TcArgs &g, Control *ctl, const CUtensorMap *map_a,
                                               const CUtensorMap *map_b, uint32_t stage0, uint32_t rank) {
    volatile int *abort_flag = &ctl->abort_flag;
    const bool leader = elect_one();
    const Deal<true> deal(g);
    const int rounds = deal.rounds(g);
    const uint32_t full_l = smem_u32(&ctl->full[0]), afull_l = smem_u32(&ctl->a_full[0]);
    // a pair counts both CTAs' bytes on the leader's barriers
    const uint32_t full0 = rank != 0 ? mapa(full_l, 0) : full_l;
    const uint32_t afull0 = rank != 0 ? mapa(afull_l, 0) : afull_l;
    const uint32_t aempty0 = smem_u32(&ctl->a_empty[0]);
    const uint32_t a_bytes = (uint32_t)g.halo * (uint32_t)g.kchunk;
    int sa = 0;
    uint32_t pa = 0, armed = 0, parity = 0, b_armed = 0;
    bool ok = true;
    for (int it = 0; ok && it < rounds; it++) {
        int mt, nt;
        deal.at(g, it, mt, nt);
        const int row = g.lead + mt * BM - g.ph * g.wp - g.pw;  // tap (0,0)
        for (int chunk = 0; chunk < g.chunks_per_tap; chunk++) {
            ok = warp_wait(aempty0 + 8u * (uint32_t)sa, pa ^ 1, abort_flag, g.error, 8, g.wait_ns);
            if (!ok) break;
            const uint32_t abar = afull0 + 8u * (uint32_t)sa;
            if (leader) {
                if (rank == 0) mbar_expect_tx(abar, 2u * a_bytes);  // abar is local here
                tma_load_2d_pair(stage0 + (uint32_t)sa * g.a_slot_bytes, map_a, chunk * g.kchunk, row, abar);
            }
            armed |= 1u << sa;
            parity = (parity & ~(1u << sa)) | (pa << sa);
            if (++sa == g.n_a_slots) { sa = 0; pa ^= 1; }
            // the chunk's filters, a barrier for each filter row (n_stages: kh * chunks)
            for (int kh = 0; it == 0 && kh < g.kh; kh++) {
                const int gr = kh * g.chunks_per_tap + chunk;
                const uint32_t bar = full0 + 8u * (uint32_t)gr;
                int brow = nt * g.n_tile + (int)rank * (g.n_tile >> 1) + kh * g.tap_kw * g.ocp16;
                uint32_t bdst = stage0 + g.b_ring_off + (uint32_t)(gr * g.tap_kw) * g.b_slot_bytes;
                if (leader) {
                    if (rank == 0) mbar_expect_tx(bar, 2u * (uint32_t)g.tap_kw * g.b_bytes);
                    for (int kw = 0; kw < g.tap_kw; kw++, brow += g.ocp16, bdst += g.b_slot_bytes)
                        tma_load_2d_pair(bdst, map_b, chunk * g.kchunk, brow, bar);
                }
                b_armed |= 1u << gr;
            }
            __syncwarp();
        }
    }
    if (rank == 0) {
        // as in producer_ring: loads already issued land before the CTA may exit
        for (int i = 0; i < g.n_stages; i++)
            if (b_armed & (1u << i)) mbar_wait_quiet(full_l + 8u * (uint32_t)i, 0, g.wait_ns);
        for (int i = 0; i < g.n_a_slots; i++)
            if (armed & (1u << i))
                mbar_wait_quiet(afull_l + 8u * (uint32_t)i, (parity >> i) & 1u, g.wait_ns);
    }
}

template <int KK>
__device__ __forceinline__ void mma_role_block(const TcArgs &g, Control *ctl, uint32_t tmem_base,
                                               uint32_t stage0, int who) {
    volatile int *abort_flag = &ctl->abort_flag;
    const bool leader = elect_one();
    const int rounds = Deal<true>(g).rounds(g);
    if (rounds == 0) return;
    const uint64_t hi = (uint64_t)g.desc_hi << 32;
    const uint32_t a_lo0 = ((stage0 >> 4) & 0x3FFF) | (1u << 16);
    const uint32_t b_lo0 = (((stage0 + g.b_ring_off) >> 4) & 0x3FFF) | (1u << 16);
    const uint32_t a_units = g.a_slot_bytes >> 4, b_units = g.b_slot_bytes >> 4;
    const uint32_t row_units = (uint32_t)g.kchunk >> 4;  // one position further
    const uint32_t full0 = smem_u32(&ctl->full[0]);
    const uint32_t afull0 = smem_u32(&ctl->a_full[0]), aempty0 = smem_u32(&ctl->a_empty[0]);
    int sa = 0, b = 0;
    uint32_t pa = 0, acc_phase = 0;
    bool ok = true;
    for (int it = 0; it < rounds; it++) {
        const uint32_t d_tmem = tmem_base + (uint32_t)b * g.acc_step;
        if (who == 0)
            ok = warp_wait(smem_u32(&ctl->acc_empty[b]), acc_phase ^ 1, abort_flag, g.error, 2, g.wait_ns);
        else
            ok = warp_wait(smem_u32(&ctl->started[b]), acc_phase, abort_flag, g.error, 6, g.wait_ns);
        if (ok && who == 0 && g.shared_cols && it > 0)
            ok = warp_wait(smem_u32(&ctl->shared_free), (uint32_t)(it - 1) & 1u, abort_flag, g.error,
                           7, g.wait_ns);
        // Two teams share three accumulators in turn. A team whose tile has the accumulator of another's would take a
        // commit that was lost for its own tile's, and hand the accumulator on; here it is found missing.
        if (ok && who == 0 && g.n_acc == 3 && it >= 3)
            ok = warp_wait(smem_u32(&ctl->acc_full[b]), acc_phase ^ 1, abort_flag, g.error, 5, g.wait_ns);
        if (!ok) break;
        for (int chunk = 0; chunk < g.chunks_per_tap; chunk++) {
            ok = warp_wait(afull0 + 8u * (uint32_t)sa, pa, abort_flag, g.error, 9, g.wait_ns);
            if (!ok) break;
            const int kk = chunk == g.chunks_per_tap - 1 ? g.kk_last : KK;
            // with two issuers each takes every other filter row of the tile (and some of each chunk: kh > 1)
            for (int kh = g.issuers > 1 ? (chunk * g.kh + who) & 1 : 0; kh < g.kh; kh += g.issuers) {
                const int gr = kh * g.chunks_per_tap + chunk;
                if (it == 0)
                    ok = warp_wait(full0 + 8u * (uint32_t)gr, 0, abort_flag, g.error, 3, g.wait_ns);
                if (!ok) break;
                fence_after();
                if (leader) {
                    uint64_t adesc =
                        hi | (uint64_t)(a_lo0 + (uint32_t)sa * a_units + (uint32_t)(kh * g.wp) * row_units);
                    uint64_t bdesc = hi | (uint64_t)(b_lo0 + (uint32_t)(gr * g.tap_kw) * b_units);
                    for (int kw = 0; kw < g.tap_kw; kw++, adesc += row_units, bdesc += b_units) {
#pragma unroll
                        for (int k = 0; k < KK; k++) {
                            if (k < kk) {
                                mma_mxf4<true>(d_tmem, adesc + (uint64_t)(2 * k),
                                               bdesc + (uint64_t)(2 * k), g.idesc,
                                               tmem_base + kScaleCol, (chunk | kh | kw | k) == 0 ? 0u : 1u);
                            }
                        }
                        if ((chunk | kh | kw) == 0 && g.issuers > 1) commit_pair(smem_u32(&ctl->started[b]));
                    }
                    if (kh + g.issuers >= g.kh) commit_pair(aempty0 + 8u * (uint32_t)sa);
                }
                __syncwarp();
            }
            if (!ok) break;
            if (++sa == g.n_a_slots) { sa = 0; pa ^= 1u; }
        }
        if (!ok) break;
        if (leader && !(g.drop_commit && it == 0 && blockIdx.x == 0)) {
            commit_pair(smem_u32(&ctl->acc_full[b]));
        }
        __syncwarp();
        if (++b == g.n_acc) { b = 0; acc_phase ^= 1u; }
    }
    if (leader) commit_pair_here(smem_u32(&ctl->drain[who]));
    mbar_wait_quiet(smem_u32(&ctl->drain[who]), 0, g.wait_ns);
}

// Position tiles of 16-byte columns (resident filters): the packed bytes of all positions that any tap
// of a tile reads, 128 + (kh-1) wp + kw-1 of them, are loaded once, as [column][position][16 bytes]:
// a box of 16 bytes by all positions for each column, from a plain map of the frame.
// That is the tensor core's unswizzled K-major form (eight positions of a column are a core matrix of
// 128 contiguous bytes, the next eight follow, the next column is plane_pitch * 16 further on), in
// which a tap is a start address: 16 bytes per position. A filter row's taps read neighbouring
// positions, so byte 32 s of its operand (what the s-th instruction starts at) is column
// 32 s % pos_bytes / 16 of position 32 s / pos_bytes, and the column after a position's last one is
// the next position's first: with an odd number of columns that one is loaded again, a position on.
__device__ __forceinline__ void producer_planes(const TcArgs &g, Control *ctl,
                                                const CUtensorMap *map_a, const CUtensorMap *map_b,
                                                uint32_t stage0, uint32_t rank) {
    volatile int *abort_flag = &ctl->abort_flag;
    const bool leader = elect_one();
    const Deal<true> deal(g);
    const int rounds = deal.rounds(g);
    const uint32_t full_l = smem_u32(&ctl->full[0]), afull_l = smem_u32(&ctl->a_full[0]);
    // a pair counts both CTAs' bytes on the leader's barriers
    const uint32_t full0 = rank != 0 ? mapa(full_l, 0) : full_l;
    const uint32_t afull0 = rank != 0 ? mapa(afull_l, 0) : afull_l;
    const uint32_t aempty0 = smem_u32(&ctl->a_empty[0]);
    const uint32_t a_bytes = (uint32_t)(g.planes * g.plane_rows) * 16u;
    const int columns = g.pos_bytes >> 4;
    int sa = 0;
    uint32_t pa = 0, armed = 0, parity = 0;
    int b_sent = 0;
    bool ok = true;
    for (int it = 0; it < rounds; it++) {
        int mt, nt;
        deal.at(g, it, mt, nt);
        ok = warp_wait(aempty0 + 8u * (uint32_t)sa, pa ^ 1, abort_flag, g.error, 8, g.wait_ns);
        if (!ok) break;
        const uint32_t abar = afull0 + 8u * (uint32_t)sa;
        if (leader) {
            if (rank == 0) mbar_expect_tx(abar, 2u * a_bytes);  // abar is local here
            const int row = g.lead + mt * BM - g.ph * g.wp - g.pw;
            uint32_t adst = stage0 + (uint32_t)sa * g.a_slot_bytes;
            for (int c = 0; c < g.planes; c++, adst += (uint32_t)g.plane_pitch * 16u) {
                const bool next = c == columns;
                tma_load_2d_pair(adst, map_a, next ? 0 : 16 * c, next ? row + 1 : row, abar);
            }
        }
        armed |= 1u << sa;
        parity = (parity & ~(1u << sa)) | (pa << sa);
        if (++sa == g.n_a_slots) { sa = 0; pa ^= 1; }
        if (it == 0) {  // the filters, a barrier for each share of the groups
            const int brow0 = nt * g.n_tile + (int)rank * (g.n_tile >> 1);
            const int groups = g.kh * g.chunks_per_tap;
            for (int part = 0, gr = 0; part < g.n_stages; part++) {
                const int end = groups * (part + 1) / g.n_stages;
                const uint32_t bar = full0 + 8u * (uint32_t)part;
                if (leader && rank == 0) mbar_expect_tx(bar, 2u * (uint32_t)(end - gr) * g.b_bytes);
                for (; gr < end; gr++) {
                    const int row = gr / g.chunks_per_tap, chunk = gr - row * g.chunks_per_tap;
                    if (leader)
                        tma_load_2d_pair(stage0 + g.b_ring_off + (uint32_t)gr * g.b_slot_bytes, map_b,
                                         chunk * g.kchunk, brow0 + row * g.ocp16, bar);
                }
            }
            b_sent = g.n_stages;
        }
        __syncwarp();
    }
    if (rank == 0) {
        // as in producer_ring: loads already issued land before the CTA may exit
        for (int i = 0; i < b_sent; i++) mbar_wait_quiet(full_l + 8u * (uint32_t)i, 0, g.wait_ns);
        for (int i = 0; i < g.n_a_slots; i++)
            if (armed & (1u << i))
                mbar_wait_quiet(afull_l + 8u * (uint32_t)i, (parity >> i) & 1u, g.wait_ns);
    }
}

// Two issuers take alternate groups (a chunk of a filter row). Nothing but a tile's first instruction
// and the barriers around the tile ties them to each other: both see every position tile and every
// accumulator, and of a filter barrier there is only one phase. What a group costs an issuer is mostly the
// chain of scalar instructions around its MMAs (750 cycles and 80 for each instruction, alone, on layers of 64
// filters; the tensor pipe needs 128 an instruction on AlexNet conv2): working the starts out once instead of
// dividing in every group took conv2 on 128 images from 42.9 to 42.0 us a pass among others, 96 channels on
// 75 images from 27.7 to 27.1 and on one stream from 33.3 to 32.3. A table of 32 starts is one a lane.
template <int KK, bool LONG>
__device__ __forceinline__ void mma_role_planes(const TcArgs &g, Control *ctl, uint32_t tmem_base,
                                                uint32_t stage0, int who) {
    volatile int *abort_flag = &ctl->abort_flag;
    const bool leader = elect_one();
    const int rounds = Deal<true>(g).rounds(g);
    if (rounds == 0) return;
    const int groups = g.kh * g.chunks_per_tap;
    const uint64_t a_hi = (uint64_t)g.plane_desc_hi << 32, b_hi = (uint64_t)g.desc_hi << 32;
    const uint32_t lbo = (uint32_t)g.plane_pitch;  // from a column to the next, in 16 bytes
    const uint32_t a_lo0 = ((stage0 >> 4) & 0x3FFF) | (lbo << 16);
    const uint32_t b_lo0 = (((stage0 + g.b_ring_off) >> 4) & 0x3FFF) | (1u << 16);
    const uint32_t a_units = g.a_slot_bytes >> 4, b_units = g.b_slot_bytes >> 4;
    const uint32_t full0 = smem_u32(&ctl->full[0]);
    const uint32_t afull0 = smem_u32(&ctl->a_full[0]), aempty0 = smem_u32(&ctl->a_empty[0]);
    // Where the instructions of a filter row's chunks start, from its first position and column: a lane
    // works one out, so that no group has to divide. Rows of more than 32 instructions (over 1 KB) have
    // the chunk's worked out by KK lanes in every group (LONG; with the question asked in the loop conv2
    // took 43.6 us instead of 43.5).
    auto start_at = [&](int byte) {
        const int pos = byte / g.pos_bytes;
        return (uint32_t)((byte - pos * g.pos_bytes) >> 4) * lbo + (uint32_t)pos;
    };
    const int lane = threadIdx.x & 31;
    uint32_t start_of = start_at(lane / KK * g.kchunk + lane % KK * 32);
    int sa = 0, b = 0;
    uint32_t pa = 0, acc_phase = 0;
    bool ok = true;
    for (int it = 0; it < rounds; it++) {
        const uint32_t d_tmem = tmem_base + (uint32_t)b * g.acc_step;
        if (who == 0) {
            ok = warp_wait(smem_u32(&ctl->acc_empty[b]), acc_phase ^ 1, abort_flag, g.error, 2, g.wait_ns);
            if (ok && g.shared_cols && it > 0)
                ok = warp_wait(smem_u32(&ctl->shared_free), (uint32_t)(it - 1) & 1u, abort_flag,
                               g.error, 7, g.wait_ns);
        } else {  // the instruction that overwrites the accumulator has been executed
            ok = warp_wait(smem_u32(&ctl->started[b]), acc_phase, abort_flag, g.error, 6, g.wait_ns);
        }
        if (ok) ok = warp_wait(afull0 + 8u * (uint32_t)sa, pa, abort_flag, g.error, 9, g.wait_ns);
        if (!ok) break;
        fence_after();
        const uint32_t tile = a_lo0 + (uint32_t)sa * a_units;
        int row = who / g.chunks_per_tap, chunk = who - row * g.chunks_per_tap;
        for (int gr = who; gr < groups; gr += 2) {
            if (it == 0) {  // the share of the filters that the group belongs to
                int part = 0;
                while (groups * (part + 1) / g.n_stages <= gr) part++;
                ok = warp_wait(full0 + 8u * (uint32_t)part, 0, abort_flag, g.error, 3, g.wait_ns);
                if (!ok) break;
                fence_after();
            }
            const int kk = chunk == g.chunks_per_tap - 1 ? g.kk_last : KK;
            if (LONG) start_of = start_at(chunk * g.kchunk + lane % KK * 32);
            uint32_t start[KK];
#pragma unroll
            for (int k = 0; k < KK; k++)
                start[k] = __shfl_sync(0xffffffffu, start_of, (LONG ? 0 : chunk * KK) + k);
            if (leader) {
                const uint32_t at = tile + (uint32_t)(row * g.wp);
                const uint64_t bdesc = b_hi | (uint64_t)(b_lo0 + (uint32_t)gr * b_units);
#pragma unroll
                for (int k = 0; k < KK; k++) {
                    if (k < kk)
                        mma_mxf4<true>(d_tmem, a_hi | (uint64_t)(at + start[k]), bdesc + (uint64_t)(2 * k),
                                       g.idesc, tmem_base + kScaleCol, (gr | k) == 0 ? 0u : 1u);
                }
                if (gr == 0) commit_pair(smem_u32(&ctl->started[b]));
            }
            __syncwarp();
            chunk += 2;
            while (chunk >= g.chunks_per_tap) { chunk -= g.chunks_per_tap; row++; }
        }
        if (!ok) break;
        if (leader) {
            commit_pair(aempty0 + 8u * (uint32_t)sa);
            if (!(g.drop_commit && it == 0 && blockIdx.x == 0)) commit_pair(smem_u32(&ctl->acc_full[b]));
        }
        __syncwarp();
        if (++sa == g.n_a_slots) { sa = 0; pa ^= 1u; }
        if (++b == g.n_acc) { b = 0; acc_phase ^= 1u; }
    }
    if (leader) commit_pair_here(smem_u32(&ctl->drain[who]));
    mbar_wait_quiet(smem_u32(&ctl->drain[who]), 0, g.wait_ns);
}

// KK = tcgen05.mma instructions per pipeline stage (kchunk / 32).
// PAIR: the grid is made of clusters of two CTAs that share tiles of 256 positions x N filters
// (tcgen05 cta_group::2). Each CTA loads its own 128 positions and its half of the filter tile,
// the leader (rank 0) issues one M = 256 instruction for both, and each CTA's epilogue drains its
// own tensor memory. A stage is a third smaller per CTA that way (32 KB instead of 48 KB at
// N = 256), which is what the kernel is short of: at one stage per 512 cycles a single CTA pulls
// 94 B/clk from L2, four fifths of what the SM's port delivers.
template <int KK, bool PAIR, int EPI, bool EMITS>
__global__ void __launch_bounds__(threads_of(EPI), 1)
conv_tcgen05_kernel(const __grid_constant__ CUtensorMap map_a,
                    const __grid_constant__ CUtensorMap map_b, const TcArgs g) {
    extern __shared__ uint8_t smem_raw[];
    // stages need the swizzle atom's alignment (1024 B); the control block sits in front
    uint8_t *base = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    Control *ctl = (Control *)base;
    uint8_t *stages = base + kControlBytes;

    // warp-uniform, and known to be: the roles below run on whole warps
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const uint32_t rank = PAIR ? cluster_ctarank() : 0u;

    if (threadIdx.x == 0) {
        for (int s = 0; s < g.n_stages; s++) {
            mbar_init(smem_u32(&ctl->full[s]), 1);
            mbar_init(smem_u32(&ctl->empty[s]), 1);
        }
        for (int a = 0; a < g.n_a_slots; a++) {
            mbar_init(smem_u32(&ctl->a_full[a]), 1);
            mbar_init(smem_u32(&ctl->a_empty[a]), (uint32_t)g.issuers);
        }
        for (int b = 0; b < g.n_acc; b++) {
            mbar_init(smem_u32(&ctl->acc_full[b]), (uint32_t)g.issuers);
            // single CTA: one arrival per epilogue thread; pair: one per epilogue warp of both
            mbar_init(smem_u32(&ctl->acc_empty[b]), (uint32_t)((PAIR ? 2 : 32) * EPI / g.teams));
            mbar_init(smem_u32(&ctl->started[b]), 1);
        }
        for (int i = 0; i < 2; i++) mbar_init(smem_u32(&ctl->drain[i]), 1);
        mbar_init(smem_u32(&ctl->shared_free), PAIR ? 8 : 4);  // one arrival per lane quadrant
        ctl->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        // the descriptors are launch parameters: fetch them while the predecessor still runs
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(&map_b) : "memory");
    }
    if (warp == 1) {
        // Each CTA allocates all of its own tensor memory, so the accumulators sit at the same
        // address in both CTAs of a pair.
        tmem_alloc(smem_u32(&ctl->tmem_base), kTmemCols);
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem_base = ctl->tmem_base;
    if (warp >= 2 && warp < 6)
        fill_scales(tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + kScaleCol, 16);
    // Everything above touched only this CTA's own shared and tensor memory and the launch
    // parameters. What earlier kernels of the stream produced is read by the TMA producer and
    // the epilogue warps, each after its own dependency_wait(); the MMA issuer reads shared
    // memory only.
    const bool alpha_in_smem = g.ocp16 <= kAlphaSmem;
    fence_before();
    __syncthreads();
    if (PAIR) {  // the partner's barriers exist before anything is sent to them
        cluster_arrive();
        cluster_wait();
    }
    fence_after();
    // Every CTA of this grid is resident from the start, so a dependent grid may be launched as
    // soon as all of them have got here: its CTAs move in as these exit (SMs with one tile fewer
    // exit a round early) and set themselves up; they wait for this grid's results themselves.
    dependency_release();

    const uint32_t stage0 = smem_u32(stages);

    if (warp == 0) {
        // ---- TMA producer ----
        dependency_wait();
        if constexpr (PAIR) {
            if (g.planes) producer_planes(g, ctl, &map_a, &map_b, stage0, rank);
            else if (g.block && g.resident) producer_block(g, ctl, &map_a, &map_b, stage0, rank);
            else if (g.halo) producer_halo(g, ctl, &map_a, &map_b, stage0, rank);
            else producer_ring<PAIR>(g, ctl, &map_a, &map_b, stage0, rank);
        } else {
            producer_ring<PAIR>(g, ctl, &map_a, &map_b, stage0, rank);
        }
    } else if (warp == 1 || warp == 2 + EPI) {
        const int who = warp == 1 ? 0 : 1;
        if (who < g.issuers && rank == 0) {
            if constexpr (PAIR) {
                // filter rows of more than 32 instructions have chunks of 128 bytes
                if (KK == 4 && g.planes && g.chunks_per_tap * KK > 32)
                    mma_role_planes<KK, true>(g, ctl, tmem_base, stage0, who);
                else if (g.planes) mma_role_planes<KK, false>(g, ctl, tmem_base, stage0, who);
                else if (KK == 4 && g.block && g.resident) mma_role_block<KK>(g, ctl, tmem_base, stage0, who);
                else if (g.resident) mma_role_resident<KK>(g, ctl, tmem_base, stage0);
                else if (g.halo) mma_role_halo<KK>(g, ctl, tmem_base, stage0, who);
                else mma_role<KK, PAIR>(g, ctl, tmem_base, stage0, who);
            } else {
                mma_role<KK, PAIR>(g, ctl, tmem_base, stage0, who);
            }
        }
        __syncwarp();
    } else {
        // ---- epilogue warps: stage alpha among themselves, then drain accumulators ----
        dependency_wait();
        if (alpha_in_smem) {
            for (int i = threadIdx.x - 64; i < g.ocp16; i += 32 * EPI)
                ctl->alpha[i] = i < g.oc ? __ldg(g.alpha + i) : 0.f;
            bar_sync(5, 32 * EPI);
        }
        epilogue_role<PAIR, EPI, EMITS>(g, ctl, tmem_base, warp, lane, alpha_in_smem);
    }

    fence_before();
    __syncthreads();
    if (PAIR) {
        // Neither CTA leaves while the other may still read its shared or tensor memory or
        // signal its barriers.
        cluster_arrive();
        cluster_wait();
    }
    if (warp == 1) {
        fence_after();
        tmem_free(tmem_base, kTmemCols);
    }
}

// ---- host side ---------------------------------------------------------------------------------

using Kernel = void (*)(CUtensorMap, CUtensorMap, TcArgs);
constexpr int kSingle = 0, kPair = 1, kPairEmits = 2, kPairFew = 3;  // forms; by MMAs of a chunk 4, 2 and 1
const Kernel kKernels[3][4] = {
    {conv_tcgen05_kernel<4, false, kEpiWarps, false>, conv_tcgen05_kernel<4, true, kEpiWarps, false>,
     conv_tcgen05_kernel<4, true, kEpiWarps, true>, conv_tcgen05_kernel<4, true, kFewEpiWarps, false>},
    {conv_tcgen05_kernel<2, false, kEpiWarps, false>, conv_tcgen05_kernel<2, true, kEpiWarps, false>,
     conv_tcgen05_kernel<2, true, kEpiWarps, true>, nullptr},
    {conv_tcgen05_kernel<1, false, kEpiWarps, false>, conv_tcgen05_kernel<1, true, kEpiWarps, false>,
     conv_tcgen05_kernel<1, true, kEpiWarps, true>, nullptr}};

// The opt-in to large dynamic shared memory, once per device and kernel.
cudaError_t opt_in(int d, int per_stage, int form) {
    static std::atomic<bool> opted_in[64][3][4];
    std::atomic<bool> &done = opted_in[d][per_stage][form];
    if (done.load(std::memory_order_acquire)) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(kKernels[per_stage][form],
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e == cudaSuccess) done.store(true, std::memory_order_release);
    return e;
}

// CTA pairs that can be resident together, asked once per device (a CTA has an SM to itself in every form).
int resident_pairs(int d, int sms) {
    static std::atomic<int> pair_count[64];
    int slots = pair_count[d].load(std::memory_order_relaxed);
    if (slots) return slots;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (sms / 2));
    cfg.blockDim = dim3(threads_of(kEpiWarps));
    cfg.dynamicSmemBytes = 227 * 1024 - 1024;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (opt_in(d, 0, kPair) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&slots, kKernels[0][kPair], &cfg) != cudaSuccess || slots <= 0) {
        (void)cudaGetLastError();
        slots = sms / 2;
    }
    pair_count[d].store(slots, std::memory_order_relaxed);
    return slots;
}

}  // namespace

cudaError_t launch_conv_tcgen05(const Plan &p, const void *bin_src, const void *bin_w,
                                const float *alpha, const float *k, const float *a, float *k_out,
                                float *dst, int32_t *sums, int *error_word, cudaStream_t s,
                                const ChainTarget *next, const ConvSelfTest *test) {
    if (p.q_total == 0) return cudaSuccess;
    const int m_tiles = (int)((p.q_total + BM - 1) / BM);
    int dev = 0;
    cudaGetDevice(&dev);
    static std::atomic<int> sm_count[64];
    const int d = dev & 63;
    int sms = sm_count[d].load(std::memory_order_relaxed);
    if (!sms) {
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        sm_count[d].store(sms, std::memory_order_relaxed);
    }
    TcArgs g;
    g.alpha = alpha; g.kmap = k; g.amap = a; g.kmap_out = k_out; g.dst = dst; g.sums = sums;
    g.error = error_word;
    g.inv_khw = p.inv_khw; g.ih = p.ih; g.iw = p.iw; g.kh = p.kh;
    g.q_total = p.q_total;
    g.m_tiles = m_tiles;
    // channels-wise: a tap, or the kw taps of a filter row one after the other
    const int tap_bytes = p.cat ? p.kw * p.icp : p.row_bytes;
    const int tap_values = p.cat ? 2 * (p.kw - 1) * p.icp + p.ic : p.ic;
    g.tap_kw = p.cat ? 1 : p.kw;
    g.taps = p.kh * g.tap_kw;
    g.kchunk = p.kchunk; g.chunks_per_tap = div_up_i(tap_bytes, p.kchunk);
    g.kk_last = (tap_values - (g.chunks_per_tap - 1) * 2 * p.kchunk + 63) / 64;
    const int kk = p.kchunk / 32;
    const int steps = g.taps * ((g.chunks_per_tap - 1) * kk + g.kk_last);  // MMAs of a tile
    // CTA pairs when the layer is more than one round of tiles (measured with 8-bit operands on
    // AlexNet conv4: 35.0 against 36.9 us at 256 images, 24.3 against 24.9 at 128) and a filter tile splits
    // into two UMMA-sized halves. With a single round the pair's longer hand-shakes cost more than its lighter
    // loads save: a pass on one image 13.5 against 12.4 us with the present operands, on 32 images 17.5
    // against 16.6.
    // Chained layers, whose CTAs carry a pixel's state across all of its filter tiles, store next to nothing,
    // and a CTA alone keeps up with the tensor pipe while its loads are whole: pairs where they are not, which
    // is where operand rows end inside a 32-byte sector or the last of several chunks of a row is partly empty
    // (a stage's hand-over for fewer MMAs), and where a position tile is enough work for the pair's longer
    // hand-shakes: cycles of the tensor pipe for all of its filter tiles. More are asked for with no more position
    // tiles than SMs, which singles share out at once and without a second round. Two layers chained, the first
    // one's CTAs alone over pairs, 603 chains of 5 to 34 pixels a side, 16 to 640 channels, 2 x 2 to 7 x 7 filters, 64
    // to 512 of them, a pass on one stream and among others (narrow: positions of up to 128 bytes):
    //   on pairs: odd rows, more tiles, narrow, 4000 cycles    107  0.92 to 1.21, mean 1.06   0.91 to 1.20, mean 1.04
    //     the same, wide                                        58  0.99 to 1.55, mean 1.20   0.97 to 1.56, mean 1.15
    //     odd rows, fewer tiles, narrow, 8000                   31  0.96 to 1.15, mean 1.05   0.94 to 1.14, mean 1.02
    //     the same, wide, 5500                                  43  0.98 to 1.46, mean 1.11   0.94 to 1.57, mean 1.09
    //     part of a chunk, more tiles, 5500                     63  0.96 to 1.19, mean 1.06   0.94 to 1.16, mean 1.04
    //     the same, fewer, wide, 8000, 6000 below half the SMs  29  0.95 to 1.11, mean 1.01   0.96 to 1.30, mean 1.00
    //   alone: the same kinds with fewer cycles, 4000 and more 142  0.91 to 1.15, mean 0.98   0.88 to 1.07, mean 0.96
    //     with fewer than 4000                                  84  0.90 to 1.19, mean 0.96   0.82 to 1.11, mean 0.94
    //     whole chunks and even rows                            46  0.86 to 1.25, mean 0.96   0.79 to 1.12, mean 0.94
    // conv3, conv4 and conv5 on 128 images, conv4 on pairs: 57.4 -> 54.4 us on one stream, 43.4 among others
    // either way.
    const bool odd_rows = p.row_bytes % 32 != 0, wide = p.row_bytes > 128, more = m_tiles > sms;
    const bool part_chunk = p.n_tile >= 96 && g.chunks_per_tap > 1 && tap_bytes % p.kchunk != 0;
    const long chained_cycles = (long)steps * p.ocp16 / 2;
    const bool chained_pair =
        p.kh > 1 && (p.icp % 32 != 0 || part_chunk) &&
        (more     ? chained_cycles >= (odd_rows ? 4000 : 5500)
         : wide   ? chained_cycles >= (odd_rows ? 5500 : m_tiles > sms / 2 ? 8000 : 6000)
                  : odd_rows && chained_cycles >= 8000);
    const bool pair = p.n_tile % 32 == 0 && m_tiles >= 2 &&
                      (next ? chained_pair : (long)m_tiles * (p.ocp16 / p.n_tile) > sms);
    const int groups = g.kh * g.chunks_per_tap;
    // as many ring buffers as fit beside the control block
    const size_t room = 227 * 1024 - 1024 - kControlBytes;
    // Results that the epilogue stores float by float (channels-last, filters no multiple of four or a result between
    // two 16-byte boundaries): a warp store is 4 bytes in each of 32 rows, and eight of them in turn fill a sector,
    // which takes the longer the less L1 there is. That is what shared memory leaves of 256 KB: 28 KB beside more than
    // 196 KB (with the system's 1 KB a block), 60 KB beside up to that. Position tiles for all filter rows are the
    // larger ones and give up tiles in flight or filter buffers for it, if two and four are left. More than 196 KB
    // over up to it, on one stream and among others, layers of 224 to 768 channels, 10 to 512 filters, 9 to 40 pixels:
    //   resident filters (and three accumulators)  79  0.98 to 1.29, mean 1.10  1.00 to 1.21, mean 1.08
    //   streamed ones, 224 and 256 a tile          18  1.00 to 1.21, mean 1.06  1.00 to 1.18, mean 1.06
    // 210 filters on 448 channels of 37 x 37, 76 images, 217 -> 179 us on one stream, with a tile for each filter row
    // 181. (Results in whole sectors, 40 layers: 0.97 to 1.02.)
    const bool scattered = p.dst_nhwc && !next && ((p.oc & 3) != 0 || ((uintptr_t)dst & 15) != 0);
    const size_t near_room = scattered ? 195 * 1024 - 1024 - kControlBytes : room;
    // A tap as a row offset into a position tile is known to work for the 128-byte swizzle only
    // (issue_probe checks that one). Narrower rows come with several taps a filter row when a layer
    // that was asked onto the image-row kernel ends a chain; it takes the plain ring.
    const bool row_offsets_ok = g.tap_kw == 1 || (g.tap_kw <= 9 && p.kchunk == 128);
    // Position tiles of a filter row, and of all filter rows (where those are rows of 128 bytes, in one box,
    // with a barrier for each filter row's and chunk's filters; a single filter row is the other form).
    const uint32_t halo_rows = (uint32_t)(g.tap_kw > 1 ? BM + 8 : BM);
    const int block_rows = BM + (g.kh - 1) * p.wp + g.tap_kw - 1;
    const uint32_t row_slot = (halo_rows * p.kchunk + 1023) & ~1023u;
    const uint32_t block_slot = (uint32_t)(block_rows * p.kchunk + 1023) & ~1023u;
    const auto filter_bytes = [&](int n) {  // a CTA's filters of a tile of n, all of their operands
        return (size_t)groups * g.tap_kw * (((pair ? n / 2 : n) * p.kchunk + 1023) & ~1023);
    };
    const auto filters_fit = [&](int n) { return filter_bytes(n) + 3 * (size_t)row_slot <= room; };
    const auto block_fits = [&](int n) {
        return g.kh > 1 && p.kchunk == 128 && block_rows <= 256 && groups <= kMaxStages &&
               filter_bytes(n) + 2 * (size_t)block_slot <= room;
    };
    // A tile of half the filters, if that half stays in shared memory beside such tiles (below) and the whole
    // would not: its filters are loaded once instead of for each position tile, which pays for reading the
    // positions twice where
    // - a position's row ends inside a 32-byte sector, or
    // - a pair has three tiles or fewer, or a tile keeps the tensor pipe for less than 5000 cycles (the others
    //   have eight epilogue warps).
    // Whole over half, 3 x 3 and 3 x 2 filters on 5 to 40 pixels, 257 to 512 channels, on one stream and among others:
    //   rows that end inside a sector, 4 tiles a pair and more, 5000 cycles
    //                                    44 layers  1.06 to 1.31, mean 1.15   1.03 to 1.24, mean 1.10
    //   the others                       70 layers  1.02 to 1.22, mean 1.10   0.98 to 1.12, mean 1.05
    // conv4 on 256 images 41.6 -> 35.6 us on one stream, 39 -> 36 among others. Even rows with four long tiles a pair
    // are left out because the tests hold them to eight epilogue warps, with which halves have not been measured (VGG,
    // half the width and sixteen warps: 1.055 and 1.025). (Half of a whole that stays resident: of 256 filters with up
    // to 1.4 tiles a pair 1.08 and 1.02, with more 0.96 and 0.93; of 192 1.02 and 0.95; of 128 0.92 and 0.90.)
    // Results stored float by float, of which halves make two stretches of a row: of 192 filters (8 layers) 1.01 to
    // 1.21, mean 1.13, and 1.01 to 1.19, mean 1.07, of 256 (10) 0.88 to 1.11, mean 1.00, and 0.86 to 1.09, mean 0.99.
    int n_tile = p.n_tile;
    const int pair_units = (m_tiles + 1) / 2, half_tiles = 2 * (p.ocp16 / p.n_tile);
    const int slots = pair ? resident_pairs(d, sms) : sms;
    const int half_grid = slots - slots % half_tiles;  // pairs that keep to one filter tile, as below
    if (pair && !next && !p.cat && g.kh >= 3 && n_tile >= 192 && n_tile % 64 == 0 && row_offsets_ok &&
        !filters_fit(n_tile) && filters_fit(n_tile / 2) && block_fits(n_tile / 2) && half_grid > 0 &&
        pair_units * half_tiles > slots &&
        div_up_i(pair_units * half_tiles, half_grid) == div_up_i(pair_units * half_tiles, slots) &&
        !(scattered && n_tile == 256) &&
        (p.row_bytes % 32 != 0 || div_up_i(pair_units * half_tiles / 2, slots) <= 3 ||
         (long)steps * n_tile / 2 < 5000))
        n_tile /= 2;
    const int b_rows = pair ? n_tile / 2 : n_tile;  // filter rows a CTA loads per stage
    g.n_tiles = p.ocp16 / n_tile;
    g.n_tile = n_tile;
    g.kw = p.kw; g.ph = p.ph; g.pw = p.pw; g.wp = p.wp; g.hp = p.hp; g.lead = p.lead;
    g.oh = p.oh; g.ow = p.ow; g.oc = p.oc; g.ocp16 = p.ocp16;
    g.by_frame = FastDiv((uint32_t)(p.hp * p.wp)); g.by_wp = FastDiv((uint32_t)p.wp);
    g.dst_nhwc = p.dst_nhwc;
    g.emit_bin = nullptr; g.emit_a = nullptr; g.n_inner = 0;
    g.wait_ns = test && test->wait_ns ? test->wait_ns : 2000000000ull;
    g.drop_commit = test ? test->drop_commit : 0;
    g.e_wp = g.e_hp = g.e_lead = g.e_icp = 0; g.e_inv_ic = 0.f;
    if (next) {
        g.emit_bin = (uint8_t *)next->bin_src; g.emit_a = next->a;
        g.e_wp = next->wp; g.e_hp = next->hp; g.e_lead = next->lead; g.e_icp = next->icp;
        g.e_inv_ic = next->inv_ic;
        g.n_inner = 1;
    }
    // M = 256 for a pair: 128 rows in each CTA
    g.idesc = mxf4_idesc(pair ? 2 * BM : BM, (uint32_t)n_tile);
    g.shared_cols = n_tile > kAccStep;
    g.acc_step = (uint32_t)(n_tile < kAccStep ? n_tile : kAccStep);
    // matrix descriptor, upper half: stride between 8-row groups (8 * kchunk bytes, in 16-byte
    // units), descriptor version 1, swizzle mode
    const uint32_t sbo = (uint32_t)(8 * p.kchunk) >> 4;
    const uint32_t layout = p.kchunk == 128 ? 2u : p.kchunk == 64 ? 4u : 6u;
    g.desc_hi = sbo | (1u << 14) | (layout << 29);
    g.a_bytes = (uint32_t)(BM * p.kchunk);
    g.tx_bytes = g.a_bytes + (uint32_t)(b_rows * p.kchunk);  // per CTA
    g.stage_bytes = (g.tx_bytes + 1023u) & ~1023u;
    g.issuers = g.taps * g.chunks_per_tap < 2 ? 1 : 2;
    // Eight epilogue warps instead of sixteen where a pair has four tiles or more and each keeps the tensor
    // pipe busy for 5000 cycles or more: the stores have the next tile's MMAs to hide behind either way, all
    // but the last tile's. The time with sixteen over that with eight, layers of 28 x 28 with 128, 256 and 512
    // filters and four to eight tiles a pair, a pass among others and on one stream (runs differ by 0.5 %):
    //   5760 to 9216 cycles  0.98 to 1.02, mean 1.006   1.00 to 1.02, mean 1.012
    //   4224 to 4608         0.94 to 1.01, mean 0.99    1.00 to 1.02, mean 1.004
    //   fewer                0.98 to 1.03, mean 1.00    1.00 to 1.09, mean 1.013
    // conv2 on 128 images (5120 cycles, six tiles) 43.3 -> 42.7 us among others, VGG (9216, six) 71.6 -> 71.2.
    // With two or three tiles 0.90 to 1.07.
    const long tile_cycles = (long)steps * n_tile / 2;
    const int pair_tiles = div_up_i(((m_tiles + 1) / 2) * g.n_tiles, sms / 2);
    const bool few = pair && !next && kk == 4 && tile_cycles >= 5000 && pair_tiles >= 4;
    const int epi = few ? kFewEpiWarps : kEpiWarps;
    const int per_stage = kk == 4 ? 0 : kk == 2 ? 1 : 2;
    const int form = few ? kPairFew : !pair ? kSingle : next ? kPairEmits : kPair;
    const Kernel kernel = kKernels[per_stage][form];
    const cudaError_t opted = opt_in(d, per_stage, form);
    if (opted != cudaSuccess) return opted;
    const int units = (pair ? (m_tiles + 1) / 2 : m_tiles) * (next ? 1 : g.n_tiles);
    int grid = units < slots ? units : slots;
    // Fewer pairs, if that costs no further round, so that each keeps to one filter tile.
    const int one_nt = grid - grid % g.n_tiles;
    const bool same_nt = pair && (!next || g.n_tiles == 1) && one_nt > 0 && div_up_i(units, one_nt) == div_up_i(units, grid);
    g.planes = 0; g.plane_rows = 0; g.plane_pitch = 0; g.pos_bytes = p.icp; g.plane_desc_hi = 0;
    g.halo = 0; g.block = 0; g.resident = 0; g.n_a_slots = 0; g.a_slot_bytes = 0; g.b_ring_off = 0; g.b_slot_bytes = 0;
    g.b_bytes = (uint32_t)(b_rows * p.kchunk);
    bool halo = pair && g.tap_kw >= 2 && row_offsets_ok && g.issuers <= g.tap_kw;
    // Filters stay in shared memory if a pair works on several tiles of the same ones and their
    // operands leave room for three position tiles of 128-byte rows. Kernel alone, conv3 on 256 images
    // 25.4 -> 23.0 us (six such tiles in flight), conv1 on 64 images 26.1 -> 25.5 (eight).
    const int walk = same_nt ? div_up_i(units, one_nt) : 1;  // tiles of a pair
    const size_t all_b = filter_bytes(n_tile);
    if (walk > 1 && row_offsets_ok && filters_fit(n_tile)) {
        // Position tiles as 16-byte columns: layers whose filter rows are one operand row (Plan::cat), if
        // the positions of all taps are one box (256 rows) and two tiles fit. AlexNet conv2 on 128
        // images, kernel alone: 42.6 -> 40.3 us from loading 16 KB a tile instead of 160, 33.8 with two
        // issuers. What pays for the columns is that a tile is loaded once for all filter rows and that
        // two issuers share it; what they cost is requests of 16 bytes and a first tile that has to land
        // whole. Columns against 128-byte rows, kernel alone, over 1756 layers of 3 to 224 channels, 16
        // to 512 filters, 1 to 7 filter rows and up to 17 tiles a pair:
        //   one or two filter rows                                      0.89 to 1.17, median 1.01
        //   more, two tiles a pair and more than 32 channels            0.95 to 1.10, median 1.01
        //   more, 33 to 64 channels, three operand rows, 64 filters     1.00 to 1.02, median 1.02
        //   more, filters that would not be resident beside rows        0.94 to 1.10, median 1.00
        //   the others                                                  0.73 to 1.04, median 0.94
        // Only the last take columns; layers of the fourth kind stream their filters. Filters of ten and more
        // columns, whose rows may be more than 1 KB, gain more, not less: 13 x 6 on 167 channels 218 us a
        // pass, 315 as rows; 33 x 3 on 39 57 and 73; 25 x 3 on 214 129 and 174.
        const int columns = p.icp / 16, planes = columns + (columns & 1);
        const int rows = BM + (g.kh - 1) * p.wp + p.kw - 1;
        const int pitch = (rows + 7) & ~7;  // a load lands on a multiple of 128 bytes
        const uint32_t col_slot = (uint32_t)(planes * pitch * 16 + 1023) & ~1023u;
        const bool as_columns = p.cat && g.kh >= 3 && (walk >= 3 || p.icp == 16) &&
                                !(p.icp == 32 && groups == 3 && n_tile <= 64) && rows <= 256 &&
                                all_b + 2 * (size_t)col_slot <= room;
        uint32_t tile_slot = row_slot;
        g.resident = 1;
        if (as_columns) {
            g.issuers = 2;
            g.planes = planes; g.plane_rows = rows; g.plane_pitch = pitch;
            g.plane_desc_hi = 8u | (1u << 14);  // 128 bytes from eight positions to the next, no swizzle
            g.n_stages = groups < kMaxStages ? groups : kMaxStages;  // barriers of the filters
        } else {
            g.issuers = 1;
            g.block = block_fits(n_tile);
            // Two issuers where the taps of a filter row keep the tensor pipe for less time than one needs for them,
            // about 500 cycles and 30 an instruction. One over two, 57 layers of 2 x 2 to 4 x 4 filters on 64 to
            // 512 channels, 1 to 6 tiles a pair, on one stream and among others:
            //   up to 800 cycles, three rows and more, or 96 filters and fewer  1.00 to 1.15   0.99 to 1.15
            //   up to 800 cycles, two rows, 128 and more                        0.95 to 1.03   0.96 to 1.03
            //   more                                                            0.98 to 1.00   0.99 to 1.00
            // conv4 on 256 images 40.1 -> 35.6 us on one stream, 37.5 -> 36 among others; conv1 has
            // three rows of 144 cycles.
            if (g.block && g.tap_kw * kk * n_tile / 2 <= 800 && (g.kh > 2 || n_tile <= 96)) g.issuers = 2;
            g.halo = g.block ? block_rows : (int)halo_rows;
            g.n_stages = g.block ? groups : 2;
            if (g.block) tile_slot = block_slot;
        }
        g.a_slot_bytes = as_columns ? col_slot : tile_slot; g.b_slot_bytes = (g.b_bytes + 1023u) & ~1023u;
        g.n_a_slots = (int)((room - all_b) / g.a_slot_bytes);
        if (g.block && near_room >= all_b + 2 * (size_t)g.a_slot_bytes)
            g.n_a_slots = (int)((near_room - all_b) / g.a_slot_bytes);
        if (g.n_a_slots > kMaxASlots) g.n_a_slots = kMaxASlots;
        g.b_ring_off = (uint32_t)g.n_a_slots * g.a_slot_bytes;
        grid = one_nt;
        halo = true;
    }
    if (halo && !g.resident) {
        // Three position tiles, for all filter rows where they are one box, else for one (136 positions); the
        // rest of the room for filter tiles. For one over for all, 160 layers of 6 to 32 pixels, 230 to 1024
        // channels and 144 to 768 filters, on one stream and among others (odd rows: those that end inside a
        // 32-byte sector):
        //   fewer than 25 taps, tiles of up to 192 filters  55  0.98 to 1.16, mean 1.06  1.01 to 1.16, mean 1.06
        //   the same, of more, up to four filter rows       50  0.94 to 1.08, mean 1.02  0.97 to 1.10, mean 1.02
        //   the same, five and six filter rows of 256        3  1.00 to 1.05, mean 1.03  1.00 to 1.04, mean 1.02
        //   25 and 49 taps, even rows, up to 224            19  0.96 to 1.08, mean 1.03  0.96 to 1.06, mean 1.02
        //   the same, tiles of 256                           6  1.00 to 1.01, mean 1.01  0.99 to 1.02, mean 1.00
        //   25 and 49 taps, odd rows, fewer than 192         4  1.00 to 1.06, mean 1.03  1.01 to 1.05, mean 1.04
        //   the same, 192 and more                          23  0.86 to 1.07, mean 0.95  0.91 to 1.04, mean 0.96
        // The last keep theirs (probably since loads of a chunk that ends inside a sector are slow, as chained layers
        // show too, and all taps of such a chunk would follow one another). So do 256 filters with five filter rows
        // and more, for which it is no gain.
        const bool long_runs = g.taps >= 25 && p.row_bytes % 32 != 0 && n_tile >= 192;
        g.block = g.kh > 1 && p.kchunk == 128 && block_rows <= 256 && (g.kh < 5 || !g.shared_cols) && !long_runs;
        g.halo = g.block ? block_rows : BM + 8;
        g.n_a_slots = 3;
        g.a_slot_bytes = (uint32_t)(g.halo * p.kchunk + 1023) & ~1023u;
        g.b_slot_bytes = (g.b_bytes + 1023u) & ~1023u;
        g.b_ring_off = (uint32_t)g.n_a_slots * g.a_slot_bytes;
        g.n_stages = (int)((room - g.b_ring_off) / g.b_slot_bytes);
        if (g.block && near_room >= g.b_ring_off + 4 * (size_t)g.b_slot_bytes)
            g.n_stages = (int)((near_room - g.b_ring_off) / g.b_slot_bytes);
        if (g.n_stages > kMaxStages) g.n_stages = kMaxStages;
        if (g.n_stages < 4) { g.halo = 0; g.block = 0; halo = false; }
    }
    if (!halo) {
        g.n_stages = (int)(room / g.stage_bytes);
        if (g.n_stages > kMaxStages) g.n_stages = kMaxStages;
    }
    if (g.issuers == 2 && g.n_stages > 2 && !g.resident) g.n_stages &= ~1;
    if (g.n_stages < 2) return cudaErrorNotSupported;
    CUtensorMap map_a, map_b;
    // a position's row is tap_bytes long but only icp further than the one before it
    const bool a_ok =
        g.planes ? encode_bytes_2d(&map_a, bin_src, (uint64_t)p.rows, (uint64_t)p.icp,
                                   (uint64_t)p.icp, 16, (uint32_t)g.plane_rows)
                 : encode_bytes_2d(&map_a, bin_src, (uint64_t)(p.rows - (p.cat ? p.kw - 1 : 0)),
                                   (uint64_t)tap_bytes, (uint64_t)p.icp, (uint32_t)p.kchunk,
                                   (uint32_t)(halo ? g.halo : BM));
    if (!a_ok ||
        !encode_bytes_2d(&map_b, bin_w, (uint64_t)g.taps * p.ocp16, (uint64_t)tap_bytes,
                         (uint64_t)p.tap_pitch, (uint32_t)p.kchunk, (uint32_t)b_rows))
        return cudaErrorNotSupported;

    size_t smem = 1024 + kControlBytes +
                  (g.resident ? (size_t)g.b_ring_off + (size_t)groups * g.tap_kw * g.b_slot_bytes
                   : halo ? (size_t)g.b_ring_off + (size_t)g.n_stages * g.b_slot_bytes
                        : (size_t)g.n_stages * g.stage_bytes);
    // At least 120 KB of shared memory so that one CTA owns the SM and all 512 TMEM columns.
    if (smem < 120 * 1024) smem = 120 * 1024;
    // As many accumulators as fit (at most four), and one epilogue team for each of two or four of
    // them if a CTA has that many tiles. With all 16 warps on every tile AlexNet conv3 (256
    // images) took 41.3 us per pass, conv1 (64 images) 86, with two teams 37.7 and 79. The chained
    // epilogue carries per-pixel state from one filter tile to the next: one team.
    const int rounds = g.n_inner ? 1 : div_up_i(units, grid);
    g.n_acc = g.shared_cols || g.n_inner ? 2 : (int)kScaleCol / n_tile;
    if (g.n_acc > kMaxAcc) g.n_acc = kMaxAcc;
    // (Two instead of three beside position tiles for all filter rows: 0.95 to 1.01 times as fast on one stream, mean
    // 0.99, over 40 layers of 112 to 512 filters; 0.91 to 1.03, mean 0.97, over 27 with results stored float by float.)
    g.teams = g.n_acc == 4 && rounds >= 4 && !few ? 4 : rounds >= 2 ? 2 : 1;
    g.by_acc = FastDiv((uint32_t)g.n_acc);
    note_launch();
    return launch_overlapped(kernel, dim3((pair ? 2 : 1) * grid), dim3(threads_of(epi)), smem, s,
                             pair ? 2 : 1, map_a, map_b, g);
}

}  // namespace xb200
