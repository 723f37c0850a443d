// Inline-PTX wrappers shared by the tensor-core convolution kernels: mbarriers with bounded waits,
// TMA tile loads, bulk stores, tcgen05 MMA / commit / tensor-memory loads.
#pragma once

#include <cuda.h>
#include <cstdint>

namespace xb200 {
namespace tc {

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// Non-blocking look at a barrier phase. Issued ahead of other work, its result is there by the
// time it is needed, which takes the barrier's round trip out of a single thread's critical path.
__device__ __forceinline__ uint32_t mbar_test(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok;
}

__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// Waits for a barrier phase, giving up after limit_ns or as soon as another role of the CTA has
// given up. Returns false in that case, after recording `code` in *error (first failure wins).
static __device__ __noinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag,
                                       int *error, int code, unsigned long long limit_ns) {
    if (mbar_try_wait(bar, parity)) return true;
    if (*abort_flag) return false;
    const unsigned long long t0 = global_ns();
    for (;;) {
        for (int i = 0; i < 64; i++)
            if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
        if (global_ns() - t0 > limit_ns) {
            *abort_flag = 1;
            atomicCAS(error, 0, code);
            return false;
        }
    }
}

// The same for a whole converged warp, with one answer for all its lanes. The issuing roles (TMA
// loads, MMAs) run on whole warps and let one elected lane issue: descriptors and barrier addresses
// then stay in uniform registers, which the instructions take them from. With the whole role inside
// `if (lane == 0)` a pipeline stage (wait, four MMAs, commit) took an issuer 640 cycles instead of 455
// (800 instead of 640 with halo tiles), which bound every tile of fewer than 256 filters and many of
// 256; in pairs of issuers a tile of AlexNet conv4 8800 instead of 7500 (tensor pipe: 6900).
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag,
                                          int *error, int code, unsigned long long limit_ns) {
    bool ok = mbar_try_wait(bar, parity);
    if (!ok) ok = mbar_wait(bar, parity, abort_flag, error, code, limit_ns);
    return __all_sync(0xffffffffu, ok);
}
// One lane of a converged warp, always the same one.
__device__ __forceinline__ bool elect_one() {
    uint32_t one;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(one));
    return one != 0;
}

// The last thing a role does: wait for its loads or MMAs in flight, bounded, without recording anything.
// Mostly there is nothing left to wait for, and the timer is not read then (18 reads of it, a filter tile
// each, cost a pass of one image 0.06 us).
__device__ __forceinline__ void mbar_wait_quiet(uint32_t bar, uint32_t parity,
                                                unsigned long long limit_ns) {
    if (mbar_try_wait(bar, parity)) return;
    const unsigned long long t0 = global_ns();
    while (!mbar_try_wait(bar, parity))
        if (global_ns() - t0 > limit_ns) break;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int c0, int c1,
                                            uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(bar)
        : "memory");
}

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap *map, int c0, int c1,
                                            int c2, int c3, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3, %4, %5}], [%6];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
        : "memory");
}

// ---- CTA pairs (cluster of two, tcgen05 cta_group::2) ----------------------------------------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// Address of the same shared-memory location in CTA `rank` of the cluster (shared::cluster window).
__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_arrive() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait() {
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Arrival on a barrier of another CTA of the cluster (address from mapa) that hands over tensor
// memory: the reads before it are complete (tcgen05.wait::ld) and ordered by fence_before(), so the
// arrival is relaxed. As a release at cluster scope it also waited until the thread's earlier
// result stores had reached L2, 2500 to 3500 cycles during which the next tile's MMAs stood still
// (a tile of AlexNet conv4 takes 8500): the kernel on conv4 with 256 images 27.4 -> 25.6 us.
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr)
                 : "memory");
}
// Tile load of a CTA pair: the data lands in the executing CTA's shared memory, the byte count is
// reported to `bar`, which may live in either CTA of the pair (shared::cluster address).
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap *map, int c0, int c1,
                                                 uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(bar)
        : "memory");
}
// Arrives on the barrier at this offset in both CTAs of the pair once every tcgen05.mma issued
// so far by this thread has completed.
__device__ __forceinline__ void commit_pair(uint32_t bar) {
    const uint16_t both = 3;
    asm volatile(
        "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 "
        "[%0], %1;"
        ::"r"(bar), "h"(both)
        : "memory");
}
// The same on this CTA's barrier alone: for a wait that the other CTA, which may leave meanwhile, has
// no part in.
__device__ __forceinline__ void commit_pair_here(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 ::"r"(bar)
                 : "memory");
}

// Shared memory -> global memory, `bytes` a multiple of 16, both addresses 16-byte aligned.
// Completion is tracked per thread in bulk groups.
__device__ __forceinline__ void bulk_store(void *gdst, uint32_t ssrc, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                 ::"l"(gdst), "r"(ssrc), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// every bulk store of this thread has read its shared-memory source
__device__ __forceinline__ void bulk_wait_read() {
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
// every bulk store of this thread is complete
__device__ __forceinline__ void bulk_wait_all() {
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}
// orders this thread's ordinary shared-memory writes before later bulk copies that read them
__device__ __forceinline__ void fence_async_smem() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void mma_i8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc,
                                       uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// ---- 4-bit floats (kind::mxf4) ----------------------------------------------------------------
// K = 64 e2m1 values per instruction, twice the rate of the 8-bit kinds for the same bytes.
// Every block of 32 values along K has a scale in tensor memory; the library's scales are all
// 2^0 (byte 0x7F), so where a row's scale lies inside the columns given does not matter.
// Accumulation is in fp32 and exact: sums of +-1 are tested up to 2^24 (tests/test_large_sums_gpu.py).
// 8780 Tera-operations/s (kind::i8: 4480; csrc/probe/pipe_probe.cu).
constexpr uint32_t kScaleOne = 0x7F7F7F7Fu;
// instruction descriptor: A and B e2m1, both K-major, scales ue8m0, D fp32; n a multiple of 16
__host__ __device__ constexpr uint32_t mxf4_idesc(uint32_t m, uint32_t n) {
    return (1u << 7) | (1u << 10) | ((n >> 3) << 17) | (1u << 23) | ((m >> 4) << 24);
}
template <bool PAIR>
__device__ __forceinline__ void mma_mxf4(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc,
                                         uint32_t idesc, uint32_t scales, uint32_t accumulate) {
    if (PAIR)
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %5, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::mxf4.block_scale.scale_vec::2X "
            "[%0], %1, %2, %3, [%4], [%4], p;\n\t}"
            ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(scales), "r"(accumulate)
            : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.ne.b32 p, %5, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X "
            "[%0], %1, %2, %3, [%4], [%4], p;\n\t}"
            ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(scales), "r"(accumulate)
            : "memory");
}
// Writes one value to this warp's 32 lanes of `cols` columns (a multiple of 8).
__device__ __forceinline__ void fill_columns(uint32_t taddr, int cols, uint32_t value) {
    for (int c = 0; c < cols; c += 8)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1};"
                     ::"r"(taddr + (uint32_t)c), "r"(value)
                     : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// Writes the block scales: this warp's 32 lanes of `cols` columns (a multiple of 16). All four
// quadrants of lanes have to be written before the first mma_mxf4.
__device__ __forceinline__ void fill_scales(uint32_t taddr, int cols) {
    fill_columns(taddr, cols, kScaleOne);
}

// Arrives on the barrier once every tcgen05.mma issued so far by this thread has completed.
__device__ __forceinline__ void commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 ::"r"(bar)
                 : "memory");
}

__device__ __forceinline__ void ld16(uint32_t taddr, uint32_t *v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
          "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
          "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
}

__device__ __forceinline__ void ld32(uint32_t taddr, uint32_t *v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]),
          "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]),
          "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]),
          "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]),
          "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
}

__device__ __forceinline__ void wait_ld() {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t smem_result, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_result), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t base, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols)
                 : "memory");
}

// Named barrier among `threads` threads of the CTA (ids 1..15; 0 is __syncthreads).
__device__ __forceinline__ void bar_sync(int id, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int threads) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

}  // namespace tc

// ---- host side: tensor-map encoding (shared by the convolution launchers) ------------------------
// A byte matrix of `rows` rows of row_bytes, `pitch` bytes apart (rows may overlap), boxes of
// box_rows x box_bytes, swizzle span = box_bytes (boxes of 16 bytes are not swizzled).
bool encode_bytes_2d(CUtensorMap *map, const void *ptr, uint64_t rows, uint64_t row_bytes,
                     uint64_t pitch, uint32_t box_bytes, uint32_t box_rows);
// A [d3][d2][d1][row_bytes] byte tensor (strides in bytes for d1, d2, d3), boxes of
// 1 x box2 x box1 x box_bytes, swizzle span = box_bytes; out-of-range elements read as zero.
bool encode_bytes_4d(CUtensorMap *map, const void *ptr, uint64_t row_bytes, uint64_t d1,
                     uint64_t d2, uint64_t d3, uint64_t s1, uint64_t s2, uint64_t s3,
                     uint32_t box_bytes, uint32_t box1, uint32_t box2);

}  // namespace xb200
