// Launchers of the device kernels. Each takes the Plan, raw device pointers and a stream, and
// returns the CUDA status of the launch; none allocates or synchronises.
#pragma once

#include <atomic>

#include <cuda_runtime.h>

#include "plan.hpp"

namespace xb200 {

// Kernels launched by this library in this process (benchmark accounting).
extern std::atomic<long> g_kernel_launches;
inline void note_launch(int n = 1) { g_kernel_launches.fetch_add(n, std::memory_order_relaxed); }

// Launch with programmatic stream serialisation: the grid may be scheduled while the previous
// kernel of the stream is still draining, so that its set-up (and the launch latency itself)
// runs under the predecessor's tail. Kernels launched this way call dependency_wait() before
// they touch anything an earlier kernel may have written (packed filters among it: that the kernel which
// writes them has ended does not make them visible, the wait does) or may still be reading. All kernels of a
// pass are launched like this (measured: 2-3 us per forward pass for the convolution, another 0.8 us for the
// tiled binarizer in back-to-back passes); those that pack weights are not.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_overlapped(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                                     cudaStream_t s, int cluster, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cluster > 1) {  // thread-block clusters of `cluster` CTAs along x
        attr[1].id = cudaLaunchAttributeClusterDimension;
        attr[1].val.clusterDim.x = (unsigned)cluster;
        attr[1].val.clusterDim.y = 1;
        attr[1].val.clusterDim.z = 1;
        cfg.numAttrs = 2;
    }
    return cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
}

// n / d for n < 2^31 by a multiplication and a shift (the round-up method: Granlund and
// Montgomery, "Division by invariant integers using multiplication", 1994).
struct FastDiv {
    uint32_t mul, shift;
    FastDiv() = default;
    explicit FastDiv(uint32_t d) {
        shift = 0;
        while ((1ull << shift) < d) shift++;
        mul = (uint32_t)(((1ull << 32) * ((1ull << shift) - d)) / d + 1);
    }
#ifdef __CUDACC__
    __device__ __forceinline__ uint32_t operator()(uint32_t n) const {
        return (__umulhi(n, mul) + n) >> shift;
    }
#endif
};

#ifdef __CUDACC__
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t d;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
    return d;
}

// The +-1 nibbles (e2m1: 0x2, and 0xA where the top bit of the word is set) of eight words, the
// first in the lowest nibble. A selector nibble of 0xB / 0xF replicates the top bit of byte 3 of
// the first / second operand, so eight words cost six byte permutes and two logic operations.
__device__ __forceinline__ uint32_t sign_nibbles(const uint32_t *v) {
    const uint32_t even = prmt(prmt(v[0], v[2], 0xFBFBu), prmt(v[4], v[6], 0xFBFBu), 0x5410u);
    const uint32_t odd = prmt(prmt(v[1], v[3], 0xFBFBu), prmt(v[5], v[7], 0xFBFBu), 0x5410u);
    return (((even & 0x0F0F0F0Fu) | (odd & 0xF0F0F0F0u)) & 0x88888888u) | 0x22222222u;
}
// The same with only the first `n` words present (n < 0 counts as none): the others are 0.
__device__ __forceinline__ uint32_t first_nibbles(uint32_t word, int n) {
    return n >= 8 ? word : n <= 0 ? 0u : word & (0xFFFFFFFFu >> (4 * (8 - n)));
}

// (S * alpha) * K in upstream's order, S as the bits of a float. The + 0 comes before the products: it
// makes a sum of zero +0 whatever sign the adder gave it, and leaves the -0 that a negative S times an
// alpha of zero is (a filter of zeros; the next layer reads that sign).
__device__ __forceinline__ float scaled(uint32_t s, float alpha, float k) {
    return __fmul_rn(__fmul_rn(__fadd_rn(__uint_as_float(s), 0.f), alpha), k);
}

// Lets the next kernel of the stream start its set-up now ...
__device__ __forceinline__ void dependency_release() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
// ... and blocks until every earlier kernel of the stream has completed and its writes are
// visible. A no-op for grids launched the ordinary way.
__device__ __forceinline__ void dependency_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
#endif

// ---- self-tests ------------------------------------------------------------------------------
// `test` (normally null) shortens a kernel's wait limit and makes one CTA lose the commit that
// publishes its first accumulator, so that a test can watch a bounded wait run out: the kernel returns
// by itself with *error_word set and the results of the call invalid. The one-launch pass can lose an
// arrival of its packed operand instead, or, like the one-launch maps, the turns at which running sums
// are handed on.
struct ConvSelfTest {
    unsigned long long wait_ns;  // 0: the normal limit (2 s)
    int drop_commit;
    int drop_operand, drop_turn;
};

// ---- activations -----------------------------------------------------------------------------
// One pass over the fp32 source: sign bits into the family's packed layout and, when `a` is not
// null, the per-pixel mean |x| map. Replaces upstream src/bcast_binarize_data.cpp:43-73 and the
// first loop of src/bcast_calculate_k.cpp:49-66.
cudaError_t launch_binarize_data(const Plan &p, const float *src, void *bin_src, float *a,
                                 cudaStream_t s);
// The same for a folded layer (Plan::fold); launch_binarize_data sends those here.
cudaError_t launch_fold(const Plan &p, const float *src, void *bin_src, float *a, cudaStream_t s);
// The mean |x| map alone (calculate_k called on its own).
cudaError_t launch_mean_abs(const Plan &p, const float *src, float *a, cudaStream_t s);
// K = box filter of A over the filter window / (KH*KW), zero outside the image.
// Replaces the second loop of upstream src/bcast_calculate_k.cpp:69-85.
cudaError_t launch_box_filter(const Plan &p, const float *a, float *k, cudaStream_t s);

// Both in one launch, for the small layers that maps_ok() names (maps.cu). `error_word` as for the
// convolutions below.
bool maps_ok(const Plan &p);
cudaError_t launch_maps(const Plan &p, const float *src, float *a, float *k, int *error_word,
                        cudaStream_t s, const ConvSelfTest *test = nullptr);

// ---- weights ---------------------------------------------------------------------------------
// Sign-pack into the family's layout, alpha[oc] = mean |w|, op_c[oh][ow] = IC * taps inside.
// Replaces upstream src/bcast_binarize_weights.cpp:54-142.
cudaError_t launch_binarize_weights(const Plan &p, const float *w, void *bin_w, float *alpha,
                                    int32_t *op_c, cudaStream_t s);

// to = sign(from) * mean(from) over `elems` device floats (upstream
// src/binarize_weights_float.cpp:3-25), with a fixed summation shape. Block sums pass through the
// result, or, where it is small or also the source, through a kilobyte of stream-ordered scratch.
cudaError_t launch_binarize_weights_float(long elems, const float *from, float *to,
                                          cudaStream_t s);

// ---- convolution -----------------------------------------------------------------------------
// dst = ((float)S * alpha) * K with S the signed agreement count over in-bounds taps
// (upstream src/default/bcast_convolution_default.cpp:60-103). When `sums` is not null the raw
// integers S are written there (NCHW int32) and dst is left alone.
cudaError_t launch_conv_popc(const Plan &p, const uint32_t *bin_src, const uint32_t *bin_w,
                             const float *alpha, const float *k, const int32_t *op_c, float *dst,
                             int32_t *sums, cudaStream_t s);

// The same contract on the tensor cores (tcgen05.mma kind::mxf4 over +-1 nibbles, plan.hpp's framed
// layout). `error_word` is a device int the kernel sets non-zero if one of its bounded waits
// ran out; it is never cleared by the kernel. With k == nullptr the epilogue box-filters K from
// the mean-|x| map `a` itself (same arithmetic as launch_box_filter) and records it in k_out,
// which saves the separate stencil launch in the fused forward call.
//
// `next` chains two layers in the packed domain: instead of storing floats, the epilogue writes
// the sign of every result into the following layer's frame and the mean |result| over the
// filters into its mean-|x| map, which is what that layer's binarize_data and the first half of
// its calculate_k would have produced from the stored floats (upstream
// src/bcast_binarize_data.cpp:43-73, src/bcast_calculate_k.cpp:49-66). The signs are exact; the
// mean is summed per group of filters and folded in a fixed order, so it is reproducible but
// rounds differently from upstream's strictly sequential sum.
struct ChainTarget {
    void *bin_src;        // the next layer's res[bin_src]
    float *a;             // the next layer's res[a]
    int wp, hp, lead, icp;  // its frame geometry (Plan)
    float inv_ic;         // its Plan::inv_ic
};
cudaError_t launch_conv_tcgen05(const Plan &p, const void *bin_src, const void *bin_w,
                                const float *alpha, const float *k, const float *a, float *k_out,
                                float *dst, int32_t *sums, int *error_word, cudaStream_t s,
                                const ChainTarget *next = nullptr,
                                const ConvSelfTest *test = nullptr);

// A forward pass of a small layer in one launch (conv_whole.cu): packs the source, leaves frame and
// maps as launch_binarize_data and the convolution would, and stores the result. For the layers that
// whole_ok() names.
bool whole_ok(const Plan &p);
cudaError_t launch_conv_whole(const Plan &p, const float *src, void *bin_src, const void *bin_w,
                              const float *alpha, float *a, float *k, float *dst, int *error_word,
                              cudaStream_t s, const ConvSelfTest *test = nullptr);

// The same contract (without chaining) with the operand roles swapped: 128 filters on the UMMA M
// side, whole output rows of one image on the N side (Plan::img_*, conv_tcgen05_img.cu). Reads
// the same packed operands as launch_conv_tcgen05; the forward pass uses it when Plan::img is set.
cudaError_t launch_conv_tcgen05_img(const Plan &p, const void *bin_src, const void *bin_w,
                                    const float *alpha, const float *k, const float *a,
                                    float *k_out, float *dst, int32_t *sums, int *error_word,
                                    cudaStream_t s, const ConvSelfTest *test = nullptr);

}  // namespace xb200
