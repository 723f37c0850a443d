// What the position-tile launcher hands the driver, without a GPU: its object files are linked against
// stand-ins for the few CUDA runtime calls it makes (a device of 148 SMs and 74 pairs of them, or
// as many pairs as the variable PAIRS says). For
// each layer on the command line (mb,oc,ic,ih,iw,kh,kw,sh,sw,ph,pw, and 1 for channels-last results) one line of
// JSON: the tensor maps it asked for, the launch, and the parameters that say which form of the kernel runs.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>

#include "conv_tile_args.cuh"
#include "kernels.cuh"

namespace xb200 {
std::atomic<long> g_kernel_launches{0};
}

static std::string g_maps, g_launch;

static CUresult fake_encode(CUtensorMap *map, CUtensorMapDataType, cuuint32_t rank, void *ptr,
                            const cuuint64_t *dim, const cuuint64_t *stride, const cuuint32_t *box,
                            const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle swizzle,
                            CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
    memset(map, 0, sizeof *map);
    char text[512];
    int n = snprintf(text, sizeof text, "%s{\"ptr\": %llu, \"swizzle\": %d", g_maps.empty() ? "" : ", ",
                     (unsigned long long)(uintptr_t)ptr, (int)swizzle);
    auto list = [&](const char *name, auto *v, unsigned count) {
        n += snprintf(text + n, sizeof text - n, ", \"%s\": [", name);
        for (unsigned i = 0; i < count; i++)
            n += snprintf(text + n, sizeof text - n, "%s%llu", i ? ", " : "", (unsigned long long)v[i]);
        n += snprintf(text + n, sizeof text - n, "]");
    };
    list("dim", dim, rank);
    list("stride", stride, rank - 1);
    list("box", box, rank);
    g_maps += std::string(text) + "}";
    return CUDA_SUCCESS;
}

extern "C" {
cudaError_t cudaGetDriverEntryPoint(const char *, void **fn, unsigned long long,
                                    cudaDriverEntryPointQueryResult *q) {
    *fn = (void *)fake_encode;
    *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : 0;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveClusters(int *n, const void *, const cudaLaunchConfig_t *) {
    const char *pairs = getenv("PAIRS");
    *n = pairs ? atoi(pairs) : 74;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *, void **args) {
    const xb200::TcArgs &g = *(const xb200::TcArgs *)args[2];
    const bool pair = c->numAttrs > 1 && c->attrs[1].val.clusterDim.x == 2;
    char text[512];
    snprintf(text, sizeof text,
             "\"grid\": %u, \"smem\": %zu, \"pair\": %s, \"planes\": %d, \"plane_rows\": %d, "
             "\"resident\": %d, \"halo\": %d, \"a_slots\": %d, \"stages\": %d, \"issuers\": %d, "
             "\"groups\": %d, \"kchunk\": %d, \"tap_kw\": %d, \"m_tiles\": %d, \"n_tiles\": %d, "
             "\"shared_cols\": %d, \"accumulators\": %d, \"epilogue_warps\": %u",
             c->gridDim.x, c->dynamicSmemBytes, pair ? "true" : "false", g.planes, g.plane_rows,
             g.resident, g.halo, g.n_a_slots, g.n_stages, g.issuers, g.kh * g.chunks_per_tap, g.kchunk,
             g.tap_kw, g.m_tiles, g.n_tiles, g.shared_cols, g.n_acc,
             c->blockDim.x / 32 - 3);
    g_launch = text;
    return cudaSuccess;
}
// referenced by the objects' registration code and host stubs, never needed here
cudaError_t cudaLaunchKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t) { abort(); }
unsigned __cudaPopCallConfiguration(dim3 *, dim3 *, size_t *, void *) { abort(); }
void **__cudaRegisterFatBinary(void *) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *,
                            dim3 *, int *) {}
}

int main(int argc, char **argv) {
    for (int i = 1; i < argc; i++) {
        xnor_nn_convolution_t c;
        memset(&c, 0, sizeof c);
        int last = 0;
        if (sscanf(argv[i], "%d,%d,%d,%d,%d,%d,%d,%d,%d,%d,%d,%d", &c.mb, &c.oc, &c.ic, &c.ih, &c.iw, &c.kh,
                   &c.kw, &c.sh, &c.sw, &c.ph, &c.pw, &last) < 11)
            return 2;
        c.oh = (c.ih + 2 * c.pw - c.kh) / c.sh + 1;
        c.ow = (c.iw + 2 * c.pw - c.kw) / c.sw + 1;
        c.src_format = xnor_nn_data_format_nchw;
        c.dst_format = last ? xnor_nn_data_format_nhwc : xnor_nn_data_format_nchw;
        c.weights_format = xnor_nn_weights_format_oihw;
        xb200::Plan plan;
        xb200::make_plan(&plan, &c, xb200::kAuto);
        const xb200::Plan view = xb200::conv_view(plan);
        g_maps.clear();
        g_launch.clear();
        if (plan.family != xb200::kTcgen05 || plan.img) {
            printf("{\"served\": false}\n");
            continue;
        }
        // addresses that no other layer of the run has: encodings are kept by them
        char *at = (char *)((uintptr_t)(3 * i + 1) << 36);
        const cudaError_t e = xb200::launch_conv_tcgen05(
            view, at, at + (1ull << 36), nullptr, nullptr, nullptr, nullptr, (float *)(at + (2ull << 36)),
            nullptr, nullptr, nullptr);
        printf("{\"served\": %s, \"activations\": %llu, \"rows\": %ld, \"icp\": %d, %s%s\"maps\": [%s]}\n",
               e == cudaSuccess ? "true" : "false", (unsigned long long)(uintptr_t)at, view.rows, view.icp,
               g_launch.c_str(), g_launch.empty() ? "" : ", ", g_maps.c_str());
    }
    return 0;
}
