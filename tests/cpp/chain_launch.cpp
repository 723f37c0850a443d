// What the position-tile launcher does with the first of two chained layers: tile_launch.cpp's stand-ins, and
// for each layer on the command line (mb,oc,ic,ih,iw,kh,kw,ph,pw) one line of JSON with its launch.
#define main tile_launch_main
#include "tile_launch.cpp"
#undef main

int main(int argc, char **argv) {
    for (int i = 1; i < argc; i++) {
        xnor_nn_convolution_t c;
        memset(&c, 0, sizeof c);
        if (sscanf(argv[i], "%d,%d,%d,%d,%d,%d,%d,%d,%d", &c.mb, &c.oc, &c.ic, &c.ih, &c.iw, &c.kh, &c.kw,
                   &c.ph, &c.pw) != 9)
            return 2;
        c.sh = c.sw = 1;
        c.oh = c.ih + 2 * c.ph - c.kh + 1;
        c.ow = c.iw + 2 * c.pw - c.kw + 1;
        c.src_format = c.dst_format = xnor_nn_data_format_nchw;
        c.weights_format = xnor_nn_weights_format_oihw;
        xb200::Plan plan;
        xb200::make_plan(&plan, &c, xb200::kAuto);
        g_launch.clear();
        char *at = (char *)((uintptr_t)(3 * i + 1) << 36);
        xb200::ChainTarget next = {at + (2ull << 36), (float *)(at + (5ull << 35)), 16, 16, 0, 128, 1.f};
        const cudaError_t e = xb200::launch_conv_tcgen05(plan, at, at + (1ull << 36), nullptr, nullptr, nullptr,
                                                         nullptr, nullptr, nullptr, nullptr, nullptr, &next);
        printf("{\"served\": %s, %s}\n", e == cudaSuccess ? "true" : "false", g_launch.c_str());
    }
    return 0;
}
