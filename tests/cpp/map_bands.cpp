// Which pixels the blocks of calculate_k in one launch read (map_bands.cuh, pixel_tasks.cuh), with tile_launch.cpp's
// stand-ins: for each layer on the command line (mb,oc,ic,ih,iw,kh,kw,sh,sw,ph,pw) one line of JSON with the least and
// the greatest pixel that any lane reads, the pixels of the source, blocks without a pixel, the rows of A that
// one block leaves in the map and that others leave too or none does, and the limits of a block.
#define main tile_launch_main
#include "tile_launch.cpp"
#undef main

#include <algorithm>
#include <vector>

#include "map_bands.cuh"
#include "pixel_tasks.cuh"

int main(int argc, char **argv) {
    using namespace xb200;
    for (int i = 1; i < argc; i++) {
        xnor_nn_convolution_t c;
        memset(&c, 0, sizeof c);
        if (sscanf(argv[i], "%d,%d,%d,%d,%d,%d,%d,%d,%d,%d,%d", &c.mb, &c.oc, &c.ic, &c.ih, &c.iw, &c.kh,
                   &c.kw, &c.sh, &c.sw, &c.ph, &c.pw) != 11)
            return 2;
        c.oh = (c.ih + 2 * c.pw - c.kh) / c.sh + 1;
        c.ow = (c.iw + 2 * c.pw - c.kw) / c.sw + 1;
        Plan plan;
        make_plan(&plan, &c, kAuto);
        bands::MapArgs g;
        if (!bands::maps_shape(plan, &g)) {
            printf("{\"served\": false}\n");
            continue;
        }
        g.hw = c.ih * c.iw; g.ih = c.ih; g.iw = c.iw; g.sh = c.sh; g.ph = c.ph;
        long least = 0, most = 0, last = 0;
        int empty = 0, groups = 0, tasks = 0, wrong = 0;
        std::vector<int> owners((size_t)c.mb * c.ih);
        for (int block = 0; block < c.mb * g.bands; block++) {
            const bands::Band b = bands::band_of(g, block);
            empty += b.tasks == 0;
            groups = std::max(groups, b.groups);
            tasks = std::max(tasks, b.tasks);
            last = std::max(last, (long)b.last);
            for (int gr = 0; gr < (b.tasks ? b.groups : 0); gr++)
                for (int lane = 0; lane < 32; lane++) {
                    const int px = tasks::lane_pixel(b.first, b.last, gr, lane);
                    least = std::min(least, (long)px);
                    most = std::max(most, (long)px);
                }
            for (int px = b.first; px < b.last; px += c.iw) {  // as maps_kernel has it
                const int y = (px - b.n * g.hw) / c.iw;
                if (y >= b.own0 && y < b.own1) owners[(size_t)b.n * c.ih + y]++;
            }
        }
        for (int n : owners) wrong += n != 1;
        printf("{\"served\": true, \"least\": %ld, \"most\": %ld, \"last\": %ld, \"pixels\": %ld, \"blocks\": %d, "
               "\"empty\": %d, \"groups\": %d, \"tasks\": %d, \"rows_not_left_once\": %d}\n",
               least, most, last, (long)c.mb * g.hw, c.mb * g.bands, empty, groups, tasks, wrong);
    }
    return 0;
}
