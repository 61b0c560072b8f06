// Prints trace_plan's choice for each "spheres rays both_outputs" triple given.
#include "venu_internal.h"

#include <cstdio>
#include <cstdlib>

int main(int argc, char** argv) {
    for (int i = 1; i + 2 < argc; i += 3) {
        const venu::TracePlan p =
            venu::trace_plan((uint32_t)std::strtoul(argv[i], nullptr, 10), (uint32_t)std::strtoul(argv[i + 1], nullptr, 10),
                             argv[i + 2][0] == '1', 152u);
        std::printf("%u %u %d\n", p.per_warp, p.grid, (int)p.walk);
    }
    return 0;
}
