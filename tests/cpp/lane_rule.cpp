// Prints which variant of the lane density pass the rule takes for each (particles, warps, judge) given.
#include <cstdio>
#include <cstdlib>

#include "../../watercube_gb300/csrc/wc_lanes.h"

int main(int argc, char** argv) {
    for (int i = 1; i + 2 < argc; i += 3) {
        const uint32_t n = (uint32_t)std::atoi(argv[i]), warps = (uint32_t)std::atoi(argv[i + 1]);
        std::puts((std::atoi(argv[i + 2]) ? wc::judge_pairs(n, warps) : wc::lane_pairs(n, warps)) ? "pairs" : "one");
    }
}
