// Exact FP32 tiles of more than 32 lanes (reads of 641-4,096 positions), one read per
// group, gcp mode: one warp with two or three parts in turn, and blocks of 8 warps.
#include "fp32_tile.cuh"

namespace phmm {

void register_long_gcp(std::vector<ConfigInfo>& out) {
    register_long<2, 11, 24, true, true>(out);
    register_long<3, 17, 22, true, true>(out);
    register_long<8, 3, 16, true, false>(out);
}

}  // namespace phmm
