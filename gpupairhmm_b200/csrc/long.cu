// Exact FP32 tiles of more than 32 lanes (reads of 641-4,096 positions), one read per
// group, default mode: one warp with two or three parts in turn, and blocks of 8 warps.
#include "fp32_tile.cuh"

namespace phmm {

void register_long(std::vector<ConfigInfo>& out) {
    register_long<2, 11, 24, false, true>(out);
    register_long<3, 17, 22, false, true>(out);
    register_long<8, 3, 16, false, false>(out);
}

}  // namespace phmm
