// Exact-tile instantiations for groups of 8 lanes (packed FP32, default mode).
#include "fp32_tile.cuh"

namespace phmm {

void register_tile_g8(std::vector<ConfigInfo>& out) { register_tiles<8, 5, 20, false>(out); }

}  // namespace phmm
