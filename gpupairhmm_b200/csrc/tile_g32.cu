// Exact-tile instantiations for groups of 32 lanes (packed FP32, default mode).
#include "fp32_tile.cuh"

namespace phmm {

void register_tile_g32(std::vector<ConfigInfo>& out) { register_tiles<32, 2, 20, false>(out); }

}  // namespace phmm
