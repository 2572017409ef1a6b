// Exact-tile instantiations for groups of 16 lanes (packed FP32, default mode).
#include "fp32_tile.cuh"

namespace phmm {

void register_tile_g16(std::vector<ConfigInfo>& out) { register_tiles<16, 11, 20, false>(out); }

}  // namespace phmm
