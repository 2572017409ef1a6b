// Exact-tile instantiations for groups of 8 lanes (packed FP32, gcp mode).
#include "fp32_tile.cuh"

namespace phmm {

void register_tile_gcp_g8(std::vector<ConfigInfo>& out) { register_tiles<8, 5, 20, true>(out); }

}  // namespace phmm
