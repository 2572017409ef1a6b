// Exact-tile instantiations for groups of 32 lanes (packed FP32, gcp mode).
#include "fp32_tile.cuh"

namespace phmm {

void register_tile_gcp_g32(std::vector<ConfigInfo>& out) { register_tiles<32, 2, 20, true>(out); }

}  // namespace phmm
