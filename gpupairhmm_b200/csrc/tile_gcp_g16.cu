// Exact-tile instantiations for groups of 16 lanes (packed FP32, gcp mode).
#include "fp32_tile.cuh"

namespace phmm {

void register_tile_gcp_g16(std::vector<ConfigInfo>& out) { register_tiles<16, 11, 20, true>(out); }

}  // namespace phmm
