// Exact-tile instantiations of the FP64 pass for groups of 32 lanes.
#include "fp64_tile.cuh"

namespace phmm {

void register_tile64_g32(std::vector<Fp64Config>& out) { register_tiles64<32, 2, 20>(out); }

}  // namespace phmm
