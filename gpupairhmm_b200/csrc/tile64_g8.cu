// Exact-tile instantiations of the FP64 pass for groups of 8 lanes.
#include "fp64_tile.cuh"

namespace phmm {

void register_tile64_g8(std::vector<Fp64Config>& out) { register_tiles64<8, 5, 20>(out); }

}  // namespace phmm
