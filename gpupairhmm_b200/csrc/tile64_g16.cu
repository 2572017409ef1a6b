// Exact-tile instantiations of the FP64 pass for groups of 16 lanes.
#include "fp64_tile.cuh"

namespace phmm {

void register_tile64_g16(std::vector<Fp64Config>& out) { register_tiles64<16, 11, 20>(out); }

}  // namespace phmm
