// Exact tiles of the FP64 pass over blocks of 4 and 8 warps (reads of 641-4,096
// positions), both tiers, gcp mode.
#include "fp64_tile.cuh"

namespace phmm {

void register_long64_gcp(std::vector<Fp64Config>& out) {
    register_long64<4, 6, 16, true, false>(out);   // many pairs: scaled tier
    register_long64<8, 3, 16, true, true>(out);
}

}  // namespace phmm
