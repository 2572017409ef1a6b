// Exact tiles of the FP64 pass over blocks of 4 and 8 warps (reads of 641-4,096
// positions), both tiers, default mode.
#include "fp64_tile.cuh"

namespace phmm {

void register_long64(std::vector<Fp64Config>& out) {
    register_long64<4, 6, 16, false, false>(out);   // many pairs: scaled tier
    register_long64<8, 3, 16, false, true>(out);
}

}  // namespace phmm
