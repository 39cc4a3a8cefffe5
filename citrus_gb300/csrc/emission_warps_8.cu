// The emission of 5 to 8 groups (emission_warps.cuh).
#include "emission_warps.cuh"

namespace citrus {

int emission_warps_8(const EmissionCall& c) {
  return launch_emission_warps<8>(c);
}

}  // namespace citrus
