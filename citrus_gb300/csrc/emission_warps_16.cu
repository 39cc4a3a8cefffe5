// The emission of 9 to 16 groups (emission_warps.cuh).
#include "emission_warps.cuh"

namespace citrus {

int emission_warps_16(const EmissionCall& c) {
  return launch_emission_warps<16>(c);
}

}  // namespace citrus
