// The emission of 1 to 4 groups (emission_warps.cuh).
#include "emission_warps.cuh"

namespace citrus {

int emission_warps_4(const EmissionCall& c) {
  return c.tb.G <= 1 ? launch_emission_warps<1>(c) : c.tb.G <= 2 ? launch_emission_warps<2>(c) : launch_emission_warps<4>(c);
}

}  // namespace citrus
