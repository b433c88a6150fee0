// Resident step kernel of groups of CTAs: every mesh class in one kernel.
#include "bd_resident.cuh"

namespace bd {
BD_RES_INSTANTIATE_KIND(-1, RES_GROUPS)
}  // namespace bd
