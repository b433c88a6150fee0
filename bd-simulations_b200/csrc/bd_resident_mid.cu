// Resident step kernels: meshes of 64 to 256.
#include "bd_resident.cuh"

namespace bd {
BD_RES_INSTANTIATE(6)
BD_RES_INSTANTIATE(7)
BD_RES_INSTANTIATE(8)
}  // namespace bd
