// Resident step kernels: meshes with a factor 3 and power-of-two meshes up to 32.
#include "bd_resident.cuh"

namespace bd {
BD_RES_INSTANTIATE(0)
BD_RES_INSTANTIATE(3)
BD_RES_INSTANTIATE(4)
BD_RES_INSTANTIATE(5)
}  // namespace bd
