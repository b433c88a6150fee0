// Resident step kernels: meshes of 3 * 2^k points a side, 48 to 768.
#include "bd_resident.cuh"

namespace bd {
BD_RES_INSTANTIATE(20)
BD_RES_INSTANTIATE(21)
BD_RES_INSTANTIATE(22)
BD_RES_INSTANTIATE(23)
BD_RES_INSTANTIATE(24)
}  // namespace bd
