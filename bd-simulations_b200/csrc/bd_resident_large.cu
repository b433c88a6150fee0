// Resident step kernels: meshes of 512 and 1024.
#include "bd_resident.cuh"

namespace bd {
BD_RES_INSTANTIATE(9)
BD_RES_INSTANTIATE(10)
}  // namespace bd
