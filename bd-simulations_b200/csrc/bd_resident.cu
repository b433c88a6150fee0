// Dispatch of the resident step kernels by mesh size.
#include "bd_kernels.h"

namespace bd {

template <int LZ, int KIND>
int resident_attributes_t();
template <int LZ, int KIND>
int resident_held_t(size_t smem, int cs, int nsm, int* n);
template <int LZ, int KIND>
int launch_resident_t(const ResArgs& A, int nclusters, int cs, int grid, size_t smem, cudaStream_t s);

int resident_attributes(int lz, int kind) {
  if (kind == RES_GROUPS) return resident_attributes_t<-1, RES_GROUPS>();
  switch (lz) {
#define BD_CASE(L)                                                                                      \
  case L:                                                                                               \
    return kind == RES_SINGLE ? resident_attributes_t<L, RES_SINGLE>() : resident_attributes_t<L, RES_CLUSTERS>();
    BD_RES_SIZES(BD_CASE)
#undef BD_CASE
    default:
      return (int)cudaErrorInvalidValue;
  }
}

int resident_held(int lz, int kind, size_t smem, int cs, int device, int* n) {
  *n = 0;
  int nsm = 0;
  cudaError_t e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) return (int)e;
  if (kind == RES_GROUPS) return resident_held_t<-1, RES_GROUPS>(smem, 0, nsm, n);
  switch (lz) {
#define BD_CASE(L)                                                       \
  case L:                                                                \
    return kind == RES_SINGLE ? resident_held_t<L, RES_SINGLE>(smem, cs, nsm, n)      \
                              : resident_held_t<L, RES_CLUSTERS>(smem, cs, nsm, n);
    BD_RES_SIZES(BD_CASE)
#undef BD_CASE
    default:
      return (int)cudaErrorInvalidValue;
  }
}

int launch_resident(int lz, int kind, const ResArgs& A, int nclusters, int cs, int grid, size_t smem,
                    cudaStream_t s) {
  if (kind == RES_GROUPS) return launch_resident_t<-1, RES_GROUPS>(A, 0, 0, grid, smem, s);
  switch (lz) {
#define BD_CASE(L)                                                             \
  case L:                                                                      \
    return kind == RES_SINGLE ? launch_resident_t<L, RES_SINGLE>(A, nclusters, cs, grid, smem, s) \
                              : launch_resident_t<L, RES_CLUSTERS>(A, nclusters, cs, grid, smem, s);
    BD_RES_SIZES(BD_CASE)
#undef BD_CASE
    default:
      return (int)cudaErrorInvalidValue;
  }
}

}  // namespace bd
