// pair_warp.h -- launch shape shared by the warp-per-unit pair kernels
// (sigma_pair_warp.cu, sigma_pair_warp64.cu).
#pragma once

#include <cstdint>

#include "internal.h"

namespace doci {

struct PwShape {
  uint32_t D;
  int L, N, na, nquads;
  long spin_limit;
  uint32_t n[16];    // C(P, j), 0 from j = P + 1
  uint32_t off[16];  // first set of j elements in the tables
};
PwShape pair_warp_shape(const doci_ham *h);
int ham_build_kdigits(doci_ham *h);
// the last pass of the reproducible form (sigma_pair_warp.cu)
template <typename T>
int launch_sum_slabs(const doci_ham *h, const T *slab, T *y, cudaStream_t st);

inline int cuda_ok(const char *what) {
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? static_cast<int>(DOCI_OK) : cuda_status(e, what);
}

}  // namespace doci
