// warp_sums.cuh -- sums of many FP64 values over a warp.
//
// Reducing K values one after the other takes 5 K shuffle-and-add steps on all
// 32 lanes, and FP64 adds run at two lanes per clock and SM on GB300: for the
// 33 projections of a block of 8 warps that is about 10 us per block, more
// than the pass's own reads on a small vector.  Here the lanes split the
// values instead: in the first step a lane keeps half of them and hands the
// other half to its partner 16 lanes away, then a quarter, and so on, so K
// values take K - 1 + (5 - log2 K) adds.  The order is fixed.
#pragma once

#include <cuda_runtime.h>

namespace doci {

// K a power of two <= 32: the sum of v[lane >> (5 - log2 K)] over the warp's
// lanes, in every lane; v is overwritten
template <int K>
__device__ __forceinline__ double warp_sum_pow2(double *v) {
  const int lane = threadIdx.x & 31;
  int o = 16;
#pragma unroll
  for (int k = K; k > 1; k >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < k / 2; ++i) {
      const double keep = up ? v[i + k / 2] : v[i], send = up ? v[i] : v[i + k / 2];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  double s = v[0];
#pragma unroll
  for (; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// out[k] = the sum of v[k] over the warp's lanes, k < NK (v is overwritten)
template <int NK>
__device__ __forceinline__ void warp_sums(double *v, double *out) {
  constexpr int K = NK >= 32 ? 32 : NK >= 16 ? 16 : NK >= 8 ? 8 : NK >= 4 ? 4 : NK >= 2 ? 2 : 1;
  constexpr int kStep = 32 / K;
  const double s = warp_sum_pow2<K>(v);
  const int lane = threadIdx.x & 31;
  if ((lane & (kStep - 1)) == 0) out[lane / kStep] = s;
  if constexpr (NK > K) warp_sums<NK - K>(v + K, out + K);
}

}  // namespace doci
