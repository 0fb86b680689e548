// warp_sums.cuh -- sums of many FP64 (or FP32) values over a warp, in FP64.
//
// Reducing K values one after the other takes 5 K shuffle-and-add steps on all
// 32 lanes, and FP64 adds run at 1/64 of the FP32 rate on GB300: for the
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

// The same for FP32 values, summed as unevaluated pairs s + e of floats: each
// addition's rounding error (Knuth's two-sum, exact) goes to e, whose own
// rounding is 2^-24 of terms already 2^-24 small.  Eight FP32 instructions take
// the place of a conversion and an FP64 add that holds its quarter of the SM
// for 64 clocks.  Values whose sums could leave FP32's range, or infinities
// (two-sum makes them NaN), are summed in FP64.
__device__ __forceinline__ void pair_add(float &s, float &e, float t) {
  const float r = __fadd_rn(s, t), z = __fadd_rn(r, -s);
  e = __fadd_rn(e, __fadd_rn(__fadd_rn(s, -__fadd_rn(r, -z)), __fadd_rn(t, -z)));
  s = r;
}

template <int K>
__device__ __forceinline__ double warp_sum_pow2(float *v) {
  const int lane = threadIdx.x & 31;
  float big = 0.f;
#pragma unroll
  for (int i = 0; i < K; ++i) big = fmaxf(big, fabsf(v[i]));
  if (__any_sync(0xffffffffu, big > 0x1p120f)) {
    double d[K];
#pragma unroll
    for (int i = 0; i < K; ++i) d[i] = static_cast<double>(v[i]);
    return warp_sum_pow2<K>(d);
  }
  float e[K];
#pragma unroll
  for (int i = 0; i < K; ++i) e[i] = 0.f;
  int o = 16;
#pragma unroll
  for (int k = K; k > 1; k >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < k / 2; ++i) {
      const float send = up ? v[i] : v[i + k / 2];
      float s = up ? v[i + k / 2] : v[i], c = 0.f;
      if (k < K) c = (up ? e[i + k / 2] : e[i]) + __shfl_xor_sync(0xffffffffu, up ? e[i] : e[i + k / 2], o);
      pair_add(s, c, __shfl_xor_sync(0xffffffffu, send, o));
      v[i] = s;
      e[i] = c;
    }
  }
  float s = v[0], c = e[0];
#pragma unroll
  for (; o > 0; o >>= 1) {
    const float t = __shfl_xor_sync(0xffffffffu, s, o);
    c += __shfl_xor_sync(0xffffffffu, c, o);
    pair_add(s, c, t);
  }
  return static_cast<double>(s) + static_cast<double>(c);
}

template <int NK>
__device__ __forceinline__ void warp_sums(float *v, double *out) {
  constexpr int K = NK >= 32 ? 32 : NK >= 16 ? 16 : NK >= 8 ? 8 : NK >= 4 ? 4 : NK >= 2 ? 2 : 1;
  constexpr int kStep = 32 / K;
  const double s = warp_sum_pow2<K>(v);
  const int lane = threadIdx.x & 31;
  if ((lane & (kStep - 1)) == 0) out[lane / kStep] = s;
  if constexpr (NK > K) warp_sums<NK - K>(v + K, out + K);
}

}  // namespace doci
