// Pieces of the TFCE sweep shared by its two forms (tfce_sweep.cu,
// tfce_basin.cu): the threshold table, the threshold weight and the increment,
// with the reference's types and roundings.
#pragma once

#include <math_constants.h>

#include "common.cuh"

namespace tfgb {

constexpr int kMaxSteps = 128;

__host__ __device__ constexpr int64_t align16(int64_t x) { return (x + 15) / 16 * 16; }

__device__ inline void set_err(int32_t* err, int32_t code) { atomicCAS(err, 0, code); }

// HH = pow(T, H) as a float (fast_tfce.hpp:70), correctly rounded: T*T for
// H == 2 (exact product, one rounding), otherwise the double-precision power
// rounded once to float.  The reference calls the host libm's powf, which is
// not always correctly rounded (glibc: <= 0.82 ulp), so at rare thresholds
// its HH can sit one float ulp away from this value.
__device__ inline float pow_h(float T, float H) {
  if (H == 2.0f) return __fmul_rn(T, T);
  if (H == 1.0f) return T;
  return __double2float_rn(pow(static_cast<double>(T), static_cast<double>(H)));
}

// pow((double)extent, E) as the reference computes it (fast_tfce.hpp:77).
__device__ inline double extent_power(int32_t extent, float E) {
  if (E == 0.5f) return sqrt(static_cast<double>(extent));
  if (E == 2.0f) return static_cast<double>(extent) * static_cast<double>(extent);
  return pow(static_cast<double>(extent), static_cast<double>(E));
}

// The threshold table of one sweep: T = tmx, tmx - dT, ... while T >= 0 with
// dT = tmx / 100 in float (fast_tfce.hpp:34-39).  Returns the step count (0
// when there is no positive finite maximum).
__device__ inline int threshold_table(float tmx, float* T_out, int32_t* err) {
  int L = 0;
  if (tmx > 0.0f && isfinite(tmx)) {
    const float dT = __fdiv_rn(tmx, 100.0f);
    float T = tmx;
    while (T >= 0.0f) {
      if (L >= kMaxSteps) {
        set_err(err, kDevTooManySteps);
        return 0;
      }
      T_out[L++] = T;
      T = __fsub_rn(T, dT);
    }
  }
  return L;
}

__device__ inline float block_max(float v, float* red) {
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  if (w == 0) {
    v = (l < (int)(blockDim.x >> 5)) ? red[l] : -INFINITY;
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (l == 0) red[0] = v;
  }
  __syncthreads();
  const float r = red[0];
  __syncthreads();
  return r;
}

}  // namespace tfgb
