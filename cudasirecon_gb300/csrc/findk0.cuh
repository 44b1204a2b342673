// findk0's peak refinement on the device (gpuFunctionsImpl.cu:306-372), with
// the reference host code's separately rounded float operations.
#pragma once
#include "kernels.h"

namespace simrecon {

#ifdef __CUDACC__

// fitparabola, gpuFunctionsImpl.cu:479-495
__device__ __forceinline__ float fitparabola_rn(float a1, float a2, float a3)
{
  const float slope = __fmul_rn(0.5f, __fsub_rn(a3, a1));
  const float curve = __fsub_rn(__fadd_rn(a3, a1), __fmul_rn(2.f, a2));
  if (curve == 0.f) return 0.f;
  const float peak = __fdiv_rn(-slope, curve);
  if (peak > 1.5f || peak < -1.5f) return 0.f;
  return peak;
}

__device__ __forceinline__ float2 polar_rn(float mag, float angle)
{
  return make_float2(__fmul_rn(mag, cosf(angle)), __fmul_rn(mag, sinf(angle)));
}

// findk0's tail (gpuFunctionsImpl.cu:345-371): peak = {ix, iy, a1x, a2, a3x,
// a1y, a3y}; k0 = the parabola-refined peak, moved by a period towards the
// guess, over fitorder2.  k1 = k0 through (|k0|, atan2) and back: the vector
// the search's first getmodamp rebuilds the overlaps at.
__device__ __forceinline__ void findk0_finish(const float* pk, float2 guess, int nx, int ny, float dkx, float dky,
                                              int fitorder2, float2* k0out, float2* k1out)
{
  const int xcent = (int)pk[0], ycent = (int)pk[1];
  float peakx = __fadd_rn(fitparabola_rn(pk[2], pk[3], pk[4]), (float)xcent);
  float peaky = __fadd_rn(fitparabola_rn(pk[5], pk[3], pk[6]), (float)ycent);
  if (__fdiv_rn(guess.x, dkx) < __fsub_rn(peakx, (float)(nx / 2))) peakx = __fsub_rn(peakx, (float)nx);
  if (__fdiv_rn(guess.x, dkx) > __fadd_rn(peakx, (float)(nx / 2))) peakx = __fadd_rn(peakx, (float)nx);
  if (__fdiv_rn(guess.y, dky) < __fsub_rn(peaky, (float)(ny / 2))) peaky = __fsub_rn(peaky, (float)ny);
  if (__fdiv_rn(guess.y, dky) > __fadd_rn(peaky, (float)(ny / 2))) peaky = __fadd_rn(peaky, (float)ny);
  const float2 k0 = make_float2(__fmul_rn(peakx, __fdiv_rn(dkx, (float)fitorder2)),
                                __fmul_rn(peaky, __fdiv_rn(dky, (float)fitorder2)));
  *k0out = k0;
  const float mag = __fsqrt_rn(__fadd_rn(__fmul_rn(k0.x, k0.x), __fmul_rn(k0.y, k0.y)));
  *k1out = polar_rn(mag, atan2f(k0.y, k0.x));
}

#endif  // __CUDACC__

}  // namespace simrecon
