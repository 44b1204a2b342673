// Per-pixel load steps shared by the ingest kernels: section order, flat field.
#pragma once
#include "kernels.h"

namespace simrecon {

#ifdef __CUDACC__

__device__ __forceinline__ int raw_section(int d, int p, int z, int nz, int ndirs, int nph, int fastSI)
{
  // loadImageData section order, cudaSirecon.cpp:1374-1382
  return fastSI ? (z * ndirs * nph + d * nph + p) : (d * nz * nph + z * nph + p);
}

template <typename T>
__device__ __forceinline__ float flat(const T* __restrict__ plane, const IngestArgs& a, int y, int x)
{
  float v = (float)plane[(size_t)y * a.nx + x];
  float bg = a.bg ? __ldg(a.bg + (size_t)y * a.nx + x) : a.bgconst;
  float sl = a.slope ? __ldg(a.slope + (size_t)y * a.nx + x) : 1.0f;
  return (v - bg - a.bgextra) * sl * a.inscale;
}

// flat() for a raw value already loaded
__device__ __forceinline__ float flat_v(float v, const IngestArgs& a, int y, int x)
{
  float bg = a.bg ? __ldg(a.bg + (size_t)y * a.nx + x) : a.bgconst;
  float sl = a.slope ? __ldg(a.slope + (size_t)y * a.nx + x) : 1.0f;
  return (v - bg - a.bgextra) * sl * a.inscale;
}

#endif  // __CUDACC__

}  // namespace simrecon
