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

// What the CTAs of blockIdx.y transform: a raw section and the plane of spec it
// goes to.  The whole stack is taken in plane order (the y pass follows in the
// reverse of it), a part of it in section order.
struct IngestPlane {
  int section, plane;  // plane id = (d*nph + p)*nz + z
};
__device__ __forceinline__ IngestPlane ingest_plane(const IngestArgs& a)
{
  int d, p, z;
  if (a.nsec == 0) {
    const int pl = blockIdx.y, dp = pl / a.nz;
    z = pl - dp * a.nz;
    d = dp / a.nphases;
    p = dp - d * a.nphases;
    return IngestPlane{raw_section(d, p, z, a.nz, a.ndirs, a.nphases, a.fastSI), pl};
  }
  const int s = a.sec0 + blockIdx.y, q = s / a.nphases;
  p = s - q * a.nphases;
  if (a.fastSI) {
    z = q / a.ndirs;
    d = q - z * a.ndirs;
  } else {
    d = q / a.nz;
    z = q - d * a.nz;
  }
  return IngestPlane{s, (d * a.nphases + p) * a.nz + z};
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
