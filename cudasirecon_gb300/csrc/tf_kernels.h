// Kernels compiled per factor pair of the two-factor transforms (tf_fft.cuh):
// one entry per length, spread over several translation units
// (k_tf_0.cu .. k_tf_7.cu) that build in parallel.
#pragma once
#include "filter.cuh"
#include "kernels.h"
#include "tf_fft.cuh"

namespace simrecon {

struct AsmX2Launch {
  const AssembleArgs* a;
  const Slot* slots;
  const int *p0, *pn, *pz;
  int nplanes;
  bool real;
};

constexpr int kMoMaxPhases = 9;
// makeotf's band separation and x half of the transform of every band
struct MoRowsArgs {
  const float* psf;  // [nz * nph][ny][n], phase fastest
  const float* bg;   // [nz * nph]
  int ny, nz, nph;
  float m[kMoMaxPhases * kMoMaxPhases];  // band = sum over phases of m[band * nph + phase] * section
  float2* bands;     // [nph][nz][ny][n/2+1]
};

// Every function returns a CUDA error code (0: launched).
struct TfKernels {
  int r1, r2;
  // zoomed x transform, ramps and sums of the assembly (even lengths; else null)
  int (*asm_x)(const AsmX2Launch& l, const TfPlan& pl, cudaStream_t s);
  // both overlaps' rows, inverse-transformed along x
  int (*ovl_x)(const OverlapArgs& a, const TfPlan& pl, cudaStream_t s);
  // inverse y transform of the overlap rows, products summed over groups of
  // kz planes; `columns`: columns per CTA (ovl_y_columns)
  int (*ovl_y)(const OverlapArgs& a, const TfPlan& pl, int planes_per_group, int groups, cudaStream_t s);
  int ovl_y_columns;
  // forward transform along the middle axis of [nplanes][n][ncol], in place
  int (*fft_cols)(float2* data, int ncol, int nplanes, const TfPlan& pl, cudaStream_t s);
  // forward transform of the conjugated rows of in[nrows][n]
  int (*fft_rows_conj)(const float2* in, float2* out, int nrows, const TfPlan& pl, cudaStream_t s);
  // flat field, edge blends and the x half of the 2D transform of every raw plane
  int (*ingest_x)(const IngestArgs& a, const TfPlan& pl, cudaStream_t s);
  int (*mo_rows)(const MoRowsArgs& a, const TfPlan& pl, cudaStream_t s);
};
// the kernels of length n and its plan; null where n has no factor pair
const TfKernels* tf_kernels(int n, TfPlan* plan);

// radial tables of two orders in the overlap build's shared memory
constexpr int kOvlTabMax = 1023;  // largest nxotf (32 KB)

}  // namespace simrecon
