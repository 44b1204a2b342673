// Short z transforms of any length with a compiled pair (R1, R2): R2 = 1 up to
// 32 planes (the whole line in one thread's registers), else R1 R2 as a
// two-factor transform through shared memory.
#pragma once
#include "kernels.h"
#include "reg_fft.cuh"

namespace simrecon {

// X(N, R1) of every length; R2 = N / R1
#define SIMRECON_Z_SIZES(X)                                                                                     \
  X(2, 2) X(3, 3) X(4, 4) X(5, 5) X(6, 6) X(7, 7) X(8, 8) X(9, 9) X(10, 10) X(12, 12) X(14, 14) X(15, 15)       \
  X(16, 16) X(18, 18) X(20, 20) X(21, 21) X(24, 24) X(25, 25) X(27, 27) X(28, 28) X(30, 30) X(32, 32) X(35, 7)  \
  X(36, 6) X(40, 8) X(42, 7) X(45, 9) X(48, 8) X(49, 7) X(50, 10) X(54, 9) X(56, 8) X(60, 10) X(63, 9) X(64, 8)

constexpr bool z_length_ok(int n)
{
#define SIMRECON_Z_OK(N, R1) \
  if (n == N) return true;
  SIMRECON_Z_SIZES(SIMRECON_Z_OK)
#undef SIMRECON_Z_OK
  return false;
}

// Separation and forward z transform of every direction, in place (nphases 3
// or 5, z_length_ok(nz)); tw: the plan's table of nz twiddles
int launch_separate_z(float2* spec, const float* scale, const float* sepmat, size_t plane, int nz, int ndirs,
                      int nphases, const float2* tw, cudaStream_t s);
// inverse z transform of S (planes of `active`, bit z), real part -> out
// (z_length_ok(Z)); split: S has its columns split by parity
int launch_asm_zn(const float2* S, float* out, int X, int Y, int Z, unsigned long long active, const float2* tw,
                  int split, cudaStream_t s);

// forward z transform of nbands volumes [nz][plane], in place (z_length_ok(nz))
int launch_z_forward(float2* data, int nz, int nbands, size_t plane, const float2* tw, cudaStream_t s);

}  // namespace simrecon
