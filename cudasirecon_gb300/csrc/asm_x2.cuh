// Zoomed x transform, phase ramp and weighted sum of the doubled-grid assembly
// (k_assemble2.cu), compiled per factor pair: the kernel's sums stay in
// registers over the plane's slots, so their count is a compile-time number.
// (One kernel that switched between the compiled sizes at run time spilled 2
// to 4 KB a thread and took minutes to build.)
// The pairs of all even lengths up to 1024 are spread over four translation
// units (k_asm_x2_0.cu .. _3.cu) to build in parallel.
// Per volume, against the Stockham stages on the doubled length: 1024^2 x 64
// 22.5 -> 3.2 ms, 640 x 384 x 30 2.61 -> 0.51 ms, 1024 x 960 0.243 -> 0.050 ms.
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
  TfPlan pl;
  cudaStream_t s;
};
// launch if the plan's pair belongs to the part; false otherwise
bool asm_x2_part0(const AsmX2Launch& l);
bool asm_x2_part1(const AsmX2Launch& l);
bool asm_x2_part2(const AsmX2Launch& l);
bool asm_x2_part3(const AsmX2Launch& l);

#define SIMRECON_X2_PAIRS_0(X) \
  X(8, 8) X(12, 8) X(12, 10) X(12, 12) X(14, 12) X(20, 10) X(16, 15) X(18, 15) X(20, 15) X(25, 14) \
  X(28, 14) X(28, 16) X(25, 20) X(28, 20) X(30, 21) X(28, 25) X(32, 24) X(30, 28) X(32, 30)
#define SIMRECON_X2_PAIRS_1(X) \
  X(9, 8) X(10, 10) X(14, 9) X(15, 10) X(15, 12) X(15, 14) X(25, 10) X(20, 14) X(20, 16) X(20, 18) \
  X(20, 20) X(25, 18) X(24, 21) X(24, 24) X(32, 20) X(30, 24) X(28, 28) X(32, 27) X(32, 32)
#define SIMRECON_X2_PAIRS_2(X) \
  X(10, 8) X(12, 9) X(16, 8) X(16, 10) X(16, 12) X(18, 12) X(18, 14) X(18, 16) X(18, 18) X(21, 18) \
  X(21, 20) X(24, 20) X(32, 16) X(28, 21) X(27, 24) X(30, 25) X(32, 25) X(32, 28)
#define SIMRECON_X2_PAIRS_3(X) \
  X(10, 9) X(14, 8) X(14, 10) X(18, 9) X(14, 14) X(16, 14) X(16, 16) X(21, 14) X(21, 16) X(24, 16) \
  X(24, 18) X(27, 18) X(27, 20) X(25, 24) X(28, 24) X(28, 27) X(30, 27) X(30, 30)

#ifdef __CUDACC__

// Geometry of a factor pair: W output rows per CTA of at most 128 threads
template <int R1, int R2>
struct X2 {
  static constexpr int N = R1 * R2, LD = R2 | 1;
  static constexpr int W = 64 / R1 > 0 ? 64 / R1 : 1;
  static constexpr int kItems = 2 * R1 * W;  // (row, parity, k1)
  static constexpr int kThreads = (kItems + 31) / 32 * 32;
  static constexpr int kBuf = kItems * LD;
  static constexpr size_t kSmem = 2 * (size_t)kBuf * sizeof(float2);
  // registers: the sums, one slot's stage-2 values and the next slot's loads
  static constexpr int kRegs = 4 * R2 + 2 * R1 + 45;
  static constexpr int kCtas = 65536 / (kThreads * kRegs) > 4 ? 4 : 65536 / (kThreads * kRegs);
};

// Thread (row, parity, k1) keeps the sums of its R2 output columns
// x = 2 (k1 + R1 k2) + parity over the plane's slots.  Stage 1 loads straight
// from T, the next slot's values before this slot's second stage (both
// parities' threads read the same ones, the second from L1); the exchange has
// two halves, so a slot costs one barrier.
// REAL output (Z = 1): the real part is the result itself.
template <int R1, int R2>
__global__ void __launch_bounds__(X2<R1, R2>::kThreads, X2<R1, R2>::kCtas)
    k_asm_x2(AssembleArgs a, const int* __restrict__ plane_slot0, const int* __restrict__ plane_nslot,
             const Slot* __restrict__ slots, const int* __restrict__ plane_zout, const float2* __restrict__ tw,
             const float2* __restrict__ twh, int real)
{
  using G = X2<R1, R2>;
  constexpr int N = G::N, X = 2 * N, LD = G::LD;
  extern __shared__ __align__(16) float2 sm[];
  const int Y = a.Y;
  const int pidx = gridDim.y - 1 - blockIdx.y;  // last-written slots first: they are still in L2
  const int s0 = plane_slot0[pidx], ns = plane_nslot[pidx], zout = plane_zout[pidx];
  const int y0 = blockIdx.x * G::W;
  // stage-1 item: j fastest, then parity, then row; stage-2 item: k1 fastest
  const int q1 = threadIdx.x / R2, j = threadIdx.x - q1 * R2, b1 = q1 & 1, l1 = q1 >> 1;
  const int q2 = threadIdx.x / R1, k1 = threadIdx.x - q2 * R1, b2 = q2 & 1, l2 = q2 >> 1;
  const bool act1 = l1 < G::W && y0 + l1 < Y, act2 = l2 < G::W && y0 + l2 < Y;
  const int yr2 = y0 + l2;
  float2 acc[R2];
#pragma unroll
  for (int k2 = 0; k2 < R2; ++k2) acc[k2] = make_float2(0.f, 0.f);
  float2 v[R1];
  auto load = [&](int si) {
    const float2* trow = a.T + ((size_t)(s0 + si) * Y + y0 + l1) * N;
#pragma unroll
    for (int e = 0; e < R1; ++e) {
      const int i = j + R2 * e;
      const bool neg = i > N / 2;
      v[e] = act1 ? trow[neg ? i - N / 2 - 1 : i + N / 2 - 1] : make_float2(0.f, 0.f);
    }
  };
  load(0);
  const float2* twp = b1 ? twh : tw;
  for (int si = 0; si < ns; ++si) {
    float2* buf = sm + (si & 1) * G::kBuf;
    if (act1) {
      if (b1) {
#pragma unroll
        for (int e = 0; e < R1; ++e)
          if (j + R2 * e > N / 2) v[e] = make_float2(-v[e].x, -v[e].y);
        tf_half_shift<R1, +1>(v);
      }
      reg_dft<R1, +1>(v);
      tf_twiddle<R1, +1>(v, twp, R2, j);
      float2* ex = buf + q1 * R1 * LD + j;
#pragma unroll
      for (int k = 0; k < R1; ++k) ex[k * LD] = v[k];
    }
    if (si + 1 < ns) load(si + 1);
    __syncthreads();
    if (act2) {
      float2 u[R2];
      const float2* ex = buf + (q2 * R1 + k1) * LD;
#pragma unroll
      for (int q = 0; q < R2; ++q) u[q] = ex[q];
      reg_dft<R2, +1>(u);
      const Slot sl = slots[s0 + si];
      if (sl.dir < 0) {  // the summed order-0 slot: ramp 1, weight 1
#pragma unroll
        for (int k2 = 0; k2 < R2; ++k2) acc[k2] = cadd(acc[k2], u[k2]);
      } else {
        const int ro = sl.dir * a.norders + sl.order;
        const float w = sl.order == 0 ? 1.f : 2.f;
        float2 ey = __ldg(a.ey + (size_t)ro * Y + yr2);
        ey.x *= w;
        ey.y *= w;
        const float2* exr = a.ex + (size_t)ro * X + b2 * N + k1;
#pragma unroll
        for (int k2 = 0; k2 < R2; ++k2) {
          const float2 e = cmul(__ldg(exr + R1 * k2), ey);
          const float2 t = cmul(u[k2], e);
          acc[k2].x += t.x;
          acc[k2].y += t.y;
        }
      }
    }
  }
  if (!act2) return;
  if (real) {
    float* dst = a.out + ((size_t)zout * Y + yr2) * X + 2 * k1 + b2;
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) dst[2 * R1 * k2] = acc[k2].x;
  } else {
    float2* dst = a.S + ((size_t)zout * Y + yr2) * X + b2 * N + k1;
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) dst[R1 * k2] = acc[k2];
  }
}

template <int R1, int R2>
inline bool asm_x2_run(const AsmX2Launch& l)
{
  using G = X2<R1, R2>;
  if (l.pl.r1 != R1 || l.pl.r2 != R2) return false;
  allow_dynamic_smem((const void*)k_asm_x2<R1, R2>, G::kSmem);
  k_asm_x2<R1, R2><<<dim3((l.a->Y + G::W - 1) / G::W, l.nplanes), G::kThreads, G::kSmem, l.s>>>(
      *l.a, l.p0, l.pn, l.slots, l.pz, l.pl.tw, l.pl.twh, l.real);
  return true;
}

#endif  // __CUDACC__

}  // namespace simrecon
