// Two-factor transforms of the lengths n = R1 * R2 with both factors among 16
// compiled DFT sizes: most lengths from 64 to 1024, and 256, 512 and 1024 where
// their own kernels were slower.
//
//   X[k1 + R1 k2] = sum_j W_n^(j k1) W_R2^(j k2) sum_e x[j + R2 e] W_R1^(e k1)
//
// Stage 1: the thread for (line, j < R2) takes x[j + R2 e] (e < R1), runs an
// in-register DFT of R1 points, multiplies by W_n^(j k1) and leaves the R1
// values in shared memory; stage 2: the thread for (line, k1 < R1) takes the
// R2 values over j, runs an in-register DFT of R2 points and holds X[k1 + R1 k2].
// One shared-memory round trip and two barriers per tile, where the Stockham
// stages make one per radix and two more to fill and empty the tile.
//
// The kernels are compiled per pair (tf_kernels.cuh, instantiated in
// k_tf_0.cu .. k_tf_7.cu).  k_asm_y2 alone chooses R1 and R2 at run time
// (tf_switch: a branch that the whole CTA takes alike), as its filter is most of
// its code; its registers are those of the largest size it may take, hence its
// two classes MR = 16 and 32.
//
// Half-shifted form: the outputs of a transform zero-padded to twice its
// length fall into two of length n, the even ones of x and the odd ones of
// x[i] exp(DIR i pi k_i / n) with k_i the signed frequency i or i - n.  With
// i = j + R2 e the factor is exp(DIR i pi e / R1) (a constant of the DFT)
// times exp(DIR i pi j / n) (part of the stage twiddle), negated for k_i < 0.
#pragma once
#include "reg_fft.cuh"

namespace simrecon {

struct TfPlan {
  int n, r1, r2;
  const float2* tw;   // [r1][r2]: exp(-2 pi i j k1 / n) at k1 * r2 + j
  const float2* twh;  // the same times exp(-i pi j / n)
};
// r1 >= r2 from the compiled sizes with r1 * r2 = n, the pair with the smallest r1
bool tf_factor(int n, int* r1, int* r2);
// plan with device twiddles, cached per (device, n); false where n has no pair
bool get_tf_plan(int n, TfPlan* plan);

// The path that `site` runs length n by: what the launchers take and what
// SRX_fftPath reports.  The lengths of the assembly's x and y sites are those of
// the doubled grid, the z separation's those of 5-phase stacks.
int fft_path(FftSite site, int n);
// neither a force, the environment nor the plan cache names the register path
// or the Stockham stages for length n at `site`
bool fft_plan_open(FftSite site, int n);
// whether `site` has a two-factor kernel for length n that a plan may choose
bool fft_two_factor_choice(FftSite site, int n);

constexpr int kTfSizes[] = {8, 9, 10, 12, 14, 15, 16, 18, 20, 21, 24, 25, 27, 28, 30, 32};
// k_asm_y2's class of a plan: the largest DFT it needs
inline int tf_class(const TfPlan& p) { return p.r1 <= 16 ? 16 : 32; }

#ifdef __CUDACC__

// f.template operator()<R>() for the compiled size R == r, r <= MR
template <int MR, typename F>
__device__ __forceinline__ void tf_switch(int r, F&& f)
{
  switch (r) {
#define SIMRECON_TF_CASE(R) \
  case R:                   \
    if constexpr (R <= MR) f.template operator()<R>(); \
    break;
    SIMRECON_TF_CASE(8)
    SIMRECON_TF_CASE(9)
    SIMRECON_TF_CASE(10)
    SIMRECON_TF_CASE(12)
    SIMRECON_TF_CASE(14)
    SIMRECON_TF_CASE(15)
    SIMRECON_TF_CASE(16)
    SIMRECON_TF_CASE(18)
    SIMRECON_TF_CASE(20)
    SIMRECON_TF_CASE(21)
    SIMRECON_TF_CASE(24)
    SIMRECON_TF_CASE(25)
    SIMRECON_TF_CASE(27)
    SIMRECON_TF_CASE(28)
    SIMRECON_TF_CASE(30)
    SIMRECON_TF_CASE(32)
#undef SIMRECON_TF_CASE
  }
}

// v[e] *= exp(DIR i pi e / R): the half shift's constant part
template <int R, int DIR>
__device__ __forceinline__ void tf_half_shift(float2* v)
{
#pragma unroll
  for (int e = 1; e < R; ++e) v[e] = cmul(v[e], w_root<2 * R>(e, DIR));
}

// v[k1] *= W_n^(j k1) from the plan's table tw, k1 * r2 + j (k1 = 0: 1)
template <int R, int DIR>
__device__ __forceinline__ void tf_twiddle(float2* v, const float2* __restrict__ tw, int r2, int j)
{
#pragma unroll
  for (int k1 = 1; k1 < R; ++k1) {
    float2 w = __ldg(tw + k1 * r2 + j);
    if (DIR > 0) w.y = -w.y;
    v[k1] = cmul(v[k1], w);
  }
}

// the same from tw or, half shifted, twh (whose k1 = 0 is not 1)
template <int R, int DIR>
__device__ __forceinline__ void tf_twiddle_half(float2* v, const float2* __restrict__ tw, int r2, int j)
{
#pragma unroll
  for (int k1 = 0; k1 < R; ++k1) {
    float2 w = __ldg(tw + k1 * r2 + j);
    if (DIR > 0) w.y = -w.y;
    v[k1] = cmul(v[k1], w);
  }
}

#endif  // __CUDACC__

}  // namespace simrecon
