// The assembly's inverse z transform and makeotf's forward one for the z
// lengths of z_fft.cuh.
#include "z_fft.cuh"

namespace simrecon {

namespace {

constexpr int kThreads = 256;

// where column x of a row of S is (the doubled-grid x pass stores the even
// columns, then the odd ones)
__device__ __forceinline__ size_t s_index(size_t t, int X, int split)
{
  if (!split) return t;
  const unsigned x = (unsigned)(t % X);
  return t - x + (x & 1) * (X >> 1) + (x >> 1);
}

// R2 = 1: one thread per output column (of the Y x X plane taken as one run)
// reads its in-band planes, transforms them in registers and stores the real
// parts.  Bound by HBM: 640 x 384 x 30: 0.62 ms with the Stockham stages,
// 0.058 ms here (6.0 TB/s).
template <int N>
__global__ void __launch_bounds__(kThreads) k_asm_zr(const float2* __restrict__ S, float* __restrict__ out, int X,
                                                   size_t n, unsigned long long active, int split)
{
  const size_t t = (size_t)blockIdx.x * kThreads + threadIdx.x;
  if (t >= n) return;
  const float2* src = S + s_index(t, X, split);
  float2 v[N];
#pragma unroll
  for (int z = 0; z < N; ++z) v[z] = (active >> z & 1) ? src[z * n] : make_float2(0.f, 0.f);
  reg_dft<N, +1>(v);
#pragma unroll
  for (int z = 0; z < N; ++z) out[z * n + t] = v[z].x;
}

// R2 > 1: 64 columns per CTA, two factors
constexpr int kW = 64;
template <int N, int R1>
__global__ void __launch_bounds__(kThreads) k_asm_z2(const float2* __restrict__ S, float* __restrict__ out, int X,
                                                   size_t n, unsigned long long active,
                                                   const float2* __restrict__ tw, int split)
{
  constexpr int R2 = N / R1;
  __shared__ float2 sm[N * kW];
  const size_t t0 = (size_t)blockIdx.x * kW;
  for (int it = threadIdx.x; it < R2 * kW; it += kThreads) {
    const int c = it % kW, j = it / kW;
    const size_t t = t0 + c;
    const float2* src = S + (t < n ? s_index(t, X, split) : 0);
    float2 v[R1];
#pragma unroll
    for (int e = 0; e < R1; ++e) {
      const int z = j + R2 * e;
      v[e] = (t < n && (active >> z & 1)) ? src[z * n] : make_float2(0.f, 0.f);
    }
    reg_dft<R1, +1>(v);
#pragma unroll
    for (int k1 = 1; k1 < R1; ++k1) {
      float2 w = __ldg(tw + j * k1);
      w.y = -w.y;
      v[k1] = cmul(v[k1], w);
    }
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) sm[(k1 * R2 + j) * kW + c] = v[k1];
  }
  __syncthreads();
  for (int it = threadIdx.x; it < R1 * kW; it += kThreads) {
    const int c = it % kW, k1 = it / kW;
    float2 u[R2];
#pragma unroll
    for (int j = 0; j < R2; ++j) u[j] = sm[(k1 * R2 + j) * kW + c];
    reg_dft<R2, +1>(u);
    if (t0 + c < n) {
#pragma unroll
      for (int k2 = 0; k2 < R2; ++k2) out[(k1 + R1 * k2) * n + t0 + c] = u[k2].x;
    }
  }
}

// Forward z transform in place: a thread per line, or the two factors over a
// tile of kW lines.  Bound by memory: 128 x 65 x 64 x 5 bands (21 MB, in L2)
// 10.5 us, 32 us by k_mo_fft_cols over full rows.
template <int N, int R1>
__global__ void __launch_bounds__(kThreads) k_z_forward(float2* data, size_t n, const float2* __restrict__ tw)
{
  constexpr int R2 = N / R1;
  float2* base = data + (size_t)blockIdx.y * N * n;
  if constexpr (R2 == 1) {
    const size_t t = (size_t)blockIdx.x * kThreads + threadIdx.x;
    if (t >= n) return;
    float2 v[N];
#pragma unroll
    for (int z = 0; z < N; ++z) v[z] = base[z * n + t];
    reg_dft<N, -1>(v);
#pragma unroll
    for (int z = 0; z < N; ++z) base[z * n + t] = v[z];
  } else {
    __shared__ float2 sm[N * kW];
    const size_t t0 = (size_t)blockIdx.x * kW;
    for (int it = threadIdx.x; it < R2 * kW; it += kThreads) {
      const int c = it % kW, j = it / kW;
      float2 v[R1];
#pragma unroll
      for (int e = 0; e < R1; ++e) v[e] = t0 + c < n ? base[(j + R2 * e) * n + t0 + c] : make_float2(0.f, 0.f);
      reg_dft<R1, -1>(v);
#pragma unroll
      for (int k1 = 1; k1 < R1; ++k1) v[k1] = cmul(v[k1], __ldg(tw + j * k1));
#pragma unroll
      for (int k1 = 0; k1 < R1; ++k1) sm[(k1 * R2 + j) * kW + c] = v[k1];
    }
    __syncthreads();
    for (int it = threadIdx.x; it < R1 * kW; it += kThreads) {
      const int c = it % kW, k1 = it / kW;
      float2 u[R2];
#pragma unroll
      for (int j = 0; j < R2; ++j) u[j] = sm[(k1 * R2 + j) * kW + c];
      reg_dft<R2, -1>(u);
      if (t0 + c < n) {
#pragma unroll
        for (int k2 = 0; k2 < R2; ++k2) base[(k1 + R1 * k2) * n + t0 + c] = u[k2];
      }
    }
  }
}

template <int N, int R1>
int run_forward(float2* data, int nbands, size_t n, const float2* tw, cudaStream_t s)
{
  constexpr int per = N == R1 ? kThreads : kW;
  k_z_forward<N, R1><<<dim3((unsigned)((n + per - 1) / per), nbands), kThreads, 0, s>>>(data, n, tw);
  return (int)cudaGetLastError();
}

template <int N, int R1>
int run(const float2* S, float* out, int X, size_t n, unsigned long long active, const float2* tw, int split,
        cudaStream_t s)
{
  if constexpr (N == R1)
    k_asm_zr<N><<<(unsigned)((n + kThreads - 1) / kThreads), kThreads, 0, s>>>(S, out, X, n, active, split);
  else
    k_asm_z2<N, R1><<<(unsigned)((n + kW - 1) / kW), kThreads, 0, s>>>(S, out, X, n, active, tw, split);
  return (int)cudaGetLastError();
}

}  // namespace

int launch_asm_zn(const float2* S, float* out, int X, int Y, int Z, unsigned long long active, const float2* tw,
                  int split, cudaStream_t s)
{
  const size_t n = (size_t)X * Y;
  switch (Z) {
#define SIMRECON_Z_CASE(N, R1) \
  case N:                      \
    return run<N, R1>(S, out, X, n, active, tw, split, s);
    SIMRECON_Z_SIZES(SIMRECON_Z_CASE)
#undef SIMRECON_Z_CASE
  }
  return -1;
}

int launch_z_forward(float2* data, int nz, int nbands, size_t plane, const float2* tw, cudaStream_t s)
{
  switch (nz) {
#define SIMRECON_Z_CASE(N, R1) \
  case N:                      \
    return run_forward<N, R1>(data, nbands, plane, tw, s);
    SIMRECON_Z_SIZES(SIMRECON_Z_CASE)
#undef SIMRECON_Z_CASE
  }
  return -1;
}

}  // namespace simrecon
