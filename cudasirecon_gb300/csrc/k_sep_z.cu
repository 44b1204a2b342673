// Band separation and forward z transform for the z lengths of z_fft.cuh.
#include "z_fft.cuh"

namespace simrecon {

namespace {

constexpr int kThreads = 256;
constexpr int kW = 32;  // columns per CTA, of the (ky, kx) plane taken as one run

// A CTA takes kW consecutive elements of a direction's (ky, kx) plane through
// every z and phase.  First each thread separates one (z, column): the nph
// phases loaded together, scaled, mixed, left in shared memory as [band][z];
// then each thread transforms one (band, column) line, in registers (R2 = 1)
// or as the two factors in place: the thread for j reads and writes back the
// slots j + R2 e, so one buffer and one more barrier do.  Bound by HBM: read
// and written once.  640 x 384 x 30 x 15: 0.94 ms with the Stockham stages on
// [z][band] tiles, 0.187 ms here (4.7 TB/s).
template <int N, int R1, int NPH>
__global__ void __launch_bounds__(kThreads) k_separate_zn(float2* spec, const float* __restrict__ scale,
                                                        const float* __restrict__ sepmat, size_t plane,
                                                        const float2* __restrict__ tw)
{
  constexpr int R2 = N / R1;
  extern __shared__ __align__(16) float2 sm[];  // [NPH][N][kW]
  __shared__ float M[NPH * NPH];
  __shared__ float sc[NPH * N];
  const int d = blockIdx.y;
  for (int i = threadIdx.x; i < NPH * NPH; i += kThreads) M[i] = sepmat[i];
  for (int i = threadIdx.x; i < NPH * N; i += kThreads) sc[i] = scale ? scale[d * NPH * N + i] : 1.f;
  __syncthreads();
  const size_t e0 = (size_t)blockIdx.x * kW;
  const int nc = (int)(plane - e0 < kW ? plane - e0 : kW);
  float2* base = spec + (size_t)d * NPH * N * plane + e0;
  for (int t = threadIdx.x; t < N * kW; t += kThreads) {
    const int c = t % kW, z = t / kW;
    float2 in[NPH];
#pragma unroll
    for (int p = 0; p < NPH; ++p)
      in[p] = c < nc ? base[((size_t)p * N + z) * plane + c] : make_float2(0.f, 0.f);
#pragma unroll
    for (int p = 0; p < NPH; ++p) {
      const float s = sc[p * N + z];
      in[p] = make_float2(in[p].x * s, in[p].y * s);
    }
#pragma unroll
    for (int b = 0; b < NPH; ++b) {
      float2 acc = make_float2(0.f, 0.f);
#pragma unroll
      for (int p = 0; p < NPH; ++p) {
        const float m = M[b * NPH + p];
        acc.x += m * in[p].x;
        acc.y += m * in[p].y;
      }
      sm[(b * N + z) * kW + c] = acc;
    }
  }
  __syncthreads();
  if constexpr (R2 > 1) {
    for (int t = threadIdx.x; t < NPH * R2 * kW; t += kThreads) {
      const int c = t % kW, r = t / kW, b = r / R2, j = r - b * R2;
      float2* line = sm + (b * N + j) * kW + c;
      float2 v[R1];
#pragma unroll
      for (int e = 0; e < R1; ++e) v[e] = line[R2 * e * kW];
      reg_dft<R1, -1>(v);
#pragma unroll
      for (int k1 = 1; k1 < R1; ++k1) v[k1] = cmul(v[k1], __ldg(tw + j * k1));
#pragma unroll
      for (int k1 = 0; k1 < R1; ++k1) line[R2 * k1 * kW] = v[k1];
    }
    __syncthreads();
  }
  // R2 = 1: item (band, column) of R1 = N points; else (band, k1, column) of R2
  constexpr int K = R2 > 1 ? R1 : 1, L = R2 > 1 ? R2 : N;
  for (int t = threadIdx.x; t < NPH * K * kW; t += kThreads) {
    const int c = t % kW, r = t / kW, b = r / K, k1 = r - b * K;
    const float2* line = sm + (b * N + k1 * L) * kW + c;
    float2 u[L];
#pragma unroll
    for (int j = 0; j < L; ++j) u[j] = line[j * kW];
    reg_dft<L, -1>(u);
    if (c < nc) {
#pragma unroll
      for (int k2 = 0; k2 < L; ++k2) base[((size_t)b * N + k1 + K * k2) * plane + c] = u[k2];
    }
  }
}

template <int N, int R1, int NPH>
int run(float2* spec, const float* scale, const float* sepmat, size_t plane, int ndirs, const float2* tw,
        cudaStream_t s)
{
  constexpr size_t bytes = (size_t)NPH * N * kW * sizeof(float2);
  allow_dynamic_smem((const void*)k_separate_zn<N, R1, NPH>, bytes);
  k_separate_zn<N, R1, NPH><<<dim3((unsigned)((plane + kW - 1) / kW), ndirs), kThreads, bytes, s>>>(spec, scale,
                                                                                                 sepmat, plane, tw);
  return (int)cudaGetLastError();
}

}  // namespace

int launch_separate_z(float2* spec, const float* scale, const float* sepmat, size_t plane, int nz, int ndirs,
                      int nphases, const float2* tw, cudaStream_t s)
{
  switch (nz) {
#define SIMRECON_Z_CASE(N, R1)                                                              \
  case N:                                                                                   \
    return nphases == 5 ? run<N, R1, 5>(spec, scale, sepmat, plane, ndirs, tw, s)           \
                        : nphases == 3 ? run<N, R1, 3>(spec, scale, sepmat, plane, ndirs, tw, s) : -1;
    SIMRECON_Z_SIZES(SIMRECON_Z_CASE)
#undef SIMRECON_Z_CASE
  }
  return -1;
}

}  // namespace simrecon
