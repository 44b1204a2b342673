// The kernels of tf_kernels.h for one factor pair (R1, R2), R1 >= R2.
#pragma once
#include "ingest_dev.cuh"
#include "tf_kernels.h"

namespace simrecon {

#ifdef __CUDACC__

// ------------------------------------------------------------------ columns
// W adjacent columns of length N per CTA.  Here the smaller factor is the first
// stage's: more threads with fewer loads each keep the reads going (512 rows:
// 0.28 against 0.34 ms per 512^2 x 48 volume).  Stage-1 item (column fastest,
// j < R1), stage-2 item (column fastest, k1 < R2); the k1 pitch is an odd
// multiple of W: the stage-2 reads of a half-warp hit distinct banks.
template <int R1, int R2>
struct TfCol {
  static constexpr int N = R1 * R2;
  static constexpr int W = R1 <= 16 ? 16 : 8;
  static constexpr int LD = (R1 | 1) * W;
  static constexpr int kThreads = (R1 * W + 31) / 32 * 32;
  static constexpr size_t kSmem = (size_t)R2 * LD * sizeof(float2);
  // a stage's values and addresses
  static constexpr int kRegs = 2 * R1 + 52;
  static constexpr int kCtas = 65536 / (kThreads * kRegs) > 6 ? 6 : 65536 / (kThreads * kRegs);
};

// Forward transform along the middle axis of [nplanes][N][ncol], in place:
// loaded and stored once, rows of 64 or 128 bytes (a last column tile may be
// ragged).  Bound by HBM: 640 x 384 x 30 spectra 0.785 -> 0.185 ms (4.8 TB/s)
// against the Stockham stages, 1024 x 960 0.067 -> 0.020 ms.
template <int R1, int R2>
__global__ void __launch_bounds__(TfCol<R1, R2>::kThreads, TfCol<R1, R2>::kCtas)
    k_tf_cols(float2* data, int ncol, const float2* __restrict__ tw)
{
  using G = TfCol<R1, R2>;
  constexpr int N = G::N, W = G::W;
  extern __shared__ __align__(16) float2 sm[];
  const int c0 = blockIdx.x * W;
  // planes in the reverse of the order the x pass wrote them: the last ones
  // written are still in L2 when the first CTAs read them
  const int plane = gridDim.y - 1 - blockIdx.y;
  float2* base = data + (size_t)plane * N * ncol + c0;
  const int c = threadIdx.x % W, q = threadIdx.x / W;
  const bool in = c0 + c < ncol;
  if (q < R1) {  // x[q + R1 e]
    float2 v[R2];
#pragma unroll
    for (int e = 0; e < R2; ++e) v[e] = in ? base[(size_t)(q + R1 * e) * ncol + c] : make_float2(0.f, 0.f);
    reg_dft<R2, -1>(v);
#pragma unroll
    for (int k1 = 1; k1 < R2; ++k1) v[k1] = cmul(v[k1], __ldg(tw + q * R2 + k1));  // W_N^(q k1)
#pragma unroll
    for (int k1 = 0; k1 < R2; ++k1) sm[k1 * G::LD + q * W + c] = v[k1];
  }
  __syncthreads();
  if (q < R2) {
    float2 u[R1];
#pragma unroll
    for (int j = 0; j < R1; ++j) u[j] = sm[q * G::LD + j * W + c];
    reg_dft<R1, -1>(u);
    if (in) {
#pragma unroll
      for (int k2 = 0; k2 < R1; ++k2) base[(size_t)(q + R2 * k2) * ncol + c] = u[k2];
    }
  }
}

// --------------------------------------------------------------------- rows
// W lines per CTA of about 128 threads: stage-1 item (j fastest, line),
// stage-2 item (k1 fastest, line).  The same memory holds the lines and then
// the exchange.
template <int R1, int R2>
struct TfRow {
  static constexpr int N = R1 * R2;
  static constexpr int LD = R2 | 1;
  static constexpr int W = 128 / R1;  // 4 .. 16
  static constexpr int kThreads = (W * R1 + 31) / 32 * 32;
  static constexpr int kElems = W * R1 * LD;  // >= W * N
  static constexpr size_t kSmem = (size_t)((kElems + 1) & ~1) * sizeof(float2);
};

// lines in sm[l * N + i] (all written, before a barrier) -> stage-2 values
// u[k2] = X[k1 + R1 k2] of item (l, k1) of this thread
template <int R1, int R2, int DIR>
__device__ __forceinline__ void tf_row_lines(float2* sm, const float2* __restrict__ tw, float2* u)
{
  using G = TfRow<R1, R2>;
  const int l1 = threadIdx.x / R2, j = threadIdx.x - l1 * R2;
  const int l2 = threadIdx.x / R1, k1 = threadIdx.x - l2 * R1;
  float2 v[R1];
  if (l1 < G::W) {
#pragma unroll
    for (int e = 0; e < R1; ++e) v[e] = sm[l1 * G::N + j + R2 * e];
  }
  __syncthreads();  // the lines are taken before the exchange overwrites them
  if (l1 < G::W) {
    reg_dft<R1, DIR>(v);
    tf_twiddle<R1, DIR>(v, tw, R2, j);
#pragma unroll
    for (int k = 0; k < R1; ++k) sm[(l1 * R1 + k) * G::LD + j] = v[k];
  }
  __syncthreads();
  if (l2 < G::W) {
#pragma unroll
    for (int q = 0; q < R2; ++q) u[q] = sm[(l2 * R1 + k1) * G::LD + q];
    reg_dft<R2, DIR>(u);
  }
}

// forward transform of the conjugated rows (the cross-correlation's first half)
template <int R1, int R2>
__global__ void __launch_bounds__(TfRow<R1, R2>::kThreads)
    k_tf_rows_conj(const float2* __restrict__ in, float2* __restrict__ out, int nrows, const float2* __restrict__ tw)
{
  using G = TfRow<R1, R2>;
  extern __shared__ __align__(16) float2 sm[];
  const int r0 = blockIdx.x * G::W;
  const int n = min(G::W, nrows - r0) * G::N;
  for (int t = threadIdx.x; t < G::W * G::N; t += G::kThreads) {
    const float2 v = t < n ? in[(size_t)r0 * G::N + t] : make_float2(0.f, 0.f);
    sm[t] = make_float2(v.x, -v.y);
  }
  __syncthreads();
  float2 u[R2];
  tf_row_lines<R1, R2, -1>(sm, tw, u);
  const int l = threadIdx.x / R1, k1 = threadIdx.x - l * R1;
  if (l < G::W && r0 + l < nrows) {
    float2* dst = out + (size_t)(r0 + l) * G::N + k1;
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) dst[R1 * k2] = u[k2];
  }
}

// One CTA: W complex lines, each two raw rows as real and imaginary part:
// flat field and both edge blends in shared memory, the transform, the split
// of the two real spectra (the steps of k_ingest_x).  Latency-bound, the
// shared-memory passes in line: 640 x 384 x 30 0.685 -> 0.464 ms against the
// Stockham stages (0.400 with paired additions), 300 x 192 x 40 (one
// direction) 0.083 -> 0.044 ms.
template <typename T, int R1, int R2>
__global__ void __launch_bounds__(TfRow<R1, R2>::kThreads)
    k_tf_ingest(const __grid_constant__ IngestArgs a, const float2* __restrict__ tw)
{
  using G = TfRow<R1, R2>;
  constexpr int N = G::N, nxh = N / 2 + 1;
  extern __shared__ __align__(16) float2 sm[];
  const int ny = a.ny;
  const IngestPlane ip = ingest_plane(a);
  const int pl = ip.plane;
  const int y0 = blockIdx.x * 2 * G::W;
  const T* plane = (const T*)a.raw + (size_t)ip.section * N * ny;
  float* smr = (float*)sm;  // row r at x -> smr[2*((r>>1)*N + x) + (r&1)]
  const int napo = a.napodize;
  const bool plainbg = !a.bg && !a.slope;
  for (int t = threadIdx.x; t < G::W * 2 * (N / 2); t += G::kThreads) {
    const int r = t / (N / 2), x0 = (t - r * (N / 2)) * 2;
    const int y = y0 + r;
    float v[2] = {0.f, 0.f};
    if (y < ny) {
      float w0, w1;
      if constexpr (sizeof(T) == 2) {
        const ushort2 u = __ldg((const ushort2*)(plane + (size_t)y * N + x0));
        w0 = (float)u.x;
        w1 = (float)u.y;
      } else {
        const float2 u = __ldg((const float2*)(plane + (size_t)y * N + x0));
        w0 = u.x;
        w1 = u.y;
      }
      if (plainbg) {
        v[0] = (w0 - a.bgconst - a.bgextra) * 1.0f * a.inscale;
        v[1] = (w1 - a.bgconst - a.bgextra) * 1.0f * a.inscale;
      } else {
        v[0] = flat_v(w0, a, y, x0);
        v[1] = flat_v(w1, a, y, x0 + 1);
      }
      // top / bottom edge blend (apodize_x_kernel)
      const bool top = y < napo, bot = (ny - 1 - y) < napo;
      if (top || bot) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const float diff = (flat(plane, a, ny - 1, x0 + i) - flat(plane, a, 0, x0 + i)) / 2.0f;
          if (top) v[i] += diff * a.apofact[y];
          if (bot) v[i] -= diff * a.apofact[ny - 1 - y];
        }
      }
    }
    float* dst = smr + 2 * ((r >> 1) * N + x0) + (r & 1);
    dst[0] = v[0];
    dst[2] = v[1];
  }
  __syncthreads();
  // left / right edge blend (apodize_y_kernel) from the blended row ends: one
  // thread per row takes the difference, all of them apply it
  if (napo > 0) {
    __shared__ float diffr[2 * G::W];
    if (threadIdx.x < 2 * G::W) {
      const int r = threadIdx.x;
      diffr[r] = (smr[2 * ((r >> 1) * N + N - 1) + (r & 1)] - smr[2 * ((r >> 1) * N) + (r & 1)]) / 2.0f;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < 2 * G::W * 2 * napo; t += G::kThreads) {
      const int r = t / (2 * napo), q = t - r * 2 * napo;
      const int l = q < napo ? q : q - napo, x = q < napo ? l : N - 1 - l;
      float* e = &smr[2 * ((r >> 1) * N + x) + (r & 1)];
      const float f = diffr[r] * a.apofact[l];
      if (q < napo) *e += f;
      else *e -= f;
    }
    __syncthreads();
  }
  float2 u[R2];
  tf_row_lines<R1, R2, -1>(sm, tw, u);
  __syncthreads();  // the exchange is taken: the lines go back in place
  {
    const int l = threadIdx.x / R1, k1 = threadIdx.x - l * R1;
    if (l < G::W) {
#pragma unroll
      for (int k2 = 0; k2 < R2; ++k2) sm[l * N + k1 + R1 * k2] = u[k2];
    }
  }
  __syncthreads();
  float2* dst = a.spec + (size_t)pl * ny * nxh;
  for (int t = threadIdx.x; t < G::W * nxh; t += G::kThreads) {
    const int l = t / nxh, k = t - l * nxh;
    const float2 zk = sm[l * N + k], zn = sm[l * N + (k == 0 ? 0 : N - k)];
    const float2 A = make_float2(0.5f * (zk.x + zn.x), 0.5f * (zk.y - zn.y));
    const float2 B = make_float2(0.5f * (zk.y + zn.y), -0.5f * (zk.x - zn.x));
    const int y = y0 + 2 * l;
    if (y < ny) dst[(size_t)y * nxh + k] = A;
    if (y + 1 < ny) dst[(size_t)(y + 1) * nxh + k] = B;
  }
}

// makeotf: two rows of one band as a complex line, the band separated from the
// phases' rows as they are loaded (k_mo_separate's operations; the phases come
// from L2 for all bands but the first), half spectra out.  Bound by the loads
// of nph sections per band: 128^2 x 64 x 5 35 us, where the separation into
// full complex rows and their transform took 18 + 43 us and left twice the
// bytes to the y and z transforms.
template <int R1, int R2>
__global__ void __launch_bounds__(TfRow<R1, R2>::kThreads)
    k_tf_mo_rows(const __grid_constant__ MoRowsArgs a, const float2* __restrict__ tw)
{
  using G = TfRow<R1, R2>;
  constexpr int N = G::N, nxh = N / 2 + 1;
  extern __shared__ __align__(16) float2 sm[];
  const int z = blockIdx.y, b = blockIdx.z, y0 = blockIdx.x * 2 * G::W;
  const size_t nxy = (size_t)a.ny * N;
  const float* psf = a.psf + (size_t)z * a.nph * nxy;
  float* smr = (float*)sm;  // row r at x -> smr[2*((r>>1)*N + x) + (r&1)]
#pragma unroll 4
  for (int t = threadIdx.x; t < 2 * G::W * N; t += G::kThreads) {
    const int r = t / N, x = t - r * N, y = y0 + r;
    float acc = 0.f;
    if (y < a.ny) {
      float v[kMoMaxPhases];
#pragma unroll
      for (int j = 0; j < kMoMaxPhases; ++j) v[j] = j < a.nph ? __ldg(psf + j * nxy + (size_t)y * N + x) : 0.f;
#pragma unroll
      for (int j = 0; j < kMoMaxPhases; ++j)
        if (j < a.nph) {
          v[j] = __fsub_rn(v[j], __ldg(a.bg + z * a.nph + j));
          acc = a.nph == 1 ? v[j] : __fadd_rn(acc, __fmul_rn(v[j], a.m[b * a.nph + j]));
        }
    }
    smr[2 * ((r >> 1) * N + x) + (r & 1)] = acc;
  }
  __syncthreads();
  float2 u[R2];
  tf_row_lines<R1, R2, -1>(sm, tw, u);
  __syncthreads();  // the exchange is taken: the lines go back in place
  {
    const int l = threadIdx.x / R1, k1 = threadIdx.x - l * R1;
    if (l < G::W) {
#pragma unroll
      for (int k2 = 0; k2 < R2; ++k2) sm[l * N + k1 + R1 * k2] = u[k2];
    }
  }
  __syncthreads();
  float2* dst = a.bands + ((size_t)b * a.nz + z) * a.ny * nxh;
  for (int t = threadIdx.x; t < G::W * nxh; t += G::kThreads) {
    const int l = t / nxh, k = t - l * nxh;
    const float2 zk = sm[l * N + k], zn = sm[l * N + (k == 0 ? 0 : N - k)];
    const int y = y0 + 2 * l;
    if (y < a.ny) dst[(size_t)y * nxh + k] = make_float2(0.5f * (zk.x + zn.x), 0.5f * (zk.y - zn.y));
    if (y + 1 < a.ny) dst[(size_t)(y + 1) * nxh + k] = make_float2(0.5f * (zk.y + zn.y), -0.5f * (zk.x - zn.x));
  }
}

// ----------------------------------------------------------------- overlaps
// radial table of one kz: order slot o at [o * (nxotf + 1)], entry i the OTF
// interpolated to kz at radial bins i and i + 1 (flat indices clamped to the
// table's end like otf_lookup_rr's; entry nxotf stands for every bin past the
// end).  The kz index is not negative (launch_overlaps).
__device__ __forceinline__ void ovl_build_tab(const OverlapArgs& a, const OvlItem& it, const OtfKz& kz, float4* tab)
{
  const int nxo = a.otf.nxotf, nzo = a.otf.nzotf, last = nxo * nzo - 1;
  for (int t = threadIdx.x; t < 2 * (nxo + 1); t += blockDim.x) {
    const int o = t / (nxo + 1), i = t - o * (nxo + 1);
    const float2* otf = o ? it.otf2 : it.otf1;
    const float az = kz.az;
    auto at = [&](int r) {
      const float2 p = __ldg(otf + min(r * nzo + kz.iz, last)), q = __ldg(otf + min(r * nzo + kz.izp, last));
      return make_float2(p.x * (1 - az) + q.x * az, p.y * (1 - az) + q.y * az);
    };
    const float2 t0 = at(i), t1 = at(i + 1);
    tab[t] = make_float4(t0.x, t0.y, t1.x, t1.y);
  }
}

__device__ __forceinline__ float2 ovl_tab_lookup(const float4* tab, int nxotf, float krindex)
{
  const int ir = (int)floorf(krindex);
  const float ar = krindex - ir;
  const float4 t = tab[min(ir, nxotf)];
  return make_float2((1 - ar) * t.x + ar * t.z, (1 - ar) * t.y + ar * t.w);
}

// Element j of overlap `ov` on row i of plane zb before the x transform (the
// element of k_fit.cu's ovl_value, the OTF from the plane's radial tables)
__device__ __forceinline__ float2 ovl_element(const OverlapArgs& a, const OvlItem& it, float2 ks, int ov, int z0, int i, int j,
                                              const float4* tab, float rdk)
{
  const int nx = a.nx, ny = a.ny, nz = a.nz, nxh = nx / 2 + 1;
  float x1f = (float)j, y1f = (float)i;
  if (x1f > nx / 2) x1f -= nx;
  if (y1f > ny / 2) y1f -= ny;
  x1f *= a.dkx;
  y1f *= a.dky;
  const float r1sq = x1f * x1f + y1f * y1f;
  if (ov == 0 ? !(r1sq <= a.r2_le) : !(r1sq < a.r2_lt)) return make_float2(0.f, 0.f);
  // the partner pixel: overlap 0 at k - shift, overlap 1 at k + shift
  const float x2f = ov == 0 ? x1f - ks.x : x1f + ks.x, y2f = ov == 0 ? y1f - ks.y : y1f + ks.y;
  const float r2sq = x2f * x2f + y2f * y2f;
  if (!(r2sq <= a.r2_le)) return make_float2(0.f, 0.f);
  const int nxo = a.otf.nxotf;
  const float4* own = ov == 0 ? tab : tab + nxo + 1;
  const float4* other = ov == 0 ? tab + nxo + 1 : tab;
  const float2 o1 = ovl_tab_lookup(own, nxo, sqrtf(r1sq) * rdk);
  const float2 o2 = ovl_tab_lookup(other, nxo, sqrtf(r2sq) * rdk);
  // |OTF(order1)| > otfcutoff and |OTF(order2)| * factor > otfcutoff
  const float m1 = cmag2(o1), m2 = cmag2(o2);
  if (ov == 0 ? !(m1 > a.m_le && m2 >= a.m_f) : !(m1 >= a.m_f && m2 > a.m_le)) return make_float2(0.f, 0.f);
  const float rroot = 1.f / sqrtf(m1 + m2);
  const float2 fact = make_float2(o2.x * rroot, o2.y * rroot);
  const bool conj = j > nx / 2;
  const int jin = conj ? nx - j : j;
  const int iin = conj && i ? ny - i : i;
  int zin = conj ? -z0 : z0;
  if (zin < 0) zin += nz;
  const size_t bplane = (size_t)ny * nxh;
  const size_t indin = (size_t)zin * bplane + (size_t)iin * nxh + jin;
  const int ob = ov == 0 ? it.order1 : it.order2;
  float2 vre = it.bands[(ob == 0 ? 0 : (size_t)(2 * ob - 1) * nz * bplane) + indin];
  float2 vim = ob == 0 ? make_float2(0.f, 0.f) : it.bands[(size_t)(2 * ob) * nz * bplane + indin];
  if (conj) {
    vre.y = -vre.y;
    vim.y = -vim.y;
  }
  vre = cmul(vre, fact);
  vim = cmul(vim, fact);
  return make_float2(vre.x - vim.y, vre.y + vim.x);
}

// W lines (line = 2 * row + overlap) of one kz plane per CTA.  Bound by the
// elements' issue and latency; per kz plane the two radial OTF tables replace
// 16 scattered loads and the kz interpolation of every element; rows outside
// the support are left out, and a line at a time leaves its row's arithmetic to
// the uniform registers.  Nine builds of 640 x 384 x 30: 1.40 ms by the
// Stockham stages, 0.37 with every row, 0.33 with a line per few threads, 0.31
// now; of 1024^2 x 64 2.16 and 1.98.
template <int R1, int R2>
__global__ void __launch_bounds__(TfRow<R1, R2>::kThreads)
    k_tf_ovl_x(const __grid_constant__ OverlapArgs a, const float2* __restrict__ tw)
{
  using G = TfRow<R1, R2>;
  constexpr int N = G::N;
  extern __shared__ __align__(16) float2 sm[];
  float4* tab = (float4*)(sm + ((G::kElems + 1) & ~1));
  const int ny = a.ny, nzb = 2 * a.zdc + 1;
  const int zb = blockIdx.y, z0 = zb - a.zdc;
  const int L0 = blockIdx.x * G::W, nl = min(G::W, 2 * ny - L0);
  const float rdk = 1.f / a.otf.dkrotf;
  const OvlItem& it = a.item[blockIdx.z];
  const float2 ks = ovl_shift(it);
  const bool empty = z0 == 0 && a.nokz0;
  // lines without an element are left out
  auto dead = [&](int l) { return ovl_plane_dead(a, zb) || ovl_row_dead(a, ks, (L0 + l) & 1, (L0 + l) >> 1); };
  if (!__syncthreads_or(threadIdx.x < nl && !dead(threadIdx.x))) return;
  if (!empty) ovl_build_tab(a, it, otf_kz(a.otf, z0), tab);
  __syncthreads();
  // a line at a time, whose row is the same for the whole CTA, unless that
  // leaves more than a seventh of the threads' turns idle
  constexpr int kTurns = (N + G::kThreads - 1) / G::kThreads * G::kThreads;
  if constexpr (7 * (kTurns - N) <= N) {
    for (int l = 0; l < G::W; ++l) {
      const bool live = !empty && l < nl && !dead(l);
      const int ov = (L0 + l) & 1, i = (L0 + l) >> 1;
#pragma unroll 2
      for (int j = threadIdx.x; j < N; j += G::kThreads)
        sm[l * N + j] = live ? ovl_element(a, it, ks, ov, z0, i, j, tab, rdk) : make_float2(0.f, 0.f);
    }
  } else {
    for (int t = threadIdx.x; t < G::W * N; t += G::kThreads) {
      const int l = t / N, j = t - l * N;
      float2 v = make_float2(0.f, 0.f);
      if (!empty && l < nl) v = ovl_element(a, it, ks, (L0 + l) & 1, z0, (L0 + l) >> 1, j, tab, rdk);
      sm[t] = v;
    }
  }
  __syncthreads();
  float2 u[R2];
  tf_row_lines<R1, R2, +1>(sm, tw, u);
  const int l = threadIdx.x / R1, k1 = threadIdx.x - l * R1;
  if (l < nl && !dead(l)) {
    const int L = L0 + l;
    float2* dst = it.ovl + ((size_t)(L & 1) * nzb + zb) * ny * N + (size_t)(L >> 1) * N + k1;
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) dst[R1 * k2] = u[k2];
  }
}

// W columns of both overlaps per CTA and group of kz planes: item (column
// fastest, overlap, j or k1).  In the second stage the threads of a column's
// two overlaps sit W lanes apart; they exchange half of their values by
// shuffles, so each sums conj(X) Y of every other k2 in registers over the
// planes and neither holds both overlaps.  Nine pairs of 1024^2 x 64: 11.2 ms
// by the Stockham stages, 2.2 reading every row and with FP64 sums, 1.92 now
// (2.5 TB/s of the overlap rows); of 640 x 384 x 30 1.29, 0.30, 0.26 ms.
template <int R1, int R2>
struct TfOvlY {
  static constexpr int N = R1 * R2;
  static constexpr int W = R1 <= 16 ? 8 : 4;
  static constexpr int LD = (R2 | 1) * 2 * W;  // k1 pitch, both overlaps
  static constexpr int kThreads = (2 * R1 * W + 31) / 32 * 32;
  static constexpr size_t kSmem = (size_t)R1 * LD * sizeof(float2);
  static constexpr int kHalf = (R2 + 1) / 2;
  static constexpr int kRegs = (2 * R1 > 2 * R2 + 2 * kHalf ? 2 * R1 + 2 * kHalf : 2 * R2 + 4 * kHalf) + 40;
  static constexpr int kCtas0 = 65536 / (kThreads * kRegs);
  static constexpr int kCtas = kCtas0 < 1 ? 1 : kCtas0 > 4 ? 4 : kCtas0;
};

template <int R1, int R2>
__global__ void __launch_bounds__(TfOvlY<R1, R2>::kThreads, TfOvlY<R1, R2>::kCtas)
    k_tf_ovl_y(const __grid_constant__ OverlapArgs a, const float2* __restrict__ tw, int planes_per_group)
{
  using G = TfOvlY<R1, R2>;
  constexpr int N = G::N, W = G::W, LD = G::LD;
  extern __shared__ __align__(16) float2 sm[];
  __shared__ double red[32];
  const int nx = a.nx, nzb = 2 * a.zdc + 1;
  const int c0 = blockIdx.x * W;
  const int zb0 = blockIdx.y * planes_per_group, zb1 = min(nzb, zb0 + planes_per_group);
  const int c = threadIdx.x % W, ov = threadIdx.x / W & 1, q = threadIdx.x / (2 * W);
  const bool in = c0 + c < nx;
  const size_t vol = (size_t)nzb * N * nx;
  const OvlItem& it = a.item[blockIdx.z];
  const float2* src0 = it.ovl + (size_t)ov * vol + c0 + c;
  float2 acc[G::kHalf];
#pragma unroll
  for (int i = 0; i < G::kHalf; ++i) acc[i] = make_float2(0.f, 0.f);
  float sq = 0.f, sqe = 0.f;  // a float pair: the FP64 adder has a sixtyfourth of the FP32 rate
  unsigned live = 0;          // the thread's rows with elements
  if (in && q < R2) {
    const float2 ks = ovl_shift(it);
#pragma unroll
    for (int e = 0; e < R1; ++e) live |= (ovl_row_dead(a, ks, ov, q + R2 * e) ? 0u : 1u) << e;
  }
  for (int zb = zb0; zb < zb1; ++zb) {
    if (ovl_plane_dead(a, zb)) continue;
    if (q < R2) {
      const float2* src = src0 + (size_t)zb * N * nx;
      float2 v[R1];
#pragma unroll
      for (int e = 0; e < R1; ++e) v[e] = live >> e & 1 ? src[(size_t)(q + R2 * e) * nx] : make_float2(0.f, 0.f);
      reg_dft<R1, +1>(v);
      tf_twiddle<R1, +1>(v, tw, R2, q);
#pragma unroll
      for (int k = 0; k < R1; ++k) sm[k * LD + q * 2 * W + ov * W + c] = v[k];
    }
    __syncthreads();
    float2 u[R2];
    const bool act = q < R1;
#pragma unroll
    for (int j = 0; j < R2; ++j) u[j] = act ? sm[q * LD + j * 2 * W + ov * W + c] : make_float2(0.f, 0.f);
    reg_dft<R2, +1>(u);
    float ps = 0.f;
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) ps += cmag2(u[k2]);
    pair_sum(sq, sqe, ps);
#pragma unroll
    for (int i = 0; i < G::kHalf; ++i) {
      // overlap 0's thread keeps k2 = 2 i, overlap 1's keeps 2 i + 1
      const float2 odd = 2 * i + 1 < R2 ? u[2 * i + 1] : make_float2(0.f, 0.f);
      const float2 send = ov ? u[2 * i] : odd;
      const float2 got = make_float2(__shfl_xor_sync(0xffffffffu, send.x, W), __shfl_xor_sync(0xffffffffu, send.y, W));
      const float2 X = ov ? got : u[2 * i], Y = ov ? odd : got;
      // conj(X) * Y, as reductionKernel's xsy (gpuFunctionsImpl.cu:1177-1178)
      acc[i].x += X.x * Y.x + X.y * Y.y;
      acc[i].y += X.x * Y.y - X.y * Y.x;
    }
    __syncthreads();
  }
  if (in && q < R1) {
    float2* dst = it.ppart + (size_t)blockIdx.y * N * nx + c0 + c;
#pragma unroll
    for (int i = 0; i < G::kHalf; ++i)
      if (2 * i + ov < R2) dst[(size_t)(q + R1 * (2 * i + ov)) * nx] = acc[i];
  }
  const double st = pair_value(sq, sqe);
  const double tx = block_sum_d(ov ? 0.0 : st, red);
  const double ty = block_sum_d(ov ? st : 0.0, red);
  if (threadIdx.x == 0) {
    const int cta = blockIdx.y * gridDim.x + blockIdx.x;
    it.sums[2 * cta] = tx;
    it.sums[2 * cta + 1] = ty;
  }
}

// ----------------------------------------------------------------- assembly
// Zoomed x transform, phase ramp and weighted sum of the doubled-grid assembly
// (k_assemble2.cu).  The sums stay in registers over the plane's slots, so
// their count is a compile-time number (one kernel that switched between the
// compiled sizes at run time spilled 2 to 4 KB a thread and took minutes to
// build).
// Per volume, against the Stockham stages on the doubled length: 1024^2 x 64
// 22.5 -> 2.9 ms, 640 x 384 x 30 2.61 -> 0.46 ms, 1024 x 960 0.243 -> 0.043 ms.
//
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
  static constexpr int kRegs = 4 * R2 + 2 * R1 + 52;
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
      tf_twiddle_half<R1, +1>(v, twp, R2, j);
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

// ---------------------------------------------------------------- launchers
template <int R1, int R2>
struct TfEntry {
  static int asm_x(const AsmX2Launch& l, const TfPlan& pl, cudaStream_t s)
  {
    using G = X2<R1, R2>;
    allow_dynamic_smem((const void*)k_asm_x2<R1, R2>, G::kSmem);
    k_asm_x2<R1, R2><<<dim3((l.a->Y + G::W - 1) / G::W, l.nplanes), G::kThreads, G::kSmem, s>>>(
        *l.a, l.p0, l.pn, l.slots, l.pz, pl.tw, pl.twh, l.real);
    return (int)cudaGetLastError();
  }
  static int ovl_x(const OverlapArgs& a, const TfPlan& pl, cudaStream_t s)
  {
    using G = TfRow<R1, R2>;
    const size_t bytes = G::kSmem + 2 * (size_t)(a.otf.nxotf + 1) * sizeof(float4);
    allow_dynamic_smem((const void*)k_tf_ovl_x<R1, R2>, bytes);
    k_tf_ovl_x<R1, R2><<<dim3((2 * a.ny + G::W - 1) / G::W, 2 * a.zdc + 1, a.nitems), G::kThreads, bytes, s>>>(a, pl.tw);
    return (int)cudaGetLastError();
  }
  static int ovl_y(const OverlapArgs& a, const TfPlan& pl, int ppg, int groups, cudaStream_t s)
  {
    using G = TfOvlY<R1, R2>;
    allow_dynamic_smem((const void*)k_tf_ovl_y<R1, R2>, G::kSmem);
    k_tf_ovl_y<R1, R2><<<dim3((a.nx + G::W - 1) / G::W, groups, a.nitems), G::kThreads, G::kSmem, s>>>(a, pl.tw, ppg);
    return (int)cudaGetLastError();
  }
  static int fft_cols(float2* data, int ncol, int nplanes, const TfPlan& pl, cudaStream_t s)
  {
    using G = TfCol<R1, R2>;
    allow_dynamic_smem((const void*)k_tf_cols<R1, R2>, G::kSmem);
    k_tf_cols<R1, R2><<<dim3((ncol + G::W - 1) / G::W, nplanes), G::kThreads, G::kSmem, s>>>(data, ncol, pl.tw);
    return (int)cudaGetLastError();
  }
  static int fft_rows_conj(const float2* in, float2* out, int nrows, const TfPlan& pl, cudaStream_t s)
  {
    using G = TfRow<R1, R2>;
    allow_dynamic_smem((const void*)k_tf_rows_conj<R1, R2>, G::kSmem);
    k_tf_rows_conj<R1, R2><<<(nrows + G::W - 1) / G::W, G::kThreads, G::kSmem, s>>>(in, out, nrows, pl.tw);
    return (int)cudaGetLastError();
  }
  static int ingest_x(const IngestArgs& a, const TfPlan& pl, cudaStream_t s)
  {
    using G = TfRow<R1, R2>;
    const dim3 g((a.ny + 2 * G::W - 1) / (2 * G::W), a.nsec ? a.nsec : a.ndirs * a.nphases * a.nz);
    if (a.raw_is_u16) {
      allow_dynamic_smem((const void*)k_tf_ingest<uint16_t, R1, R2>, G::kSmem);
      k_tf_ingest<uint16_t, R1, R2><<<g, G::kThreads, G::kSmem, s>>>(a, pl.tw);
    } else {
      allow_dynamic_smem((const void*)k_tf_ingest<float, R1, R2>, G::kSmem);
      k_tf_ingest<float, R1, R2><<<g, G::kThreads, G::kSmem, s>>>(a, pl.tw);
    }
    return (int)cudaGetLastError();
  }
  static int mo_rows(const MoRowsArgs& a, const TfPlan& pl, cudaStream_t s)
  {
    using G = TfRow<R1, R2>;
    allow_dynamic_smem((const void*)k_tf_mo_rows<R1, R2>, G::kSmem);
    k_tf_mo_rows<R1, R2><<<dim3((a.ny + 2 * G::W - 1) / (2 * G::W), a.nz, a.nph), G::kThreads, G::kSmem, s>>>(a, pl.tw);
    return (int)cudaGetLastError();
  }
  static constexpr bool even = R1 * R2 % 2 == 0;
  template <bool E>
  static constexpr TfKernels make()
  {
    if constexpr (E)
      return {R1, R2, asm_x, ovl_x, ovl_y, TfOvlY<R1, R2>::W, fft_cols, fft_rows_conj, ingest_x, mo_rows};
    else
      return {R1, R2, nullptr, ovl_x, ovl_y, TfOvlY<R1, R2>::W, fft_cols, fft_rows_conj, nullptr, nullptr};
  }
  static constexpr TfKernels kernels() { return make<even>(); }
};

#endif  // __CUDACC__

}  // namespace simrecon
