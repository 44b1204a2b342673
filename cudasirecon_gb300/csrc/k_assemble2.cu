// Assembly with the grid doubled in x and y (zoomfact 2), for any image
// length with a two-factor plan (tf_fft.cuh).
//
// A transform zero-padded to twice its length is two of its own length: the
// even outputs come from the data, the odd ones from the data times half a
// sample's phase.  So neither axis runs the doubled transform: no zeros are
// read, multiplied or kept in shared memory, and the 2048-point lines of a
// 1024 image are 1024-point ones.  The tables of slots and planes, T and the
// order of the sums are those of k_assemble.cu; only S has its columns split
// by parity, S[zout][yr][x & 1][x >> 1], so that the x pass stores runs
#include <algorithm>

#include "assemble.h"
#include "tf_kernels.h"

namespace simrecon {

namespace {

constexpr int kThreads = 256;

// Zoomed y transform of W columns of one slot per CTA.
//
// FILT: the Wiener filter inside the band load, each filtered value formed
// once (the reasons are k_asm_y4f's, k_assemble.cu); else bands that are
// filtered already.  The CTA's ny x W values sit row-major in shared memory;
// every stage-1 thread (parity, j, column) takes its R1 rows from there, and
// both parities' stage-1 results then overwrite them, so the tile costs the
// same shared memory as a doubled column would.  W is 8 where 2 R2 W threads
// fit in the CTA, else 4 (a 32-byte sector of a row of T).
// Bound by the filter's issue slots and latency (the register bounds of the two
// classes spill 52 and 196 bytes a thread around the transforms).  Filter + y
// transform per volume, before (k_filter and the Stockham stages) and now:
// 640 x 384 x 30 2.87 -> 0.64 ms, 1024 x 960 0.293 -> 0.080 ms, 1024^2 x 64 25.3 ->
// 6.2 ms (with tables of values and steps; 2 % more since).
// At 256/512/1024 output rows the compiled k_asm_y4f stays: 1.31 against
// 1.45 ms per 512^2 x 48 volume (0.98 now).
template <bool FILT, int MR>
__global__ void __launch_bounds__(kThreads, MR <= 16 ? 4 : 3) k_asm_y2(AssembleArgs a, const Slot* __restrict__ slots,
                                                                    TfPlan pl, int lw,
                                                                    const __grid_constant__ FilterArgs fa,
                                                                    const __grid_constant__ FilterK fk)
{
  extern __shared__ __align__(16) float2 sm[];
  const Slot sl = slots[blockIdx.y];
  const int nx = a.nx, ny = a.ny, nz = a.nz, nxh = nx / 2 + 1;
  const int W = 1 << lw, c0 = a.tx0 + (blockIdx.x << lw);
  const int R1 = pl.r1, R2 = pl.r2;
  const int ld = (R2 | 1) << lw;  // k1 pitch of the exchange: odd multiple of W, conflict-free reads
  const size_t plane = (size_t)ny * nxh;
  const int order = sl.order;
  const int d0 = sl.dir < 0 ? 0 : sl.dir;
  const float2* br = a.bands + ((size_t)d0 * a.nphases + (order == 0 ? 0 : 2 * order - 1)) * nz * plane;
  const float2* bi = order == 0 ? nullptr : a.bands + ((size_t)d0 * a.nphases + 2 * order) * nz * plane;
  const size_t dstride = (size_t)a.nphases * nz * plane;  // next direction's band 0
  const int no = a.norders;
  // the row-major values, then the exchange of both parities over them
  float2* tab = sm + 2 * R1 * ld;  // [2][no][nxotf]
  if constexpr (FILT) {
    if (c0 < a.cx0 || c0 >= a.cx1) {  // no data: zeros for the x pass
      for (int t = threadIdx.x; t < a.Y << lw; t += kThreads) {
        const int c = c0 + (t & (W - 1));
        if (c < nx) a.T[((size_t)blockIdx.y * a.Y + (t >> lw)) * nx + c] = make_float2(0.f, 0.f);
      }
      return;
    }
    __shared__ FilterTerms terms;
    build_filter_tab(fa, no, sl.kz, tab);
    build_filter_terms(fa, fk, d0, order, sl.kz, c0 - (nx / 2 - 1), min(W, nx - c0), terms);
    FilterSlot fsl{br, bi, plane, dstride, nx, ny, nz, order, d0, sl.kz};
    load_fit(fa, fsl);
    __syncthreads();
#pragma unroll 1
    for (int t = threadIdx.x; t < (ny / 2) << lw; t += kThreads) {
      const int r = 2 * (t >> lw), w = t & (W - 1);
      const int c = c0 + w;
      float2 v0 = make_float2(0.f, 0.f), v1 = v0;
      if (c < nx) filtered_rows(fa, fk, fsl, terms, tab, c - (nx / 2 - 1), r, v0, v1);
      sm[(r << lw) + w] = v0;
      sm[((r + 1) << lw) + w] = v1;
    }
  } else {
    for (int t = threadIdx.x; t < ny << lw; t += kThreads) {
      const int r = t >> lw, w = t & (W - 1);
      const int c = c0 + w;
      float2 v = make_float2(0.f, 0.f);
      if (c < nx) {
        int x = c - (nx / 2 - 1), y = r <= ny / 2 ? r : r - ny, z = sl.kz;
        const bool conj = x < 0;
        if (conj) {
          x = -x;
          y = -y;
          z = -z;
        }
        if (y < 0) y += ny;
        if (z < 0) z += nz;
        const size_t indin = (size_t)z * plane + (size_t)y * nxh + x;
        if (order == 0) {
          v = br[indin];
          if (sl.dir < 0)
            for (int d = 1; d < a.ndirs; ++d) {
              const float2 u = br[d * dstride + indin];
              v.x += u.x;
              v.y += u.y;
            }
          if (conj) v.y = -v.y;
        } else {
          float2 re = br[indin], im = bi[indin];
          if (conj) {
            re.y = -re.y;
            im.y = -im.y;
          }
          v = make_float2(re.x - im.y, re.y + im.x);
        }
      }
      sm[t] = v;
    }
  }
  __syncthreads();
  {  // stage 1: thread (parity b, j, column c)
    const int it = threadIdx.x, c = it & (W - 1), jb = it >> lw;
    const bool act = jb < 2 * R2;
    const int b = jb >= R2, j = jb - b * R2;
    tf_switch<MR>(R1, [&]<int R>() {
      float2 v[R];
#pragma unroll
      for (int e = 0; e < R; ++e) {
        const int r = j + R2 * e;
        v[e] = act ? sm[(r << lw) + c] : make_float2(0.f, 0.f);
        if (b && r > ny / 2) v[e] = make_float2(-v[e].x, -v[e].y);
      }
      __syncthreads();  // the values are taken before the exchange overwrites them
      if (act) {
        if (b) tf_half_shift<R, +1>(v);
        reg_dft<R, +1>(v);
        tf_twiddle_half<R, +1>(v, b ? pl.twh : pl.tw, R2, j);
        float2* ex = sm + b * R1 * ld;
#pragma unroll
        for (int k1 = 0; k1 < R; ++k1) ex[k1 * ld + (j << lw) + c] = v[k1];
      }
    });
  }
  __syncthreads();
  float2* dst = a.T + (size_t)blockIdx.y * a.Y * nx + c0;
  tf_switch<MR>(R2, [&]<int R>() {
    for (int it = threadIdx.x; it < (2 * R1) << lw; it += kThreads) {
      const int c = it & (W - 1), kb = it >> lw;
      const int b = kb >= R1, k1 = kb - b * R1;
      const float2* ex = sm + b * R1 * ld + k1 * ld + c;
      float2 u[R];
#pragma unroll
      for (int j = 0; j < R; ++j) u[j] = ex[j << lw];
      reg_dft<R, +1>(u);
      if (c0 + c < nx) {
        float2* o = dst + (size_t)(2 * k1 + b) * nx + c;
        const size_t step = (size_t)2 * R1 * nx;
#pragma unroll
        for (int k2 = 0; k2 < R; ++k2) o[k2 * step] = u[k2];
      }
    }
  });
}

}  // namespace

bool asm_y2_supported(const AssembleArgs& a)
{
  int r1, r2;
  return a.Y == 2 * a.ny && a.ny % 2 == 0 && tf_factor(a.ny, &r1, &r2);
}

bool asm_x2_supported(const AssembleArgs& a)
{
  int r1, r2;
  return a.X == 2 * a.nx && a.nx % 2 == 0 && tf_factor(a.nx, &r1, &r2);
}

int launch_asm_y2(const AssembleArgs& a, const void* d_slots, int nslots, const FilterArgs* filt, cudaStream_t s)
{
  TfPlan pl;
  if (!get_tf_plan(a.ny, &pl)) return -1;
  const int lw = 2 * pl.r2 * 8 <= kThreads ? 3 : 2;
  const size_t ld = (size_t)(pl.r2 | 1) << lw;
  const size_t elems = 2 * pl.r1 * ld;
  const size_t tabb = filt ? filter_tab_bytes(filt->norders, filt->otf.nxotf) : 0;
  const size_t bytes = elems * sizeof(float2) + tabb;
  const dim3 g((a.tx1 - a.tx0 + (1 << lw) - 1) >> lw, nslots);
  const Slot* slots = (const Slot*)d_slots;
  auto go = [&]<bool FILT>() {
    const FilterArgs fa = filt ? *filt : FilterArgs{};
    const FilterK fk = filt ? make_filter_k(*filt) : FilterK{};
    auto run = [&]<int MR>() {
      allow_dynamic_smem((const void*)k_asm_y2<FILT, MR>, bytes);
      k_asm_y2<FILT, MR><<<g, kThreads, bytes, s>>>(a, slots, pl, lw, fa, fk);
    };
    if (tf_class(pl) == 16) run.template operator()<16>();
    else run.template operator()<32>();
  };
  if (filt) go.template operator()<true>();
  else go.template operator()<false>();
  return (int)cudaGetLastError();
}

int launch_asm_x2(const AssembleArgs& a, const void* d_slots, const int* d_p0, const int* d_pn, const int* d_pz,
                  int nplanes, bool real, cudaStream_t s)
{
  TfPlan pl;
  const TfKernels* k = tf_kernels(a.nx, &pl);
  if (!k || !k->asm_x) return -1;
  return k->asm_x(AsmX2Launch{&a, (const Slot*)d_slots, d_p0, d_pn, d_pz, nplanes, real}, pl, s);
}

}  // namespace simrecon
