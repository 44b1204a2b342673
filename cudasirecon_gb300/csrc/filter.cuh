// The Wiener filter's per-pixel arithmetic (filterbands_kernel1,
// gpuFunctionsImpl.cu:1443-1644), shared by the filter pass and by the
// assembly kernels that filter the bands as they load them.
#pragma once
#include <cmath>

#include "kernels.h"
#include "thresholds.h"

namespace simrecon {

// Per-launch constants derived on the host from FilterArgs (reciprocals and
// products the per-term arithmetic would otherwise recompute per element).
struct FilterK {
  float rnv[kMaxDirs * kMaxOrders];    // 1 / noisevar
  float kxo[kMaxDirs * kMaxOrders];    // order * k0x of each direction
  float kyo[kMaxDirs * kMaxOrders];
  float rdkrotf;                       // 1 / dkrotf
  float min_dkr, rmin_dkr, supp_r;     // suppression radius (1/um) and its unit
  float rrcut;                         // 1 / rdistcutoff
  // exact squared-radius forms of the reference's float-radius decisions
  // (sqrtf is correctly rounded and monotonic): sqrtf(r2) < rdistcutoff
  // <=> r2 < r2_in, sqrtf(r2) <= suppRadius <=> r2 <= r2_supp
  float r2_in, r2_supp;
  float rapo, rzapo;                   // 1 / apocutoff, 1 / zapocutoff
  // every direction's order-0 noise factor is the same (the reference's are
  // all 1): the order-0 Wiener denominator is then one sum for all directions
  int order0_shared;
};

// One transformed plane: band (dir, order) at signed kz, summed into output
// plane zout.  dir < 0 marks the order-0 slot of a plane: the order-0 bands
// of all directions summed before the transforms (their phase ramps are all
// 1, so the sum commutes with the inverse FFTs).
struct Slot {
  int dir, order, kz, zout;
};

inline FilterK make_filter_k(const FilterArgs& a)
{
  FilterK k{};
  const int no = a.norders;
  for (int d = 0; d < a.ndirs; ++d)
    for (int o = 0; o < no; ++o) {
      const int i = d * no + o;
      k.rnv[i] = 1.f / a.noisevar[i];
      k.kxo[i] = o * a.k0[d].x;
      k.kyo[i] = o * a.k0[d].y;
    }
  k.rdkrotf = 1.f / a.otf.dkrotf;
  k.min_dkr = a.dkx < a.dky ? a.dkx : a.dky;
  k.rmin_dkr = 1.f / k.min_dkr;
  k.supp_r = a.supp_radius * k.min_dkr;
  k.rrcut = 1.f / a.rdistcutoff;
  k.r2_in = r2_below(a.rdistcutoff);
  k.r2_supp = r2_atmost(k.supp_r);
  k.rapo = 1.f / a.apocutoff;
  k.rzapo = a.zapocutoff > 0 ? 1.f / a.zapocutoff : 0.f;
  k.order0_shared = 1;
  for (int d = 1; d < a.ndirs; ++d)
    if (a.noisevar[d * no] != a.noisevar[0]) k.order0_shared = 0;
  return k;
}

// Every looked-up radius is <= rdistcutoff (filter_rows and sum_terms hold the
// pixels outside at the edge), so the table is never left when
// floor(rdistcutoff / dkrotf) + 3 <= nxotf (+ 3: a cross term's interpolation
// radius comes from an approximate square root and may pass rdistcutoff by
// an ulp) and no kz index, |kz| <= nz/2, leaves it along kz; otherwise the
// lookups clamp
inline bool filter_needs_clamp(const FilterArgs& a, const FilterK& k)
{
  return !(std::floor(a.rdistcutoff * k.rdkrotf) + 3 <= a.otf.nxotf) ||
         !(a.nz == 1 || (a.nz / 2) * (double)a.otf.kzscale + 1.0 < a.otf.nzotf);
}

// Two pixels of column kx on the data rows r0 and r0 + 1, as a thread of the
// fused assembly filters them: rows in transform order, row r at ky = r or
// r - ny; row ny/2 holds the pixel ky = -ny/2 for the filter (both passes of
// the reference index rows as y in [-ny/2, ny/2 - 1]).
struct FilterRows {
  int ky[2];
  float yf[2], rd[2];
  bool in[2];  // a row of the image, inside the support
  // The radii at which the pixels' own OTF is looked up.  A pixel outside goes
  // through the filter with its neighbour and is dropped there; it can lie dky
  // beyond the support, more bins than filter_needs_clamp leaves where the image
  // is short against the OTF, so its lookup stays at the edge.  (Formed where it
  // is used: held in rd, the pass of 640 x 384 x 30 took 0.670 instead of
  // 0.641 ms.)
  __host__ __device__ __forceinline__ float2 own(float cutoff) const
  {
    return make_float2(fminf(rd[0], cutoff), fminf(rd[1], cutoff));
  }
};
__host__ __device__ __forceinline__ FilterRows filter_rows(float dky, float cutoff, int ny, float x1f, int r0)
{
  FilterRows p;
#ifdef __CUDACC__
#pragma unroll
#endif
  for (int i = 0; i < 2; ++i) {
    const int r = r0 + i;
    p.ky[i] = r <= ny / 2 ? r : r - ny;
    const int kyf = p.ky[i] == ny / 2 ? -(ny / 2) : p.ky[i];
    p.yf[i] = kyf * dky;
    p.rd[i] = sqrtf(x1f * x1f + p.yf[i] * p.yf[i]);
    p.in[i] = r < ny && p.rd[i] <= cutoff;
  }
  return p;
}

// The terms of the Wiener denominator that a CTA's pixels can meet, in shared
// memory: p = (-shift y twice, |amp|^2 / noisevar twice), aligned pairs for the
// paired instructions; q = (shift x, first entry of the order's radial table).
// Three runs: side orders whose suppressed centre no column of the CTA reaches
// (up to nplain), the other side orders (up to nside), order 0 (up to n).  A
// term whose support no column reaches is left out.
struct FilterTerms {
  float4 p[kMaxDirs * (2 * kMaxOrders - 1)];
  float2 q[kMaxDirs * (2 * kMaxOrders - 1)];
  int nplain, nside, n;
};

// Shared memory of the radial tables, [2][norders][nxotf].  Entries are the
// values alone: with the step to the next bin beside each (one 16-byte load a
// lookup) the tables took twice the space and twice the building, the fused
// kernels lost a CTA per SM from 66 bins on, and 512^2 x 48 took 1.23 ms at 129
// bins and 2.51 at 513, against 1.02 and 1.41.  At 65 bins the wider entries cost
// or gained little: 0.98 either way there, 1024^2 x 8 0.76 against 0.78 with
// values, 640 x 384 x 30 0.66 against 0.64.
inline size_t filter_tab_bytes(int norders, int nxotf) { return 2 * (size_t)norders * nxotf * sizeof(float2); }
// The fused kernels' tables at most: with the transform buffer of 1024 rows two
// CTAs stay resident on an SM (three up to 129 bins and three orders)
constexpr size_t kFusedTabMax = 32 * 1024;

// |x| of a term's distance at column x1f, (x1f + kxo) - sx, less what rounding
// or a fused product can move it: a term is left out of a CTA's list, or taken
// for an unsuppressed one, only where no rounding of the per-pixel test can
// disagree.
__host__ __device__ __forceinline__ float filter_x_least(float x1f, float kxo, float sx)
{
  const float slack = 1e-6f * (fabsf(x1f) + fabsf(kxo) + fabsf(sx));  // 16 units of the largest sum
  return fmaxf(fabsf(x1f + kxo - sx) - slack, 0.f);
}

// the switches fixed at compile time on the table path
inline int filter_flags(const FilterArgs& a)
{
  return (a.suppress ? 1 : 0) | (a.dampen0 ? 2 : 0) | (a.filteroverlaps ? 4 : 0);
}

#ifdef __CUDACC__

__device__ __forceinline__ float dev_suppress(float x)
{
  float x6 = x * x * x;
  x6 *= x6;
  return 1.f / (1 + 20000 / (x6 + 20));  // float division: correctly rounded, like the double one rounded
}

// Wiener scale of pixel (x1f, y1f, z0) of band (dir, order): the body of
// filterbands_kernel1 (gpuFunctionsImpl.cu:1504-1592) without the final
// conjamp factor.  ND/NO: compile-time direction and order counts (0: use
// the runtime values).
// OTF value of order o at radial index krindex in the plane's kz: from the
// plane's radial table (TAB; its entries are the kz interpolation of the
// bilinear lookup, so the result is the same interpolation), else the
// bilinear lookup itself.
// The bin is the integer nearest to krindex - 1/2, taken from the mantissa of
// a sum with 1.5 * 2^23 (additions on the FP32 pipe; float-to-int and back
// are quarter-rate): a krindex on a bin boundary may give the bin below with
// ar = 1, the same value.  krindex < nxotf, far below 2^22.
template <bool CLAMP, bool TAB>
__device__ __forceinline__ float2 filter_otf(const FilterArgs& a, const float2* tabz, int o, float krindex,
                                             const OtfKz& kzi)
{
  if (TAB) {
    const float m = (krindex - 0.5f) + 12582912.f;
    const int ir = __float_as_int(m) - 0x4B400000;
    const float ar = krindex - (m - 12582912.f);
    const float2* t = tabz + o * a.otf.nxotf + ir;
    const float2 t0 = t[0], t1 = t[1];
    return make_float2(fmaf(ar, t1.x - t0.x, t0.x), fmaf(ar, t1.y - t0.y, t0.y));
  }
  return otf_lookup_rr<CLAMP>(a.otf.otf[o], a.otf, krindex, kzi);
}

// FL >= 0: the suppress (bit 0), dampen-order-0 (bit 1) and filter-overlaps
// (bit 2) switches fixed at compile time; FL < 0: read from the arguments.
// termw: |amp|^2 / noisevar of every (direction, order) (FitDev::termw, in
// registers on the compile-time paths); ampmag2: |amp|^2 of this band.
template <int ND, int NO, bool CLAMP, bool TAB, int FL>
__device__ __forceinline__ float2 filter_scale(const FilterArgs& a, const FilterK& k, const float* termw,
                                               float ampmag2, int dir, int order, int z0, float rdist1, float x1f,
                                               float y1f, const float2* tabz)
{
  const bool suppress = FL >= 0 ? (FL & 1) != 0 : a.suppress != 0;
  const bool dampen0 = FL >= 0 ? (FL & 2) != 0 : a.dampen0 != 0;
  const bool filteroverlaps = FL >= 0 ? (FL & 4) != 0 : a.filteroverlaps != 0;
  const int nd = ND ? ND : a.ndirs, no = NO ? NO : a.norders;
  const float xabs = x1f + k.kxo[dir * no + order], yabs = y1f + k.kyo[dir * no + order];
  const OtfKz kzi = otf_kz(a.otf, z0);
  // order-0 damping's axial part |z0 / zdc0|^3, the same for every term
  const float zf = fabsf(z0 / (float)a.zdc[0]);
  const float zf3 = zf * zf * zf;
  float2 otf1 = filter_otf<CLAMP, TAB>(a, tabz, order, rdist1 * k.rdkrotf, kzi);
  float weight = otf1.x * otf1.x + otf1.y * otf1.y;
  if (order != 0) weight *= ampmag2;
  float dampfact = k.rnv[dir * no + order];
  if (suppress && order != 0 && rdist1 <= k.supp_r)
    dampfact *= dev_suppress(rdist1 * k.rmin_dkr);
  else if (!dampen0 && suppress && order == 0 && rdist1 <= k.supp_r)
    dampfact *= dev_suppress(rdist1 * k.rmin_dkr);
  else if (dampen0 && order == 0) {
    const float rf = rdist1 * k.rrcut;
    dampfact *= rf * rf + zf3;
  }
  if (order == 0 && z0 == 0 && a.nokz0) dampfact = 0;
  weight *= dampfact;
  float sumweight = weight;
#pragma unroll
  for (int dir2 = 0; dir2 < nd; dir2++) {
#pragma unroll
    for (int order2 = -(no - 1); order2 < no; order2++) {
      if (dir2 == dir && order2 == order) continue;
      if (!filteroverlaps && !(order2 == 0 && order == 0)) continue;
      const int ao2 = order2 < 0 ? -order2 : order2;
      const float sx = order2 < 0 ? -k.kxo[dir2 * no + ao2] : k.kxo[dir2 * no + ao2];
      const float sy = order2 < 0 ? -k.kyo[dir2 * no + ao2] : k.kyo[dir2 * no + ao2];
      const float x2 = xabs - sx, y2 = yabs - sy;
      const float r2 = x2 * x2 + y2 * y2;
      if (r2 < k.r2_in) {  // rdist2 < rdistcutoff
        const float rdist2 = sqrt_approx(r2);
        const float2 otf2 = filter_otf<CLAMP, TAB>(a, tabz, ao2, rdist2 * k.rdkrotf, kzi);
        float w = (otf2.x * otf2.x + otf2.y * otf2.y) * termw[dir2 * no + ao2];
        if (suppress && order2 != 0 && r2 <= k.r2_supp)
          w *= dev_suppress(rdist2 * k.rmin_dkr);
        else if (!dampen0 && suppress && order2 == 0 && r2 <= k.r2_supp)
          w *= dev_suppress(rdist2 * k.rmin_dkr);
        else if (dampen0 && order2 == 0) {
          const float rf = rdist2 * k.rrcut;
          w *= rf * rf + zf3;
        }
        if (a.nokz0 && order2 == 0 && z0 == 0) w = 0.0f;
        sumweight += w;
      }
    }
  }
  sumweight += a.wiener2;
  const float f = dampfact / sumweight;
  float2 scale = make_float2(otf1.x * f, -otf1.y * f);
  if (a.apodizeoutput) {
    float rdistabs = sqrtf(xabs * xabs + yabs * yabs);
    float rho;
    float zdistabs = abs(z0);
    const float ra = rdistabs * k.rapo;
    if (a.zapocutoff > 0 && a.bessel) {  // gpuFunctionsImpl.cu:1572-1577
      const float rhox = xabs * k.rrcut, rhoy = yabs * k.rapo, rhoz = zdistabs * k.rzapo;
      rho = sqrtf(rhox * rhox + rhoy * rhoy + rhoz * rhoz);
    } else if (a.zapocutoff > 0) {
      const float rz = zdistabs * k.rzapo;
      rho = sqrtf(ra * ra + rz * rz);
    } else {
      rho = ra;
    }
    if (rho > 1.f) rho = 1.0f;
    float apofact = 1.f;
    if (a.apodizeoutput == 1) apofact = cosf(1.57079632679f * rho);
    else if (a.apodizeoutput == 2) apofact = 1.0f - rho;
    scale.x *= apofact;
    scale.y *= apofact;
  }
  return scale;
}

// ------------------------------------------------------ pairs of pixels
// Two float operations in one instruction (each half rounded as the scalar one)
__device__ __forceinline__ float2 add2(float2 a, float2 b)
{
  float2 r;
  asm("add.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<unsigned long long&>(r))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
  return r;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b)
{
  float2 r;
  asm("mul.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<unsigned long long&>(r))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
  return r;
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c)
{
  float2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(reinterpret_cast<unsigned long long&>(r))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)),
        "l"(reinterpret_cast<unsigned long long&>(c)));
  return r;
}
__device__ __forceinline__ float2 dup2(float v) { return make_float2(v, v); }

// |OTF|^2 of order slot T at two radial indices (filter_otf's table lookup)
__device__ __forceinline__ float2 otf_mag2_pair(const float2* T, float2 kri)
{
  const float2 m = add2(add2(kri, dup2(-0.5f)), dup2(12582912.f));
  const float2 ar = fma2(add2(m, dup2(-12582912.f)), dup2(-1.f), kri);
  const float2 *t0 = T + (__float_as_int(m.x) - 0x4B400000), *t1 = T + (__float_as_int(m.y) - 0x4B400000);
  const float2 a0 = t0[0], b0 = t0[1], a1 = t1[0], b1 = t1[1];
  const float2 v0 = fma2(dup2(ar.x), csub(b0, a0), a0);
  const float2 v1 = fma2(dup2(ar.y), csub(b1, a1), a1);
  return make_float2(fmaf(v0.x, v0.x, v0.y * v0.y), fmaf(v1.x, v1.x, v1.y * v1.y));
}

// square root for the interpolation radius of a pair (subnormal squares flushed)
__device__ __forceinline__ float2 sqrt_pair(float2 x)
{
  float2 r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(x.x));
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(x.y));
  return r;
}

// built by the CTA's first warp; a barrier must follow.  kx0: the CTA's first
// column, ncol of them.
__device__ __forceinline__ void build_filter_terms(const FilterArgs& a, const FilterK& k, int dir, int order, int kz,
                                                   int kx0, int ncol, FilterTerms& out)
{
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x, no = a.norders, per = 2 * no - 1, all = a.ndirs * per;
  const float kxo = __ldg(a.fit->kxo + dir * no + order);
  int n = 0;
  for (int run = 0; run < 3; ++run) {  // plain side orders, suppressed ones, order 0
    for (int i0 = 0; i0 < all; i0 += 32) {
      const int i = i0 + lane, d2 = i / per, o2 = i - d2 * per - (no - 1), ao = abs(o2);
      bool use = i < all && (o2 == 0) == (run == 2) && !(d2 == dir && o2 == order);
      if (!a.filteroverlaps && !(o2 == 0 && order == 0)) use = false;
      if (o2 == 0 && a.nokz0 && kz == 0) use = false;
      float sx = 0.f, sy = 0.f, w = 0.f;
      if (use) {
        sx = __ldg(a.fit->kxo + d2 * no + ao);
        sy = __ldg(a.fit->kyo + d2 * no + ao);
        if (o2 < 0) {
          sx = -sx;
          sy = -sy;
        }
        w = __ldg(a.fit->termw + d2 * no + ao);
        bool reach = false, supp = false;
        for (int c = 0; c < ncol; ++c) {
          float x1f = (kx0 + c) * a.dkx;
          if (order == 0) x1f = fabsf(x1f);  // order 0 is filtered at the stored element's own pixel
          const float x2 = filter_x_least(x1f, kxo, sx);
          reach = reach || x2 * x2 < k.r2_in;
          supp = supp || (a.suppress && x2 * x2 <= k.r2_supp);
        }
        use = reach && (run == 2 || supp == (run == 1));
      }
      const unsigned m = __ballot_sync(0xffffffffu, use);
      if (use) {
        const int at = n + __popc(m & ((1u << lane) - 1));
        out.p[at] = make_float4(-sy, -sy, w, w);
        out.q[at] = make_float2(sx, __int_as_float(ao * a.otf.nxotf));
      }
      n += __popc(m);
    }
    if (lane == 0) (run == 0 ? out.nplain : run == 1 ? out.nside : out.n) = n;
  }
}

// One run of the term list: the sum of the terms' weights at two pixels
enum : int { kTermPlain = 0, kTermSuppressed = 1, kTermOrder0 = 2 };
template <int KIND>
__device__ __forceinline__ float2 sum_terms(const FilterArgs& a, const FilterK& k, const FilterTerms& terms, int i0,
                                            int i1, float xabs, float2 yabs, float zf3, const float2* tabz, float2 sum)
{
#pragma unroll 1
  for (int i = i0; i < i1; ++i) {
    const float4 p = terms.p[i];
    const float2 q = terms.q[i];
    const float x2 = xabs - q.x;
    const float2 y2 = add2(yabs, make_float2(p.x, p.y));
    const float2 r2 = fma2(y2, y2, dup2(x2 * x2));
    const bool in0 = r2.x < k.r2_in, in1 = r2.y < k.r2_in;  // rdist2 < rdistcutoff
    if (in0 || in1) {
      // the one outside (if any) is looked up at the edge and dropped
      const float2 rd = sqrt_pair(make_float2(fminf(r2.x, k.r2_in), fminf(r2.y, k.r2_in)));
      float2 w = mul2(otf_mag2_pair(tabz + __float_as_int(q.y), mul2(rd, dup2(k.rdkrotf))), make_float2(p.z, p.w));
      if (KIND == kTermOrder0 && a.dampen0) {
        const float2 rf = mul2(rd, dup2(k.rrcut));
        w = mul2(w, fma2(rf, rf, dup2(zf3)));
      } else if (KIND == kTermSuppressed || (KIND == kTermOrder0 && a.suppress)) {
        if (r2.x <= k.r2_supp) w.x *= dev_suppress(rd.x * k.rmin_dkr);
        if (r2.y <= k.r2_supp) w.y *= dev_suppress(rd.y * k.rmin_dkr);
      }
      sum = add2(sum, make_float2(in0 ? w.x : 0.f, in1 ? w.y : 0.f));
    }
  }
  return sum;
}

// The slot whose plane a CTA of the fused assembly filters
struct FilterSlot {
  const float2 *br, *bi;  // order 0: band of direction 0 and null
  size_t plane, dstride;
  int nx, ny, nz, order, dir, kz;
  float ampmag2;
  float2 conjamp;
  float kxo, kyo, rapo;  // the fit's values for (dir, order): FitDev
};
// the fit's part of the slot (dir = 0 for the summed order 0)
__device__ __forceinline__ void load_fit(const FilterArgs& a, FilterSlot& f)
{
  const int i = f.dir * a.norders + f.order;
  f.ampmag2 = 0.f;
  f.conjamp = make_float2(1.f, 0.f);
  if (f.order != 0) {
    f.ampmag2 = __ldg(a.fit->ampmag2 + i);
    const float2 am = __ldg(a.fit->amp + i);
    f.conjamp = make_float2(am.x, -am.y);
  }
  f.kxo = __ldg(a.fit->kxo + i);
  f.kyo = __ldg(a.fit->kyo + i);
  f.rapo = __ldg(&a.fit->rapo);
}

// filter_scale's Wiener scale (table path) of two pixels of one column, (x1f,
// y1f.x) and (x1f, y1f.y).  Two pixels of neighbouring rows take nearly always
// the same side of a term's support test, share the x half of the distance,
// and their additions and products pair up in one instruction each.  The terms
// are a loop over the CTA's list: unrolled over directions and orders the code
// did not fit the instruction cache, whose misses were the largest stall
// (2.6 of 8 warps an issue), and a third of its tests were for terms out of
// the columns' reach.
__device__ __forceinline__ void filter_scale_pair(const FilterArgs& a, const FilterK& k, const FilterTerms& terms,
                                                  const FilterSlot& f, int z0, float2 rdist1, float x1f, float2 y1f,
                                                  const float2* tabz, float2& s0, float2& s1)
{
  const int order = f.order, i1 = f.dir * a.norders + order;
  const float ampmag2 = f.ampmag2;
  const float xabs = x1f + f.kxo;
  const float2 yabs = add2(y1f, dup2(f.kyo));
  const float zf = fabsf(z0 / (float)a.zdc[0]);
  const float zf3 = zf * zf * zf;
  float2 sum = make_float2(0.f, 0.f);
  sum = sum_terms<kTermPlain>(a, k, terms, 0, terms.nplain, xabs, yabs, zf3, tabz, sum);
  sum = sum_terms<kTermSuppressed>(a, k, terms, terms.nplain, terms.nside, xabs, yabs, zf3, tabz, sum);
  sum = sum_terms<kTermOrder0>(a, k, terms, terms.nside, terms.n, xabs, yabs, zf3, tabz, sum);
  const bool dampen0 = a.dampen0 != 0;
  const bool drop0 = a.nokz0 && z0 == 0;
  auto finish = [&](float r1, float yabs1, float others) {
    const float2 otf1 = filter_otf<false, true>(a, tabz, order, r1 * k.rdkrotf, OtfKz{});
    float weight = otf1.x * otf1.x + otf1.y * otf1.y;
    if (order != 0) weight *= ampmag2;
    float dampfact = k.rnv[i1];
    if (dampen0 && order == 0) {
      const float rf = r1 * k.rrcut;
      dampfact *= rf * rf + zf3;
    } else if (a.suppress && r1 <= k.supp_r) {
      dampfact *= dev_suppress(r1 * k.rmin_dkr);
    }
    if (order == 0 && drop0) dampfact = 0;
    const float q = dampfact / (weight * dampfact + others + a.wiener2);
    float2 scale = make_float2(otf1.x * q, -otf1.y * q);
    if (a.apodizeoutput) {
      const float ra = sqrtf(xabs * xabs + yabs1 * yabs1) * f.rapo;
      float rho = ra;
      if (a.zapocutoff > 0) {
        const float rz = abs(z0) * k.rzapo;
        rho = sqrtf(ra * ra + rz * rz);
      }
      if (rho > 1.f) rho = 1.0f;
      float apofact = 1.f;
      if (a.apodizeoutput == 1) apofact = cosf(1.57079632679f * rho);
      else if (a.apodizeoutput == 2) apofact = 1.0f - rho;
      scale.x *= apofact;
      scale.y *= apofact;
    }
    return scale;
  };
  s0 = finish(rdist1.x, yabs.x, sum.x);
  s1 = finish(rdist1.y, yabs.y, sum.y);
}

// Filtered values of column kx on the data rows r0 and r0 + 1 (r0 + 1 may be
// past the end), filter_rows' pixels
__device__ __forceinline__ void filtered_rows(const FilterArgs& fa, const FilterK& fk, const FilterSlot& f,
                                              const FilterTerms& terms, const float2* tab, int kx, int r0, float2& v0,
                                              float2& v1)
{
  v0 = v1 = make_float2(0.f, 0.f);
  const int nd = fa.ndirs, no = fa.norders;
  const int nxh = f.nx / 2 + 1;
  const float x1f = kx * fa.dkx;
  const bool conj = kx < 0;
  int z = conj ? -f.kz : f.kz;
  if (z < 0) z += f.nz;
  const FilterRows p = filter_rows(fa.dky, fa.rdistcutoff, f.ny, x1f, r0);
  const int(&ky)[2] = p.ky;
  const float(&yf)[2] = p.yf;
  const bool(&in)[2] = p.in;
  size_t ind[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    int y = conj ? -ky[i] : ky[i];
    if (y < 0) y += f.ny;
    ind[i] = (size_t)z * f.plane + (size_t)y * nxh + (conj ? -kx : kx);
  }
  if (!in[0] && !in[1]) return;
  if (f.order == 0) {
    // each direction's order-0 band at the stored element's own pixel
    const float xs = conj ? -x1f : x1f;
    const float2 ys = make_float2(conj ? (float)(-ky[0]) * fa.dky : yf[0], conj ? (float)(-ky[1]) * fa.dky : yf[1]);
    const int zs = conj ? -f.kz : f.kz;
    const float2* tz = tab + (conj ? no * fa.otf.nxotf : 0);
    // one denominator for every direction (fk.order0_shared): direction d's own
    // term and the (d, 0) term its sum skips are the same OTF value
    float2 b0 = in[0] ? f.br[ind[0]] : make_float2(0.f, 0.f), b1 = in[1] ? f.br[ind[1]] : make_float2(0.f, 0.f);
    for (int d = 1; d < nd; ++d) {
      if (in[0]) b0 = cadd(b0, f.br[d * f.dstride + ind[0]]);
      if (in[1]) b1 = cadd(b1, f.br[d * f.dstride + ind[1]]);
    }
    float2 s0, s1;
    filter_scale_pair(fa, fk, terms, f, zs, p.own(fa.rdistcutoff), xs, ys, tz, s0, s1);
    v0 = cmul(b0, s0);
    v1 = cmul(b1, s1);
    if (conj) {
      v0.y = -v0.y;
      v1.y = -v1.y;
    }
  } else {
    const float2 zero = make_float2(0.f, 0.f);
    float2 re0 = in[0] ? f.br[ind[0]] : zero, im0 = in[0] ? f.bi[ind[0]] : zero;
    float2 re1 = in[1] ? f.br[ind[1]] : zero, im1 = in[1] ? f.bi[ind[1]] : zero;
    float2 s0, s1;
    filter_scale_pair(fa, fk, terms, f, f.kz, p.own(fa.rdistcutoff), x1f, make_float2(yf[0], yf[1]), tab, s0, s1);
    if (conj) {
      re0.y = -re0.y;
      im0.y = -im0.y;
      re1.y = -re1.y;
      im1.y = -im1.y;
    }
    v0 = cmul(make_float2(re0.x - im0.y, re0.y + im0.x), cmul(s0, f.conjamp));
    v1 = cmul(make_float2(re1.x - im1.y, re1.y + im1.x), cmul(s1, f.conjamp));
  }
  if (!in[0]) v0 = make_float2(0.f, 0.f);
  if (!in[1]) v1 = make_float2(0.f, 0.f);
}

// The radial tables of plane zp: each order's OTF interpolated to kz = zp
// (pass 0) and to the conjugate pass's kz = -zp (pass 1) along kr:
// [2][no][nxotf]
__device__ __forceinline__ void build_filter_tab(const FilterArgs& a, int no, int zp, float2* tab)
{
  const int nxo = a.otf.nxotf, nzo = a.otf.nzotf;
  for (int t = threadIdx.x; t < 2 * no * nxo; t += blockDim.x) {
    const int pass = t / (no * nxo), r = t - pass * no * nxo, o = r / nxo, ir = r - o * nxo;
    const OtfKz kz = otf_kz(a.otf, pass ? -zp : zp);
    const float2 va = __ldg(a.otf.otf[o] + ir * nzo + kz.iz), vb = __ldg(a.otf.otf[o] + ir * nzo + kz.izp);
    tab[t] = make_float2(va.x * (1 - kz.az) + vb.x * kz.az, va.y * (1 - kz.az) + vb.y * kz.az);
  }
}

#endif  // __CUDACC__

}  // namespace simrecon
