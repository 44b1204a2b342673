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

// Every looked-up radius is <= rdistcutoff, so the table is never left when
// floor(rdistcutoff / dkrotf) + 3 <= nxotf (+ 3: a cross term's interpolation
// radius comes from an approximate square root and may pass rdistcutoff by
// an ulp) and no kz index, |kz| <= nz/2, leaves it along kz; otherwise the
// lookups clamp
inline bool filter_needs_clamp(const FilterArgs& a, const FilterK& k)
{
  return !(std::floor(a.rdistcutoff * k.rdkrotf) + 3 <= a.otf.nxotf) ||
         !(a.nz == 1 || (a.nz / 2) * (double)a.otf.kzscale + 1.0 < a.otf.nzotf);
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
// A table entry is (t[ir], t[ir + 1] - t[ir]): one 16-byte load and two FMAs.
// The bin is the integer nearest to krindex - 1/2, taken from the mantissa of
// a sum with 1.5 * 2^23 (additions on the FP32 pipe; float-to-int and back
// are quarter-rate): a krindex on a bin boundary may give the bin below with
// ar = 1, the same value.  krindex < nxotf, far below 2^22.
template <bool CLAMP, bool TAB>
__device__ __forceinline__ float2 filter_otf(const FilterArgs& a, const float4* tabz, int o, float krindex,
                                             const OtfKz& kzi)
{
  if (TAB) {
    const float m = (krindex - 0.5f) + 12582912.f;
    const int ir = __float_as_int(m) - 0x4B400000;
    const float ar = krindex - (m - 12582912.f);
    const float4 t = tabz[o * a.otf.nxotf + ir];
    return make_float2(fmaf(ar, t.z, t.x), fmaf(ar, t.w, t.y));
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
                                               float y1f, const float4* tabz)
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

// The radial tables of plane zp: each order's OTF interpolated to kz = zp
// (pass 0) and to the conjugate pass's kz = -zp (pass 1) along kr, with the
// step to the next bin: [2][no][nxotf]
__device__ __forceinline__ void build_filter_tab(const FilterArgs& a, int no, int zp, float4* tab)
{
  const int nxo = a.otf.nxotf, nzo = a.otf.nzotf;
  for (int t = threadIdx.x; t < 2 * no * nxo; t += blockDim.x) {
    const int pass = t / (no * nxo), r = t - pass * no * nxo, o = r / nxo, ir = r - o * nxo;
    const OtfKz kz = otf_kz(a.otf, pass ? -zp : zp);
    auto at = [&](int i) {
      const float2 va = __ldg(a.otf.otf[o] + i * nzo + kz.iz), vb = __ldg(a.otf.otf[o] + i * nzo + kz.izp);
      return make_float2(va.x * (1 - kz.az) + vb.x * kz.az, va.y * (1 - kz.az) + vb.y * kz.az);
    };
    const float2 t0 = at(ir), t1 = at(ir + 1 < nxo ? ir + 1 : ir);
    tab[t] = make_float4(t0.x, t0.y, t1.x - t0.x, t1.y - t0.y);
  }
}

#endif  // __CUDACC__

}  // namespace simrecon
