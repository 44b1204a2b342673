// The pattern-vector search on the device: findk0's peak refinement and
// fitk0andmodamps' line searches (gpuFunctionsImpl.cu:306-372, 874-1044)
// without a host round trip.
//
// findk0_finish     the cross-correlation peak's parabola fits and the
//                   wrap-around choice -> k0 (findk0.cuh)
// k_k0_search       one thread-block cluster per direction (all directions in
//                   one launch, side by side on the GPU): the angle and
//                   magnitude line searches with their parabola fits and the
//                   final modulation amplitude.  The cluster's CTAs
//                   evaluate batches of candidate k0s over the overlap map P
//                   (each CTA one tile of P, its partial sums written into
//                   the leader CTA's shared memory); one thread of the
//                   leader runs the sequential search between batches.
//
// The search visits the same float32 angles and magnitudes as the reference
// (float-accumulated steps from the start value) and makes its decisions
// and parabola fits with separately rounded float operations, as the
// reference's host code does.  The candidate values themselves come from the
// device's cosf/sinf/atan2f, which may differ from a host libm in the last
// bit, and the phase factors from float sincospi of an exactly reduced
// argument (the host-driven evaluation uses double sincos), so the fitted k0
// matches the host-driven search to a few 1e-5 pixel, not bit for bit.
#include <cooperative_groups.h>

#include "findk0.cuh"
#include "kernels.h"

namespace cg = cooperative_groups;

namespace simrecon {

namespace {

// fitxyparabola, gpuFunctionsImpl.cu:1022-1044
__device__ float fitxyparabola_rn(float x1, float y1, float x2, float y2, float x3, float y3)
{
  if (x1 == x2 || x2 == x3 || x3 == x1) return 0.f;
  const float xbar1 = __fmul_rn(0.5f, __fadd_rn(x1, x2));
  const float xbar2 = __fmul_rn(0.5f, __fadd_rn(x2, x3));
  const float slope1 = __fdiv_rn(__fsub_rn(y2, y1), __fsub_rn(x2, x1));
  const float slope2 = __fdiv_rn(__fsub_rn(y3, y2), __fsub_rn(x3, x2));
  const float curve = __fdiv_rn(__fsub_rn(slope2, slope1), __fsub_rn(xbar2, xbar1));
  if (curve == 0.f) return 0.f;
  return __fsub_rn(xbar2, __fdiv_rn(slope2, curve));
}

constexpr int kSCmax = 16;    // CTAs per cluster at most: one direction's search
constexpr int kST = 512;      // threads per CTA
constexpr int kSW = kST / 32;
constexpr int kSB = 32;       // candidates per batch at most
constexpr long long kSearchWide = 256 * 256;
constexpr int kSL = 1024;     // line cache: steps -kSL..kSL from the start value
// first batch of a line: the start and 3 to 12 steps each way (line_start),
// later batches 8 steps further along the climb
constexpr int kSLine0Min = 3, kSLine0Max = 12;
constexpr int kSLineK = 8;
// every batch but the two line starts and the final evaluation extends a
// climb by kSLineK steps, so this bounds the batches of a search
constexpr int kSMaxBatches = 2 * (2 * kSL / kSLineK + 2) + 4;

enum : int { kPhaseAngle = 0, kPhaseMag = 1, kPhaseFinal = 2, kPhaseDone = 3 };

struct SearchLine {
  float val[2 * kSL + 1];  // |modamp|^2 at step j (index j + kSL)
  float pos[2 * kSL + 1];  // the angle or magnitude at step j
  unsigned char have[2 * kSL + 1];
};

struct __align__(16) SearchCtl {
  int nbatch;                // candidates of the current batch; 0: finished
  int vary_angle;            // 1: pos[] are angles at magnitude `fixed`; 0: magnitudes at angle `fixed`
  float fixed;
  int pad;
  float pos[kSB];            // the batch's positions along its line
  int j[kSB];                // their line steps
  float4 khl[kSB];           // candidate vectors k1 * fitorder2 * dxy as float pairs: x hi, lo, y hi, lo
  double red[kSCmax][kSB][2];  // every CTA's partial XStarY (leader only)
  double res[kSB][2];        // the batch's XStarY (leader only)
};

struct ClimbResult {
  int need;   // 1: step `j` is not evaluated yet
  int j;
  float fit;  // fitxyparabola of the last three points
  float x1, amp1;
};

// One line search of fitk0andmodamps (gpuFunctionsImpl.cu:902-942 for the
// angle, 944-985 for the magnitude), replayed from the line's cached values;
// x1 / amp1 carry over from the previous line as in the reference (declared
// once, not reset between the two searches).
__device__ __forceinline__ ClimbResult run_climb(const SearchLine& L, float x1, float amp1)
{
  ClimbResult r{0, 0, 0.f, x1, amp1};
  auto has = [&](int j) { return j >= -kSL && j <= kSL && L.have[j + kSL]; };
  if (!has(0)) return ClimbResult{1, 0, 0.f, x1, amp1};
  if (!has(1)) return ClimbResult{1, 1, 0.f, x1, amp1};
  float x2 = L.pos[kSL], amp2 = L.val[kSL];
  float x3 = L.pos[kSL + 1], amp3 = L.val[kSL + 1];
  int steps = 0;
  if (amp3 > amp2) {
    int j = 1;
    while (amp3 > amp2 && steps < kMaxClimbSteps) {
      amp1 = amp2;
      x1 = x2;
      amp2 = amp3;
      x2 = x3;
      ++j;
      ++steps;
      if (!has(j)) return ClimbResult{1, j, 0.f, x1, amp1};
      x3 = L.pos[j + kSL];
      amp3 = L.val[j + kSL];
    }
  } else {
    float a = amp3;
    amp3 = amp2;
    amp2 = a;
    a = x3;
    x3 = x2;
    x2 = a;
    int j = 0;
    while (amp3 > amp2 && steps < kMaxClimbSteps) {
      amp1 = amp2;
      x1 = x2;
      amp2 = amp3;
      x2 = x3;
      --j;
      ++steps;
      if (!has(j)) return ClimbResult{1, j, 0.f, x1, amp1};
      x3 = L.pos[j + kSL];
      amp3 = L.val[j + kSL];
    }
  }
  r.fit = fitxyparabola_rn(x1, amp1, x2, amp2, x3, amp3);
  r.x1 = x1;
  r.amp1 = amp1;
  return r;
}

// Leader state, held by thread 0 of CTA 0 across batches
struct Controller {
  int phase;
  int status;
  int ncand;           // candidates evaluated
  float k0mag, k0angle, delta_angle, delta_mag;
  float afit, mfit;    // fitted angle, magnitude
  float x1, amp1;      // carried between the lines
  float angle_px;      // pixels of the overlaps' spectrum per step of angle, of magnitude
  float mag_px;
};

// Steps each way that a line's first batch evaluates: the cross-correlation's
// parabola leaves the start within about 0.4 pixel of the peak, and the climb
// looks one or two steps past it.  Every step costs a pass of FMAs over P, a
// missing one a further batch.
__device__ __forceinline__ int line_start(float px_per_step)
{
  const int n = (int)ceilf(0.4f / px_per_step) + 2;
  return min(max(n, kSLine0Min), kSLine0Max);
}

// position of step j from its neighbour towards the start (float-accumulated
// like the reference's angle += deltaangle)
__device__ __forceinline__ void set_pos(SearchLine& L, int j, float base, float delta)
{
  if (j == 0) L.pos[kSL] = base;
  else if (j > 0) L.pos[j + kSL] = __fadd_rn(L.pos[j - 1 + kSL], delta);
  else L.pos[j + kSL] = __fsub_rn(L.pos[j + 1 + kSL], delta);
}

// queue steps j, j+s, ... (or the start batch) of the current line; the
// candidate vectors are formed by the leader's threads in parallel
__device__ __forceinline__ void request_line(const Controller& c, SearchLine& L, SearchCtl& ctl, int j)
{
  const bool ang = c.phase == kPhaseAngle;
  const float base = ang ? c.k0angle : c.k0mag;
  const float delta = ang ? c.delta_angle : c.delta_mag;
  int n = 0;
  auto add = [&](int jj) {
    if (jj < -kSL || jj > kSL || L.have[jj + kSL]) return;
    set_pos(L, jj, base, delta);
    ctl.pos[n] = L.pos[jj + kSL];
    ctl.j[n] = jj;
    ++n;
  };
  if (j == 0) {  // a new line: nothing is evaluated yet
    const int n0 = line_start(ang ? c.angle_px : c.mag_px);
    float up = base, dn = base;
    L.pos[kSL] = ctl.pos[0] = base;
    ctl.j[0] = 0;
    for (int i = 1; i <= n0; ++i) {
      up = __fadd_rn(up, delta);
      dn = __fsub_rn(dn, delta);
      L.pos[kSL + i] = ctl.pos[i] = up;
      L.pos[kSL - i] = ctl.pos[n0 + i] = dn;
      ctl.j[i] = i;
      ctl.j[n0 + i] = -i;
    }
    n = 2 * n0 + 1;
  } else {
    const int s = j > 0 ? 1 : -1;
    for (int i = 0; i < kSLineK; ++i) add(j + s * i);
  }
  ctl.vary_angle = ang;
  ctl.fixed = ang ? c.k0mag : c.afit;
  ctl.nbatch = n;
}

// Advance the search over the finished batch (its values are in the line),
// queue the next batch (or none).  Runs on one thread; lines[0] is the angle line, lines[1] the
// magnitude line.
__device__ __forceinline__ void control(Controller& c, SearchLine* lines, SearchCtl& ctl, const K0SearchArgs& a, int dir)
{
  const int nb = ctl.nbatch;
  if (c.phase == kPhaseFinal && nb > 0) {
    // getmodamp at the fitted (angle, magnitude): the amplitude of fitorder2
    double* slot = a.slot[dir];
    slot[0] = ctl.res[0][0];
    slot[1] = ctl.res[0][1];
    slot[2] = a.sumxy[dir][0];
    slot[3] = a.sumxy[dir][1];
    *a.k0fit[dir] = polar_rn(c.mfit, c.afit);
    c.phase = kPhaseDone;
    ctl.nbatch = 0;
    return;
  }
  ctl.nbatch = 0;
  while (c.phase == kPhaseAngle || c.phase == kPhaseMag) {
    SearchLine& L = lines[c.phase == kPhaseAngle ? 0 : 1];
    const ClimbResult r = run_climb(L, c.x1, c.amp1);
    if (r.need) {
      if (r.j < -kSL || r.j > kSL) {  // beyond the line cache: the host search takes over
        c.status = 1;
        c.phase = kPhaseDone;
        return;
      }
      request_line(c, L, ctl, r.j);
      return;
    }
    c.x1 = r.x1;
    c.amp1 = r.amp1;
    if (c.phase == kPhaseAngle) {
      c.afit = r.fit;
      c.phase = kPhaseMag;
      continue;
    }
    c.mfit = r.fit;
    c.phase = kPhaseFinal;
    ctl.pos[0] = c.mfit;
    ctl.j[0] = 0;
    ctl.vary_angle = 0;
    ctl.fixed = c.afit;
    ctl.nbatch = 1;
  }
}

// Phase factor e^{i 2 pi m k dxy} for m = x - n/2 (an integer or a half
// integer, exact in float): m * (k dxy) split into a float product, its exact
// rounding error (fmaf) and the low part of k dxy, reduced to [-1/2, 1/2]
// turns before sincospif -- a phase error of a few 1e-7 rad at any m.
__device__ __forceinline__ float2 phase_factor(int x, int n, float hi, float lo)
{
  const float fm = 0.5f * (float)(2 * x - n);
  const float p = fm * hi;
  const float e = fmaf(fm, hi, -p);
  const float t = fmaf(fm, lo, e);
  const float r = (p - rintf(p)) + t;
  float s, c;
  sincospif(2.f * r, &s, &c);
  return make_float2(c, s);
}

// XStarY partial sums of CC candidates over this CTA's tile: per row the x
// sum with the x phase factors, times the row's y factor; kRows rows per pass
// share the x factors (with two, their shared-memory reads took as long as the
// FMAs), and the next loads of P are in flight meanwhile.  acc: per-thread sums.
constexpr int kRows = 4;
__device__ __forceinline__ unsigned long long pack2(float x, float y)
{
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v)
{
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c)
{
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
template <int CC>
__device__ __forceinline__ void tile_sums(const float2* __restrict__ pmap, int nx, const float2* ex, const float2* ey,
                                          int tw, int th, int tp, int warp, int lane, float2 (&acc)[CC])
{
#pragma unroll
  for (int k = 0; k < CC; ++k) acc[k] = make_float2(0.f, 0.f);
  // rows and columns past the tile repeat its last: their x factors are zero
  // and their rows' sums are not taken
  auto load = [&](int y, int x, float2 (&p)[kRows]) {
    const float2* col = pmap + min(x, tw - 1);
#pragma unroll
    for (int r = 0; r < kRows; ++r) p[r] = __ldg(col + min(y + r, th - 1) * nx);
  };
  float2 p[kRows];
  load(kRows * warp, lane, p);
  for (int y = kRows * warp; y < th; y += kRows * kSW) {
    unsigned long long r[kRows][CC];  // (re, im): both parts of a product's sum in one paired FMA
#pragma unroll
    for (int q = 0; q < kRows; ++q)
#pragma unroll
      for (int k = 0; k < CC; ++k) r[q][k] = 0;
    for (int x = 0; x < tw; x += 32) {
      unsigned long long a[kRows], b[kRows];
#pragma unroll
      for (int q = 0; q < kRows; ++q) {
        a[q] = pack2(p[q].x, p[q].x);
        b[q] = pack2(-p[q].y, p[q].y);
      }
      if (x + 32 < tw) load(y, x + 32 + lane, p);
      else load(y + kRows * kSW, lane, p);
      const float2* el = ex + x + lane;
#pragma unroll
      for (int k = 0; k < CC; ++k) {
        const float2 e = el[k * tp];
        const unsigned long long f = pack2(e.x, e.y), g = pack2(e.y, e.x);
#pragma unroll
        for (int q = 0; q < kRows; ++q) r[q][k] = fma2(a[q], f, fma2(b[q], g, r[q][k]));
      }
    }
#pragma unroll
    for (int q = 0; q < kRows; ++q)
      if (y + q < th) {
#pragma unroll
        for (int k = 0; k < CC; ++k) {
          const float2 e = ey[k * th + y + q], v = unpack2(r[q][k]);
          acc[k].x += v.x * e.x - v.y * e.y;
          acc[k].y += v.x * e.y + v.y * e.x;
        }
      }
  }
}

// (s, e) + (t, f), the rounding error of the sum kept
__device__ __forceinline__ void pair_add(float& s, float& e, float t, float f)
{
  const float u = __fadd_rn(s, t), b = __fsub_rn(u, s);
  e = __fadd_rn(__fadd_rn(e, f), __fadd_rn(__fsub_rn(s, __fsub_rn(u, b)), __fsub_rn(t, b)));
  s = u;
}

// The CTA's sums of CC candidates into the leader's partial-sum table at
// candidate c0: the threads' float sums transposed through shared memory, a
// warp per value, its lanes' shares and the lanes added as float pairs (48
// bits; the FP64 adder runs at a sixtyfourth of the FP32 rate here, and chains
// of it were the longest part of a batch on a small map).
template <int CC>
__device__ __forceinline__ void tile_reduce(const float2 (&acc)[CC], float* sacc, SearchCtl* lead, int rank, int c0,
                                            int n, int tid)
{
  constexpr int V = 2 * CC, kPitch = V + 1;
  static_assert(V <= kSW, "a warp per value");
  __syncthreads();  // the last pass has read its sums
#pragma unroll
  for (int k = 0; k < CC; ++k) {
    sacc[tid * kPitch + 2 * k] = acc[k].x;
    sacc[tid * kPitch + 2 * k + 1] = acc[k].y;
  }
  __syncthreads();
  const int v = tid >> 5, lane = tid & 31;
  if (v >= 2 * n) return;
  float x[kSW];
#pragma unroll
  for (int i = 0; i < kSW; ++i) x[i] = sacc[(i * 32 + lane) * kPitch + v];
  float s = x[0], e = 0.f, t = x[1], f = 0.f;
#pragma unroll
  for (int i = 2; i < kSW; i += 2) {
    pair_add(s, e, x[i], 0.f);
    pair_add(t, f, x[i + 1], 0.f);
  }
  pair_add(s, e, t, f);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    pair_add(s, e, __shfl_xor_sync(0xffffffffu, s, o), __shfl_xor_sync(0xffffffffu, e, o));
  // (a sum past the float range that a double would hold does not get here: the
  // correlation's peak, whose square is a float, is infinite long before)
  if (lane == 0) lead->red[rank][c0 + (v >> 1)][v & 1] = pair_value(s, e);
}

template <int CC>
__device__ void chunk(const float2* __restrict__ pmap, int nx, const float2* ex, const float2* ey, int tw, int th,
                      int tp, float* sacc, SearchCtl* lead, int rank, int c0, int n)
{
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float2 acc[CC];
  tile_sums<CC>(pmap, nx, ex, ey, tw, th, tp, warp, lane, acc);
  tile_reduce<CC>(acc, sacc, lead, rank, c0, n, tid);
}

// C: candidates of one pass; SC: CTAs per cluster; ntab candidates' phase
// tables at a time.
// Bound by latency on small maps (three batches, each two cluster barriers, the
// control thread, the phase tables and the reduction), by the issue of the sums
// on large ones: a pass of 8 candidates over 256 x 240 of P takes 39k cycles,
// half of them issuing.  Search of three directions with 25 candidates a first
// batch, doubles shuffled through the warps and 8 CTAs; with passes of up to 16
// candidates over two rows, their tables and segment sums in double each; and
// now: 128^2 131, 41, 33 us; 512^2 215, 63, 50; 1024 x 960 433, 127, 91 us.
// (128 registers a thread; passes of 8 spill 28 and 40 bytes at 16 and 8 CTAs.)
template <int C, int SC>
__global__ void __launch_bounds__(kST, 1) k_k0_search(const __grid_constant__ K0SearchArgs a, int ntab)
{
  cg::cluster_group cluster = cg::this_cluster();
  const unsigned rank = cluster.block_rank();
  const int dir = blockIdx.x / SC;  // one cluster per direction
  __shared__ SearchCtl ctl;
  __shared__ SearchLine lines[2];
  __shared__ float4 khl[kSB];
  __shared__ int nloc;
  extern __shared__ float2 tab[];  // phase tables [ntab][tp], [ntab][th], then the reduction's transposed sums
  SearchCtl* lead = cluster.map_shared_rank(&ctl, 0);
  const int tid = threadIdx.x;
  const int nx = a.nx, ny = a.ny;
  // tile of P: SC / 4 column parts x 4 row quarters
  constexpr int TX = SC / 4;
  const int tx = rank % TX, ty = rank / TX;
  const int x0 = tx * nx / TX, x1 = (tx + 1) * nx / TX;
  const int y0 = ty * ny / 4, y1 = (ty + 1) * ny / 4;
  const int tw = x1 - x0, th = y1 - y0, tp = (tw + 31) & ~31;
  float* sacc = (float*)(tab + (size_t)ntab * (((nx + TX - 1) / TX + 31 & ~31) + (ny + 3) / 4));
  const float2* __restrict__ pmap = a.pmap[dir] + (size_t)y0 * nx + x0;

  __shared__ Controller held;  // the control thread's, between the batches
  float sx = 1.f;  // sum |X|^2
  if (rank == 0) {
    sx = __double2float_rn(a.sumxy[dir][0]);
    for (int i = tid; i < 2 * kSL + 1; i += kST) lines[0].have[i] = lines[1].have[i] = 0;
    if (tid == 0) {
      Controller c{};
      const float2 k0 = *a.k0find[dir];
      c.phase = kPhaseAngle;
      c.k0mag = __fsqrt_rn(__fadd_rn(__fmul_rn(k0.x, k0.x), __fmul_rn(k0.y, k0.y)));
      c.k0angle = atan2f(k0.y, k0.x);
      c.delta_angle = a.delta_angle;
      c.delta_mag = a.delta_mag;
      // the overlaps beat at k0 * fitorder2; one pixel is 1 / (n dxy)
      const float ext = (float)max(nx, ny) * a.dxy * (float)a.fitorder2;
      c.angle_px = c.k0mag * a.delta_angle * ext;
      c.mag_px = a.delta_mag * ext;
      ctl.nbatch = 0;
      held = c;
    }
  }
  const float fac = (float)a.fitorder2;
  int it = 0;
  for (; it < kSMaxBatches; ++it) {
    if (rank == 0) {
      __syncthreads();  // the line has the previous batch's values; the line caches are clear
      if (tid == 0) {
        Controller c = held;
        control(c, lines, ctl, a, dir);
        c.ncand += ctl.nbatch;
        held = c;
      }
      __syncthreads();
      // the candidate vectors (getmodamp: k1 = mag (cosf, sinf)(angle), times
      // fitorder2 - fitorder1) and, once for all CTAs, their double products
      // with the pixel size (FP64 is slow on this GPU)
      if (tid < ctl.nbatch) {
        const float2 k1 = ctl.vary_angle ? polar_rn(ctl.fixed, ctl.pos[tid]) : polar_rn(ctl.pos[tid], ctl.fixed);
        const double kx = (double)__fmul_rn(k1.x, fac) * (double)a.dxy;
        const double ky = (double)__fmul_rn(k1.y, fac) * (double)a.dxy;
        const float hx = (float)kx, hy = (float)ky;
        ctl.khl[tid] = make_float4(hx, (float)(kx - (double)hx), hy, (float)(ky - (double)hy));
      }
    }
    cluster.sync();  // the batch (or the end) is visible to every CTA
    if (tid == 0) nloc = lead->nbatch;
    if (tid < kSB) khl[tid] = lead->khl[tid];
    __syncthreads();
    const int nb = nloc;
    if (nb == 0) break;
    for (int g0 = 0; g0 < nb; g0 += ntab) {
      const int ng = min(ntab, nb - g0);
      const int np = ng == 1 ? 1 : (ng + C - 1) / C * C;  // whole passes: the padding's sums are not kept
      float2* ex = tab;                    // [np][tp]
      float2* ey = tab + (size_t)np * tp;  // [np][th]
      if (g0 > 0) __syncthreads();         // the tables are read
      for (int e = tid; e < np * (tp + th); e += kST) {
        const int k = e / (tp + th), r = e - k * (tp + th);
        const float4 kk = khl[min(g0 + k, nb - 1)];
        if (r >= tp) ey[k * th + (r - tp)] = phase_factor(y0 + (r - tp), ny, kk.z, kk.w);
        else ex[k * tp + r] = r < tw ? phase_factor(x0 + r, nx, kk.x, kk.y) : make_float2(0.f, 0.f);
      }
      __syncthreads();
      for (int c0 = 0; c0 < ng; c0 += C) {
        const int n = min(C, ng - c0);
        if (n > 1) chunk<C>(pmap, nx, ex + c0 * tp, ey + c0 * th, tw, th, tp, sacc, lead, rank, g0 + c0, n);
        else chunk<1>(pmap, nx, ex + c0 * tp, ey + c0 * th, tw, th, tp, sacc, lead, rank, g0 + c0, n);
      }
    }
    cluster.sync();  // every CTA's partial sums are in the leader
    if (rank == 0 && tid < 2 * kSB) {
      double v[SC];
#pragma unroll
      for (int r = 0; r < SC; ++r) v[r] = tid < 2 * nb ? ctl.red[r][tid >> 1][tid & 1] : 0.0;
#pragma unroll
      for (int h = SC / 2; h > 0; h >>= 1)
#pragma unroll
        for (int r = 0; r < h; ++r) v[r] += v[r + h];
      if (tid < 2 * nb) ctl.res[tid >> 1][tid & 1] = v[0];
      const float m = __fdiv_rn(__double2float_rn(v[0]), sx);
      const float my = __shfl_down_sync(0xffffffffu, m, 1);
      if (tid < 2 * nb && !(tid & 1)) {  // the step's |modamp|^2 (the final evaluation's place is not read)
        SearchLine& L = lines[ctl.vary_angle ? 0 : 1];
        L.val[ctl.j[tid >> 1] + kSL] = __fadd_rn(__fmul_rn(m, m), __fmul_rn(my, my));
        L.have[ctl.j[tid >> 1] + kSL] = 1;
      }
    }
  }
  // no CTA leaves while another may still read the leader's shared memory
  cluster.sync();
  if (rank == 0 && tid == 0) {
    Controller c = held;
    if (c.phase != kPhaseDone && c.status == 0) c.status = 2;  // batch limit reached
    atomicAdd(a.info, c.ncand);
    if (c.status) atomicOr(a.info + 1, c.status);
  }
}

}  // namespace

// CTAs per cluster: sixteen where P gives each at least 4096 elements (smaller
// maps are all barriers and control, which more CTAs lengthen); a non-portable
// size, so only where the device can hold such a cluster
static int search_ctas(int nx, int ny) { return (long long)nx * ny >= kSearchWide ? 16 : 8; }

// Dynamic shared memory: ntab candidates' phase tables (x in whole warps) and a
// pass's sums
static size_t search_smem(int nx, int ny, int C, int ntab, int sc)
{
  const size_t tp = (((size_t)nx + sc / 4 - 1) / (sc / 4) + 31) / 32 * 32, th = ((size_t)ny + 3) / 4;
  return ntab * (tp + th) * sizeof(float2) + (size_t)kST * (2 * C + 1) * sizeof(float);
}

// Candidates whose phase tables are built together, all of a batch where 164 KB
// hold them; 0: not even four fit
static int search_tables(int nx, int ny, int sc)
{
  for (int n : {32, 24, 16, 8, 4})
    if (search_smem(nx, ny, n > 4 ? 8 : 4, n, sc) <= 164 * 1024) return n;
  return 0;
}

// Up to 1024^2 maps (a tile of at most 512 x 256 per CTA).  Larger maps
// take the host-driven search, whose candidate batches run on every SM: one
// cluster per direction would spend milliseconds per batch on a 1024 x 512
// tile.
bool k0_search_supported(int nx, int ny)
{
  return nx >= 64 && ny >= 8 && (long long)nx * ny <= 1024LL * 1024 && search_tables(nx, ny, 8) > 0 &&
         4 * (((size_t)nx + 1) / 2 + ((size_t)ny + 3) / 4) * sizeof(float2) + kST * 9 * sizeof(float) <= 160 * 1024;
}

int launch_k0_search(const K0SearchArgs& a, cudaStream_t s, long long* launches)
{
  if (a.nx < 64 || a.ny < 8 || a.ndirs < 1 || a.ndirs > kMaxDirs) return -1;
  auto go = [&](auto kern, int C, int ntab, int sc) -> int {
    const size_t smem = search_smem(a.nx, a.ny, C, ntab, sc);
    // raised only (under a lock): handles of other shapes launch concurrently
    allow_dynamic_smem((const void*)kern, smem);
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = sc;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.gridDim = dim3(sc * a.ndirs);
    cfg.blockDim = dim3(kST);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (sc > 8) {
      if (cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
        (void)cudaGetLastError();
        return -2;
      }
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) {
        (void)cudaGetLastError();
        return -2;
      }
    }
    return (int)cudaLaunchKernelEx(&cfg, kern, a, ntab);
  };
  KernelTimer* kt = kernel_timer();
  if (kt) kt->begin(s);
  auto by_chunk = [&]<int SC>() {
    const int ntab = search_tables(a.nx, a.ny, SC);
    if (ntab >= 8) return go(k_k0_search<8, SC>, 8, ntab, SC);
    return ntab == 4 ? go(k_k0_search<4, SC>, 4, 4, SC) : -1;
  };
  int rc = -2;
  if (search_ctas(a.nx, a.ny) == 16) rc = by_chunk.template operator()<16>();
  if (rc == -2) rc = by_chunk.template operator()<8>();
  if (rc != 0) return rc;
  if (kt) kt->end("k_k0_search", s, (double)a.ndirs * a.nx * a.ny * sizeof(float2));
  if (launches) *launches += 1;
  return (int)cudaGetLastError();
}

}  // namespace simrecon
