"""CPU: the radial-table entries that the fused Wiener filter reads for the two
pixels of a pair (csrc/filter.cuh), over image heights that are short and long
against the OTF.  One of the two pixels may lie outside the support; its entry
has to be in the table all the same."""
import host_probe

PROBE = r"""
#include <algorithm>
#include <cstdio>
#include "filter.cuh"
using namespace simrecon;
int main()
{
  long long pairs = 0, outside = 0;
  int worst = -1 << 30;
  for (int nxotf : {33, 65, 129, 257, 513})
    for (int ny : {64, 72, 96, 128, 250, 512, 1024})
      for (float part : {0.4f, 0.86f, 0.975f, 0.985f, 0.995f}) {
        const float dxy = 0.08f;
        FilterArgs a{};
        a.norders = a.ndirs = 1;
        a.nx = a.ny = ny;
        a.nz = 1;
        a.dkx = a.dky = 1.f / (ny * dxy);
        a.rdistcutoff = part / (2.f * dxy);  // of the highest frequency
        a.otf.nxotf = nxotf;
        a.otf.nzotf = 1;
        a.otf.dkrotf = 1.f / (dxy * (nxotf - 1) * 2);
        a.otf.kzscale = 1.f;
        a.noisevar[0] = 1.f;
        a.apocutoff = 1.f;
        const FilterK k = make_filter_k(a);
        if (filter_needs_clamp(a, k)) continue;  // not taken by the fused filter
        for (int kx = 0; kx <= ny / 2; ++kx)
          for (int r = 0; r < ny; r += 2) {
            const FilterRows p = filter_rows(a.dky, a.rdistcutoff, ny, kx * a.dkx, r);
            if (!p.in[0] && !p.in[1]) continue;  // neither is looked up
            ++pairs;
            outside += !p.in[0] + !p.in[1];
            const float2 own = p.own(a.rdistcutoff);
            for (float r : {own.x, own.y}) worst = std::max(worst, (int)std::floor(r * k.rdkrotf) - (nxotf - 1));
          }
      }
  std::printf("%lld %lld %d\n", pairs, outside, worst);
}
"""


def test_pair_lookups_stay_in_the_table(tmp_path):
    pairs, outside, worst = (int(v) for v in host_probe.run(PROBE, tmp_path).split())
    assert pairs > 100000 and outside > 1000
    assert worst < 0  # a lookup reads its entry and the next; the last is nxotf - 1


SHARED = r"""
#include <cstdio>
#include "col_fft.cuh"
#include "filter.cuh"
using namespace simrecon;
int main()
{
  const size_t fixed = ColFft<1024, 32, 8>::kSmemElems * sizeof(float2) + sizeof(FilterTerms);
  const size_t sm = 228 * 1024, reserved = 1024;  // of an SM; per CTA
  for (int nxotf : {65, 129}) std::printf("%zu ", sm / (fixed + filter_tab_bytes(3, nxotf) + reserved));
  std::printf("%zu\n", sm / (fixed + kFusedTabMax + reserved));
}
"""


def test_fused_filter_keeps_its_ctas(tmp_path):
    """1024 output rows, three orders: three CTAs per SM with the OTFs of 128-
    and 256-pixel PSFs, two with the largest tables that are taken."""
    assert [int(v) for v in host_probe.run(SHARED, tmp_path).split()] == [3, 3, 2]


TERMS = r"""
#include <cmath>
#include <cstdio>
#include <random>
#include "filter.cuh"
using namespace simrecon;
int main()
{
  std::mt19937 g(7);
  auto u = [&](float a, float b) { return a + (b - a) * (float)(g() / 4294967296.0); };
  long long near = 0, missed = 0, kept = 0, far = 0;
  for (int t = 0; t < 400000; ++t) {
    const int n = 64 << (g() % 6), kx = (int)(g() % n) - n / 2;
    const float dkx = 1.f / (n * u(0.04f, 0.12f)), kxo = u(-10.f, 10.f);
    // a column whose distance is the bound, to a few units in the last place
    const float r = g() % 2 ? u(3.f, 7.f) : 10 * dkx;
    float sx = (float)((double)kx * dkx + kxo + (g() % 2 ? r : -r));
    for (int i = (int)(g() % 7); i > 0; --i) sx = std::nextafter(sx, g() % 2 ? 1e9f : -1e9f);
    const float r2 = r * r;
    // the distance as a compiler may form it: separate, or the product fused
    const float x1f = kx * dkx;
    const float d[2] = {x1f + kxo - sx, std::fma((float)kx, dkx, kxo) - sx};
    const float least = filter_x_least(x1f, kxo, sx);
    for (float x : d) {
      const bool in = x * x <= r2 || std::fma(x, x, 0.f) < r2;
      near += in;
      missed += in && !(least * least <= r2);
    }
    const float away = 1.001f * r;  // well outside: the term is not kept
    const float sf = x1f + kxo + away;
    const float lf = filter_x_least(x1f, kxo, sf);
    if (r > 3.f) ++far, kept += lf * lf <= r2;
  }
  std::printf("%lld %lld %lld %lld\n", near, missed, far, kept);
}
"""


def test_terms_are_left_out_only_out_of_reach(tmp_path):
    near, missed, far, kept = (int(v) for v in host_probe.run(TERMS, tmp_path).split())
    assert near > 100000 and far > 100000
    assert missed == 0 and kept == 0
