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
            for (int i = 0; i < 2; ++i) {
              outside += !p.in[i];
              worst = std::max(worst, (int)std::floor(p.rd[i] * k.rdkrotf) - (nxotf - 1));
            }
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
