"""GPU: SRX_fitCounts counts each overlap build once, with the search on the
device and without a search."""
import pytest

import cudasirecon_gb300 as sr
from cudasirecon_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


# per direction: at the guess, at the refined k0, then every order but the
# fitted one; without a search every order once
@pytest.mark.parametrize("nz,search,builds", [(8, 1, 3 * (2 + 1)), (1, 1, 3 * 2), (8, 0, 3 * 2), (1, 0, 3 * 1)])
def test_builds_are_counted_once(nz, search, builds):
    twod = nz == 1
    o = syn.Optics(nphases=3 if twod else 5)
    raw = syn.simulate(64, 64, nz, o, seed=3, n_filaments=10).raw
    r = sr.Reconstructor(64, 64, raw.shape[0], syn.config_text(o, twod=twod, extra={"wiener": 0.00048828125}),
                         syn.ra_otf(o, nx_psf=64, nz_psf=24, norders=2 if twod else 3, twod=twod))
    r.recon_params().bSearchforvector = search
    r.set_raw(raw)
    r.load_and_rescale(0, 0)
    r.set_cur_time(0)
    c0 = r.fit_counts()
    r.process()
    c1 = r.fit_counts()
    r.close()
    assert c1["overlap_builds"] - c0["overlap_builds"] == builds
    assert c1["k0_searches"] - c0["k0_searches"] == 3 * search
