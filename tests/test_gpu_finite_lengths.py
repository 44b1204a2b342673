"""GPU: lengths whose other comparisons have no finite answer (a volume of two
planes with kz = 0 dropped and the order-0 damping divides 0 by 0), on inputs
that have one: kz = 0 kept and the damping off, against the FP64 oracle, which
must be finite.  Also lengths of the transformable range without a factor pair
beside ones with.  Bars: rel-L2 <= 1e-4, k0 within 1e-3 pixel."""
import warnings

import numpy as np
import pytest

import cudasirecon_gb300 as sr
from cudasirecon_gb300 import synthetic as syn
from oracle.sirecon_oracle import SIMReconOracle

pytestmark = pytest.mark.gpu

KZ0 = {"wiener": 0.00048828125, "dampenOrder0": 0}


# two and three planes; 252 = 18 x 14 rows and columns; 98 and 490 have no pair
@pytest.mark.parametrize("nx,ny,nz,extra", [(72, 64, 2, KZ0), (72, 64, 3, KZ0), (72, 64, 4, {"wiener": 0.00048828125}),
                                            (64, 252, 6, {}), (252, 64, 5, {}), (64, 252, 4, KZ0), (98, 70, 9, {}),
                                            (490, 64, 5, {}), (64, 490, 5, {})])
def test_volume_matches_a_finite_oracle(nx, ny, nz, extra):
    o = syn.Optics()
    raw = syn.simulate(nx, ny, nz, o, seed=11 + nz, n_filaments=20).raw
    cfg = syn.config_text(o, extra=extra)
    otf = syn.ra_otf(o, nx_psf=64, nz_psf=24)
    q = SIMReconOracle(nx, ny, raw.shape[0], cfg, otf)
    q.set_raw(raw)
    q.load_and_rescale(0)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        q.process()
    assert np.isfinite(q.result).all() and np.isfinite(q.k0).all()
    r = sr.Reconstructor(nx, ny, raw.shape[0], cfg, otf)
    r.set_raw(raw)
    r.load_and_rescale(0, 0)
    r.set_cur_time(0)
    r.process()
    out, k0 = r.result(), r.fit()[0]
    r.close()
    assert np.abs(k0 - q.k0).max() * max(nx, ny) * 0.08 <= 1e-3
    assert np.linalg.norm(out - q.result) <= 1e-4 * np.linalg.norm(q.result)
