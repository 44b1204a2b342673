"""GPU: volumes whose kz range leaves the OTF (a PSF step above one over the
axial cutoff: the lookups' wrapped kz index is negative and clamps to the
table's first entry) against the FP64 oracle, with row lengths that have a
compiled overlap kernel.  Bar: the volume's parity tolerance (rel-L2 <= 1e-4)
and k0 within 1e-3 pixel."""
import warnings

import numpy as np
import pytest

import cudasirecon_gb300 as sr
from cudasirecon_gb300 import synthetic as syn
from oracle.sirecon_oracle import SIMReconOracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz,dz_psf", [(96, 80, 9, 0.8), (64, 72, 8, 0.8), (256, 64, 7, 1.0), (96, 80, 12, 1.0)])
def test_kz_beyond_the_otf_matches_oracle(nx, ny, nz, dz_psf):
    o = syn.Optics()
    raw = syn.simulate(nx, ny, nz, o, seed=5, n_filaments=20).raw
    cfg = syn.config_text(o, dz_psf=dz_psf)
    otf = syn.ra_otf(o, nx_psf=64, nz_psf=24)
    q = SIMReconOracle(nx, ny, raw.shape[0], cfg, otf)
    q.set_raw(raw)
    q.load_and_rescale(0)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        q.process()
    assert np.isfinite(q.result).all()
    r = sr.Reconstructor(nx, ny, raw.shape[0], cfg, otf)
    r.set_raw(raw)
    r.load_and_rescale(0, 0)
    r.set_cur_time(0)
    r.process()
    out, k0 = r.result(), r.fit()[0]
    r.close()
    assert np.abs(k0 - q.k0).max() * max(nx, ny) * 0.08 <= 1e-3
    assert np.linalg.norm(out - q.result) <= 1e-4 * np.linalg.norm(q.result)
