"""GPU: reconstructions whose lengths take the two-factor transforms
(csrc/tf_fft.cuh) against the FP64 oracle: the smallest and largest factors,
widths that leave a column tile or a row group partly empty, a length without
a factor pair next to one with, one direction, and the filter switches that
are read from the arguments.  Bar: the parity tolerance of the volume
(rel-L2 <= 1e-4) with k0 within 1e-3 pixel."""
import warnings

import numpy as np
import pytest

import cudasirecon_gb300 as sr
from cudasirecon_gb300 import synthetic as syn
from oracle.sirecon_oracle import SIMReconOracle

pytestmark = pytest.mark.gpu


def close(out, want):
    """rel-L2 within the parity bar; where the oracle has no finite value (an
    overlap without a kz plane gives 0 / 0) neither has the product."""
    if not np.isfinite(want).any():
        return not np.isfinite(out).any()
    return np.linalg.norm(out - want) / np.linalg.norm(want) <= 1e-4


def close_k0(k0, want, n):
    if not np.isfinite(want).any():
        return True
    return np.abs(k0 - want).max() * n * 0.08 <= 1e-3


def both(nx, ny, nz, extra=None, ndirs=3):
    o = syn.Optics(nphases=5 if nz > 1 else 3)
    raw = syn.simulate(nx, ny, nz, o, seed=5 + nx + ny, n_filaments=20, ndirs=ndirs).raw
    kv = {"ndirs": ndirs, "k0angles": ",".join("%.6f" % a for a in o.angles[:ndirs])}
    if nz == 1:
        kv["wiener"] = 0.00048828125
    kv.update(extra or {})
    cfg = syn.config_text(o, twod=nz == 1, extra=kv)
    otf = syn.ra_otf(o, nx_psf=64, nz_psf=24) if nz > 1 else syn.ra_otf(o, nx_psf=128, norders=2, twod=True)
    r = sr.Reconstructor(nx, ny, raw.shape[0], cfg, otf)
    r.set_raw(raw)
    r.load_and_rescale(0, 0)
    r.set_cur_time(0)
    r.process()
    out, (k0, _) = r.result().copy(), r.fit()
    r.close()
    q = SIMReconOracle(nx, ny, raw.shape[0], cfg, otf)
    q.set_raw(raw)
    q.load_and_rescale(0)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        q.process()
    return out, q.result, k0, q.k0


# 64 = 8 x 8, 72 = 9 x 8, 90 = 10 x 9, 98 and 70 have no pair, 162 = 18 x 9, 196 = 14 x 14,
# 210 = 15 x 14, 252 = 18 x 14, 294 = 21 x 14, 150 has none
@pytest.mark.parametrize("nx,ny,nz", [(64, 72, 8), (90, 98, 9), (70, 162, 6), (196, 64, 5), (210, 90, 6),
                                      (64, 252, 4), (294, 80, 6), (150, 100, 10)])
def test_volume_matches_oracle(nx, ny, nz):
    out, want, k0, wk0 = both(nx, ny, nz)
    assert close(out, want)
    assert close_k0(k0, wk0, max(nx, ny))


# 1024 = 32 x 32, 768 = 32 x 24, 896 = 32 x 28, 400 = 20 x 20, 640 = 32 x 20, 486 = 27 x 18
@pytest.mark.parametrize("nx,ny", [(1024, 128), (128, 1024), (768, 486), (400, 896), (640, 300)])
def test_frame_matches_oracle(nx, ny):
    out, want, k0, wk0 = both(nx, ny, 1)
    assert close(out, want)
    assert close_k0(k0, wk0, max(nx, ny))


@pytest.mark.parametrize("extra,ndirs", [({"nosuppress": 0}, 3), ({"dampenOrder0": 0}, 3), ({}, 1),
                                         ({"nofilterovlps": 0}, 1), ({"dampenOrder0": 0, "equalizez": 1}, 1)])
def test_filter_switches_match_oracle(extra, ndirs):
    out, want, _, _ = both(96, 80, 8, extra, ndirs)
    assert close(out, want)
