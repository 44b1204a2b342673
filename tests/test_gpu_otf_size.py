"""GPU: the fused filter against the filter as its own pass with OTF tables of
larger PSFs: 129 and 257 radial bins, and the last size the fused kernels take
and the first they leave, in the kernels of doubled and of compiled column
lengths.  Tolerance: the one of the same comparison at 65 bins."""
from functools import lru_cache

import numpy as np
import pytest

import cudasirecon_gb300 as sr
from cudasirecon_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


@lru_cache(maxsize=None)
def pages(nxotf):
    return syn.ra_otf(syn.Optics(), nx_psf=2 * (nxotf - 1), nz_psf=12)


def volume(nx, ny, nz, otf, fused):
    o = syn.Optics()
    raw = syn.simulate(nx, ny, nz, o, seed=nx + ny, n_filaments=10).raw
    r = sr.Reconstructor(nx, ny, raw.shape[0], syn.config_text(o), otf)
    r.set_filter_fusion(fused)
    r.set_raw(raw)
    r.load_and_rescale(0, 0)
    r.set_cur_time(0)
    r.process()
    out = r.result().copy()
    r.close()
    return out


# 682 bins of three orders fill the 32 KB of tables, 683 do not fit
@pytest.mark.parametrize("nxotf", [129, 257, 682, 683])
@pytest.mark.parametrize("nx,ny", [(96, 512), (128, 80), (96, 1024)])
def test_fused_filter_with_large_otfs(nx, ny, nxotf):
    otf = pages(nxotf)
    assert otf.shape[1] == nxotf
    a, b = volume(nx, ny, 6, otf, True), volume(nx, ny, 6, otf, False)
    assert np.isfinite(a).all()
    assert np.linalg.norm(a - b) < 2e-6 * np.linalg.norm(b)
