"""GPU: the z transforms of every kind of length, batches of more directions
than one launch takes, stacks uploaded in parts, and makeotf's half-spectrum
transforms, each at the sizes where a kernel changes or leaves lanes empty.
Bars: the volume's parity tolerance (rel-L2 <= 1e-4), makeotf's (rel-L2 and
max-abs of the peak <= 1e-5), and equal bits where only the order of the
launches differs."""
import os
import sys
import warnings

import numpy as np
import pytest

import cudasirecon_gb300 as sr
from cudasirecon_gb300 import synthetic as syn
from oracle.sirecon_oracle import SIMReconOracle

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "oracle"))

pytestmark = pytest.mark.gpu

ANGLES = (-0.8043, -1.8555, 0.2388, 0.75, -1.3)


def setup(nx, ny, nz, ndirs, extra=None):
    o = syn.Optics(angles=ANGLES[:ndirs])
    raw = syn.simulate(nx, ny, nz, o, seed=11 + nz + ndirs, n_filaments=20, ndirs=ndirs).raw
    cfg = syn.config_text(o, extra={"ndirs": ndirs, **(extra or {})})
    return raw, cfg, syn.ra_otf(o, nx_psf=64, nz_psf=24)


def product(raw, cfg, otf, whole=False):
    r = sr.Reconstructor(raw.shape[2], raw.shape[1], raw.shape[0], cfg, otf)
    if whole:  # a profiled upload goes up in one piece
        r.set_profiling(True)
    r.set_raw(raw)
    r.load_and_rescale(0, 0)
    r.set_cur_time(0)
    r.process()
    out = r.result().copy()
    r.close()
    return out


def close(out, want):
    if not np.isfinite(want).any():  # an overlap without a kz plane: 0 / 0 in both
        return not np.isfinite(out).any()
    return np.linalg.norm(out - want) / np.linalg.norm(want) <= 1e-4


def matches_oracle(raw, cfg, otf):
    q = SIMReconOracle(raw.shape[2], raw.shape[1], raw.shape[0], cfg, otf)
    q.set_raw(raw)
    q.load_and_rescale(0)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore")
        q.process()
    return close(product(raw, cfg, otf), q.result)


# in registers (2 to 32), as two factors (35 to 64), and beyond the list (33, 70);
# 72 x 64 planes leave the column tiles partly empty
@pytest.mark.parametrize("nz", [2, 7, 15, 32, 35, 49, 64, 70])
def test_z_length_matches_oracle(nz):
    assert matches_oracle(*setup(72, 64, nz, 1))


# 4 = 3 + 1 and 5 = 3 + 2 directions per launch
@pytest.mark.parametrize("ndirs", [2, 4, 5])
def test_direction_count_matches_oracle(ndirs):
    assert matches_oracle(*setup(72, 64, 6, ndirs))


# sections of 0.5 or 1 MB, parts of 8 or 4: the last part of a direction is longer
@pytest.mark.parametrize("nz,ndirs,dtype,extra", [(9, 3, np.uint16, {}), (9, 1, np.float32, {}),
                                                  (6, 3, np.uint16, {"fastSI": 1})])
def test_upload_in_parts_gives_the_same_bits(nz, ndirs, dtype, extra):
    raw, cfg, otf = setup(512, 512, nz, ndirs, extra)
    raw = np.ascontiguousarray(raw.astype(dtype))
    assert np.array_equal(product(raw, cfg, otf), product(raw, cfg, otf, whole=True))


# pairs and a z length of the list; 70 and 98 have no pair; one plane; more
# planes than the list; rows that do not fill the last group
@pytest.mark.parametrize("nx,ny,nz,nph", [(64, 72, 35, 5), (70, 96, 8, 5), (96, 98, 8, 5), (64, 72, 70, 5),
                                          (80, 128, 1, 3), (64, 256, 4, 5)])
def test_makeotf_lengths_match_oracle(nx, ny, nz, nph):
    import makeotf_oracle as mo
    psf = syn.bead_psf_stack(nx, ny, nz, syn.Optics(nphases=nph), nphases=nph, peak_photons=5e4, seed=nx + nz)
    args = ["-angle", "0.2388", "-ls", "0.21", "-xyres", "0.08", "-zres", "0.125", "-na", "1.42", "-nimm", "1.515",
            "-wavelength", "528", "-nphases", str(nph), "-beaddiam", "0.25"]
    got = sr.make_otf(psf, args)
    want = mo.makeotf(psf, mo.MakeOTFOptions.from_args(args))
    d = got - want
    assert np.linalg.norm(d) <= 1e-5 * np.linalg.norm(want)
    assert np.abs(d).max() <= 1e-5 * np.abs(want).max()
