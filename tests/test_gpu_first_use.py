"""GPU: the first volume of a new process, whose lengths have no plan on the
device yet, against the same volume again: uploads through the default stream
(twiddles, OTF, tables) are waited for before the handle's stream reads them,
also when the first use lies inside a captured series."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CODE = """
import sys; sys.path.insert(0, {root!r})
import numpy as np
import cudasirecon_gb300 as sr
from cudasirecon_gb300 import synthetic as syn
o = syn.Optics()
nx, ny, nz = {shape}
raw = syn.simulate(nx, ny, nz, o, seed=3, n_filaments=10).raw
def handle():
    r = sr.Reconstructor(nx, ny, raw.shape[0], syn.config_text(o), syn.ra_otf(o, nx_psf=128, nz_psf=24))
    if {series}:
        r.set_ntimes(2)
        r.recon_params().bSearchforvector = 0
    return r
def volume(r):
    if {series}:
        out = np.zeros(r.out_shape, np.float32)
        r.process_series([raw, raw], [out, out.copy()])
        return out
    r.set_raw(raw); r.load_and_rescale(0, 0); r.set_cur_time(0); r.process()
    return r.result().copy()
a = handle()
first = volume(a)
again = volume(a)
b = volume(handle())
assert np.isfinite(first).all()
assert np.array_equal(first, again) and np.array_equal(first, b)
"""


@pytest.mark.parametrize("series", [0, 1])
@pytest.mark.parametrize("shape", [(640, 384, 6), (512, 512, 16), (98, 70, 9), (1000, 64, 5)])
def test_first_volume_of_a_process(shape, series):
    r = subprocess.run([sys.executable, "-c", CODE.format(root=ROOT, shape=shape, series=series)], capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-3000:]
