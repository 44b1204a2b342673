"""GPU: sums kept as float pairs at the end of the float range.  An infinite
sum stays infinite (an amplitude over it is then 0, not NaN), a sum past the
range whose mean is inside stays a number, and the bead's form factor takes
the sign of the diameter as it always did."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

import cudasirecon_gb300 as sr
from cudasirecon_gb300 import synthetic as syn

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "oracle"))

pytestmark = pytest.mark.gpu

# the amplitudes at time 0's k0 (a search's correlation peak overflows earlier)
AMPS = """
import sys, json; sys.path.insert(0, {root!r})
import numpy as np
import cudasirecon_gb300 as sr
from cudasirecon_gb300 import synthetic as syn
o = syn.Optics()
raw = syn.simulate({n}, {n}, 8, o, seed=3, n_filaments=10).raw.astype(np.float32)
flat = np.ascontiguousarray(np.repeat(raw[::5], 5, axis=0))  # no pattern: sum |X|^2 leaves the range, sum X* Y stays
r = sr.Reconstructor({n}, {n}, raw.shape[0], syn.config_text(o, extra={{"k0searchAll": 1}}),
                     syn.ra_otf(o, nx_psf=64, nz_psf=24))
r.set_ntimes(200)
out = []
for e in range(0, 112):
    r.set_raw(flat * np.float32(2.0 ** e) if e else raw)
    r.load_and_rescale(e, 0); r.set_cur_time(e); r.process()
    out.append([("nan" if np.isnan(v) else "zero" if v == 0 else "number") for v in np.ravel(r.fit()[1])])
print(json.dumps(out))
"""


def amps(n, env=None):
    r = subprocess.run([sys.executable, "-c", AMPS.format(root=ROOT, n=n)], env=dict(os.environ, **(env or {})),
                       capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stderr[-3000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


# 64 and 96 rows have both the two-factor overlap columns (pairs) and the
# staged ones, which add in double: the plan mask names the staged ones
@pytest.mark.parametrize("n", [64, 96])
def test_amplitudes_past_the_float_range(n):
    got = amps(n)
    want = amps(n, {"SIMRECON_FFT_REGISTER_SITES": "0"})
    flat = [k for row in want for k in row]
    assert "zero" in flat and "nan" in flat and "number" in flat  # the ladder crosses the range
    assert got == want


def test_makeotf_background_past_the_float_range():
    import makeotf_oracle as mo
    psf = syn.bead_psf_stack(64, 72, 8, syn.Optics(), nphases=5, peak_photons=5e4, seed=3, background=0.0)
    psf = (np.float32(3e37) + psf / psf.max() * np.float32(3e34)).astype(np.float32)  # a border's sum: about 1e41
    args = ["-angle", "0.2388", "-ls", "0.21", "-xyres", "0.08", "-zres", "0.125", "-na", "1.42", "-nimm", "1.515",
            "-wavelength", "528", "-nphases", "5", "-beaddiam", "0.1"]
    got = sr.make_otf(psf, args)
    want = mo.makeotf(psf, mo.MakeOTFOptions.from_args(args))
    d = got - want
    assert np.linalg.norm(d) <= 1e-5 * np.linalg.norm(want)
    assert np.abs(d).max() <= 1e-5 * np.abs(want).max()


@pytest.mark.parametrize("diam", [0.1, 1.5])
def test_bead_diameter_sign(diam):
    psf = syn.bead_psf_stack(64, 72, 8, syn.Optics(), nphases=5, peak_photons=5e4, seed=3)
    args = ["-angle", "0.2388", "-ls", "0.21", "-xyres", "0.08", "-zres", "0.125", "-na", "1.42", "-nimm", "1.515",
            "-wavelength", "528", "-nphases", "5", "-beaddiam"]
    assert np.array_equal(sr.make_otf(psf, args + [str(diam)]), sr.make_otf(psf, args + [str(-diam)]))
