"""GPU: makeotf on one plane with -ifixkr.  The replaced element of a bin is then
the mean of the bin and the next one (of the last bin: of the next band's
first), taken before either changes, whatever the number of bins and bands; the
expected values come from the same call without the switch."""
import numpy as np
import pytest

import cudasirecon_gb300 as sr
from cudasirecon_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


# 19 bins (one warp), 81 and 181 (several warps); one, three and five bands
@pytest.mark.parametrize("n", [36, 160, 360])
@pytest.mark.parametrize("nph", [1, 3, 5])
@pytest.mark.parametrize("kr", [1, 5])
def test_ifixkr_on_one_plane(n, nph, kr):
    psf = syn.bead_psf_stack(n, n, 1, syn.Optics(nphases=nph), nphases=nph, peak_photons=5e4, seed=3)
    args = ["-angle", "0.2388", "-ls", "0.21", "-xyres", "0.08", "-na", "1.42", "-nimm", "1.515", "-wavelength", "528",
            "-nphases", str(nph), "-beaddiam", "0.1", "-nocompen", "-5bands", "-bessel", "-ifixkz", "0"]
    flat = sr.make_otf(psf, args)
    base = flat.reshape(nph, n // 2 + 1, 2).astype(np.float64)
    want = base.copy()
    for b in range(nph):
        nxt = np.concatenate([base[b, 1:], base[b + 1, :1] if b + 1 < nph else np.zeros((1, 2))])
        want[b, kr:] = (base[b, kr:] + nxt[kr:]) / 2
    for _ in range(3):
        got = sr.make_otf(psf, args + ["-ifixkr", str(kr)]).reshape(want.shape)
        assert np.abs(got - want).max() <= 1e-6 * np.abs(want).max()
