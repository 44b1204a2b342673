"""GPU: a climb that leaves the device search's line cache.  The volume has then
been filtered and assembled with what the device left, and is fitted by the host
search and assembled again: the same bits as with the host search from the
start.  The frame is one whose coarse pattern (0.4 pixel) lets the angle climb
run past 1024 steps; the searches counted show that the second one ran."""
import numpy as np
import pytest

import cudasirecon_gb300 as sr
from cudasirecon_gb300 import synthetic as syn

pytestmark = pytest.mark.gpu


def run(device, calls=1):
    o = syn.Optics(nphases=3, ls=12.0)
    raw = syn.simulate(64, 64, 1, o, seed=4, n_filaments=10).raw
    otf = syn.ra_otf(syn.Optics(nphases=3), nx_psf=64, nz_psf=24, norders=2, twod=True)
    r = sr.Reconstructor(64, 64, raw.shape[0], syn.config_text(o, twod=True, extra={"wiener": 0.00048828125}), otf)
    r.set_device_search(device)
    res = []
    for _ in range(calls):
        c0 = r.fit_counts()
        r.set_raw(raw)
        r.load_and_rescale(0, 0)
        r.set_cur_time(0)
        r.process()
        res.append((r.result().copy(), *(np.array(v) for v in r.fit()), r.fit_counts()["k0_searches"] - c0["k0_searches"]))
    r.close()
    return res


def test_redo_gives_the_host_searchs_volume():
    (host,) = run(False)
    first, second = run(True, calls=2)
    assert host[3] == 3 and first[3] == second[3] == 6
    assert np.isfinite(host[0]).all()
    for got in (first, second):
        assert np.array_equal(got[0], host[0])
        assert np.array_equal(got[1], host[1]) and np.array_equal(got[2], host[2])
