"""GPU: a recorded FFT plan governs the assembly and makeotf where their kernels
for doubled and two-factor lengths do not need it: SRX_tuneFFT measures the
doubled rows and columns of a 64-pixel image with all three paths, a plan that
names one of the other two is followed (the filter then runs as its own pass),
and results agree to float precision either way."""
import json
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SETUP = """
import sys, json; sys.path.insert(0, {root!r})
import numpy as np
import cudasirecon_gb300 as sr
from cudasirecon_gb300 import synthetic as syn
o = syn.Optics()
raw = syn.simulate(64, 64, 12, o, seed=3, n_filaments=10).raw
r = sr.Reconstructor(64, 64, raw.shape[0], syn.config_text(o), syn.ra_otf(o, nx_psf=64, nz_psf=24))
r.set_raw(raw)
"""
TUNE = SETUP + """
print(json.dumps(r.tune_fft(1)))
"""
RUN = SETUP + """
r.set_profiling(True)
r.reset_profile()
r.load_and_rescale(0, 0); r.set_cur_time(0); r.process()
p = r.profile()
np.save({out!r}, r.result())
psf = syn.bead_psf_stack(64, 64, 32, o, nphases=5, peak_photons=5e4, seed=3)
args = ["-angle", "0.2388", "-ls", "0.21", "-xyres", "0.08", "-zres", "0.125", "-na", "1.42", "-nimm", "1.515",
        "-wavelength", "528", "-nphases", "5", "-beaddiam", "0.1"]
np.save({otf!r}, sr.make_otf(psf, args))
print(json.dumps(sorted(p["kernels"])))
"""


def py(code, cache):
    env = dict(os.environ, SIMRECON_FFT_PLAN_CACHE=str(cache))
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, r.stderr[-3000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


def test_assembly_follows_a_recorded_plan(tmp_path):
    def run(tag, cache):
        out, otf = tmp_path / f"{tag}.npy", tmp_path / f"{tag}_otf.npy"
        kernels = py(RUN.format(root=ROOT, out=str(out), otf=str(otf)), cache)
        return np.load(out), np.load(otf), kernels

    base, base_otf, kernels = run("base", tmp_path / "none.tsv")
    assert "k_asm_y_filter" in kernels and "k_filter" not in kernels
    cache = tmp_path / "fft.tsv"
    report = {(e["site"], e["n"]): e for e in py(TUNE.format(root=ROOT), cache)["sites"]}
    for site in ("assemble_x", "assemble_y"):
        e = report[(site, 128)]
        assert min(e["register_ms"], e["stockham_ms"], e["two_factor_ms"]) > 0
        assert max(e["register_ms"], e["stockham_ms"], e["two_factor_ms"]) < 1e3
    gpu = cache.read_text().split("\t")[0]
    for x, y in (("stockham", "register"), ("register", "stockham"), ("two-factor", "stockham"),
                 ("stockham", "two-factor")):
        plan = tmp_path / f"{x}_{y}.tsv"
        plan.write_text(f"{gpu}\tassemble_x\t128\t{x}\t1\t2\n{gpu}\tassemble_y\t128\t{y}\t1\t2\n"
                        f"{gpu}\tmakeotf\t32\t{x}\t1\t2\n")
        got, otf, kernels = run(f"{x}_{y}", plan)
        assert ("k_filter" in kernels) == (y != "two-factor"), (x, y, kernels)
        assert np.linalg.norm(got - base) < 2e-6 * np.linalg.norm(base)
        assert np.linalg.norm(otf - base_otf) < 2e-6 * np.linalg.norm(base_otf)
