"""CPU: SRX_fftPath names the path that a call site runs a length by, over all
four kinds, with and without a plan file.  Subprocesses without a visible GPU
(the model name then reads "unknown")."""
import json
import os
import subprocess
import sys

import cudasirecon_gb300 as sr

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

QUERY = """
import sys, json; sys.path.insert(0, {root!r})
import cudasirecon_gb300 as sr
print(json.dumps([[s, n, *sr.fft_path(s, n)] for s in sr.FFT_SITES for n in {lengths!r}]))
"""
LENGTHS = (5, 30, 32, 60, 64, 75, 80, 98, 128, 130, 150, 192, 256, 384, 490, 512, 640, 1000, 1024, 1280, 2048)


def query(tmp_path, plan="", env=None):
    cache = tmp_path / "plans.tsv"
    cache.write_text(plan)
    env = dict(os.environ, SIMRECON_FFT_PLAN_CACHE=str(cache), CUDA_VISIBLE_DEVICES="", **(env or {}))
    r = subprocess.run([sys.executable, "-c", QUERY.format(root=ROOT, lengths=LENGTHS)], env=env, capture_output=True,
                       text=True, timeout=120)
    assert r.returncode == 0, r.stderr
    return {(s, n): (p, src) for s, n, p, src in json.loads(r.stdout)}


def test_built_in_paths(tmp_path):
    q = query(tmp_path)
    assert {v[1] for k, v in q.items() if k[1] not in (32, 64, 128, 256, 512, 1024)} <= {"built-in", "stockham-only"}
    path = {k: v[0] for k, v in q.items()}
    for s in ("ingest_x", "ingest_y", "overlap_x", "overlap_y", "crosscorr_rows", "crosscorr_cols", "makeotf"):
        assert path[s, 640] == path[s, 384] == path[s, 128] == path[s, 64] == "two-factor"
        assert path[s, 490] == path[s, 98] == path[s, 1000] == path[s, 2048] == "stockham"  # no pair
        assert path[s, 32] == "register"
        assert path[s, 150] == "two-factor"  # 15 x 10
    assert path["ingest_x", 75] == "stockham" and path["ingest_y", 192] == "two-factor"
    # compiled for the length, or two-factor whatever a plan says
    for n in (256, 512, 1024):
        assert path["ingest_x", n] == path["assemble_y", n] == path["assemble_x", n] == "compiled"
        assert path["overlap_x", n] == path["crosscorr_rows", n] == "two-factor"
    assert [path["ingest_y", n] for n in (256, 512, 1024)] == ["two-factor", "two-factor", "compiled"]
    assert [path["overlap_y", n] for n in (256, 512, 1024)] == ["two-factor", "compiled", "two-factor"]
    # the doubled grid of 64, 75 (odd), 192, 320 and 640
    assert [path["assemble_x", n] for n in (128, 150, 384, 640, 1280)] == \
        ["two-factor", "stockham", "two-factor", "two-factor", "two-factor"]
    assert path["assemble_y", 64] == "register"  # images of 32 have no pair
    for s in ("separate_z", "assemble_z"):
        assert path[s, 5] == path[s, 30] == path[s, 60] == path[s, 80] == path[s, 128] == path[s, 64] == "compiled"
        assert path[s, 98] == path[s, 150] == "stockham"


def test_a_plan_decides_only_where_it_is_followed(tmp_path):
    sites = [s for s in sr.FFT_SITES]
    plan = "".join(f"unknown\t{s}\t{n}\tstockham\t1\t2\n" for s in sites for n in LENGTHS)
    base, q = query(tmp_path), query(tmp_path, plan)
    for k, (path, src) in q.items():
        if src == "tuned":
            assert path == "stockham" and k[1] in (32, 64, 128, 256, 512, 1024), k
        else:  # a plan has no say: the same path as without
            assert (path, src) == base[k], k
    tuned = {k for k, v in q.items() if v[1] == "tuned"}
    assert {("overlap_x", 128), ("overlap_y", 1024), ("crosscorr_rows", 512), ("assemble_x", 128),
            ("assemble_y", 128), ("ingest_x", 64), ("makeotf", 256)} <= tuned
    assert not tuned & {("overlap_x", 256), ("overlap_x", 1024), ("overlap_y", 256), ("overlap_y", 512),
                        ("ingest_x", 512), ("ingest_y", 256), ("ingest_y", 1024), ("assemble_x", 1024),
                        ("assemble_z", 32)}
    two = query(tmp_path, plan.replace("stockham", "two-factor"))
    assert two["crosscorr_rows", 512] == ("two-factor", "tuned")
    env = query(tmp_path, env={"SIMRECON_FFT_REGISTER_SITES": "fff"})
    assert env["overlap_x", 128] == ("register", "environment") and env["overlap_x", 640] == ("two-factor", "built-in")


def test_recorded_two_factor_is_not_reported_as_stockham(tmp_path):
    cache = tmp_path / "plans.tsv"
    cache.write_text("unknown\tcrosscorr_rows\t256\ttwo-factor\t1\t2\n")
    code = ("import sys, ctypes as C; sys.path.insert(0, %r)\nimport cudasirecon_gb300 as sr\n"
            "b = C.create_string_buffer(32)\n"
            "print(sr.load_library().SRX_fftPlanChoice(5, 256, b, 32), b.value.decode(), sr.fft_plan_choice('crosscorr_rows', 256))"
            % ROOT)
    env = dict(os.environ, SIMRECON_FFT_PLAN_CACHE=str(cache), CUDA_VISIBLE_DEVICES="")
    r = subprocess.run([sys.executable, "-c", code], env=env, capture_output=True, text=True, timeout=120)
    assert r.stdout.strip() == "2 tuned (False, 'tuned')", r.stdout + r.stderr
