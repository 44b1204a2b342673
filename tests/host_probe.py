"""Compiles a small C++ program over the product's headers with the host
compiler and returns what it prints: the parts of the kernels' arithmetic that
are plain host code as well."""
import os
import shutil
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def cuda_include():
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    return os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(nvcc))), "include")


def run(code, tmp_path):
    src, exe = tmp_path / "probe.cpp", tmp_path / "probe"
    src.write_text(code)
    cmd = ["g++", "-std=c++20", "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "cudasirecon_gb300", "csrc"),
           "-I", os.path.join(ROOT, "include"), "-I", cuda_include(), str(src), "-o", str(exe)]
    r = subprocess.run(cmd, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]
    return r.stdout
