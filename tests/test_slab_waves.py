"""The plan of a batch's slab sweeps over the SMs it may use, checked on the host (tests/slab_waves_check.cpp)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_launch_passes_its_share(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    lib = os.path.join(ROOT, "pscbfm_b200")
    exe = str(tmp_path / "slab_waves_check")
    r = subprocess.run([nvcc, "-std=c++17", "-O2", "-x", "cu", "-gencode", "arch=compute_100a,code=sm_100a",
                        "-I", os.path.join(lib, "csrc"), "-I", os.path.join(ROOT, "include"),
                        os.path.join(ROOT, "tests", "slab_waves_check.cpp"), "-o", exe,
                        "-L", lib, "-l:libbfm.so", "-Xlinker", "-rpath=" + lib], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-3000:]
    run = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and run.stdout.strip() == "ok", run.stdout + run.stderr
