"""Host-side parts of the engine's headers, compiled and run without a GPU."""

import os
import subprocess

from conftest import ROOT


def test_host_units(tmp_path):
    src = os.path.join(ROOT, "tests", "cpp", "host_units.cpp")
    exe = str(tmp_path / "host_units")
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    r = subprocess.run(["g++", "-O1", "-std=c++17", "-I", cuda, src,
                        os.path.join(ROOT, "gpu_bitruss_gb300", "csrc", "bt_plan.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
