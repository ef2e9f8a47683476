"""What the per-kernel fluxes set for a device is set for each device of the process (CPU, with a
stand-in for the CUDA runtime: tests/cpp/two_devices.cpp)."""
import os
import shutil
import subprocess

import pytest

from apophis_gb300 import _build

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_flux_launches_on_a_second_device(tmp_path):
    lib = _build.build()
    libdir, exe = os.path.dirname(lib), str(tmp_path / "two_devices")
    subprocess.check_call(["g++", "-std=c++17", "-O1", "-rdynamic", os.path.join(ROOT, "tests", "cpp", "two_devices.cpp"),
                           "-I", os.path.join(ROOT, "include"), "-I", os.path.join(CUDA, "include"),
                           "-L", libdir, "-laph_hydro", "-Wl,-rpath," + libdir,
                           "-Wl,-rpath-link," + os.path.join(CUDA, "lib64"),
                           "-Wl,-rpath," + os.path.join(CUDA, "lib64"), "-o", exe])
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
