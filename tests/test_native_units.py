"""Host-callable pieces of the CUDA sources, as C++ programs without a GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("unit", ["surface_rows", "per_device"])
def test_unit(tmp_path, unit):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = tmp_path / unit
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", "-pthread", "-I",
                    os.path.join(ROOT, "fwi_cuda_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "c_abi", unit + ".cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.startswith("ok "), out.stdout + out.stderr
