"""The scratch ring of the assembly by element matrices (micropp_gb300/csrc/assembly_ring.h): its chunks cover the layers, and
its size stays within the memory that is left.  Built with the host compiler; no GPU."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_ring_covers_the_layers_within_its_memory(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    exe = tmp_path / "ring_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-I", os.path.join(ROOT, "micropp_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "native", "ring_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
