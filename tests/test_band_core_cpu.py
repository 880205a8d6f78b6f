"""The banded core of the filter and of the alignment's score bound (storm_b200/csrc/band_core.cuh),
compiled for the host, on random cases: against the oracle's filter, against the same recurrence on
plain integers, and never below the oracle's alignment score where it claims to be a bound."""
import os
import shutil
import subprocess

import pytest

import ffi

NVCC = "/usr/local/cuda/bin/nvcc" if os.path.exists("/usr/local/cuda/bin/nvcc") else shutil.which("nvcc")


@pytest.mark.skipif(NVCC is None, reason="nvcc not available")
def test_band_core_matches_oracle(tmp_path):
    ffi.ensure_built()
    exe = str(tmp_path / "bch")
    src = os.path.join(os.path.dirname(__file__), "band_core_host.cu")
    subprocess.run([NVCC, "-std=c++17", "-O2", "-Wno-deprecated-gpu-targets", src, "-o", exe,
                    "-L" + ffi.ORACLE_DIR, "-loracle", "-Xlinker", "-rpath=" + ffi.ORACLE_DIR], check=True)
    p = subprocess.run([exe, "30000"], capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stdout + p.stderr
    assert "checked filter" in p.stdout
