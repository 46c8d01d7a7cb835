"""The library's host code overwrites no object that has constructors byte by byte
(g++'s -Wclass-memaccess, on the file that holds tables and batches; no GPU)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_no_bytes_written_over_objects(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    csrc = os.path.join(ROOT, "beampower_b200", "csrc")
    host = ["-ccbin", "/usr/bin/g++"] if os.path.exists("/usr/bin/g++") else []
    r = subprocess.run([nvcc, *host, "-O0", "-std=c++17", "--expt-relaxed-constexpr",
                        "-gencode", "arch=compute_100a,code=sm_100a",
                        "-Xcompiler", "-Werror=class-memaccess",
                        "-I", os.path.join(ROOT, "include"), "-I", csrc, "-c",
                        "-o", str(tmp_path / "bp_capi.o"), os.path.join(csrc, "bp_capi.cu")],
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]
