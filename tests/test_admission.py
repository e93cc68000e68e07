"""The order in which the server gives device memory to its jobs
(csrc/admission.h), checked on host threads by a small C++ program: while a job
waits for room no later one takes any, so a large job is not starved by a
stream of small ones.  The reference runs one job per process."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "gene-sequences-de-redundancy_gb300", "csrc")


def test_admission_order(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    exe = tmp_path / "admission_check"
    subprocess.run([gxx, "-O2", "-std=c++17", "-Wall", "-pthread", "-I", CSRC,
                    os.path.join(HERE, "admission_check.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "faults 0" in r.stdout
