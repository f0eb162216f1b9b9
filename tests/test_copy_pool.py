"""The host copy threads behind pageable transfers (cpsz_b200/csrc/copy_pool.h)
on the CPU: tests/copy_pool_check.cpp runs jobs of several threads beside one
another, also beside one whose owner waits (for the device, in the library)
between its pieces."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_jobs_run_beside_one_another(tmp_path):
    exe = str(tmp_path / "cpc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", os.path.join(ROOT, "cpsz_b200", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "copy_pool_check.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "ALL OK" in r.stdout, r.stdout + r.stderr
