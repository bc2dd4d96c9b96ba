"""exact_reciprocal() (mfg_exact.cuh), which FP64 batches form on the device at
set-up, against a 128-bit division: on the host and on the device."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "mumfim_gb300", "csrc")
SOURCE = os.path.join(HERE, "native", "reciprocal_check.cpp")


def _check(exe):
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "bad=0" in r.stdout


def test_reciprocals_on_the_host(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    exe = str(tmp_path / "reciprocal_check")
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I" + CSRC, SOURCE, "-o", exe],
                   check=True)
    _check(exe)


@pytest.mark.gpu
def test_reciprocals_on_the_device(tmp_path):
    from mumfim_gb300.build import ARCH, _cuda_home
    exe = str(tmp_path / "reciprocal_check")
    subprocess.run([os.path.join(_cuda_home(), "bin", "nvcc"), *ARCH, "-x", "cu", "-O3",
                    "-std=c++17", "--fmad=false", "-I" + CSRC, SOURCE, "-o", exe], check=True)
    _check(exe)
