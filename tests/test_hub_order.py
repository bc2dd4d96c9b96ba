"""Set-up of a mixed batch for a network with a hub: memory in proportion to its
incidences."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "mumfim_gb300", "csrc")


def test_hub_is_ordered_in_little_memory(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    from mumfim_gb300.build import _cuda_home
    try:
        cuda = _cuda_home()
    except RuntimeError:
        pytest.skip("CUDA headers not found")
    exe = str(tmp_path / "hub_order_check")
    subprocess.run([gxx, "-O1", "-std=c++17", "-I" + CSRC, "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(cuda, "include"),
                    os.path.join(HERE, "native", "hub_order_check.cpp"),
                    os.path.join(CSRC, "mfg_mixed_order.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "bad=0" in r.stdout
