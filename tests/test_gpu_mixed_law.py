"""The mixed solve's fiber law (mfg_mixed_law.cuh) gives the bits of its
definition by IEEE square roots and divisions: a small CUDA program built
from the same header compares them over every branch."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.mark.gpu
def test_law_matches_ieee_operations(tmp_path):
    from mumfim_gb300.build import ARCH, _cuda_home
    cuda = _cuda_home()
    exe = str(tmp_path / "law_check")
    subprocess.run([os.path.join(cuda, "bin", "nvcc"), *ARCH, "-O3", "-std=c++17",
                    "-I" + os.path.join(ROOT, "mumfim_gb300", "csrc"),
                    "-I" + os.path.join(ROOT, "include"),
                    os.path.join(HERE, "native", "law_check.cu"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "bad=0" in r.stdout
