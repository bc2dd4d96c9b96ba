"""The FP64 kernel's quotients and square roots (mfg_exact.cuh): correctly
rounded next to rounding boundaries (host build of the same functions), and
the general operations where they do not apply (GPU, against the oracle)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "mumfim_gb300", "csrc")


def test_quotients_and_roots_are_correctly_rounded(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    exe = str(tmp_path / "exact_check")
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I" + CSRC,
                    os.path.join(HERE, "native", "exact_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "bad=0" in r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("radius,E,damping", [
    (1e-3, 1.0, 0.5),    # the fast forms
    (1e-20, 1e30, 0.5),  # masses below 2^-100: general quotients at the nodes
    (1e-130, 1.0, 0.5),  # forces below 2^-800: general quotients on the fibers too
    (1e-157, 1.0, 0.5),  # forces below the smallest normal number
    (1e-3, 1.0, 0.0),    # no damping: zero forces at rest
])
def test_general_operations_match_oracle(lib_path, oracle, radius, E, damping):
    import mumfim_gb300 as m
    from mumfim_gb300 import synthetic as S
    from mumfim_gb300.network_io import Reaction
    coords, conn = S.knn_network(333, 4, S.geometry_seed(21, 0))
    net = m.FiberNetwork(coords, conn, [Reaction(0, radius, E, 1.0)])
    strat = [m.SolutionStrategy.ramp(205, damping)]
    F = np.array([[[1.03, 0.01, 0.0], [0.0, 0.98, 0.02], [0.01, 0.0, 1.01]]])
    g = m.BatchedFiberRVEAnalysisExplicit([net], strat)
    s = np.zeros((1, 6))
    g.run(F, s)
    o = oracle.OracleBatch([net], strat)
    _, so, _ = o.run(F)
    np.testing.assert_array_equal(s, so)
    np.testing.assert_array_equal(g.displacements(0), o.displacements(0))
    assert np.abs(g.displacements(0)).max() > 0
