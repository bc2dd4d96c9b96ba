"""The end of the nonlinear law's toe (toe_limit in mfg_toe.cuh) over the whole
range of transition ratios that a batch accepts: the limit itself (CPU), and
ratios so large that no fiber leaves the toe, which give the results of any
other ratio that no fiber reaches (GPU)."""
import os
import shutil
import subprocess
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "mumfim_gb300", "csrc")


def test_limit_is_the_largest_square(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    exe = str(tmp_path / "toe_check")
    subprocess.run([gxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I" + CSRC,
                    os.path.join(HERE, "native", "toe_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "bad=0" in r.stdout


def _solve(sizes, ratio, **options):
    import mumfim_gb300 as m
    from mumfim_gb300 import synthetic as S
    from mumfim_gb300.network_io import Reaction
    nets = [m.FiberNetwork(*S.knn_network(n, 4, S.geometry_seed(53, i)),
                           [Reaction(1, 1e-3, 1.0, 1.0, 4.0, ratio)])
            for i, n in enumerate(sizes)]
    F = np.stack([np.eye(3) + (S.uniform(S.param_seed(53, i), 9) * 0.2 - 0.1).reshape(3, 3)
                  for i in range(len(sizes))])
    strat = [m.SolutionStrategy.ramp(120, 0.5)] * len(sizes)
    if options.pop("serve", False):
        from mumfim_gb300.serving import RVEServer
        with RVEServer(nets, strat, precision="mixed") as sv:
            for r in range(len(sizes)):
                sv.submit(r, F[r])
            done = sv.drain(timeout_s=60)
        assert (done["status"] == 0).all()
        return done["sigma"][np.argsort(done["rve"])]
    g = m.BatchedFiberRVEAnalysisExplicit(nets, strat, precision="mixed", **options)
    s = np.zeros((len(sizes), 6))
    assert g.run(F, s)
    g.close()
    return s


@pytest.mark.gpu
@pytest.mark.parametrize("options", [{}, {"max_cluster_ctas": 1}, {"small_rve_solve": "node",
                                                                  "max_cluster_ctas": 1},
                                     {"serve": True}])
def test_ratios_that_no_fiber_reaches(lib_path, options):
    sizes = (200, 900, 2_500)
    want = _solve(sizes, 1e6, **dict(options))
    assert np.isfinite(want).all() and np.abs(want).max() > 0
    for ratio in (1e19, 2e19, 3.4028234e38, 1e39, 1e300, sys.float_info.max):
        np.testing.assert_array_equal(_solve(sizes, ratio, **dict(options)), want)
