"""FP64 solves split over thread-block clusters: the host-side order decodes
back to the network (CPU), and a clustered solve gives the bits of the
single-CTA one (GPU; the no-allocation solve always runs on single CTAs)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "mumfim_gb300", "csrc")


def test_parts_decode(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    from mumfim_gb300.build import _cuda_home
    try:
        cuda = _cuda_home()
    except RuntimeError:
        pytest.skip("CUDA headers not found")
    exe = str(tmp_path / "f64_order_check")
    subprocess.run([gxx, "-O1", "-std=c++17", "-I" + CSRC, "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(cuda, "include"),
                    os.path.join(HERE, "native", "f64_order_check.cpp"),
                    os.path.join(CSRC, "mfg_f64_order.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "bad=0" in r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("rves,n_min,n_max,law", [
    (1, 60, 60, 0),          # fewer free nodes per CTA than a warp
    (3, 300, 2_500, 1),      # clusters of 16, nonlinear law
    (1, 27_000, 27_000, 0),  # read-only data partly outside shared memory
    (30, 300, 3_000, 0),     # more RVEs than clusters of 16
    (70, 200, 900, 0),       # small clusters
])
@pytest.mark.parametrize("relax", [False, True])
def test_clusters_match_single_ctas(lib_path, rves, n_min, n_max, law, relax):
    import torch
    import mumfim_gb300 as m
    from mumfim_gb300 import synthetic as S
    from mumfim_gb300.network_io import Reaction
    nets, F = [], []
    for i in range(rves):
        n = int(round(n_min * (n_max / n_min) ** ((i + 0.5) / rves)))
        coords, conn = S.knn_network(n, 3 + i % 3, S.geometry_seed(31, i))
        rc = Reaction(law, 1e-3, 1.0, 1.0, 4.0, 1.05) if law else S._linear_params(31, i)
        nets.append(m.FiberNetwork(coords, conn, [rc]))
        F.append(np.eye(3) + (S.uniform(S.param_seed(31, i), 9) * 0.1 - 0.05).reshape(3, 3))
    if relax:
        strat = m.SolutionStrategy(visc_damp_coeff=2.0, residual_tol=1e-9, max_steps=203)
    else:
        strat = m.SolutionStrategy.ramp(203, 0.5)
    F_dev = torch.tensor(np.stack(F).reshape(rves, 9), device="cuda")
    out = []
    for noalloc in (False, True):
        g = m.BatchedFiberRVEAnalysisExplicit(nets, [strat] * rves)
        sigma = torch.zeros((rves, 6), dtype=torch.float64, device="cuda")
        status = torch.zeros((rves, 2), dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        run = g.run_device_noalloc if noalloc else g.run_device
        for _ in range(2):
            run(F_dev.data_ptr(), rves, sigma.data_ptr(), True, status.data_ptr())
        torch.cuda.synchronize()
        out.append((sigma.cpu().numpy(), status.cpu().numpy(),
                    [g.displacements(r) for r in range(rves)],
                    [g.coordinates(r) for r in range(rves)]))
        g.close()
    for a, b in zip(*out):
        if isinstance(a, list):
            for x, y in zip(a, b):
                np.testing.assert_array_equal(x, y)
        else:
            np.testing.assert_array_equal(a, b)
    assert np.isfinite(out[0][0]).all() and np.abs(out[0][0]).max() > 0
