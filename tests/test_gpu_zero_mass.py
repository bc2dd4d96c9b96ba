"""FP64 networks whose fiber area underflows to zero: the nodes' masses are zero
too, their accelerations 0 / 0, and the run reports a non-finite result, on
every solve and as the oracle does, instead of a converged zero stress."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("noalloc", [False, True])  # a cluster, a single CTA
def test_zero_mass_is_reported(lib_path, oracle, noalloc):
    import torch
    import mumfim_gb300 as m
    from mumfim_gb300 import synthetic as S
    from mumfim_gb300.network_io import Reaction
    coords, conn = S.knn_network(300, 4, S.geometry_seed(22, 0))
    net = m.FiberNetwork(coords, conn, [Reaction(0, 1e-170, 1.0, 1.0)])
    strat = [m.SolutionStrategy.ramp(120, 0.5)]
    F = np.array([[[1.03, 0.01, 0.0], [0.0, 0.98, 0.02], [0.01, 0.0, 1.01]]])
    _, so, _ = oracle.OracleBatch([net], strat).run(F)
    assert np.isnan(so).all()
    g = m.BatchedFiberRVEAnalysisExplicit([net], strat)
    F_dev = torch.tensor(F.reshape(1, 9), device="cuda")
    sigma = torch.zeros((1, 6), dtype=torch.float64, device="cuda")
    status = torch.zeros((1, 2), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    run = g.run_device_noalloc if noalloc else g.run_device
    run(F_dev.data_ptr(), 1, sigma.data_ptr(), True, status.data_ptr())
    torch.cuda.synchronize()
    assert np.isnan(sigma.cpu().numpy()).all()
    assert int(status.cpu().numpy().view(np.int32)[0, 0]) == 4  # MFG_E_NONFINITE
