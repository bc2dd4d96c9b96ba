"""FP64 solve of a linear law whose modulus has no exact half (the smallest
number), with a fiber area that makes its stiffness an ordinary one: the
oracle's bits, on clusters and on single CTAs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("limit", [0, 1])
def test_smallest_modulus_matches_oracle(lib_path, oracle, limit):
    import mumfim_gb300 as m
    from mumfim_gb300 import synthetic as S
    from mumfim_gb300.network_io import Reaction
    coords, conn = S.knn_network(300, 4, S.geometry_seed(23, 0))
    net = m.FiberNetwork(coords, conn, [Reaction(0, 1e150, 5e-324, 1e-300)])
    strat = [m.SolutionStrategy.ramp(120, 0.0)]
    F = np.array([[[1.03, 0.01, 0.0], [0.0, 0.98, 0.02], [0.01, 0.0, 1.01]]])
    _, so, _ = oracle.OracleBatch([net], strat).run(F)
    assert np.isfinite(so).all() and np.abs(so).max() > 0
    g = m.BatchedFiberRVEAnalysisExplicit([net], strat, max_cluster_ctas=limit)
    s = np.zeros((1, 6))
    assert g.run(F, s)
    np.testing.assert_array_equal(s, so)
