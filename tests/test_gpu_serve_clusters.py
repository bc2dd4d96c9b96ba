"""Served RVEs that one CTA would hold but a cluster of 4 takes, because the
wave ends sooner: the results are the batch run's bits, whichever of the
server's solves each RVE gets."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,law", [
    ((1_600, 3_700, 6_200), 0),                      # all on clusters
    ((900, 2_600, 4_500, 6_200, 14_900, 15_400), 1),  # two record copies and one
    (tuple(400 + 29 * i for i in range(160)), 0),    # the longest alone
    ((60, 300), 0),                                  # none: no faster on four CTAs
])
def test_served_on_clusters_matches_batch(lib_path, sizes, law):
    import mumfim_gb300 as m
    from mumfim_gb300 import synthetic as S
    from mumfim_gb300.network_io import Reaction
    from mumfim_gb300.serving import RVEServer
    nets, F = [], []
    for i, n in enumerate(sizes):
        coords, conn = S.knn_network(n, 3 + i % 3, S.geometry_seed(43, i))
        rc = Reaction(1, 1e-3, 1.0, 1.0, 4.0, 1.05) if law else S._linear_params(43, i)
        nets.append(m.FiberNetwork(coords, conn, [rc]))
        F.append(np.eye(3) + (S.uniform(S.param_seed(43, i), 9) * 0.1 - 0.05).reshape(3, 3))
    strat = [m.SolutionStrategy.ramp(203, 0.5)] * len(nets)
    g = m.BatchedFiberRVEAnalysisExplicit(nets, strat, precision="mixed")
    ref = []
    for G in (np.stack(F), np.linalg.inv(np.stack(F))):
        s = np.zeros((len(nets), 6))
        g.run(G, s)
        ref.append(s)
    with RVEServer(nets, strat, precision="mixed") as sv:
        for k, want in enumerate(ref):
            for r in range(len(nets)):
                sv.submit(r, F[r] if k == 0 else np.linalg.inv(F[r]))
            got = sv.drain()
            assert len(got) == len(nets)
            for rec in got:
                assert rec["status"] == 0 and rec["steps"] == 203
                np.testing.assert_array_equal(rec["sigma"], want[rec["rve"]])
