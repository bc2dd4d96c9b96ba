"""Served RVEs of both laws side by side, some moved to clusters of 4 because
a wave ends sooner and some not: stresses and material stiffnesses of updating
requests are the bits of a batch that solves every RVE on its own."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [
    tuple(1_800 + 270 * i for i in range(13)),             # the larger ones move
    (9_000, 5_900, 6_800, 5_000, 500, 700, 1_100, 4_100),  # beside RVEs that need a cluster
])
def test_stress_and_stiffness_of_both_laws(lib_path, sizes):
    import mumfim_gb300 as m
    from mumfim_gb300 import synthetic as S
    from mumfim_gb300.network_io import Reaction
    from mumfim_gb300.serving import RVEServer
    nets, F = [], []
    for i, n in enumerate(sizes):
        coords, conn = S.knn_network(n, 3 + i % 3, S.geometry_seed(79, i))
        rc = Reaction(1, 1e-3, 1.0, 1.0, 4.0, 1.03) if i % 2 else S._linear_params(79, i)
        nets.append(m.FiberNetwork(coords, conn, [rc]))
        F.append(np.eye(3) + (S.uniform(S.param_seed(79, i), 9) * 0.1 - 0.05).reshape(3, 3))
    F = np.stack(F)
    strat = [m.SolutionStrategy.ramp(103, 0.5)] * len(nets)
    g = m.BatchedFiberRVEAnalysisExplicit(nets, strat, precision="mixed", max_cluster_ctas=8)
    want = []
    for G in (F, np.linalg.inv(F)):
        s = np.zeros((len(nets), 6))
        assert g.run(G, s)
        want.append((s, g.computeMaterialStiffness()))
    assert np.abs(want[0][1]).max() > 0
    with RVEServer(nets, strat, precision="mixed") as sv:
        for (s, C), G in zip(want, (F, np.linalg.inv(F))):
            for r in range(len(nets)):
                sv.submit(r, G[r], stiffness=True)
            got = sv.drain(timeout_s=60)
            assert len(got) == len(nets)
            for rec in got:
                assert rec["status"] == 0 and rec["stiffness_status"] == 0
                np.testing.assert_array_equal(rec["sigma"], s[rec["rve"]])
                np.testing.assert_array_equal(rec["C"], C[rec["rve"]])
