"""RVEs in parts of a few nodes, four lanes to a node: the same bits as one CTA
per RVE, at part sizes around the limit, with parts that fill no warp, for
batches all on the linear law and for nonlinear RVEs beside linear ones."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [
    (40,), (90, 130, 470),
    # around 4, 8 and 16 parts of 256 free nodes
    (1_060,), (1_120,), (1_180,), (2_120,), (2_200,), (2_290,), (4_230,), (4_340,), (4_450,),
    (350, 900, 1_400, 2_000, 2_800, 3_600),
])
@pytest.mark.parametrize("relax", [False, True])
@pytest.mark.parametrize("linear", [False, True])
def test_split_nodes_match_one_cta(lib_path, sizes, relax, linear):
    import mumfim_gb300 as m
    from mumfim_gb300 import synthetic as S
    from mumfim_gb300.network_io import Reaction
    nets, F = [], []
    for i, n in enumerate(sizes):
        coords, conn = S.knn_network(n, 3 + i % 3, S.geometry_seed(47, i))
        rc = Reaction(1, 1e-3, 1.0, 1.0, 4.0, 1.02) \
            if i % 3 != 2 and not linear else S._linear_params(47, i)
        nets.append(m.FiberNetwork(coords, conn, [rc]))
        F.append(np.eye(3) + (S.uniform(S.param_seed(47, i), 9) * 0.2 - 0.1).reshape(3, 3))
    F = np.stack(F)
    if relax:
        strat = m.SolutionStrategy(visc_damp_coeff=2.0, residual_tol=1e-9, max_steps=202)
    else:
        strat = m.SolutionStrategy.ramp(202, 0.5)
    out = []
    for limit in (0, 1):
        g = m.BatchedFiberRVEAnalysisExplicit(nets, [strat] * len(nets), precision="mixed",
                                              max_cluster_ctas=limit)
        s = np.zeros((len(nets), 6))
        g.run(F, s)
        out.append((s, g.last_status.copy(), [g.displacements(r) for r in range(len(nets))]))
        g.close()
    (s0, st0, u0), (s1, st1, u1) = out
    assert np.isfinite(s0).all() and np.abs(s0).max() > 0
    np.testing.assert_array_equal(s0, s1)
    np.testing.assert_array_equal(st0["steps"], st1["steps"])
    np.testing.assert_array_equal(st0["status"], st1["status"])
    np.testing.assert_allclose(st0["residual"], st1["residual"], rtol=1e-9)
    for a, b in zip(u0, u1):
        np.testing.assert_array_equal(a, b)
