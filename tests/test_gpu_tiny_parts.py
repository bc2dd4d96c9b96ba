"""Small RVEs that share a size bucket with larger ones and so run on its wide
clusters, in parts of fewer nodes than a warp: the bits of one CTA per RVE,
with and without four lanes to a node. (An RVE of these sizes alone stays on
one CTA; tests/test_placement.py checks which of these take which kind.)"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,law", [
    ((60, 1_400), 0),                # 8 CTAs, split, linear
    ((60, 500, 1_400, 1_400), 2),    # 4 CTAs, not split; 16, split, nonlinear
    ((60,) + (1_400,) * 20, 0),      # 4 CTAs, not split
    ((200, 200), 1),                 # 8 CTAs, split, nonlinear
])
@pytest.mark.parametrize("relax", [False, True])
def test_tiny_parts_match_one_cta(lib_path, sizes, law, relax):
    import mumfim_gb300 as m
    from mumfim_gb300 import synthetic as S
    from mumfim_gb300.network_io import Reaction
    nets, F = [], []
    for i, n in enumerate(sizes):
        coords, conn = S.knn_network(n, 4, S.geometry_seed(59, i))
        nonlinear = i % 2 == 1 if law == 2 else law
        rc = Reaction(1, 1e-3, 1.0, 1.0, 4.0, 1.02) if nonlinear else S._linear_params(59, i)
        nets.append(m.FiberNetwork(coords, conn, [rc]))
        F.append(np.eye(3) + (S.uniform(S.param_seed(59, i), 9) * 0.2 - 0.1).reshape(3, 3))
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
