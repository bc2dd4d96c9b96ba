"""Mixed-precision batches that leave SMs idle: RVEs on wider thread-block
clusters than they need (up to 16 CTAs) and with the step's read-only data
staged in shared memory give the bits of one CTA per RVE (or, for the RVEs
that need one, of the smallest cluster)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes,law,narrow", [
    ((60, 500), 0, 1),                       # fewer nodes per CTA than a warp
    ((1_250, 1_330, 1_410, 1_490), 0, 1),    # around the staging limit of one CTA
    ((3_700, 6_200), 0, 1),                  # around two record copies, one record copy
    ((300, 1_100, 2_600, 4_000), 1, 1),      # nonlinear law: node-centric instead of pairs
    ((45_000,), 0, 8),                       # 16 CTAs, two record copies
    (tuple(400 + 37 * i for i in range(40)), 0, 1),  # some RVEs wider, some not
])
@pytest.mark.parametrize("relax", [False, True])
def test_wide_clusters_match_narrow(lib_path, sizes, law, narrow, relax):
    import mumfim_gb300 as m
    from mumfim_gb300 import synthetic as S
    from mumfim_gb300.network_io import Reaction
    nets, F = [], []
    for i, n in enumerate(sizes):
        coords, conn = S.knn_network(n, 3 + i % 3, S.geometry_seed(41, i))
        rc = Reaction(1, 1e-3, 1.0, 1.0, 4.0, 1.05) if law else S._linear_params(41, i)
        nets.append(m.FiberNetwork(coords, conn, [rc]))
        F.append(np.eye(3) + (S.uniform(S.param_seed(41, i), 9) * 0.1 - 0.05).reshape(3, 3))
    F = np.stack(F)
    if relax:
        strat = m.SolutionStrategy(visc_damp_coeff=2.0, residual_tol=1e-9, max_steps=203)
    else:
        strat = m.SolutionStrategy.ramp(203, 0.5)
    out = []
    for limit in (0, narrow):
        g = m.BatchedFiberRVEAnalysisExplicit(nets, [strat] * len(nets), precision="mixed",
                                              max_cluster_ctas=limit)
        s = np.zeros((len(nets), 6))
        for _ in range(2):
            g.run(F, s)
        C = g.computeMaterialStiffness()
        out.append((s, g.last_status.copy(), C, [g.displacements(r) for r in range(len(nets))],
                    [g.coordinates(r) for r in range(len(nets))]))
        g.close()
    (s0, st0, C0, u0, x0), (s1, st1, C1, u1, x1) = out
    np.testing.assert_array_equal(s0, s1)
    np.testing.assert_array_equal(C0, C1)
    np.testing.assert_array_equal(st0["steps"], st1["steps"])
    np.testing.assert_array_equal(st0["status"], st1["status"])
    np.testing.assert_allclose(st0["residual"], st1["residual"], rtol=1e-9)
    for r in range(len(nets)):
        np.testing.assert_array_equal(u0[r], u1[r])
        np.testing.assert_array_equal(x0[r], x1[r])
    assert np.isfinite(s0).all() and np.abs(s0).max() > 0
