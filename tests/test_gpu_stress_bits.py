"""Bits of the mixed solve's stress: the sum over the boundary rounds each
product once, together with what it is added to. The expected numbers are
those of the kernels before the sum was written out operation by operation,
when the compiler fused it (linear law, no library function involved)."""
import json
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden",
                      "mixed_stress_linear.json")


@pytest.mark.parametrize("options", [{}, {"max_cluster_ctas": 1}, {"small_rve_solve": "fiber"},
                                     {"serving_layout": True}])
def test_stress_bits(lib_path, options):
    import mumfim_gb300 as m
    from mumfim_gb300 import synthetic as S
    with open(GOLDEN) as fh:
        want = {int(n): [float.fromhex(x) for x in row] for n, row in json.load(fh).items()}
    nets = [m.FiberNetwork(*S.knn_network(n, 4, S.geometry_seed(73, n)), [S._linear_params(73, n)])
            for n in want]
    F = np.stack([np.eye(3) + (S.uniform(S.param_seed(73, n), 9) * 0.1 - 0.05).reshape(3, 3)
                  for n in want])
    g = m.BatchedFiberRVEAnalysisExplicit(nets, [m.SolutionStrategy.ramp(60, 0.5)] * len(nets),
                                          precision="mixed", **options)
    s = np.zeros((len(nets), 6))
    assert g.run(F, s)
    # one with more boundary nodes than a CTA has threads: more than a term a thread
    assert max(int((np.abs(np.abs(n.coords) - 0.5) < 1e-8).any(axis=1).sum()) for n in nets) > 1024
    np.testing.assert_array_equal(s, np.array(list(want.values())))
