"""The launch-shape tuner tries what a batch without options gets: clusters
without a limit. A tuned batch is never held to smaller clusters than an
untuned one, and an RVE that only a cluster of 16 holds stays off global
memory (GPU)."""
import inspect

import numpy as np
import pytest


def test_the_default_shape_is_a_candidate():
    from mumfim_gb300.autotune import (CANDIDATES_VERSION, DEFAULT_SHAPE, LaunchShape,
                                       candidate_shapes, tune_cluster_limit)
    assert DEFAULT_SHAPE.kwargs() == LaunchShape().kwargs()
    for nonlinear in (0.0, 0.5, 1.0):
        tried = candidate_shapes(nonlinear)
        assert any(s.max_cluster_ctas == 0 and not s.serving_layout and
                   s.small_rve_solve == "auto" for s in tried)
    assert 0 in inspect.signature(tune_cluster_limit).parameters["candidates"].default
    assert CANDIDATES_VERSION > 3  # choices made among other candidates are not reused


@pytest.mark.gpu
def test_large_rves_keep_their_wide_clusters(lib_path, tmp_path, monkeypatch):
    import mumfim_gb300 as m
    from mumfim_gb300 import synthetic as S
    from mumfim_gb300.autotune import tune_launch_shape
    monkeypatch.setenv("MFG_AUTOTUNE_CACHE", str(tmp_path / "cache.json"))
    nets = [m.FiberNetwork(*S.knn_network(70_000, 4, S.geometry_seed(71, 0)),
                           [S._linear_params(71, 0)])]
    F = np.array([[[1.02, 0.0, 0.0], [0.0, 0.99, 0.0], [0.0, 0.0, 1.0]]])
    best, report = tune_launch_shape(nets, [m.SolutionStrategy.ramp(40, 0.5)], F, steps=40,
                                     repeats=1)
    # 16 CTAs take 11 us a step of it, global memory 280 us
    assert best.max_cluster_ctas == 0 and not best.serving_layout
    rate = {(t["shape"]["max_cluster_ctas"], t["shape"]["serving_layout"]): t["fiber_steps_per_s"]
            for t in report["table"]}
    assert rate[(0, False)] > 5 * rate[(4, False)]
