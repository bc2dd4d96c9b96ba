"""mfg_device_bytes_estimate() counts what a batch keeps on the device: the parts
of the FP64 cluster solve where the batch leaves SMs idle, and no second
working set of the mixed solve before the first stiffness. A server's figure
does not change with the batch's (CPU); what a batch takes is below its
figure (GPU)."""
import numpy as np
import pytest


def _networks(n, nodes):
    import mumfim_gb300 as m
    from mumfim_gb300 import synthetic as S
    coords, conn = S.knn_network(nodes, 4, S.geometry_seed(61, 0))
    return [m.FiberNetwork(coords, conn, [S._linear_params(61, i)]) for i in range(n)]


@pytest.mark.parametrize("n,nodes,clusters", [(1, 1_000, True), (36, 4_500, True),
                                              (400, 2_000, False)])
def test_f64_batches_that_take_clusters_count_their_parts(lib_path, n, nodes, clusters):
    from mumfim_gb300.serving import device_bytes_estimate, server_bytes_estimate
    nets = _networks(n, nodes)
    batch, server = (f(nets, "f64") for f in (device_bytes_estimate, server_bytes_estimate))
    fibers = sum(net.n_fibers for net in nets)
    if clusters:  # ends, length and its reciprocal 24 B a fiber, two incidences 8 B, at least
        assert 32 * fibers < batch - server < 100 * fibers
    else:
        assert batch == server
    assert device_bytes_estimate(nets, "mixed") == server_bytes_estimate(nets, "mixed")


@pytest.mark.gpu
@pytest.mark.parametrize("precision,n,nodes", [("f64", 36, 20_000), ("f64", 60, 8_000),
                                               ("mixed", 3, 80_000), ("mixed", 36, 20_000)])
def test_batches_take_no_more_than_their_estimate(lib_path, precision, n, nodes):
    import torch
    import mumfim_gb300 as m
    from mumfim_gb300.serving import device_bytes_estimate
    F = np.eye(3)[None]

    def make(nets):
        g = m.BatchedFiberRVEAnalysisExplicit(nets, [m.SolutionStrategy.ramp(5, 0.5)] * len(nets),
                                              precision=precision)
        g.run(F, update_coords=False)
        return g

    nets = _networks(n, nodes)
    make(nets).close()  # the kernels are loaded
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    g = make(nets)
    taken = before - torch.cuda.mem_get_info()[0]
    g.close()
    # an allocation is rounded up to 2 MB: at most 32 of them
    assert 0 < taken < device_bytes_estimate(nets, precision) + 32 * 2e6
