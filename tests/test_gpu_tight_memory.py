"""A device with room for a batch but not for what only speeds it up: the batch
is created and solves with the same bits. Device memory is not used up for
this: the library is linked once more from its objects, with a cudaMalloc that
fails above a budget and counts what is held."""
import os
import subprocess
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)

pytestmark = pytest.mark.gpu

PRELUDE = """
import ctypes, sys
import numpy as np
import mumfim_gb300 as m
from mumfim_gb300 import batched, synthetic as S
L = batched.load_library(sys.argv[1])
L.fake_memory_held.restype = L.fake_memory_peak.restype = ctypes.c_size_t
L.fake_memory_more.argtypes = [ctypes.c_size_t]
NO_LIMIT = 2 ** 62
F = np.array([[1.02, 0.01, 0.0], [0.0, 0.99, 0.01], [0.01, 0.0, 1.01]])[None]

def networks(sizes):
    return [m.FiberNetwork(*S.knn_network(n, 4, S.geometry_seed(67, i)),
                           [S._linear_params(67, i)]) for i, n in enumerate(sizes)]

def batch(sizes, precision, steps=120, **options):
    before = L.fake_memory_held()
    g = m.BatchedFiberRVEAnalysisExplicit(networks(sizes), [m.SolutionStrategy.ramp(steps, 0.5)]
                                          * len(sizes), precision=precision, **options)
    return g, L.fake_memory_held() - before

def stress(g, n):
    s = np.zeros((n, 6))
    assert g.run(np.repeat(F, n, axis=0), s)
    return s
"""

F64_PLAN = PRELUDE + """
sizes = (300, 1_100, 2_000)
g, wide = batch(sizes, "f64")
want = stress(g, 3)
g.close()
g, narrow = batch(sizes, "f64", serving_layout=True)
g.close()
assert narrow < wide
L.fake_memory_more(narrow)
g, taken = batch(sizes, "f64")
assert taken == narrow
np.testing.assert_array_equal(stress(g, 3), want)
"""

F64_LIMIT = PRELUDE + """
sizes = (300, 1_100, 2_000)
g, narrow = batch(sizes, "f64", serving_layout=True)
want = stress(g, 3)
C = g.computeMaterialStiffness()
g.close()
held = {}
for limit in (1, 2, 8, 0):
    g, held[limit] = batch(sizes, "f64", max_cluster_ctas=limit)
    np.testing.assert_array_equal(stress(g, 3), want)
    np.testing.assert_array_equal(g.computeMaterialStiffness(), C)
    g.close()
# a limit of 1 keeps no parts; wider parts share more fibers, and so take more
assert narrow == held[1] < held[2] < held[8] < held[0]
"""

MIXED_STIFFNESS = PRELUDE + """
sizes = (500, 900, 1_300, 2_500, 4_000, 6_000, 9_000, 15_000) * 2
n = len(sizes)
L.fake_memory_peak()
g, plain = batch(sizes, "mixed", stiffness="sequential")
want = stress(g, n)
g.close()
# no memory for a second working set before a stiffness asks for one
L.fake_memory_more(L.fake_memory_peak() - L.fake_memory_held())
g, taken = batch(sizes, "mixed")
assert taken == plain
np.testing.assert_array_equal(stress(g, n), want)
L.fake_memory_more(NO_LIMIT)
C = g.computeMaterialStiffness()
with_own = L.fake_memory_held()
np.testing.assert_array_equal(g.computeMaterialStiffness(), C)
assert L.fake_memory_held() == with_own
g.close()
start = L.fake_memory_held()
# nor later: one byte too few for it, and the six solves share the batch's
g, _ = batch(sizes, "mixed")
stress(g, n)
L.fake_memory_more(with_own - L.fake_memory_held() - 1)
np.testing.assert_array_equal(g.computeMaterialStiffness(), C)
assert start < L.fake_memory_held() < with_own
np.testing.assert_array_equal(g.computeMaterialStiffness(), C)
L.fake_memory_more(NO_LIMIT)
stress(g, n)
assert np.isfinite(g.computeMaterialStiffness()).all()
"""

# one RVE: six solves of it fit beside one another on the clusters that one takes,
# so they need the batch's working set and six sets of what a solve writes
ONE_RVE_STIFFNESS = PRELUDE + """
g, plain = batch((4_500,), "mixed")
stress(g, 1)
before = L.fake_memory_held()
C = g.computeMaterialStiffness()
nodes, fibers = g.n_nodes(0), g.n_fibers(0)
scratch = 6 * (72 * nodes + 24 * fibers + 48 * nodes)  # (boundary: at most every node)
assert L.fake_memory_held() - before < scratch + 4096
g.close()
g, _ = batch((4_500,), "mixed", max_cluster_ctas=1)
stress(g, 1)
np.testing.assert_array_equal(g.computeMaterialStiffness(), C)
"""


@pytest.fixture(scope="module")
def limited_library(lib_path, tmp_path_factory):
    from mumfim_gb300.build import ARCH, OBJ_DIR, SOURCES, _cuda_home
    cuda = _cuda_home()
    d = tmp_path_factory.mktemp("tight")
    wrap, lib = str(d / "fake_memory.o"), str(d / "libmumfim_gpu_limited.so")
    subprocess.run(["g++", "-O1", "-std=c++17", "-fPIC", "-I" + os.path.join(cuda, "include"),
                    "-c", os.path.join(HERE, "native", "fake_memory.cpp"), "-o", wrap], check=True)
    objs = [os.path.join(OBJ_DIR, name + ".o") for name, _, _ in SOURCES]
    subprocess.run([os.path.join(cuda, "bin", "nvcc"), *ARCH, "-shared", "-cudart", "static",
                    "-Xlinker", "--wrap=cudaMalloc", "-Xlinker", "--wrap=cudaFree", *objs, wrap,
                    "-o", lib, "-lpthread", "-ldl", "-lrt"], check=True)
    return lib


def _run(script, library):
    r = subprocess.run([sys.executable, "-c", script, library], cwd=ROOT, capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def test_f64_batch_without_room_for_clusters(limited_library):
    _run(F64_PLAN, limited_library)


def test_stiffness_of_one_rve_shares_the_working_set(limited_library):
    _run(ONE_RVE_STIFFNESS, limited_library)


def test_f64_clusters_keep_to_the_limit(limited_library):
    _run(F64_LIMIT, limited_library)


def test_mixed_batch_without_room_for_a_second_working_set(limited_library):
    _run(MIXED_STIFFNESS, limited_library)
