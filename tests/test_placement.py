"""The choice of launch kinds, made on the host (mfg_mixed_place.h and
f64_cluster_size): which RVEs get which cluster on a GPU that holds 152 CTAs
or 76, 36, 15 and 7 clusters of 2, 4, 8 and 16. Also, that the batches with
which the GPU tests compare one placement with another do take different ones."""
import os
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CSRC = os.path.join(ROOT, "mumfim_gb300", "csrc")
SMS, HELD = 152, (152, 76, 36, 15, 7)
NONE, NONLINEAR, LINEAR = 0, 1, 2  # split
AUTO, NODE, FIBER = 0, 1, 2        # small solve


@pytest.fixture(scope="module")
def place(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    from mumfim_gb300.build import _cuda_home
    try:
        cuda = _cuda_home()
    except RuntimeError:
        pytest.skip("CUDA headers not found")
    exe = str(tmp_path_factory.mktemp("place") / "place_check")
    subprocess.run([gxx, "-O1", "-std=c++17", "-I" + CSRC, "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(cuda, "include"),
                    os.path.join(HERE, "native", "place_check.cpp"),
                    os.path.join(CSRC, "mfg_mixed_place.cpp"),
                    os.path.join(CSRC, "mfg_f64_order.cpp"), "-o", exe], check=True)

    def run(rves, max_cluster=16, serving=False, small_solve=AUTO, copies=1):
        """(FP64 cluster size, [(CTAs, fiber-centric, two copies, staged, split) per RVE])"""
        lines = [f"{SMS} {' '.join(map(str, HELD))} {max_cluster} {int(serving)} {small_solve} "
                 f"{copies} {len(rves)}"]
        for law, nodes, free, fibers, steps, degrees in rves:
            lines += [f"{law} {nodes} {free} {fibers} {steps}", " ".join(map(str, degrees))]
        r = subprocess.run([exe], input="\n".join(lines), capture_output=True, text=True,
                           check=True, timeout=60)
        out = r.stdout.split("\n")
        return int(out[0].split()[1]), [tuple(map(int, row.split())) for row in out[1:] if row]
    return run


def rve(nodes, law=0, k=4, steps=200):
    """An RVE as the generator makes them: a boundary share that falls with the
    size, 0.62 k fibers a node, degrees around their mean."""
    free = max(1, int(nodes * (1.0 - min(0.6, 1.0 / nodes ** (1.0 / 3.0) * 2.0))))
    fibers = int(0.62 * k * nodes)
    degrees = np.random.default_rng(nodes).poisson(1.24 * k - 2, free) + 2
    return law, nodes, free, fibers, steps, degrees


def ctas(placed):
    return [p[0] for p in placed]


# ---- batches that leave SMs idle --------------------------------------------------------------

@pytest.mark.parametrize("nodes,law,want", [
    (1_000, 0, (4, LINEAR)), (2_500, 0, (16, LINEAR)), (4_230, 0, (16, LINEAR)),
    (1_000, 1, (8, NONLINEAR)), (4_300, 1, (16, NONLINEAR)), (20_000, 0, (16, NONE)),
    (80_000, 0, (16, NONE))])
def test_one_rve_takes_a_wide_cluster(place, nodes, law, want):
    (cl, _, two_copies, _, split), = place([rve(nodes, law)])[1]
    assert split == want[1]
    assert cl == want[0] if nodes > 1_000 else cl >= want[0] // 2
    assert two_copies or nodes > 50_000


def test_batches_that_fill_the_gpu_are_not_widened(place):
    for sizes in ([4_500] * 152, [1_200] * 304, [500 + 37 * i for i in range(512)]):
        assert max(ctas(place([rve(n) for n in sizes])[1])) <= 4
        assert place([rve(n) for n in sizes])[1] == place([rve(n) for n in sizes], 8)[1]
    assert ctas(place([rve(4_500)] * 152)[1]) == [1] * 152
    assert ctas(place([rve(19_500)] * 36)[1]) == [4] * 36  # one wave


@pytest.mark.parametrize("n", [150, 300])
def test_small_nonlinear_rves_share_ctas_where_clusters_of_2_remain(place, n):
    # 38 to 76 RVEs leave room for 2 CTAs each, on which the longest row's chain
    # takes longer than two RVEs side by side on one
    for rves in (48, 64, 76):
        assert ctas(place([rve(n, 1)] * rves)[1]) == [1] * rves
    assert ctas(place([rve(n, 1)] * 32)[1]) == [4] * 32  # four lanes to a node


def test_widest_cluster_is_limited(place):
    for limit in (1, 2, 4, 8):
        for rves in ([rve(4_500)], [rve(900, 1), rve(3_000, 1)], [rve(20_000)] * 3):
            assert max(ctas(place(rves, limit)[1])) <= limit


def test_six_solves_at_once_widen_less(place):
    rves = [rve(500 + 300 * i) for i in range(32)]
    one, six = ctas(place(rves)[1]), ctas(place(rves, copies=6)[1])
    assert max(one) == 16 and max(six) == 2  # six times 32 RVEs fill the GPU
    assert max(ctas(place(rves[:8], copies=6)[1])) == 4


def test_fiber_centric_small_solve_is_kept(place):
    placed = place([rve(600), rve(900)], small_solve=FIBER)[1]
    assert all(fiber and cl == 1 for cl, fiber, *_ in placed)
    placed = place([rve(600, 1), rve(900, 1)])[1]  # chosen, not asked for: wider pays
    assert not any(fiber for _, fiber, *_ in placed)


@pytest.mark.parametrize("rves,want", [
    ([rve(1_000)], 16), ([rve(4_500)] * 36, 4), ([rve(4_500)] * 152, 2), ([rve(4_500)] * 304, 1),
    ([rve(500 + 300 * i) for i in range(64)], 4), ([rve(300)] * 2_000, 1)])
def test_f64_cluster_size(place, rves, want):
    assert place(rves)[0] == want


def test_staged_records_stay_within_their_bound(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not found")
    from mumfim_gb300.build import _cuda_home
    try:
        cuda = _cuda_home()
    except RuntimeError:
        pytest.skip("CUDA headers not found")
    exe = str(tmp_path / "stage_bound_check")
    subprocess.run([gxx, "-O1", "-std=c++17", "-I" + CSRC, "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(cuda, "include"),
                    os.path.join(HERE, "native", "stage_bound_check.cpp"),
                    os.path.join(CSRC, "mfg_mixed_order.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "bad=0" in r.stdout


# ---- serving: RVEs that one CTA holds, on clusters of 4 ---------------------------------------

def _spread(n, lo, hi):
    return [int(round(lo * (hi / lo) ** ((i * 0.6180339887498949 + 0.5) % 1.0))) for i in range(n)]


@pytest.mark.parametrize("n,lo,hi,both,want", [
    # single CTAs keep the SMs busy: a cluster would take two to three times the
    # SM time, and its CTAs wait for one another between small requests
    (150, 3_000, 6_000, False, 0), (110, 300, 6_000, True, 0), (96, 2_000, 6_000, False, 0),
    # fewer RVEs than clusters: nothing waits
    (36, 3_000, 6_000, False, 36), (13, 1_800, 5_100, True, 10),
    (53, 500, 2_200, True, 0),    # too small to be faster on four CTAs
    (600, 1_000, 6_000, False, 0)])
def test_served_on_clusters(place, n, lo, hi, both, want):
    rves = [rve(x, int(both and i % 2 == 1)) for i, x in enumerate(_spread(n, lo, hi))]
    assert ctas(place(rves, serving=True)[1]).count(4) == want


def test_few_move_beside_rves_that_need_a_cluster(place):
    sizes = _spread(96, 500, 20_000)
    rves = [rve(x, i % 2) for i, x in enumerate(sizes)]
    need = sum(9 * 4 * ((x + 1) // 2 * 2) > 220 * 1024 for x in sizes)
    moved = ctas(place(rves, serving=True)[1]).count(4) - need
    assert 1 <= moved <= 8  # the longest; all 30 that would be faster alone cost throughput


@pytest.mark.parametrize("sizes,need", [  # tests/test_gpu_serve_laws.py
    (tuple(1_800 + 270 * i for i in range(13)), 0),
    ((9_000, 5_900, 6_800, 5_000, 500, 700, 1_100, 4_100), 2)])
def test_served_batches_of_both_laws_move_some(place, sizes, need):
    placed = ctas(place([rve(n, i % 2, 3 + i % 3, 103) for i, n in enumerate(sizes)],
                        serving=True)[1])
    assert need < placed.count(4) < len(sizes)


# ---- the GPU tests that compare placements ----------------------------------------------------

@pytest.mark.parametrize("sizes,law,narrow", [
    ((1_250, 1_330, 1_410, 1_490), 0, 1), ((3_700, 6_200), 0, 1),
    ((300, 1_100, 2_600, 4_000), 1, 1), ((45_000,), 0, 8),
    (tuple(400 + 37 * i for i in range(40)), 0, 1)])
def test_wide_and_narrow_batches_differ(place, sizes, law, narrow):
    rves = [rve(n, law, 3 + i % 3, 203) for i, n in enumerate(sizes)]
    wide, held = ctas(place(rves)[1]), ctas(place(rves, narrow)[1])
    assert max(held) <= narrow < max(wide)


@pytest.mark.parametrize("sizes", [
    (90, 130, 470), (1_060,), (1_120,), (1_180,), (2_120,), (2_200,), (2_290,), (4_230,),
    (350, 900, 1_400, 2_000, 2_800, 3_600)])
@pytest.mark.parametrize("linear", [False, True])
def test_small_parts_are_split(place, sizes, linear):
    rves = [rve(n, 0 if linear or i % 3 == 2 else 1, 3 + i % 3, 202) for i, n in enumerate(sizes)]
    split = {p[4] for p in place(rves)[1]}
    assert (LINEAR if linear else NONLINEAR) in split
    assert {p[4] for p in place(rves, 1)[1]} == {NONE}


def test_tiny_rves_alone_stay_on_one_cta(place):
    assert ctas(place([rve(60), rve(500)])[1]) == [1, 1]
    assert ctas(place([rve(40)])[1]) == ctas(place([rve(40, 1)])[1]) == [1]


@pytest.mark.parametrize("sizes,law,split,cl", [  # tests/test_gpu_tiny_parts.py
    ((60, 1_400), 0, LINEAR, 8), ((60, 500, 1_400, 1_400), 2, NONE, 4),
    ((60,) + (1_400,) * 20, 0, NONE, 4), ((200, 200), 1, NONLINEAR, 8)])
def test_parts_of_fewer_nodes_than_a_warp(place, sizes, law, split, cl):
    placed = place([rve(n, i % 2 if law == 2 else law, 4, 202) for i, n in enumerate(sizes)])[1]
    assert placed[0][0] == cl and placed[0][4] == split and sizes[0] / cl < 32


@pytest.mark.parametrize("sizes,relax_wants", [
    ((60,), 16), ((27_000,), 16), (tuple(300 + 90 * i for i in range(30)), None),
    (tuple(200 + 10 * i for i in range(70)), None)])
def test_f64_batches_take_clusters(place, sizes, relax_wants):
    cl = place([rve(n, 0, 3 + i % 3, 203) for i, n in enumerate(sizes)])[0]
    assert cl > 1 and (relax_wants is None or cl == relax_wants)
