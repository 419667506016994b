"""rayhierarchy's work counters (profiling level 2) describe the form of the
leaf tests that runs without them: a small batch's warps take one leaf of a
(cluster, parent) pair each and test the members against the parent again."""
import numpy as np
import pytest

import pbg_import

pbg_import.load()
from pbrt_gb300 import accel as A  # noqa: E402

pytestmark = pytest.mark.gpu


def test_small_batch_counts(gpu_lib):
    g = np.random.default_rng(4)
    turn = g.uniform(0, 7, (32, 1)) + np.arange(3) * 2 * np.pi / 3  # one cluster of equal triangles about the origin
    tris = np.stack([0.3 * np.cos(turn), 0.3 * np.sin(turn), np.zeros((32, 3))], -1) + g.uniform(-0.01, 0.01, (32, 1, 3))
    tris = tris.astype(np.float32).reshape(32, 9)
    leaves, parents, fan = 5, 2, 4
    rays = np.zeros((8, 32 * leaves), np.float32)  # one eye, into the cluster: every node reaches every member
    rays[2] = -5.0
    rays[3:5] = g.uniform(-0.02, 0.02, (2, 32 * leaves))
    rays[5], rays[7] = 1.0, np.inf
    acc = A.MakeAccelerator("rayhierarchy", tris)
    acc.profile(2)
    acc.IntersectP(rays)
    work = acc.stats()["work"]
    acc.close()
    # the seed's pairs; each pair's members against the parent, once per leaf; the members against the leaves
    assert work["node_tests"] == parents + parents * fan * 32 + leaves * 32
    assert work["leaves"] == leaves


def test_many_pairs_count_as_a_large_batch(gpu_lib):
    """By leaves only while there are few pairs to a warp: incoherent rays on
    either side of the small batches' line do the same work (by leaves each
    member is tested against the parent four times)."""
    from pbrt_gb300 import scenes as S
    line = 1 << 19
    acc = A.MakeAccelerator("rayhierarchy", S.terrain_icospheres(seed=2, grid=20, n_spheres=2)["tris"])
    rays = S.random_rays(line + 32, -6.0, 6.0, seed=8)
    tests = []
    for n in (line, line + 32):
        acc.profile(2)
        acc.Intersect(np.ascontiguousarray(rays[:, :n]))
        tests.append(acc.stats()["work"]["node_tests"])
    acc.close()
    assert tests[0] <= 1.1 * tests[1]


@pytest.mark.parametrize("spread", [0.02, 0.2, 0.3, 3.0])
@pytest.mark.parametrize("n", [33, 4099, (1 << 19) + 7])
def test_leaves_about_the_narrow_line(gpu_lib, spread, n):
    """Nearest hits of leaves whose cones lie on either side of the line where
    the beam test and the held exact tests stop, as the naive accelerator's."""
    from pbrt_gb300 import scenes as S
    tris = S.terrain_icospheres(seed=2, grid=20, n_spheres=2)["tris"]
    g = np.random.default_rng(n)
    rays = np.zeros((8, n), np.float32)
    rays[0:3] = g.uniform(-0.1, 0.1, (3, n)) + np.array([[0.5], [4.0], [-1.0]])
    rays[3:6] = g.normal(size=(3, n)) * spread + np.array([[0.1], [-1.0], [0.05]])
    rays[7] = np.where(g.random(n) < 0.2, 4.0, np.inf)
    ref, acc = A.MakeAccelerator("naive", tris), A.MakeAccelerator("rayhierarchy", tris)
    want = ref.Intersect(rays.copy())
    for a, b in zip(acc.Intersect(rays.copy()), want):
        np.testing.assert_array_equal(a, b)
    assert (want[0] >= 0).any()
    acc.close()
    ref.close()
