"""The renderer's queues at their edges: bounce counts around the eight that
share one set of device counters, shadow slots around the four appended
together, frames without lights or hits.  ray-bvh frames keep the queue
lengths on the device; the other accelerators read them on the host."""
import numpy as np
import pytest

import pbg_import

pbg_import.load()
from pbrt_gb300 import accel as A  # noqa: E402
from pbrt_gb300 import render as R  # noqa: E402
from pbrt_gb300 import scenes as S  # noqa: E402

pytestmark = pytest.mark.gpu
QUAD = np.array([[-1, 3, -1], [1, 3, -1], [1, 3, 1], [-1, 3, 1]], np.float32)


def room():
    """A closed sphere around a few small ones: no path escapes."""
    small = S.displaced_icospheres(seed=4, n_inst=6, box=5.0)["tris"]
    v, f = S.icosphere(2)
    return np.concatenate([small, (v * 6.0)[f].reshape(-1, 9).astype(np.float32)])


def frames(tris, lights, prm, res=(61, 47), kinds=("ray-bvh", "naive", "rayhierarchy"), eye=(0.0, 0.5, -4.0), look=(0.0, 0.0, 0.0),
           params=None):
    r2c, c2w = R.perspective_camera(*res, eye, look, (0.0, 1.0, 0.0), 70.0)
    out = []
    for kind in kinds:
        acc = A.MakeAccelerator(kind, tris, params)
        for _ in range(2):  # the second frame reuses buffers, streams and counters
            img, st = R.render(acc, R.camera_struct(r2c, c2w, *res), lights, prm)
        st.pop("ms_total")
        counted = acc.stats()
        out.append((img, st, counted["rays_nearest"], counted["rays_occluded"]))
        acc.close()
    return out


def same(out):
    img, st, near, occ = out[0]
    assert (near, occ) == (2 * st["nearest_rays"], 2 * st["shadow_rays"])
    for other in out[1:]:
        np.testing.assert_array_equal(img, other[0])
        assert other[1] == st and other[2:] == (near, occ)
    return img, st


@pytest.mark.parametrize("depth", [1, 7, 8, 9, 17])
def test_path_depths(gpu_lib, depth):
    img, st = same(frames(room(), [R.quad_light(QUAD, (9.0, 8.0, 7.0), 1), R.point_light((0.0, -2.0, 0.0), (3.0, 3.0, 3.0))],
                          R.render_params("path", spp=(2, 2), jitter=True, seed=depth, max_depth=depth)))
    assert img.max() > 0 and st["bounces"] >= min(depth, 8)


@pytest.mark.parametrize("ns,two", [(1, False), (3, False), (4, True), (5, False), (9, True)])
def test_direct_slots(gpu_lib, oracle, ns, two):
    lights = [R.quad_light(QUAD, (9.0, 8.0, 7.0), ns)]
    spec = [{"type": "quad", "quad": QUAD, "L": (9.0, 8.0, 7.0), "nsamples": ns}]
    if two:
        lights.append(R.quad_light(QUAD - np.float32([0.5, 1.0, 0.0]), (4.0, 4.0, 4.0), 2))
        spec.append({"type": "quad", "quad": QUAD - np.float32([0.5, 1.0, 0.0]), "L": (4.0, 4.0, 4.0), "nsamples": 2})
    tris = room()
    img, _ = same(frames(tris, lights, R.render_params("directlighting", spp=(1, 2), jitter=True, seed=3)))
    r2c, c2w = R.perspective_camera(61, 47, (0.0, 0.5, -4.0), (0.0, 0.0, 0.0), (0.0, 1.0, 0.0), 70.0)
    want = oracle.render(tris, r2c, c2w, 61, 47, spec, spp=(1, 2), jitter=True, seed=3)
    assert img.max() > 0 and np.sqrt(np.mean((img - want) ** 2)) <= 1e-4


@pytest.mark.parametrize("integrator", ["path", "directlighting"])
def test_empty_queues(gpu_lib, integrator):
    prm = R.render_params(integrator, spp=(1, 1), jitter=False, max_depth=5)
    img, st = same(frames(room(), [], prm))  # no lights: no shadow rays
    assert st["shadow_rays"] == 0 and img.max() == 0
    away = frames(room(), [R.quad_light(QUAD, (1.0, 1.0, 1.0), 2)], prm, eye=(0.0, 0.0, -40.0), look=(0.0, 0.0, -80.0))
    img, st = same(away)  # every camera ray misses
    assert st["shadow_rays"] == 0 and img.max() == 0


@pytest.mark.parametrize("walk", [1, 2, 3, 4, 5, 6])
def test_walks(gpu_lib, walk):
    prm = R.render_params("path", spp=(1, 1), jitter=True, seed=6, max_depth=5)
    light = [R.quad_light(QUAD, (9.0, 8.0, 7.0), 1)]
    want = frames(room(), light, prm, kinds=("naive",))
    same(frames(room(), light, prm, kinds=("ray-bvh",), params={"walk": walk}) + want)
