"""rayhierarchy's grid candidates are the ones that the batch's launches take:
small batches have their own, and keep their setting apart."""
import numpy as np
import pytest

import pbg_import

pbg_import.load()
from pbrt_gb300 import accel as A  # noqa: E402
from pbrt_gb300 import scenes as S  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("anyhit", [False, True])
def test_candidates_by_batch_size(gpu_lib, anyhit):
    import torch
    acc = A.MakeAccelerator("rayhierarchy", S.terrain_icospheres(seed=2, grid=20, n_spheres=2)["tris"])
    line = 1 << 19
    rays = S.random_rays(line + 1, -6.0, 6.0, seed=1)
    o, d = (torch.from_numpy(np.ascontiguousarray(rays[k].T)).cuda() for k in ([0, 1, 2, 6], [3, 4, 5, 7]))
    torch.cuda.synchronize()
    for n, grids in ((1, {12, 32}), (line, {12, 32}), (line + 1, {16, 32})):
        r = acc.autotune(o[:n], d[:n], anyhit=anyhit, reps=1)
        got = [c["setting"] for c in r["candidates"]]
        assert {c["grid_ctas_per_sm"] for c in got} == grids and len({tuple(c.items()) for c in got}) == 6
        assert r["mismatches"] == 0
    acc.close()
