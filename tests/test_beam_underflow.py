"""Rays that start within 2^-70 of a triangle's vertex: products of such
distances underflow in the leaf's beam test, which may not call a triangle
missed there that pbrt's test hits.  Edges, origin and two directions of each
case were found by a search; a leaf's rays take the two in turn."""
import numpy as np
import pytest

import pbg_import

pbg_import.load()
from pbrt_gb300 import accel as A  # noqa: E402

pytestmark = pytest.mark.gpu
CASES = [
    [[0.7657533884048462, 0.039348162710666656, -0.23543761670589447], [0.005372796207666397, 0.6129888892173767, 0.30683743953704834],
     [6.136499125705041e-23, -5.0668343460284714e-23, 4.249563621103579e-25], [-0.5933511853218079, 0.7994687557220459, -0.0937231183052063],
     [-0.5544602274894714, 0.6848205327987671, -0.4728580117225647]],
    [[-1.113899827003479, -0.9730199575424194, -0.04590662568807602], [-0.009630115702748299, -0.659291684627533, 0.22331087291240692],
     [5.38686227795779e-23, -2.841008081684021e-23, 7.761469286748734e-23], [-0.2434466928243637, -0.9687145352363586, 0.04822752624750137],
     [0.10162375867366791, -0.9835212826728821, -0.14952774345874786]],
    [[0.9344161748886108, 1.1478631496429443, -0.6211599111557007], [0.3882651925086975, -1.2850037813186646, -0.3396981656551361],
     [2.2964791713709408e-23, -5.340043698777285e-23, 3.57783193506431e-23], [0.20884834229946136, -0.8208168148994446, -0.5316409468650818],
     [-0.1511448323726654, -0.9096078276634216, -0.38699978590011597]],
    [[-0.5560937523841858, -0.6835765838623047, 0.43160057067871094], [-0.6929013729095459, 1.0568397045135498, 0.3162277936935425],
     [8.479346752223968e-24, -3.130999661330507e-23, 2.982295278619639e-23], [-0.31694141030311584, 0.7954564094543457, -0.5165242552757263],
     [0.011629436165094376, 0.9389799237251282, -0.34377530217170715]],
]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_origin_at_a_vertex(gpu_lib, oracle, case):
    e1, e2, o, d, d2 = (np.array(x, np.float32) for x in CASES[case])
    tris = np.concatenate([np.zeros(3, np.float32), e1, e2])[None]
    n = 160  # five leaves of an image row
    rays = np.zeros((8, n), np.float32)
    rays[0:3], rays[7] = o[:, None], np.inf
    rays[3:6] = np.where(np.arange(n) % 2, d2[:, None], d[:, None])
    want = oracle.nearest(tris, rays.copy())
    assert (want[0][::2] == 0).all()
    acc = A.MakeAccelerator("rayhierarchy", tris)
    acc.Preprocess(xres=n, yres=1)
    for a, b in zip(acc.Intersect(rays.copy()), want):
        np.testing.assert_array_equal(a, b)
    acc.close()
