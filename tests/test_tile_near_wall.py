"""Warps above 2^17 node images at the nodes beside the surface, which one or a few
terms carry: a boundary layer keeps its shape under the smallest motions.

Tolerance: the last of the four weight digits is rounded at 2^-46 of a node's
denominator, the motions' at 2^-46 of the largest; with up to a thousand terms a
node that is 2 x 1000 x 2^-46 = 3e-11 of the largest motion at the very most.  (Three
digits: 7e-11 in the median and 3e-10 at most on these nodes.)"""
import numpy as np
import pytest

from idwarp_gb300 import synthetic as S
from tests.meshes import build_gpu

pytestmark = pytest.mark.gpu


def bump(pts):
    """A local motion of 0.1, elsewhere 1e-6."""
    d = np.linalg.norm(pts - pts[len(pts) // 2], axis=1)
    return pts + np.exp(-((d / 0.2) ** 2))[:, None] * np.array([0.0, 0.0, 0.1]) + 1e-6 * np.sin(3.0 * pts[:, ::-1])


@pytest.mark.parametrize("surface", [lambda p: S.wing_perturbation(p, seed=3), bump])
@pytest.mark.parametrize("lists", ["auto", "off"])
def test_nodes_beside_the_surface(built_lib, surface, lists):
    from scipy.spatial import cKDTree

    m = S.wing_shell(121, 41, 16)
    pts, x0 = np.asarray(m["pts"]), np.asarray(m["xv0"])
    assert 2 * len(x0) > 2**17
    near = np.argsort(cKDTree(pts).query(x0)[0])[: len(x0) // 5]
    xs = surface(pts)
    out = []
    for precision in ("mixed", "fp64"):
        g = build_gpu(m, {"errTol": 5e-4, "walkLists": lists}, precision=precision)
        g.setSurfaceCoordinates(xs)
        g.warpMesh()
        out.append(np.array(g.getWarpGrid()).reshape(-1, 3)[near])
    assert np.abs(out[0] - out[1]).max() <= 3e-11 * np.abs(xs - pts).max()
