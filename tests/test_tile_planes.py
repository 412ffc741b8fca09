"""Nodes on a symmetry plane stay on it to the last bit: their mirror images are
themselves, and the parts of the motion along the normal cancel.  (With several
planes the four or eight images are added in a row, and only nearly cancel.)"""
import numpy as np
import pytest

from tests.meshes import build_gpu, sphere_small, wing_small

pytestmark = pytest.mark.gpu

PLANES = [[[0.0, 0.0, 0.0], [1.0, 0.0, 0.0]], [[0.0, 0.0, 0.0], [0.0, 1.0, 0.0]], [[0.0, 0.0, 0.0], [0.0, 0.0, 1.0]]]


@pytest.mark.parametrize("lists", ["auto", "off"])
@pytest.mark.parametrize("make,axis", [(wing_small, 1), (sphere_small, 0), (sphere_small, 2)])
def test_nodes_on_the_plane(built_lib, make, axis, lists):
    m = dict(make())
    m["symmetryPlanes"] = [PLANES[axis]]
    rng = np.random.default_rng(3)
    m["xv0"] = np.array(m["xv0"])
    m["xv0"][rng.permutation(len(m["xv0"]))[: len(m["xv0"]) // 3], axis] = 0.0
    on = m["xv0"][:, axis] == 0.0
    g = build_gpu(m, {"walkLists": lists}, precision="mixed")
    g.setSurfaceCoordinates(m["xs"])
    g.warpMesh()
    xv = np.array(g.getWarpGrid()).reshape(-1, 3)
    xvd = np.asarray(g.warpDerivFwd(rng.standard_normal(np.asarray(m["pts"]).size), solverVec=False)).reshape(-1, 3)
    assert on.sum() > 300 and not xv[on, axis].any() and not xvd[on, axis].any()
