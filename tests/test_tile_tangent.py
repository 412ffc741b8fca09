"""Tangents through the tile walk (five digits of the weights and of the motions)
against the FP64 walk, at the edges of the 32-node units, for rough directions
whose gradients are thousands of times their size, and without kept digits.

Tolerance: the sums carry 2^-47 of the largest motion; a term's motion D' (r - O) +
e cancels to its size near the term, by the ratio of the mesh's extent to the
edge of a face (below 2^13 here): 2^-47 x 2^13 = 6e-11 a term, taken as 5e-10 of
the result."""
import numpy as np
import pytest

from tests.meshes import build_gpu, sphere_small, wing_small

pytestmark = pytest.mark.gpu
TOL = 5e-10


def tangents(m, dirs, **opts):
    precision = opts.pop("precision", "mixed")
    g = build_gpu(m, opts, precision=precision)
    g.setSurfaceCoordinates(m["xs"])
    g.warpMesh()
    return np.asarray(g.warpDerivFwdBatch(dirs)).reshape(len(dirs), -1)


@pytest.mark.parametrize("nvol", [1, 31, 32, 33, 65, 1000])
@pytest.mark.parametrize("make", [wing_small, sphere_small])
def test_edges_of_units(built_lib, make, nvol):
    m = dict(make())
    m["xv0"] = np.asarray(m["xv0"]).reshape(-1, 3)[-nvol:]
    d = np.random.default_rng(nvol).standard_normal((1,) + np.shape(m["pts"]))
    a, b = tangents(m, d), tangents(m, d, precision="fp64")
    assert np.linalg.norm(a - b) <= TOL * np.linalg.norm(b)
    np.testing.assert_array_equal(a, tangents(m, d, walkLists="off"))


@pytest.mark.parametrize("scale", [1e-20, 1.0, 1e15])
@pytest.mark.parametrize("make", [wing_small, sphere_small])
def test_directions(built_lib, make, scale):
    m = make()
    rng = np.random.default_rng(4)
    pts = np.asarray(m["pts"])
    d = scale * np.stack([rng.standard_normal(pts.shape), np.sin(pts[:, ::-1]), np.ones(pts.shape)])
    a, b = tangents(m, d), tangents(m, d, precision="fp64")
    for x, y in zip(a, b):
        assert np.linalg.norm(x - y) <= TOL * np.linalg.norm(y)
