"""Tile weights where the softening of the distances (d^2 + 1e-15 at surface points)
is of the size of d^2 or above it: small length units, and first cells of 1e-7.

Tolerances: those of the tangents (5e-10) and of the reverse product (1.5e-11) at
ordinary distances, as derived in their tests.  A softening added at FP32's
rounding (2^-24 of d^2) is 1e-8 off here."""
import numpy as np
import pytest

from tests.meshes import build_gpu, sphere_small, wing_small

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("unit", [1e-5, 1e-6, 1e-7])
@pytest.mark.parametrize("make", [wing_small, sphere_small])
def test_small_units(built_lib, make, unit):
    m = dict(make())
    for k in ("xv0", "pts", "xs"):
        m[k] = np.asarray(m[k]) * unit
    rng = np.random.default_rng(1)
    seed, d = rng.standard_normal(m["xv0"].size), rng.standard_normal(m["pts"].size)
    out = []
    for precision in ("mixed", "fp64"):
        g = build_gpu(m, precision=precision)
        g.setSurfaceCoordinates(m["xs"])
        g.warpMesh()
        g.warpDeriv(seed, solverVec=False)
        out.append((np.array(g.warpDerivFwd(d, solverVec=False)).ravel(), np.array(g.getdXs()).ravel()))
    for a, b, tol in zip(*out, (5e-10, 1.5e-11)):
        assert np.linalg.norm(a - b) <= tol * np.linalg.norm(b)
