"""The FP64 weight law with its FP32-seeded inverse square root, against the oracle:
denominators and warped grids at mesh sizes whose squared distances lie near the
ends of FP32's range, and at exponents off the (3, 5) branch.

Tolerance: as the FP64 parity tests', 1e-12 relative (an ulp or two a term)."""
import numpy as np
import pytest

from tests.meshes import build_gpu, build_oracle, sphere_small, wing_small

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exps", [(3.0, 5.0), (2.0, 5.0), (3.0, 3.0)])
@pytest.mark.parametrize("scale", [1e-4, 1.0, 1e12])
@pytest.mark.parametrize("make", [wing_small, sphere_small])
def test_scaled_meshes(built_lib, make, scale, exps):
    m = dict(make())
    for k in ("xv0", "pts", "xs"):
        m[k] = np.asarray(m[k]) * scale
    o = {"aExp": exps[0], "bExp": exps[1]}
    g, om = build_gpu(m, o, precision="fp64"), build_oracle(m, o)
    np.testing.assert_allclose(g.getDenominator0(), om.den0(), rtol=1e-12)
    g.setSurfaceCoordinates(m["xs"])
    g.warpMesh()
    om.set_surface_coordinates(m["xs"])
    ref = np.asarray(om.warp()).reshape(-1)
    np.testing.assert_allclose(np.asarray(g.getWarpGrid()).reshape(-1), ref, rtol=0, atol=1e-12 * np.abs(ref).max())
