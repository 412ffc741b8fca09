"""Restart files outlive a build: their check refuses an estimate that is 1e-15 off, so
the denominator estimate keeps its bits.  The digests are those of the estimate whose
terms take an IEEE square root and division, on the golden fixtures' meshes; the scales
put squared distances in and around FP32's range, where the root is formed otherwise."""
import contextlib
import hashlib
import io

import numpy as np
import pytest

from tests.test_golden import REF_OPTS, load, sym_of

pytestmark = pytest.mark.gpu

DIGESTS = {
    ("sphere_inflate", 0, 3.0, 5.0): "4ba7780f94d44326",
    ("sphere_inflate", 0, 2.0, 4.0): "eb029089bbf4164e",
    ("sphere_inflate", 0, 2.5, 5.0): "3a6463570145d835",
    ("sphere_inflate", -13, 3.0, 5.0): "ef0160c14949b189",
    ("sphere_inflate", 40, 3.0, 5.0): "aa5ee87dd62602a1",
    ("sphere_inflate", 40, 2.0, 4.0): "f9921b4685d92baf",
    ("wing_sym_shear", 0, 3.0, 5.0): "8eea27c9b90d0812",
    ("wing_sym_shear", 0, 2.0, 4.0): "81ded92637e5de30",
    ("wing_sym_shear", 0, 2.5, 5.0): "b284373dc1b4ca72",
    ("wing_sym_shear", -13, 3.0, 5.0): "e91b9b85593b0239",
    ("wing_sym_shear", 40, 3.0, 5.0): "5ae471508e3594cd",
    ("wing_sym_shear", 40, 2.0, 4.0): "5b95df469d6d8f2e",
}


@pytest.mark.parametrize("name,scale,a,b", list(DIGESTS))
def test_estimate_bits(built_lib, name, scale, a, b):
    from idwarp_gb300 import USMesh

    z = load(name)
    opts = dict(REF_OPTS, fileType="NPY", precision="fp64", evalMode="fast", aExp=a, bExp=b)
    if sym_of(z):
        opts["symmetryPlanes"] = sym_of(z)
    with contextlib.redirect_stdout(io.StringIO()):
        m = USMesh(options=opts)
        m.createCommonGrid(z["xv0"] * 2.0**scale)
        m.setSurfaceDefinition(z["pts"] * 2.0**scale, z["conn"], z["faceSizes"])
    den0 = np.ascontiguousarray(m.getDenominator0(), dtype=np.float64)
    assert hashlib.sha256(den0.tobytes()).hexdigest()[:16] == DIGESTS[name, scale, a, b]
