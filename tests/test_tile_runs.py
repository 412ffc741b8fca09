"""Lists off: a walk in several list runs of several digit runs each (their lengths cut
so that a small mesh has them), bit for bit the walk from kept digits: warps,
denominators, counters, batches and tangents.  The shortest runs are one group of 32
nodes each, a list run that ends amid a group's steps ends before it."""
import ctypes as C

import numpy as np
import pytest

from tests.meshes import build_gpu, sphere_small, wing_small

pytestmark = pytest.mark.gpu


def internal(g, name):
    v = C.c_int64(0)
    assert g.lib.idw_get_internal(g.ctx, name.encode(), C.byref(v)) == 0
    return v.value


def results(m, lists, steps):
    g = build_gpu(m, {"walkLists": lists}, precision="mixed")
    for name, n in zip(("tileListSteps", "tileDigitSteps"), steps):
        assert g.lib.idw_set_internal(g.ctx, name.encode(), n) == 0
    dirs = np.random.default_rng(3).standard_normal((2,) + np.shape(m["pts"]))
    g.setSurfaceCoordinates(m["xs"])
    g.warpMesh()
    s = g.getStats()
    out = [g.getWarpGrid(), g.getDenominator(), s["leafPairs"], s["approx"], s["visited"]]
    out.append(g.warpMeshBatch(np.stack([m["xs"], m["pts"], np.asarray(m["xs"]) * 1.01])))
    out.append(g.warpDerivFwdBatch(dirs))
    out.append(g.warpDerivFwd(dirs[0].ravel(), solverVec=False))
    return out, (internal(g, "tileListRuns"), internal(g, "tileDigitRuns"))


@pytest.mark.parametrize("steps", [(1, 1), (300, 1), (300, 100), (1000, 300), (10**6, 100)])
@pytest.mark.parametrize("make", [wing_small, sphere_small])
def test_runs_equal_kept_digits(built_lib, make, steps):
    m = make()
    kept, none = results(m, "auto", steps)
    made, (listRuns, digitRuns) = results(m, "off", steps)
    assert none == (0, 0)
    assert digitRuns > 1 and digitRuns >= listRuns and (listRuns > 1) == (steps[0] <= 1000)
    if 1 < steps[1] < steps[0]:
        assert digitRuns > listRuns
    for a, b in zip(kept, made):
        np.testing.assert_array_equal(a, b)
