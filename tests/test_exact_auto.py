"""Exact mode's default schedule on meshes far below a wave of the tiled kernel:
bitwise the walk's sums and counters, at the edges of its 256-node blocks."""
import numpy as np
import pytest

from tests.meshes import build_gpu, wing_small

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exps", [(3.0, 5.0), (2.0, 4.0)])
@pytest.mark.parametrize("nvol", [1, 127, 128, 129, 255, 256, 257, 513])
def test_auto_equals_walk(built_lib, nvol, exps):
    m = dict(wing_small())
    m["xv0"] = np.asarray(m["xv0"]).reshape(-1, 3)[:nvol]
    out = []
    for schedule in ("auto", "walk"):
        g = build_gpu(m, {"evalMode": "exact", "exactSchedule": schedule, "aExp": exps[0], "bExp": exps[1]},
                      precision="mixed")
        g.setSurfaceCoordinates(m["xs"])
        g.warpMesh()
        s = g.getStats()
        out.append((g.getWarpGrid(), g.getDenominator(), s["leafPairs"], s["preciseTerms"]))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
