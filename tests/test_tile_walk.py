"""The tile walk (idw_tile.cu): fast-mode sums at the default exponents as
tensor-core products of weight and motion digits, against the FP64 walk.

Its weights are double-float (2^-44 relative) and its sums carry three digits of
11 bits (meshes above 2^17 node images) or four: the dropped digits are below
2^-32 (2^-43) of the denominator per term, so with the few hundred terms of a
node and motions of order Ldef the positions stay within 1e-8 of Ldef0 (the
stated bar of the mixed form) with three digits and 1e-9 with four."""
import numpy as np
import pytest

from idwarp_gb300 import synthetic as S
from tests.meshes import build_gpu, sphere_small, wing_small

pytestmark = pytest.mark.gpu


def _pair(m, opts=None):
    out = []
    for prec in ("mixed", "fp64"):
        g = build_gpu(m, opts, precision=prec)
        g.setSurfaceCoordinates(m["xs"])
        g.warpMesh()
        out.append((g.getWarpGrid().reshape(-1, 3), g.getDenominator(), g.getStats()))
    (a, da, sa), (b, db, sb) = out
    assert (sa["leafPairs"], sa["approx"]) == (sb["leafPairs"], sb["approx"])
    return np.abs(a - b).max() / sb["Ldef0"], np.abs(da / db - 1.0).max(), sa


# partial and whole groups of 32 nodes, one and several groups
@pytest.mark.parametrize("n", [1, 7, 8, 31, 32, 33, 64, 1000])
@pytest.mark.parametrize("planes", [0, 1, 3])
def test_group_edges(n, planes, built_lib):
    m = dict(sphere_small())
    m["xv0"] = m["xv0"][:: len(m["xv0"]) // n][:n].copy()
    m["symmetryPlanes"] = [[[0.0, 0.0, 0.0], [1.0, 0.0, 0.0]], [[0.0, 0.0, 0.0], [0.0, 1.0, 0.0]],
                           [[0.1, 0.0, 0.2], [0.0, 0.6, 0.8]]][:planes] or None
    err, derr, _ = _pair(m)
    assert err < 1e-9 and derr < 1e-7


# lists of many lengths (bucket sizes, tolerances), other laws of the same exponents, both trees
@pytest.mark.parametrize("opts", [{"bucketSize": 1}, {"bucketSize": 40}, {"errTol": 0.0}, {"errTol": 1e-2},
                                  {"alpha": 0.0}, {"alpha": 2.0}, {"LdefFact": 0.01}, {"LdefFact": 100.0},
                                  {"treeBuild": "morton"}, {"useRotations": False}, {"mixedGate": 1.0}])
def test_options(opts, built_lib):
    err, _, st = _pair(wing_small(), opts)
    assert err < 1e-9
    assert st["preciseTerms"] == 0


def test_three_digits(built_lib):
    # 159,572 nodes: above the limit of four digits
    m = S.sphere_ogrid(n=18, layers=81)
    m["xs"] = S.sphere_perturbation(m["pts"], seed=4)
    err, derr, _ = _pair(m)
    assert err < 1e-8 and derr < 1e-7


@pytest.mark.parametrize("scale", [1e-3, 1e4])
def test_units(scale, built_lib):
    # the same wing in other length units: the scales of nodes and areas move
    m = wing_small()
    m = dict(m, xv0=m["xv0"] * scale, pts=m["pts"] * scale, xs=m["xs"] * scale)
    err, _, st = _pair(m)
    assert err < 1e-8


def test_law_change_rebuilds_the_weights(built_lib):
    m = wing_small()
    g = build_gpu(m, precision="mixed")
    for opt, val in (("LdefFact", 3.0), ("alpha", 0.5), ("errTol", 1e-3)):
        g.setSurfaceCoordinates(m["xs"])
        g.warpMesh()
        g.setOption(opt, val)
    g.warpMesh()
    f = build_gpu(m, precision="fp64")
    for opt, val in (("LdefFact", 3.0), ("alpha", 0.5), ("errTol", 1e-3)):
        f.setOption(opt, val)
    f.setSurfaceCoordinates(m["xs"])
    f.warpMesh()
    assert np.abs(g.getWarpGrid() - f.getWarpGrid()).max() < 1e-9 * f.getStats()["Ldef0"]


@pytest.mark.parametrize("count", [2, 3, 5])
def test_batch_pairs_equal_single_warps(built_lib, count):
    """Above 2^17 node images a batch takes two surfaces a walk: the same bits."""
    m = S.wing_shell(121, 41, 16)
    g = build_gpu(m, {"errTol": 1e-3}, precision="mixed")
    xs = np.stack([np.asarray(m["pts"]) * (1.0 + 0.01 * i) for i in range(count)])
    assert g.nVol * 2 > 2**17
    out = np.asarray(g.warpMeshBatch(xs)).reshape(count, -1)
    for x, a in zip(xs, out):
        g.setSurfaceCoordinates(x)
        g.warpMesh()
        np.testing.assert_array_equal(a, np.asarray(g.getWarpGrid()).reshape(-1))


def test_runs_of_groups_equal_kept_digits(built_lib):
    """With the lists off a mesh of more than 2^17 steps is walked in several runs: the same bits."""
    m = S.wing_shell(201, 61, 20)
    out = []
    for lists in ("auto", "off"):
        g = build_gpu(m, {"errTol": 1e-4, "walkLists": lists}, precision="mixed")
        g.setSurfaceCoordinates(np.asarray(m["pts"]) * 1.01)
        g.warpMesh()
        s = g.getStats()
        out.append((g.getWarpGrid(), g.getDenominator(), s["leafPairs"], s["approx"], s["visited"], s["walkListEntries"]))
    assert out[0][5] > 16 * 2**17 and out[1][5] == 0
    for a, b in zip(out[0][:5], out[1][:5]):
        np.testing.assert_array_equal(a, b)
