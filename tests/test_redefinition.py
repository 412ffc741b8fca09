"""A context whose volume and surface are redefined, larger and smaller, between
calls: its workspaces follow the sizes, whatever was asked of the first mesh.

Tolerance: grids are the fresh context's bit for bit; reverse products land with
FP64 atomics, whose order alone differs (1e-12 of the largest entry)."""
import contextlib
import io

import numpy as np
import pytest

from tests.meshes import build_gpu, sphere_small, wing_small
from idwarp_gb300 import synthetic as S

pytestmark = pytest.mark.gpu


def larger():
    m = S.sphere_ogrid(n=24, layers=10)
    m["xs"] = S.sphere_perturbation(m["pts"], seed=3)
    return m


def results(g, m):
    """A batch of three surfaces (one group), and the products of two seeds."""
    xs = np.stack([m["xs"] * (1.0 + 0.01 * i) for i in range(3)])
    grids = np.array(g.warpMeshBatch(xs))
    g.setSurfaceCoordinates(m["xs"])
    g.warpMesh()
    seeds = np.random.default_rng(4).standard_normal((2, len(m["xv0"]), 3))
    return grids, np.array(g.warpDerivBatch(seeds))


@pytest.mark.parametrize("opts", [{"precision": "mixed"}, {"precision": "mixed", "adjointPrecision": "fast"},
                                  {"precision": "mixed", "mixedGate": 1e-3},
                                  {"precision": "mixed", "evalMode": "exact"},
                                  {"precision": "mixed", "deterministic": True}, {"precision": "fp64"}])
def test_workspaces_follow_the_sizes(built_lib, opts):
    opts = dict(opts)
    precision = opts.pop("precision")
    meshes = [dict(m, symmetryPlanes=None) for m in (sphere_small(), larger(), wing_small())]
    g = None
    for m in meshes:
        if g is None:
            g = build_gpu(m, opts, precision=precision)
        else:
            with contextlib.redirect_stdout(io.StringIO()):
                g.createCommonGrid(m["xv0"])
                g.setSurfaceDefinition(m["pts"], m["conn"], m["faceSizes"])
        grids, dxs = results(g, m)
        want, dwant = results(build_gpu(m, opts, precision=precision), m)
        np.testing.assert_array_equal(grids, want)
        assert np.abs(dxs - dwant).max() <= 1e-12 * np.abs(dwant).max()


def test_other_planes_need_a_new_surface_definition(built_lib):
    from idwarp_gb300 import _lib

    g = build_gpu(sphere_small(), precision="mixed")
    p, nrm = np.zeros((1, 3)), np.array([[0.0, 1.0, 0.0]])
    assert g.lib.idw_set_symmetry_planes(g.ctx, _lib.dptr(p), _lib.dptr(nrm), 1) == 0
    assert g.lib.idw_warp_mesh(g.ctx) == _lib.IDW_ERR_STATE


def test_a_refused_grid_needs_a_new_one(built_lib):
    from idwarp_gb300 import _lib

    m = sphere_small()
    g = build_gpu(m, precision="mixed")
    x = np.full((2 * len(m["xv0"]), 3), np.nan)
    assert g.lib.idw_create_common_grid(g.ctx, _lib.dptr(x), len(x), _lib.IDW_HOST) == _lib.IDW_ERR_NONFINITE
    assert g.lib.idw_warp_mesh(g.ctx) == _lib.IDW_ERR_STATE
    with contextlib.redirect_stdout(io.StringIO()):
        g.createCommonGrid(m["xv0"])
        g.setSurfaceDefinition(m["pts"], m["conn"], m["faceSizes"])
    assert g.lib.idw_warp_mesh(g.ctx) == 0


def test_solver_indices_of_a_larger_grid(built_lib):
    """A smaller grid ends the indices that would reach past it; the others stay."""
    import ctypes as C

    from idwarp_gb300 import _lib

    m = sphere_small()
    g = build_gpu(m, precision="mixed")
    n = len(m["xv0"])
    for last, state in ((3 * n - 1, _lib.IDW_ERR_STATE), (n, 0)):
        with contextlib.redirect_stdout(io.StringIO()):
            g.createCommonGrid(m["xv0"])
        ind = np.array([0, last], dtype=np.int32)
        assert g.lib.idw_set_external_mesh_indices(g.ctx, ind.ctypes.data_as(C.POINTER(C.c_int32)), 2) == 0
        with contextlib.redirect_stdout(io.StringIO()):
            g.createCommonGrid(m["xv0"][: n // 2])
        w, s = np.arange(3.0 * (n // 2)), np.zeros(2)
        assert g.lib.idw_warp_to_solver_grid(g.ctx, _lib.dptr(w), w.size, _lib.dptr(s), 2, _lib.IDW_HOST) == state
        assert s.tolist() == ([0.0, float(n)] if state == 0 else [0.0, 0.0])
