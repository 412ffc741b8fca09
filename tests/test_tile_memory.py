"""What the tile walks keep on the device, what the other calls leave of it, and
which walk serves where the memory is not to be had (allocations refused on the
host).

Tolerances against the FP64 form: those that hold for whichever walk serves, the
gated one's 1e-8 of Ldef0 for warps and 1e-9 of the largest entry for the
double-float reverse product, and 1e-6 for its tangents."""
import ctypes as C

import numpy as np
import pytest

from idwarp_gb300 import synthetic as S
from tests.meshes import build_gpu, wing_small

pytestmark = pytest.mark.gpu


def internal(g, name):
    v = C.c_int64(0)
    assert g.lib.idw_get_internal(g.ctx, name.encode(), C.byref(v)) == 0
    return v.value


def limit(g, name, value):
    assert g.lib.idw_set_internal(g.ctx, name.encode(), value) == 0


def calls(g, m):
    """Two rounds of a warp, a reverse product, a tangent and a batch."""
    rng = np.random.default_rng(1)
    seed, tangent = rng.standard_normal(np.asarray(m["xv0"]).size), rng.standard_normal(np.asarray(m["pts"]).size)
    out = []
    for _ in range(2):
        g.setSurfaceCoordinates(m["xs"])
        g.warpMesh()
        out.append(np.array(g.getWarpGrid()).ravel())
        g.warpDeriv(seed, solverVec=False)
        out.append(np.array(g.getdXs()).ravel())
        out.append(np.array(g.warpDerivFwd(tangent, solverVec=False)).ravel())
        out.append(np.array(g.warpMeshBatch(np.stack([m["xs"], m["xs"]]))).ravel())
    return out


def close(a, b, L):
    for i, (x, y) in enumerate(zip(a, b)):
        assert np.abs(x - y).max() <= (1e-8 * L, 1e-9 * np.abs(y).max(), 1e-6 * np.abs(y).max(), 1e-8 * L)[i % 4]


@pytest.mark.parametrize("lists,basic", [("auto", 12), ("off", 7)])
@pytest.mark.parametrize("allowed", range(19))
def test_refused_allocations(built_lib, lists, basic, allowed):
    """The gated walk serves until the tile walk's own memory is there (`basic`
    allocations; off: its runs need four more), the double-float reverse product and
    the gated tangent until the fifth digits' is; with the lists off a batch that
    cannot have its four buffers goes surface by surface."""
    m = wing_small()
    f, g = build_gpu(m, precision="fp64"), build_gpu(m, {"walkLists": lists}, precision="mixed")
    limit(g, "tileAllocs", allowed)
    close(calls(g, m), calls(f, m), f.getStats()["Ldef0"])
    assert internal(g, "tileState") == (1 if allowed >= basic else -1)
    assert internal(g, "tileAllocs") == max(0, allowed - (15 if lists == "auto" else 17))


def test_refused_allocations_after_an_errtol_change(built_lib):
    m = wing_small()
    f, g = build_gpu(m, precision="fp64"), build_gpu(m, precision="mixed")
    calls(g, m)
    limit(g, "tileAllocs", 0)
    # shorter lists go where the longer ones were
    for errTol, state in ((2e-4, 1), (1e-5, -1), (1e-4, -1)):
        for mesh in (f, g):
            mesh.setOption("errTol", errTol)
        close(calls(g, m), calls(f, m), f.getStats()["Ldef0"])
        assert internal(g, "tileState") == state


def test_digits_beyond_half_of_the_free_memory(built_lib):
    """The gated walks serve both settings of walkLists, with the same bits."""
    m = wing_small()
    out = []
    for lists in ("auto", "off"):
        g = build_gpu(m, {"walkLists": lists}, precision="mixed")
        limit(g, "tileFree", 10**6)
        out.append(calls(g, m))
        assert internal(g, "tileState") == -1
    f = build_gpu(m, precision="fp64")
    close(out[0], calls(f, m), f.getStats()["Ldef0"])
    for i, (a, b) in enumerate(zip(*out)):
        if i % 4 != 1:  # reverse products land with atomics
            np.testing.assert_array_equal(a, b)


def test_a_batch_leaves_the_buffers_of_single_warps(built_lib):
    """A captured graph of a warp holds their addresses."""
    m = S.wing_shell(121, 41, 16)
    g = build_gpu(m, {"errTol": 1e-3}, precision="mixed")
    g.setSurfaceCoordinates(m["pts"])
    g.warpMesh()
    before = [internal(g, k) for k in ("tileSums", "tileMot")]
    assert all(before)
    g.warpMeshBatch(np.stack([np.asarray(m["pts"]) * (1.0 + 0.01 * i) for i in range(3)]))
    assert [internal(g, k) for k in ("tileSums", "tileMot")] == before
