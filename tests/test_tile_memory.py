"""What the tile walks keep on the device, and what the other calls leave of it."""
import ctypes as C

import numpy as np
import pytest

from idwarp_gb300 import synthetic as S
from tests.meshes import build_gpu

pytestmark = pytest.mark.gpu


def internal(g, name):
    v = C.c_int64(0)
    assert g.lib.idw_get_internal(g.ctx, name.encode(), C.byref(v)) == 0
    return v.value


def test_a_batch_leaves_the_buffers_of_single_warps(built_lib):
    """A captured graph of a warp holds their addresses.  Above 2^17 node images a
    batch takes two surfaces a walk."""
    m = S.wing_shell(121, 41, 16)
    g = build_gpu(m, {"errTol": 1e-3}, precision="mixed")
    assert 2 * g.nVol > 2**17
    g.setSurfaceCoordinates(m["pts"])
    g.warpMesh()
    before = [internal(g, k) for k in ("tileSums", "tileMot")]
    assert all(before)
    g.warpMeshBatch(np.stack([np.asarray(m["pts"]) * (1.0 + 0.01 * i) for i in range(3)]))
    assert [internal(g, k) for k in ("tileSums", "tileMot")] == before
