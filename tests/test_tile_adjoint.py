"""Reverse products from the kept weight digits against the FP64 walk and against
the double-float walk (walk lists off), at the edges of the 32-node units, at seed
counts that leave a remainder of the pairs, and at seeds of extreme size.

Tolerance: the columns carry five 11-bit digits and the weights 44 bits and more
of their own size, the sums 48 bits; moving a moment from a unit's origin to a
term loses the ratio of their distance to the node's, a few hundred on these
meshes: 2^-44 x 2^8 is 1.5e-11 of the result.  The double-float walk has an FP32
seed, so it is compared at ordinary sizes only.
"""
import numpy as np
import pytest
from tests.meshes import build_gpu, sphere_small, wing_small

pytestmark = pytest.mark.gpu
TOL = 1.5e-11


def moved(m):
    return m["pts"] + 0.01 * np.sin(3.0 * m["pts"][:, ::-1])


def products(m, seeds, **kw):
    precision = kw.pop("precision", "mixed")
    g = build_gpu(m, kw, precision=precision)
    g.setSurfaceCoordinates(moved(m))
    g.warpMesh()
    if seeds.ndim == 1:
        g.warpDeriv(seeds, solverVec=False)
        return np.array(g.getdXs()).reshape(-1), g
    return np.array(g.warpDerivBatch(seeds)).reshape(len(seeds), -1), g


def close(a, b):
    assert np.linalg.norm(a - b) <= TOL * np.linalg.norm(b)


@pytest.mark.parametrize("nvol", [1, 31, 32, 33, 65, 1000])
@pytest.mark.parametrize("make", [wing_small, sphere_small])
def test_edges_of_units(built_lib, make, nvol):
    m = dict(make())
    m["xv0"] = np.asarray(m["xv0"]).reshape(-1, 3)[-nvol:]
    d = np.random.default_rng(nvol).standard_normal(3 * nvol)
    a, g = products(m, d)
    assert g.getStats()["walkListEntries"] > 0
    close(a, products(m, d, precision="fp64")[0])
    close(a, products(m, d, walkLists="off")[0])


@pytest.mark.parametrize("count", [1, 2, 3, 5])
def test_seed_counts(built_lib, count):
    m = wing_small()
    d = np.random.default_rng(count).standard_normal((count, np.asarray(m["xv0"]).size))
    a, g = products(m, d)
    b, f = products(m, d, precision="fp64")
    for x, y in zip(a, b):
        close(x, y)
    assert g.getStats()["leafPairs"] > 0


@pytest.mark.parametrize("scale", [1e-250, 1e-40, 1e150])
def test_seed_sizes(built_lib, scale):
    """Each component, and nodes beside each other, of very different size."""
    m = sphere_small()
    n = np.asarray(m["xv0"]).size
    d = np.random.default_rng(7).standard_normal(n) * scale
    a, b = products(m, d)[0] / scale, products(m, d, precision="fp64")[0] / scale
    close(a, b)
    d = np.random.default_rng(8).standard_normal((n // 3, 3)) * np.array([1.0, 1e-30, scale])
    a, b = (products(m, d.reshape(-1), **o)[0].reshape(-1, 3) for o in ({}, {"precision": "fp64"}))
    s = np.max(np.abs(d))
    close(a / s, b / s)


def test_zero_and_single_seeds(built_lib):
    m = wing_small()
    n = np.asarray(m["xv0"]).size
    assert not products(m, np.zeros(n))[0].any()
    d = np.zeros(n)
    d[3 * 40 + 1] = 1.0
    close(products(m, d)[0], products(m, d, precision="fp64")[0])


def test_law_change_rebuilds_the_digits(built_lib):
    m = wing_small()
    d = np.random.default_rng(3).standard_normal(np.asarray(m["xv0"]).size)
    out = []
    for precision in ("mixed", "fp64"):
        _, g = products(m, d, precision=precision)
        for opt, val in (("LdefFact", 3.0), ("alpha", 0.5), ("errTol", 1e-3)):
            g.setOption(opt, val)
        g.warpMesh()
        g.warpDeriv(d, solverVec=False)
        out.append(np.array(g.getdXs()).reshape(-1))
    close(*out)


def test_large_low_parts(built_lib):
    """Nodes whose nearest point carries most of the denominator, layer by layer: the
    low part of such a weight, left unnormalised, would overflow its third digit."""
    from idwarp_gb300 import synthetic

    m = synthetic.sphere_ogrid(n=9, layers=53)
    m = dict(m, xv0=np.asarray(m["xv0"]).reshape(-1, 3)[: 488 * 12])
    n = m["xv0"].size
    d = np.random.default_rng(5).standard_normal(n)
    out = []
    for precision in ("mixed", "fp64"):
        g = build_gpu(m, {"errTol": 1e-3}, precision=precision)
        g.setSurfaceCoordinates(moved(m))
        g.warpMesh()
        g.warpDeriv(d, solverVec=False)
        out.append(np.array(g.getdXs()).reshape(-1))
    assert np.linalg.norm(out[0] - out[1]) <= 1e-12 * np.linalg.norm(out[1])


@pytest.mark.parametrize("first", [1e-3, 1e-5, 1e-7])
def test_thin_layers(built_lib, first):
    """First layers far thinner than the surface's spacing: the weight law's second
    term is up to 1e13 times its first, and the weights of close points still count."""
    from idwarp_gb300 import synthetic

    m = synthetic.wing_shell(ni=101, nj=9, nk=8, first=first)
    n = np.asarray(m["xv0"]).size
    d = np.random.default_rng(6).standard_normal(n)
    a, b = products(m, d)[0], products(m, d, precision="fp64")[0]
    assert np.linalg.norm(a - b) <= 1e-12 * np.linalg.norm(b)
