"""Option changes between calls: what the tile walks keep must follow them, in every
order.  At the first and the last step the warp, a tangent and a reverse product are
compared with those of an FP64 context that went through the same options.

Tolerances: those of the walks themselves (warp 1e-9 of Ldef0 below 2^17 node
images; tangents 5e-10, reverse products 1.5e-11 of the result, as derived in
their own tests); a stale law is off by its own effect, 1e-3 and more here."""
import numpy as np
import pytest

from tests.meshes import build_gpu, wing_small

pytestmark = pytest.mark.gpu

AUTO, OFF = {"walkLists": "auto"}, {"walkLists": "off"}
SEQUENCES = [
    [AUTO, {"walkLists": "off", "alpha": 0.6}, AUTO],
    [AUTO, {"walkLists": "off", "LdefFact": 3.0}, AUTO],
    [AUTO, {"walkLists": "off", "errTol": 1e-2}, AUTO],
    [OFF, AUTO, {"walkLists": "off", "alpha": 0.6}, {"walkLists": "off", "alpha": 0.25}, AUTO],
    [AUTO, {"precision": "fp64", "alpha": 0.6}, {"precision": "mixed"}],
    [AUTO, {"evalMode": "exact", "alpha": 0.6}, {"evalMode": "fast"}],
    [AUTO, {"adjointPrecision": "fast", "alpha": 0.6}, {"adjointPrecision": "precise"}],
    [AUTO, {"mixedGate": 1e-4, "LdefFact": 0.5}, {"mixedGate": 2e-3}],
]


@pytest.mark.parametrize("derivatives", [False, True])  # with them the fifth digits are kept from the first step on
@pytest.mark.parametrize("steps", SEQUENCES)
def test_options_in_sequence(built_lib, steps, derivatives):
    m = wing_small()
    rng = np.random.default_rng(2)
    seed, tangent = rng.standard_normal(np.asarray(m["xv0"]).size), rng.standard_normal(np.asarray(m["pts"]).size)
    g, f = build_gpu(m, precision="mixed"), build_gpu(m, precision="fp64")
    for mesh in (g, f):
        mesh.setSurfaceCoordinates(m["xs"])
    for i, opts in enumerate(steps):
        out = []
        for mesh in (g, f):
            for k, v in opts.items():
                if not (mesh is f and k == "precision"):
                    mesh.setOption(k, v)
            mesh.warpMesh()
            r = [np.array(mesh.getWarpGrid()).ravel()]
            if derivatives or i == len(steps) - 1:
                mesh.warpDeriv(seed, solverVec=False)
                r += [np.array(mesh.getdXs()).ravel(),
                      np.array(mesh.warpDerivFwd(tangent, solverVec=False)).ravel()]
            out.append(r)
        if g.getOption("precision") == "mixed" and i in (0, len(steps) - 1):
            a, b = out
            assert np.abs(a[0] - b[0]).max() < 1e-9 * g.getStats()["Ldef0"]
            for x, y, tol in zip(a[1:], b[1:], (1.5e-11, 5e-10)):
                assert np.linalg.norm(x - y) <= tol * np.linalg.norm(y)


@pytest.mark.parametrize("opts", [{"deterministic": True}, {"walkLists": "off"}, {"mixedGate": 1e-3}])
def test_errtol_change_renews_the_double_float_denominators(built_lib, opts):
    """Reverse products that sum term by term divide by denominators of their own; their
    tolerance is 1e-9 of the largest entry (a stale one is off by 4e-3)."""
    m = wing_small()
    seed = np.random.default_rng(2).standard_normal(np.asarray(m["xv0"]).size)
    g, f = build_gpu(m, opts, precision="mixed"), build_gpu(m, precision="fp64")
    for errTol in (1e-4, 1e-3):
        out = []
        for mesh in (g, f):
            mesh.setOption("errTol", errTol)
            mesh.setSurfaceCoordinates(m["xs"])
            mesh.warpMesh()
            mesh.warpDeriv(seed, solverVec=False)
            out.append(np.array(mesh.getdXs()).ravel())
        assert np.abs(out[0] - out[1]).max() <= 1e-9 * np.abs(out[1]).max()


def test_negative_weights_have_the_gated_walk(built_lib):
    """alpha < 0: weights of both signs can exceed their node's denominator, which the
    digits' range does not hold.  Nodes on a line towards the point where the
    denominator vanishes; the sums are 1e-5 of the weights' sizes off at most (FP32
    terms).  Digits of such weights are infinite and the quotients not numbers."""
    m = wing_small()
    x0, opts = np.asarray(m["xv0"]), {"alpha": -1.0, "errTol": 0.0}  # every point by itself

    def warped(x, precision):
        g = build_gpu(dict(m, xv0=x), opts, precision=precision)
        g.setSurfaceCoordinates(m["xs"])
        g.warpMesh()
        return np.array(g.getWarpGrid()).reshape(-1, 3), g.getDenominator()

    den = warped(x0, "fp64")[1]
    start, b = x0[den > 0.0][0], x0[den < 0.0][0]
    a = start
    for _ in range(3):
        line = a + np.linspace(0.0, 1.0, 301)[:, None] * (b - a)
        den = warped(line, "fp64")[1]
        k = int(np.argmax(den < 0.0))
        a, b = line[k - 1], line[k]
    x = a + np.linspace(0.0, 1.0, 201)[:, None] * (start - a)
    (got, _), (want, den) = warped(x, "mixed"), warped(x, "fp64")
    assert den.min() > 0.0 and den.min() < 1e-4 * den.max()
    assert np.isfinite(got).all()
    # N / D: an error of D counts with the quotient
    assert (np.abs(got - want) * den[:, None] <= 1e-5 * den.max() * (1.0 + np.abs(want))).all()


@pytest.mark.parametrize("ni,tile", [(201, True), (221, False)])
def test_lists_off_beyond_half_a_million_images(built_lib, ni, tile):
    """Up to 2^19 node images the walk from digits made on the way, beyond it the gated
    walk that decides as it goes (1e-8 of Ldef0; its tangents 1e-6 of the largest entry,
    its reverse products 1e-9), also after a walk from kept digits."""
    from idwarp_gb300 import synthetic as S

    m = S.wing_shell(ni, 61, 20)
    assert (2 * len(m["xv0"]) <= 2**19) == tile
    xs = S.wing_perturbation(np.asarray(m["pts"]), seed=3)
    rng = np.random.default_rng(6)
    seed, d = rng.standard_normal(np.asarray(m["xv0"]).size), rng.standard_normal(np.asarray(m["pts"]).size)
    g, f = (build_gpu(m, {"errTol": 1e-3}, precision=p) for p in ("mixed", "fp64"))

    def results(mesh):
        mesh.setSurfaceCoordinates(xs)
        mesh.warpMesh()
        r = [np.array(mesh.getWarpGrid()).ravel(), mesh.getStats()["preciseTerms"]]
        mesh.warpDeriv(seed, solverVec=False)
        return r + [np.array(mesh.getdXs()).ravel(), np.array(mesh.warpDerivFwd(d, solverVec=False)).ravel()]

    want = results(f)
    for lists in ("off", "auto", "off"):
        g.setOption("walkLists", lists)
        got = results(g)
        assert (got[1] == 0) == (tile or lists == "auto")
        assert np.abs(got[0] - want[0]).max() <= 1e-8 * g.getStats()["Ldef0"]
        for a, b, tol in zip(got[2:], want[2:], (1e-9, 1e-6)):
            assert np.abs(a - b).max() <= tol * np.abs(b).max()
