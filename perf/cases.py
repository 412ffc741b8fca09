"""The work that users of idwarp_gb300 have it do, as cases that can be timed and checked.

A case is one pass of one call sequence on one synthetic mesh of the package
(a cubed-sphere O-grid, or a NACA0012 half wing with a symmetry plane):

* ``step``     surface in, warped grid out, with host arrays (the USMesh calls
               of an optimisation script);
* ``warp``     the same through ``idwarp_gb300.autograd`` on CUDA tensors;
* ``gradient`` warp and reverse product of one seed (a torch training step);
* ``seeds``    several reverse products at the current surface (one per
               objective or constraint), device arrays through the C ABI;
* ``surfaces`` several perturbed surfaces warped in one call;
* ``tangent``  forward-mode products of one or more directions;
* ``setup``    volume grid and surface definition of a new mesh, up to its
               denominator estimate.

``listed`` gives the fixed cases, ``draw`` further ones of the same ranges,
``prepare`` / ``run`` / ``work`` make, run and count one, and ``exact``
evaluates it in FP64 with plain torch and numpy.
"""
import contextlib
import ctypes
import functools
import io
import math

import numpy as np
import torch

from idwarp_gb300 import USMesh, _lib, synthetic
from idwarp_gb300.autograd import warp

A_EXP, B_EXP, ALPHA, BUCKET, CORNER_DEG = 3, 5, 0.25, 8, 30.0  # the package's defaults


def _case(op, mesh, n1, n2, n3=0, errTol=1e-4, count=1, evalMode="fast", precision="mixed", adjoint="precise",
          tree="kd", name=None):
    c = {"op": op, "mesh": mesh, "n1": n1, "n2": n2, "n3": n3, "errTol": errTol, "count": count,
         "evalMode": evalMode, "precision": precision, "adjoint": adjoint, "tree": tree}
    return dict(c, name=name) if name else c


def listed():
    return [
        # a coarse mesh inside a host-driven optimisation loop: launches and latency
        _case("step", "wing", 41, 17, 10, errTol=5e-4, name="step_wing_7k"),
        # forward and backward of a torch loop on a small mesh
        _case("gradient", "sphere", 18, 48, name="gradient_sphere_95k"),
        # the all-double form, for users who compare with the reference digit by digit
        _case("warp", "sphere", 18, 48, precision="fp64", name="warp_fp64_sphere_95k"),
        # an ordinary mesh at the default tolerance
        _case("warp", "wing", 201, 61, 20, errTol=5e-4, name="warp_wing_245k"),
        # exact mode: every volume node against every surface node
        _case("warp", "wing", 201, 61, 20, evalMode="exact", name="exact_wing_245k"),
        # tangent of one design variable
        _case("tangent", "wing", 201, 61, 20, errTol=5e-4, name="tangent_wing_245k"),
        # objective and constraints in the faster adjoint precision
        _case("seeds", "wing", 201, 61, 20, errTol=5e-4, count=4, adjoint="fast", name="seeds4_fast_wing_245k"),
        # a new production mesh: tree, error tables, denominator estimate
        _case("setup", "wing", 401, 101, 50, name="setup_wing_2m"),
        # forward and backward of a torch loop on a production mesh
        _case("gradient", "wing", 401, 101, 50, name="gradient_wing_2m"),
        # sixteen objectives and constraints at once
        _case("seeds", "wing", 401, 101, 50, count=16, name="seeds16_wing_2m"),
        # a design sweep: eight perturbations of one mesh
        _case("surfaces", "wing", 401, 101, 50, count=8, name="surfaces8_wing_2m"),
        # the largest single mesh
        _case("warp", "wing", 577, 261, 53, name="warp_wing_8m"),
    ]


# seconds that a drawn case may cost at most (_cost): about those of the largest listed case
_COST_MOST = 0.12


def draw(rng):
    """One more case: sizes over the listed cases' range (log-uniform, odd and even), every option in use."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    while True:
        op = rng.choice(["step", "warp", "warp", "gradient", "gradient", "seeds", "surfaces", "tangent", "setup"])
        mesh = rng.choice(["wing", "wing", "sphere"])
        if mesh == "wing":
            n = (size(41, 577), size(17, 261), size(10, 64))
        else:
            n = (size(8, 60), size(12, 80), 0)
        c = _case(op, mesh, *n, errTol=rng.choice([1e-3, 5e-4, 1e-4]))
        if op in ("seeds", "surfaces", "tangent"):
            c["count"] = size(1, 16)
        if op == "warp":
            c["evalMode"], c["precision"] = rng.choice([("fast", "mixed")] * 3 + [("exact", "mixed"), ("fast", "fp64")])
        if op in ("gradient", "seeds"):
            c["adjoint"] = rng.choice(["precise", "precise", "fast"])
        if op != "setup" and rng.random() < 0.2:
            c["tree"] = "morton"
        nv, ns, _ = _sizes(c)
        if 6000 <= nv <= 8_000_000 and _cost(c) <= _COST_MOST and (op != "step" or nv <= 1_000_000):
            return c


def _sizes(c):
    """Volume nodes, surface points (with duplicates) and mirror images of a case."""
    if c["mesh"] == "wing":
        return c["n1"] * c["n2"] * c["n3"], c["n1"] * c["n2"], 2
    return (6 * c["n1"] ** 2 + 2) * (c["n2"] + 1), 6 * (c["n1"] + 1) ** 2, 1


def _pairs(c):
    """Pair interactions (leaf pairs and cluster terms) of one walk: all of them in exact mode; in fast mode about
    270 to 360 a node at errTol 1e-4 on the package's meshes, fewer with a looser tolerance."""
    nv, ns, loops = _sizes(c)
    if c["evalMode"] == "exact":
        return float(nv) * ns * loops
    return float(nv) * min(ns * loops, 300.0 * (1e-4 / c["errTol"]) ** 0.35)


def _flops(c):
    """42 operations a pair forward; 17 and 24 a seed in the reverse product; the estimate's pairs in a set-up."""
    p, k = _pairs(c), c["count"]
    if c["op"] == "gradient":
        return 42 * p + 41 * p
    if c["op"] == "seeds":
        return p * (17 + 24 * k)
    return 42 * p * (k if c["op"] in ("surfaces", "tangent") else 1)


def _cost(c):
    """Rough seconds of one pass, to bound the drawn cases."""
    if c["precision"] == "fp64":
        return _flops(c) / 1.3e12
    if c["evalMode"] == "exact":
        return _flops(c) / 2e13
    if c["op"] == "setup":
        return _sizes(c)[0] * 1e-7
    return _flops(c) / (3e12 if c["op"] in ("gradient", "seeds") else 6e12)


def work(case):
    nv, ns, _ = _sizes(case)
    k = case["count"]
    surfaces, grids = {"step": (1, 1), "warp": (1, 1), "gradient": (2, 2), "seeds": (1 + k, k), "surfaces": (k, k),
                       "tangent": (1 + k, k), "setup": (1, 0)}[case["op"]]
    # the initial grid, surfaces in or out, grids or seeds in or out; FP64 coordinates; a set-up gives one value a node
    return {"bytes": 24.0 * (nv + surfaces * ns + grids * nv) + (8.0 * nv if case["op"] == "setup" else 0.0),
            "flops": _flops(case)}


@functools.lru_cache(maxsize=2)
def _geometry(mesh, n1, n2, n3):
    if mesh == "wing":
        return synthetic.wing_shell(n1, n2, n3, first=1e-4 if n1 < 60 else 1e-5, far=10.0 if n1 < 60 else 25.0)
    return synthetic.sphere_ogrid(n=n1, layers=n2)


def _surface(case, pts, seed):
    if case["mesh"] == "wing":
        return synthetic.wing_perturbation(pts, seed=seed)
    return synthetic.sphere_perturbation(pts, seed=seed)


def _inputs(case, seed):
    """The mesh, `count` perturbed surfaces and the seeds or directions of a case (numpy, FP64)."""
    g = _geometry(case["mesh"], case["n1"], case["n2"], case["n3"])
    many = case["count"] if case["op"] == "surfaces" else 1
    xs = [_surface(case, g["pts"], seed * 16 + j) for j in range(many)]
    return g, np.stack(xs) if case["op"] == "surfaces" else xs[0]


def _normal(shape, seed, device):
    """N(0, 1) from the seed alone, made on the device."""
    g = torch.Generator(device=device).manual_seed(1000003 + seed)
    return torch.randn(shape, generator=g, dtype=torch.float64, device=device)


def prepare(case, seed):
    g, xs = _inputs(case, seed)
    options = {"fileType": "NPY", "errTol": case["errTol"], "evalMode": case["evalMode"],
               "precision": case["precision"], "adjointPrecision": case["adjoint"], "treeBuild": case["tree"],
               "aExp": float(A_EXP), "bExp": float(B_EXP), "alpha": ALPHA, "bucketSize": BUCKET,
               "cornerAngle": CORNER_DEG, "symmetryPlanes": g["symmetryPlanes"]}
    dev = torch.device("cuda", torch.cuda.current_device())
    s = {"op": case["op"], "count": case["count"]}
    with contextlib.redirect_stdout(io.StringIO()):
        mesh = s["mesh"] = USMesh(options=options)
        if case["op"] == "setup":
            # a new mesh a seed: the grid and its surface, swept by a small angle
            s["xv0"], s["pts"] = _sweep(g["xv0"], seed), _sweep(g["pts"], seed)
            s["conn"], s["faceSizes"] = g["conn"], g["faceSizes"]
            return s
        mesh.createCommonGrid(g["xv0"])
        mesh.setSurfaceDefinition(g["pts"], g["conn"], g["faceSizes"])
    nv, ns = len(g["xv0"]), len(g["pts"])
    if case["op"] == "step":
        s["xs"] = xs
        s["out"] = torch.empty(3 * nv, dtype=torch.float64, pin_memory=True).numpy()
        return s
    s["xs"] = torch.from_numpy(xs).to(dev)
    if case["op"] == "gradient":
        s["xs"].requires_grad_(True)
        s["dxv"] = _normal((nv, 3), seed, dev)
    elif case["op"] in ("seeds", "tangent"):
        mesh.setSurfaceCoordinates(s["xs"])
        mesh.warpMesh()
        n_in, n_out = (nv, ns) if case["op"] == "seeds" else (ns, nv)
        s["in"] = _normal((case["count"], n_in, 3), seed, dev)
        s["out"] = torch.empty((case["count"], n_out, 3), dtype=torch.float64, device=dev)
    elif case["op"] == "surfaces":
        s["out"] = torch.empty((case["count"], nv, 3), dtype=torch.float64, device=dev)
    return s


def _sweep(x, seed):
    """The same geometry sheared along the span by a seeded small angle (mirror symmetry is kept)."""
    t = 0.02 * np.random.default_rng(seed).standard_normal()
    y = np.array(x)
    y[:, 0] += t * np.abs(y[:, 1])
    return y


def _device_call(s, fn):
    """A C ABI call on device arrays: ctx, in, count, out, where."""
    m = s["mesh"]
    src = s["xs"] if s["op"] == "surfaces" else s["in"]
    rc = fn(m.ctx, ctypes.c_void_p(src.data_ptr()), s["count"], ctypes.c_void_p(s["out"].data_ptr()), _lib.IDW_DEVICE)
    _lib.check(m.lib, m.ctx, rc, s["op"])
    return s["out"]


def run(state):
    op, m = state["op"], state["mesh"]
    if op == "step":
        m.setSurfaceCoordinates(state["xs"])
        m.warpMesh()
        return m.getWarpGrid(out=state["out"])
    if op == "warp":
        return warp(state["xs"], m)
    if op == "gradient":
        xv = warp(state["xs"], m)
        return xv.detach(), torch.autograd.grad(xv, state["xs"], state["dxv"])[0]
    if op == "seeds":
        return _device_call(state, m.lib.idw_warp_deriv_batch)
    if op == "surfaces":
        return _device_call(state, m.lib.idw_warp_mesh_batch)
    if op == "tangent":
        return _device_call(state, m.lib.idw_warp_deriv_fwd_batch)
    m.createCommonGrid(state["xv0"])
    m.setSurfaceDefinition(state["pts"], state["conn"], state["faceSizes"])
    return m.getDenominator0()


# ---------------------------------------------------------------------------
# the same values in FP64 with plain torch and numpy: the IDWarp algorithm
# (kd tree, error tables, denominator estimate, fast or exact sums, Rodrigues
# nodal motions), vectorised over pairs of volume nodes and tree nodes
# ---------------------------------------------------------------------------
_RSTAR = np.array([2.0, 3.0, 4.0, 5.0, 7.5, 10.0, 20.0, 40.0, 80.0, 160.0, 320.0, 640.0])
_GOLD = 2.1180339887498949


def _law(lod):
    t3 = lod ** A_EXP
    return t3 + ALPHA ** B_EXP * t3 * lod ** (B_EXP - A_EXP)


def _unique(pts):
    """First occurrence and index of the unique points, in (z, y, x) order."""
    _, first, inv = np.unique(np.round(pts * 1e10).astype(np.int64), axis=0, return_index=True, return_inverse=True)
    order = np.lexsort(pts[first].T)
    rank = np.empty_like(order)
    rank[order] = np.arange(len(order))
    return first[order], rank[inv.ravel()]


def _kd_tree(x):
    """Preorder kd tree: tree order of the points and per node l, u, right child (0 for a leaf)."""
    cols, ind, nodes = x.T.tolist(), list(range(len(x))), []

    def build(lo, hi):
        me = len(nodes)
        nodes.append([lo, hi, 0])
        if hi - lo <= BUCKET:
            return me
        sample = x[ind[lo:min(hi, lo + 200) + 1]]
        v = cols[int(np.argmax(sample.max(0) - sample.min(0)))]
        k, l, u = (lo + hi) // 2, lo, hi
        while l < u:
            pivot, m = v[ind[l]], l
            for i in range(l + 1, u + 1):
                if v[ind[i]] < pivot:
                    m += 1
                    ind[m], ind[i] = ind[i], ind[m]
            ind[l], ind[m] = ind[m], ind[l]
            l, u = (m + 1 if m <= k else l), (m - 1 if m >= k else u)
        build(lo, k)
        nodes[me][2] = build(k + 1, hi)
        return me

    build(0, len(x) - 1)
    return np.array(ind), np.array(nodes)


def _faces(xu, quads):
    """Area and unit normal of each quad, from the four triangles about its centre."""
    p = xu[quads]
    r = p - p.mean(1, keepdim=True)
    c = torch.linalg.cross(r, torch.roll(r, -1, 1))
    cn = torch.sqrt((c * c).sum(-1) + 1e-15)
    n = (c / cn[..., None]).sum(1)
    return 0.5 * cn.sum(1), n / torch.sqrt((n * n).sum(-1, keepdim=True))


def _node_normals(xu, quads):
    area, n = _faces(xu, quads)
    da = (area / 4)[:, None].expand(-1, 4).reshape(-1)
    total = torch.zeros(len(xu), dtype=xu.dtype, device=xu.device).index_add(0, quads.reshape(-1), da)
    sums = torch.zeros_like(xu).index_add(0, quads.reshape(-1), da[:, None] * n.repeat_interleave(4, 0))
    return sums / total[:, None], total


def _motions(t, xu):
    """Rotation and translation (M, b) of every surface node; no derivative through undefined axes."""
    n, _ = _node_normals(xu, t["quads"])
    n0 = t["n0"]
    mag = [torch.sqrt((v * v).sum(-1, keepdim=True) + 1e-30) for v in (n0, n)]
    axis = torch.linalg.cross(n0, n)
    am = torch.sqrt((axis * axis).sum(-1, keepdim=True) + 1e-30)
    d = (n0 / mag[0] * (n / mag[1])).sum(-1, keepdim=True)
    turn = (am >= 1.4901161193847656e-08) & (d < 1.0) & ~t["corner"][:, None]
    ex = torch.tensor([1.0, 0.0, 0.0], dtype=xu.dtype, device=xu.device).expand_as(axis)
    a = torch.where(turn, axis / torch.where(turn, am, torch.ones_like(am)), ex)
    ang = torch.where(turn, torch.acos(torch.where(turn, d, torch.zeros_like(d))), torch.zeros_like(d))[..., None]
    z = torch.zeros_like(a[:, 0])
    K = torch.stack([z, -a[:, 2], a[:, 1], a[:, 2], z, -a[:, 0], -a[:, 1], a[:, 0], z], -1).reshape(-1, 3, 3)
    M = torch.eye(3, dtype=xu.dtype, device=xu.device) + torch.sin(ang) * K + (1 - torch.cos(ang)) * (K @ K)
    return M, xu - (M @ t["x"][..., None])[..., 0]


def _surface_tree(pts, conn, dev):
    """The surface definition in tree order: points, areas, normals, corners, kd tree and error tables."""
    first, link = _unique(pts)
    order, nodes = _kd_tree(pts[first])
    inv = np.empty_like(order)
    inv[order] = np.arange(len(order))
    t = {"first": torch.from_numpy(first[order]).to(dev), "quads": torch.from_numpy(inv[link[conn.reshape(-1, 4)]]).to(dev)}
    x = t["x"] = torch.from_numpy(np.ascontiguousarray(pts[first][order])).to(dev)
    t["n0"], t["A"] = _node_normals(x, t["quads"])
    dots = (_faces(x, t["quads"])[1][:, None] * t["n0"][t["quads"]]).sum(-1).abs() < math.cos(math.radians(CORNER_DEG))
    t["corner"] = torch.zeros(len(x), dtype=torch.bool, device=dev)
    t["corner"][t["quads"][dots]] = True
    t["L"] = float((x - x.mean(0)).norm(dim=1).max())
    t["l"], t["u"], t["right"] = (torch.from_numpy(nodes[:, k].copy()).to(dev) for k in range(3))
    nn = len(nodes)
    cen, orad, area = torch.zeros((nn, 3), dtype=x.dtype, device=dev), torch.zeros(nn, dtype=x.dtype, device=dev), \
        torch.zeros(nn, dtype=x.dtype, device=dev)
    err = torch.zeros((nn, 12), dtype=x.dtype, device=dev)
    o, p, ip = 1.0, _GOLD, 1.0 / _GOLD
    ball = [(a, b, c) for a in (-o, o) for b in (-o, o) for c in (-o, o)]
    ball += [q for a in (-1, 1) for b in (-1, 1) for q in ((0, a * ip, b * p), (a * ip, b * p, 0), (a * p, 0, b * ip))]
    shells = torch.tensor(_RSTAR[:, None, None] * np.array(ball)[None] / math.sqrt(3.0), device=dev).reshape(-1, 3)
    for q, (lo, hi, right) in enumerate(nodes.tolist()):
        xq, aq = x[lo:hi + 1], t["A"][lo:hi + 1]
        cen[q] = xq.mean(0)
        orad[q] = 1.0 / (xq - cen[q]).norm(dim=1).max()
        area[q] = aq.sum()
        if right:
            v = cen[q] + shells / orad[q]
            e = (_law(t["L"] / torch.cdist(v, xq, compute_mode="donot_use_mm_for_euclid_dist")) @ aq
                 - area[q] * _law(t["L"] / (v - cen[q]).norm(dim=1)))
            err[q] = (e * e).reshape(12, 20).mean(1).sqrt()
    t.update(cen=cen, orad=orad, area=area, err=err)
    return t


def _walk(t, r, tol_den):
    """Yields (is_cluster, volume index, point or tree node, weight). tol_den: errTol times the denominator estimate
    (fast sums), None for the estimate itself (clusters beyond five radii)."""
    eps = 1e-15 if tol_den is not None else 1e-16
    rstar = torch.tensor(_RSTAR, device=r.device)
    vol = torch.arange(len(r), device=r.device)
    node = torch.zeros_like(vol)
    while len(vol):
        leaf = t["right"][node] == 0
        v, q = vol[leaf], node[leaf]
        for k in range(BUCKET + 1):
            has = t["l"][q] + k <= t["u"][q]
            vi, pi = v[has], t["l"][q[has]] + k
            if len(vi):
                d = r[vi] - t["x"][pi]
                yield False, vi, pi, t["A"][pi] * _law(t["L"] / torch.sqrt((d * d).sum(-1) + eps))
        v, q = vol[~leaf], node[~leaf]
        d2 = ((r[v] - t["cen"][q]) ** 2).sum(-1)
        dist = torch.sqrt(d2 + 1e-16 if tol_den is None else d2)
        s = dist * t["orad"][q]
        if tol_den is None:
            far = s > 5.0
        else:
            i = (torch.searchsorted(rstar, s, right=True) - 1).clamp(0, 10)
            f = (s - rstar[i]) / (rstar[i + 1] - rstar[i])
            e = torch.where(s < 640.0, (1 - f) * t["err"][q, i] + f * t["err"][q, i + 1], t["err"][q, 11])
            far = (s >= 2.0) & (e < tol_den[v])
        yield True, v[far], q[far], t["area"][q[far]] * _law(t["L"] / dist[far])
        v, q = v[~far], q[~far]
        vol, node = torch.cat([v, v]), torch.cat([q + 1, t["right"][q]])


def _weights(t, r):
    """Exact mode: the weight of every surface node at every volume node."""
    d = torch.cdist(r, t["x"], compute_mode="donot_use_mm_for_euclid_dist")
    return t["A"] * _law(t["L"] / torch.sqrt(d * d + 1e-15))


def _images(planes):
    """Reflections I - 2 n n' of the mirror images (planes through the origin)."""
    out = [np.eye(3)]
    for _, n in planes or []:
        out += [R @ (np.eye(3) - 2.0 * np.outer(n, n)) for R in out]
    return out


def _members(t):
    """(tree node, point) of every member of every interior node."""
    n = t["u"] - t["l"] + 1
    n = torch.where(t["right"] > 0, n, torch.zeros_like(n))
    q = torch.repeat_interleave(torch.arange(len(n), device=n.device), n)
    at = torch.arange(len(q), device=n.device) - (n.cumsum(0) - n)[q]
    return q, t["l"][q] + at, 1.0 / n[q].double()


def _sums(case, t, xv0, planes, motions, seeds):
    """Numerators of each (M, b) in `motions`, the denominator, the denominator estimate (fast mode), and the adjoint
    (n, 3, 4) of (M, b) of each seed (formed with the denominator of a first pass)."""
    dev, fast = xv0.device, case["evalMode"] == "fast"
    chunk = 1 << 18 if fast else max(1, 40_000_000 // len(t["x"]))
    q, p, w = _members(t)

    def means(a):
        return torch.zeros((len(t["l"]),) + a.shape[1:], dtype=a.dtype, device=dev).index_add(
            0, q, a[p] * w.reshape((-1,) + (1,) * (a.dim() - 1)))

    motions = [torch.cat([M, b[..., None]], 2) for M, b in motions]  # (n, 3, 4), applied to (r, 1)
    clusters = [means(m) for m in motions]
    num = [torch.zeros_like(xv0) for _ in motions]
    den, den0 = torch.zeros(len(xv0), dtype=xv0.dtype, device=dev), torch.zeros(len(xv0), dtype=xv0.dtype, device=dev)
    mats = [torch.from_numpy(R).to(dev) for R in _images(planes)]
    adj = [[torch.zeros((n, 3, 4), dtype=xv0.dtype, device=dev) for n in (len(t["x"]), len(t["l"]))] for _ in seeds]
    for a in range(0, len(xv0), chunk):
        c = slice(a, min(len(xv0), a + chunk))
        images = [xv0[c] @ R.T for R in mats]
        ones = [torch.cat([r, torch.ones_like(r[:, :1])], 1) for r in images]
        if fast:
            for r in images:
                for _, v, _, wt in _walk(t, r, None):
                    den0[c].index_add_(0, v, wt)
        if case["op"] == "setup":
            continue
        for r, r1, R in zip(images, ones, mats):
            if not fast:
                W = _weights(t, r)
                den[c] += W.sum(1)
                for i, m in enumerate(motions):
                    num[i][c] += ((W @ m.reshape(-1, 12)).reshape(-1, 3, 4) @ r1[..., None])[..., 0] @ R
                continue
            for cluster, v, k, wt in _walk(t, r, case["errTol"] * den0[c]):
                den[c].index_add_(0, v, wt)
                for i, m in enumerate(clusters if cluster else motions):
                    num[i][c].index_add_(0, v, wt[:, None] * ((m[k] @ r1[v][..., None])[..., 0] @ R))
        for r, r1, R in zip(images, ones, mats) if seeds else ():
            rows = [(g[c] / den[c, None] @ R.T)[:, :, None] * r1[:, None] for g in seeds]
            if not fast:
                W = _weights(t, r)
                for row, ad in zip(rows, adj):
                    ad[0] += (W.T @ row.reshape(-1, 12)).reshape(-1, 3, 4)
                continue
            for cluster, v, k, wt in _walk(t, r, case["errTol"] * den0[c]):
                for row, ad in zip(rows, adj):
                    ad[int(cluster)].index_add_(0, k, wt[:, None, None] * row[v])
    for pt, cl in adj:
        pt.index_add_(0, p, cl[q] * w[:, None, None])
    return num, den, den0, [pt for pt, _ in adj]


def exact(case, seed):
    nv, ns, loops = _sizes(case)
    seeds_n = case["count"] if case["op"] in ("seeds", "tangent", "surfaces") else 1
    most = 8e9 if case["evalMode"] == "fast" else 5e10
    if case["tree"] != "kd" or ns > 45_000 or _pairs(case) * (1 + seeds_n) > most:
        return None  # the Morton tree is the package's own; the rest would take too long
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    g, xs = _inputs(case, seed)
    xv0, pts = g["xv0"], g["pts"]
    if case["op"] == "setup":
        xv0, pts = _sweep(xv0, seed), _sweep(pts, seed)
    t = _surface_tree(pts, np.asarray(g["conn"]), dev)
    xv0 = torch.from_numpy(np.ascontiguousarray(xv0)).to(dev)
    if case["op"] == "setup":
        return _sums(case, t, xv0, g["symmetryPlanes"], [], [])[2].cpu().numpy()
    xu = [torch.from_numpy(x).to(dev)[t["first"]] for x in (xs if xs.ndim == 3 else xs[None])]
    seeds = []
    if case["op"] == "tangent":
        dirs = _normal((case["count"], ns, 3), seed, dev)[:, t["first"]]
        motions = [torch.func.jvp(lambda x: _motions(t, x), (xu[0],), (d,))[1] for d in dirs]
    else:
        eye = torch.eye(3, dtype=xv0.dtype, device=dev)
        # the displacement's motion, S = (M - I) r + b
        motions = [(M - eye, b) for M, b in (_motions(t, x) for x in xu)]
    if case["op"] in ("gradient", "seeds"):
        seeds = list(_normal((nv, 3), seed, dev)[None] if case["op"] == "gradient"
                     else _normal((case["count"], nv, 3), seed, dev))
    num, den, _, adj = _sums(case, t, xv0, g["symmetryPlanes"], motions, seeds)
    moved = [n / den[:, None] for n in num]
    if case["op"] == "tangent":
        return torch.stack(moved)
    grids = [xv0 + m for m in moved]
    if case["op"] == "step":
        return grids[0].reshape(-1).cpu().numpy()
    if not seeds:
        return torch.stack(grids) if case["op"] == "surfaces" else grids[0]
    x = xu[0].clone().requires_grad_(True)
    M, b = _motions(t, x)
    out = []
    for a in adj:
        d = torch.autograd.grad((M * a[..., :3]).sum() + (b * a[..., 3]).sum(), x, retain_graph=True)[0]
        out.append(torch.zeros((ns, 3), dtype=d.dtype, device=dev).index_copy(0, t["first"], d))
    return (grids[0], out[0]) if case["op"] == "gradient" else torch.stack(out)
