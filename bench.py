"""Benchmark: IDW volume-mesh warping on a GB300.

Headline metric: volume nodes warped per second by the mixed-precision fast
(tree) warpMesh, on the 8M-volume-node / 150k-surface-node NACA0012 half-wing
shell mesh with a symmetry plane (seeded synthetic inputs; twist + FFD
surface perturbation), errTol 1e-4.  One step = setSurfaceCoordinates +
warpMesh over the whole mesh.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl gb300|reference]

`value` is timed with CUDA events on the library's stream with the inputs
resident in HBM; `e2e` runs the same step through the public USMesh API with
host arrays (surface in, warped grid out) inside the timed region.  The
`--impl reference` arm times the CPU restatement of the reference algorithm
(the oracle; the Fortran reference cannot be built here) on the host cores.
"""
import argparse
import contextlib
import ctypes as C
import io
import json
import os
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

CONFIGS = {
    # name: (ni, nj, nk) of the wing shell mesh
    "P": (577, 261, 53),   # ~8.0M volume nodes, ~150k surface nodes
    "W": (401, 101, 50),   # ~2.0M volume nodes, ~40k surface nodes
    "S": (101, 33, 20),    # small (tests / quick checks)
}
ERR_TOL = 1e-4


def _env_int(k, d):
    try:
        return int(os.environ.get(k, d))
    except ValueError:
        return d


def make_workload(cfg, seed=2):
    from idwarp_gb300 import synthetic as S

    ni, nj, nk = CONFIGS[cfg]
    m = S.wing_shell(ni, nj, nk, first=1e-5, far=25.0)
    m["xs"] = S.wing_perturbation(m["pts"], seed=seed)
    return m


WALK_LISTS = "auto"  # --walk-lists: "off" makes every walk decide as it goes
TREE_BUILD = "kd"  # --tree-build: "morton" builds the surface tree on the GPU
DETERMINISTIC = False  # --deterministic: reverse products with order-independent sums


def mesh_options(m, precision, mode="fast", tree=None):
    return {"fileType": "NPY", "precision": precision, "evalMode": mode, "errTol": ERR_TOL,
            "aExp": 3.0, "bExp": 5.0, "LdefFact": 1.0, "alpha": 0.25, "bucketSize": 8,
            "symmetryPlanes": m["symmetryPlanes"], "walkLists": WALK_LISTS, "treeBuild": tree or TREE_BUILD,
            "deterministic": DETERMINISTIC}


def build_mesh(m, precision, mode="fast", restartFile=None, tree=None):
    from idwarp_gb300 import USMesh

    o = dict(mesh_options(m, precision, mode, tree))
    if restartFile:
        o["restartFile"] = restartFile
    with contextlib.redirect_stdout(io.StringIO()):
        mesh = USMesh(options=o)
        mesh.createCommonGrid(m["xv0"])
        mesh.setSurfaceDefinition(m["pts"], m["conn"], m["faceSizes"])
    return mesh


class ClockSampler:
    """nvidia-smi clock/throttle sampling during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index):
        self.gpu = gpu_index
        self.proc = None
        self.lines = []

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.gpu), "--query-gpu=" + self.FIELDS, "--format=csv,noheader,nounits",
                 "-lms", "100"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.thread = threading.Thread(target=self._read, daemon=True)
            self.thread.start()
        except Exception:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        time.sleep(0.25)
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        sm, smax, reasons = [], None, set()
        names = ["active", "hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            parts = [p.strip() for p in ln.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                smax = float(parts[2])
            except ValueError:
                continue
            for nm, val in zip(names[1:], parts[5:9]):
                if val.lower() == "active":
                    reasons.add(nm)
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": smax, "samples": len(sm),
                "reasons": sorted(reasons)}


def _measured_peak(key):
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            return json.load(f).get(key)
    except Exception:
        return None


def fp32_peak_tflops():
    """Measured FFMA issue peak of this GPU (TFLOP/s) from a dependent-chain-free FMA probe."""
    import torch

    from idwarp_gb300 import _lib

    L = _lib.load()
    f = getattr(L, "idw_probe_ffma", None)
    if f is None:
        return None
    f.argtypes = [C.c_void_p, C.c_int, C.POINTER(C.c_double)]
    f.restype = C.c_int
    stream = torch.cuda.current_stream().cuda_stream
    out = C.c_double(0.0)
    best = 0.0
    for _ in range(3):
        if f(C.c_void_p(stream), 0, C.byref(out)) == 0:
            best = max(best, out.value)
    return best if best > 0 else None


def cpu_info():
    """CPU model and core counts of this host, recorded beside the CPU numbers."""
    model = None
    try:
        out = subprocess.run(["lscpu"], capture_output=True, text=True, timeout=10).stdout
        for ln in out.splitlines():
            if ln.startswith("Model name:"):
                model = ln.split(":", 1)[1].strip()
                break
    except Exception:
        pass
    if not model:
        try:
            with open("/proc/cpuinfo") as f:
                for ln in f:
                    if ln.lower().startswith(("model name", "cpu part")):
                        model = ln.split(":", 1)[1].strip()
                        break
        except Exception:
            pass
    try:
        usable = len(os.sched_getaffinity(0))
    except Exception:
        usable = os.cpu_count()
    return {"cpu_model": model, "nproc": os.cpu_count(), "usable_cores": usable, "machine": os.uname().machine}


def workload_config(cfg, m, mode, nunique, world):
    """The `config` object of both arms' JSON lines (the same dict, so the two
    lines name the same workload)."""
    nvol = len(m["xv0"])
    return {"workload": "wing_shell_%dx%dx%d" % CONFIGS[cfg], "volume_nodes": nvol, "surface_points": len(m["pts"]),
            "unique_surface_nodes": int(nunique), "errTol": ERR_TOL, "mode": mode,
            "symmetry_planes": len(m["symmetryPlanes"]), "surface_tree": TREE_BUILD,
            "parallelism": "replicas" if world > 1 else "single",
            "l2": "inputs %s L2 (Xv0+Xv+den0+den ~%.0f MB per step)" % (
                "larger than" if nvol * 64 > 129e6 else "fit in", nvol * 64 / 1e6)}


class OracleSample:
    """The oracle (CPU restatement of the reference) set up on a seeded sample
    of the workload's volume nodes: the volume nodes are independent given
    the surface, so a sample is a bounded piece of the same work."""

    def __init__(self, m, idx, library=None, mode="fast", tree="kd"):
        from oracle.pyoracle import OracleMesh

        o = dict(mesh_options(m, "fp64", mode, tree))
        self.idx = idx
        self.om = OracleMesh({k: o[k] for k in ("aExp", "bExp", "LdefFact", "alpha", "errTol", "evalMode",
                                                "bucketSize", "treeBuild")}, library=library)
        self.om.set_volume(m["xv0"][idx])
        planes = m["symmetryPlanes"]
        self.om.set_symmetry(np.array([p[0] for p in planes]).reshape(-1, 3),
                             np.array([p[1] for p in planes]).reshape(-1, 3))
        self.om.set_surface_definition(m["pts"], m["conn"], m["faceSizes"])
        self.xs = m["xs"]

    def step(self):
        """One step of the CPU path: surface coordinates in, the sample warped."""
        self.om.set_surface_coordinates(self.xs)
        return self.om.warp()


def run_cpu_baseline(m, budget_s=10.0, seed=0):
    """The oracle's timing build (-O3, tuned for this CPU, OpenMP on every
    usable core) warping a seeded sample of the workload's volume nodes sized
    to about budget_s, plus the same on one core over a smaller sample.
    Returns the JSON object and the sample (indices, warped nodes) that the
    parity check reuses with the checker build."""
    from oracle.build import timing_flags
    from oracle.pyoracle import max_threads, set_threads, timing_library

    L = timing_library()
    nthr = max_threads(L)
    rng = np.random.default_rng(seed)
    nvol = len(m["xv0"])
    # calibrate on 20k nodes (after one run that starts the thread pool)
    idx = np.sort(rng.choice(nvol, min(nvol, 20000), replace=False))
    s = OracleSample(m, idx, L)
    s.step()
    t0 = time.perf_counter()
    s.step()
    rate = len(idx) / (time.perf_counter() - t0)
    n = int(min(nvol, max(20000, rate * budget_s)))
    idx = np.sort(rng.choice(nvol, n, replace=False))
    s = OracleSample(m, idx, L)
    t0 = time.perf_counter()
    xv = s.step()
    dt = time.perf_counter() - t0
    # one core, about budget_s / 3 of work
    n1 = int(min(n, max(2000, rate / max(nthr, 1) * budget_s / 3)))
    s1 = OracleSample(m, idx[:n1], L)
    set_threads(1, L)
    t0 = time.perf_counter()
    s1.step()
    dt1 = time.perf_counter() - t0
    set_threads(nthr, L)
    del s1
    line = {"value": n / dt, "unit": "volume nodes/s", "cores": nthr, "kind": "port",
            "sample": "%d of %d volume nodes (seeded uniform sample), fast mode errTol %g, FP64, %.2f s per step "
                      "(setSurfaceCoordinates + warpMesh)" % (n, nvol, ERR_TOL, dt),
            "value_1core": n1 / dt1, "sample_1core": "%d nodes, %.2f s" % (n1, dt1),
            "build": "oracle/idw_oracle.cpp timing build: g++ " + timing_flags()}
    line.update(cpu_info())
    return line, idx, xv


def run_parity(m, idx, xv_timing, grids, gpu_stats_fn):
    """The GPU path against the oracle at this workload: the oracle's checker
    build (no FMA contraction) warps the sampled volume nodes; the GPU grids
    of the whole mesh are compared at the same nodes, and GPU meshes of just
    the sampled nodes give the GPU's decision counts for the same nodes.
    The timing build's difference from the checker is the case's rounding
    sensitivity (different rounding order of the same formulas)."""
    s = OracleSample(m, idx, tree=TREE_BUILD)
    xo = s.step()
    ost = s.om.stats()
    L = s.om.ldef0()
    # the timing build runs the reference's kd tree: a rounding comparison only on that tree
    sens = float(np.abs(xv_timing - xo).max() / L) if TREE_BUILD == "kd" else 0.0
    out = {"n_nodes": int(len(idx)), "sample": "the CPU baseline's sample", "Ldef": L, "surface_tree": TREE_BUILD,
           "oracle": {"leafPairs": ost["leafPairs"], "approx": ost["approx"]},
           "rounding_sensitivity_over_Ldef": sens if TREE_BUILD == "kd" else None}
    del s
    ok = True
    for prec, bar in (("mixed", 1e-8), ("fp64", 1e-12)):
        st = gpu_stats_fn(prec, idx)
        res = {"leafPairs": st["leafPairs"], "approx": st["approx"],
               "leafPairs_equal": st["leafPairs"] == ost["leafPairs"], "approx_equal": st["approx"] == ost["approx"],
               "bar_over_Ldef": max(bar, 4 * sens)}
        e = np.abs(st["xv"] - xo).max(axis=1) / L
        res["sample_mesh_max_err_over_Ldef"] = float(e.max())
        res["sample_mesh_rms_err_over_Ldef"] = float(np.sqrt(np.mean(e ** 2)))
        g = grids.get(prec)
        if g is not None:
            e = np.abs(g[idx] - xo).max(axis=1) / L
            res["max_err_over_Ldef"] = float(e.max())
            res["rms_err_over_Ldef"] = float(np.sqrt(np.mean(e ** 2)))
        worst = max(res["sample_mesh_max_err_over_Ldef"], res.get("max_err_over_Ldef", 0.0))
        res["pass"] = bool(res["leafPairs_equal"] and res["approx_equal"] and worst <= res["bar_over_Ldef"])
        ok = ok and res["pass"]
        out[prec] = res
    out["pass"] = ok
    return out


def replica_throughput(ms_step, units_per_rank, world, device):
    """Whole-job throughput of ``world`` replicas that each processed
    ``units_per_rank`` units per step: the step time is the maximum over the
    ranks (all-reduce MAX when a process group is up).  Returns (max ms, units/s)."""
    import torch

    t = torch.tensor([float(ms_step)], dtype=torch.float64, device=device)
    if world > 1:
        torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MAX)
    ms_max = float(t.item())
    return ms_max, world * units_per_rank / (ms_max * 1e-3)


def _timed(fn, reps, stream):
    import torch

    fn()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(reps):
        fn()
    e1.record(stream)
    torch.cuda.synchronize()
    return e0.elapsed_time(e1) / reps


def run_suite():
    """The measurement table: S1 sphere, W wing, P wing errTol sweep; one JSON line per row.

    Per row: GPU mixed and FP64 times (CUDA events on the library's stream,
    device-resident surface), the precision error of the mixed form against
    FP64 on the same tree and decisions, the algorithmic error of fast against
    exact mode, and the oracle on the host cores (all threads, and one) on a
    seeded sample of volume nodes."""
    import torch

    from idwarp_gb300 import _lib
    from idwarp_gb300 import synthetic as S
    from oracle.pyoracle import OracleMesh, max_threads, set_threads

    stream = torch.cuda.current_stream()
    nthreads = max_threads()

    def gpu_mesh(m, prec, mode, errTol):
        o = mesh_options(m, prec, mode)
        o["errTol"] = errTol
        with contextlib.redirect_stdout(io.StringIO()):
            g = USMesh_(o)
            g.createCommonGrid(m["xv0"])
            g.setSurfaceDefinition(m["pts"], m["conn"], m["faceSizes"])
        g.lib.idw_set_stream(g.ctx, C.c_void_p(stream.cuda_stream))
        return g

    def cpu_rate(m, mode, errTol, threads, budget):
        set_threads(threads)
        rng = np.random.default_rng(7)
        nvol = len(m["xv0"])
        n = min(nvol, 2000 if mode == "exact" else 20000)
        for attempt in range(2):
            idx = np.sort(rng.choice(nvol, n, replace=False))
            o = dict(mesh_options(m, "fp64", mode))
            o["errTol"] = errTol
            om = OracleMesh({k: o[k] for k in ("aExp", "bExp", "LdefFact", "alpha", "errTol", "evalMode", "bucketSize")})
            om.set_volume(m["xv0"][idx])
            if m.get("symmetryPlanes"):
                planes = m["symmetryPlanes"]
                om.set_symmetry(np.array([p[0] for p in planes]), np.array([p[1] for p in planes]))
            om.set_surface_definition(m["pts"], m["conn"], m["faceSizes"])
            om.set_surface_coordinates(m["xs"])
            t0 = time.perf_counter()
            om.warp()
            dt = time.perf_counter() - t0
            if attempt == 0 and dt < budget and n < nvol:
                n = int(min(nvol, n * budget / max(dt, 1e-3)))
                continue
            break
        set_threads(nthreads)
        return n / dt, n

    from idwarp_gb300 import USMesh as USMesh_

    sph = S.sphere_ogrid(n=18, layers=48)
    sph["xs"] = S.sphere_perturbation(sph["pts"], seed=0)
    rows = [("S1_sphere_95k", sph, [1e-4]), ("W_wing_2M", make_workload("W"), [1e-4]),
            ("P_wing_8M", make_workload("P"), [1e-3, 1e-4, 1e-5])]
    for name, m, tols in rows:
        nvol = len(m["xv0"])
        for errTol in tols:
            res = {"row": name, "volume_nodes": nvol, "surface_points": len(m["pts"]), "errTol": errTol}
            xs_dev = torch.tensor(m["xs"], dtype=torch.float64, device="cuda")
            grids = {}
            # exact mode does not depend on errTol: once per mesh
            modes = ["fast", "exact"] if (name != "P_wing_8M" or errTol == 1e-4) else ["fast"]
            for mode in modes:
                for prec in ("mixed", "fp64"):
                    if prec == "fp64" and mode == "exact" and nvol > 3e5:
                        continue  # minutes of FP64 pairs; the mixed exact result stands in
                    g = gpu_mesh(m, prec, mode, errTol)

                    def step(g=g):
                        g.lib.idw_set_surface_coordinates(g.ctx, C.c_void_p(xs_dev.data_ptr()), xs_dev.numel(),
                                                          _lib.IDW_DEVICE)
                        g.lib.idw_warp_mesh(g.ctx)

                    ms = _timed(step, 2 if (prec == "fp64" or mode == "exact") else 5, stream)
                    grids[(mode, prec)] = g.getWarpGrid().reshape(-1, 3)
                    st = g.getStats()
                    res["%s_%s_ms" % (mode, prec)] = ms
                    res["%s_%s_nodes_per_s" % (mode, prec)] = nvol / (ms * 1e-3)
                    res["%s_PI" % mode] = st["leafPairs"] + st["approx"]
                    if errTol == 1e-4 and name != "P_wing_8M" and (mode == "fast" or prec == "mixed"):
                        rng = np.random.default_rng(1)
                        seed = torch.tensor(rng.normal(size=3 * nvol), device="cuda")
                        dxs = torch.empty(3 * len(m["pts"]), dtype=torch.float64, device="cuda")

                        def deriv(g=g):
                            g.lib.idw_warp_deriv_batch(g.ctx, C.c_void_p(seed.data_ptr()), 1, C.c_void_p(dxs.data_ptr()),
                                                       _lib.IDW_DEVICE)

                        res["warpDeriv1_%s_%s_ms" % (mode, prec)] = _timed(deriv, 2, stream)
                    del g
                Ldef = None
            # precision error (same tree, same decisions) and algorithmic error
            ref = grids[("fast", "fp64")]
            gL = gpu_mesh(m, "fp64", "fast", errTol)
            Ldef = gL.getStats()["Ldef0"]
            del gL
            e = np.abs(grids[("fast", "mixed")] - ref).max(axis=1) / Ldef
            res["fast_mixed_vs_fp64_max_over_Ldef"] = float(e.max())
            res["fast_mixed_vs_fp64_rms_over_Ldef"] = float(np.sqrt(np.mean(e ** 2)))
            if ("exact", "fp64") in grids:
                e = np.abs(grids[("exact", "mixed")] - grids[("exact", "fp64")]).max(axis=1) / Ldef
                res["exact_mixed_vs_fp64_max_over_Ldef"] = float(e.max())
                exact_ref = grids[("exact", "fp64")]
            elif ("exact", "mixed") in grids:
                exact_ref = grids[("exact", "mixed")]
            else:
                exact_ref = None
            if exact_ref is not None:
                res["fast_fp64_vs_exact_max_over_Ldef"] = float((np.abs(ref - exact_ref).max(axis=1) / Ldef).max())
            # against the FP64 exact oracle (the reference's exact mode) on a
            # seeded sample of volume nodes, about 1e9 pair evaluations
            st0 = gpu_mesh(m, "mixed", "fast", errTol)
            nloop, nuniq = st0.getStats()["nLoop"], st0.getStats()["nUnique"]
            del st0
            nsamp = int(min(nvol, max(500, 1e9 / (nloop * nuniq))))
            idx = np.sort(np.random.default_rng(11).choice(nvol, nsamp, replace=False))
            o = dict(mesh_options(m, "fp64", "exact"))
            om = OracleMesh({k: o[k] for k in ("aExp", "bExp", "LdefFact", "alpha", "errTol", "evalMode", "bucketSize")})
            om.set_volume(m["xv0"][idx])
            if m.get("symmetryPlanes"):
                planes = m["symmetryPlanes"]
                om.set_symmetry(np.array([p[0] for p in planes]), np.array([p[1] for p in planes]))
            om.set_surface_definition(m["pts"], m["conn"], m["faceSizes"])
            om.set_surface_coordinates(m["xs"])
            xo = om.warp()
            res["oracle_exact_sample_nodes"] = nsamp
            for (mode, prec), grid in grids.items():
                e = np.abs(grid[idx] - xo).max(axis=1) / Ldef
                res["%s_%s_vs_oracle_exact_max_over_Ldef" % (mode, prec)] = float(e.max())
                res["%s_%s_vs_oracle_exact_rms_over_Ldef" % (mode, prec)] = float(np.sqrt(np.mean(e ** 2)))
            del om
            # the oracle on the host cores
            budget = 6.0
            r_all, n_all = cpu_rate(m, "fast", errTol, nthreads, budget)
            r_one, n_one = cpu_rate(m, "fast", errTol, 1, budget / 2)
            res["cpu_fast_nodes_per_s_all_cores"] = r_all
            res["cpu_fast_nodes_per_s_1_core"] = r_one
            res["cpu_cores"] = nthreads
            res["cpu_sample_nodes"] = [n_all, n_one]
            print(json.dumps(res), flush=True)
            del grids
    return 0


def run_suite_tree():
    """Error report of the Morton tree (treeBuild "morton", built on the GPU)
    against the reference kd tree, one JSON line per mesh and errTol: set-up
    and tree build times, tree shape, the mixed fast walk (first warp, which
    records its decisions, and the replayed steady state), its work, and its
    error against mixed exact mode (max and RMS of |dx| / Ldef0 over every
    volume node)."""
    import torch

    from idwarp_gb300 import USMesh
    from idwarp_gb300 import _lib
    from idwarp_gb300 import synthetic as S

    stream = torch.cuda.current_stream()

    def gpu_mesh(m, mode, errTol, tree):
        o = mesh_options(m, "mixed", mode, tree)
        o["errTol"] = errTol
        t0 = time.perf_counter()
        with contextlib.redirect_stdout(io.StringIO()):
            g = USMesh(o)
            g.createCommonGrid(m["xv0"])
            g.setSurfaceDefinition(m["pts"], m["conn"], m["faceSizes"])
        torch.cuda.synchronize()
        setup = time.perf_counter() - t0
        g.lib.idw_set_stream(g.ctx, C.c_void_p(stream.cuda_stream))
        return g, setup

    sph = S.sphere_ogrid(n=18, layers=48)
    sph["xs"] = S.sphere_perturbation(sph["pts"], seed=0)
    rows = [("S1_sphere_95k", sph, [1e-4]), ("W_wing_2M", make_workload("W"), [1e-3, 1e-4, 1e-5]),
            ("P_wing_8M", make_workload("P"), [1e-4])]
    for name, m, tols in rows:
        nvol = len(m["xv0"])
        xs_dev = torch.tensor(m["xs"], dtype=torch.float64, device="cuda")

        def step(g):
            g.lib.idw_set_surface_coordinates(g.ctx, C.c_void_p(xs_dev.data_ptr()), xs_dev.numel(), _lib.IDW_DEVICE)
            g.lib.idw_warp_mesh(g.ctx)

        ge, _ = gpu_mesh(m, "exact", 1e-4, "kd")
        exact_ms = _timed(lambda: step(ge), 1, stream)
        xe = ge.getWarpGrid().reshape(-1, 3).copy()
        L = ge.getStats()["Ldef0"]
        del ge
        for errTol in tols:
            res = {"row": name, "volume_nodes": nvol, "surface_points": len(m["pts"]), "errTol": errTol,
                   "exact_mixed_ms": exact_ms}
            for tree in ("kd", "morton"):
                g, setup = gpu_mesh(m, "fast", errTol, tree)
                st = g.getStats()
                t = g.getTree()
                torch.cuda.synchronize()
                t0 = time.perf_counter()
                step(g)
                torch.cuda.synchronize()
                first = time.perf_counter() - t0
                ms = _timed(lambda: step(g), 5, stream)
                st2 = g.getStats()
                e = np.abs(g.getWarpGrid().reshape(-1, 3) - xe).max(axis=1) / L
                res.update({
                    "%s_setup_s" % tree: setup, "%s_tree_build_ms" % tree: st["treeBuildMs"],
                    "%s_tree_nodes" % tree: int(st["nTreeNodes"]), "%s_leaves" % tree: int(t["isLeaf"].sum()),
                    "%s_max_depth" % tree: int(st["maxDepth"]), "%s_first_warp_ms" % tree: 1e3 * first,
                    "%s_warp_ms" % tree: ms, "%s_nodes_per_s" % tree: nvol / (ms * 1e-3),
                    "%s_leafPairs_per_node" % tree: st2["leafPairs"] / nvol,
                    "%s_approx_per_node" % tree: st2["approx"] / nvol,
                    "%s_vs_exact_max_over_Ldef" % tree: float(e.max()),
                    "%s_vs_exact_rms_over_Ldef" % tree: float(np.sqrt(np.mean(e ** 2)))})
                del g
            print(json.dumps(res), flush=True)
    return 0


def run_suite_d(steps=50, sample=200000, directions=5):
    """Differentiation at scale: the two-body mesh (wing 577x261x53 + sphere
    158x79: 19.96M volume nodes, 302k surface points), 50 Adam steps on 48
    FFD coefficients minimising sum(1/max(V_cell, eps)) through the
    differentiable warp (mixed precision).  Gradient checks:
      * central differences (h = 1e-6) on 5 random directions at the
        undeformed surface, with the reference's rotation derivative (zero on
        the degenerate rotation axes of an undeformed surface) and with
        rotations off;
      * the same at the deformed surface after the loop, where every wing
        node's rotation axis is well defined;
      * the GPU's reverse product against the oracle's (the reference's
        warpDeriv restated, FP64) at the deformed surface: dXv = the
        objective's gradient restricted to a seeded sample of volume nodes
        (dXs is linear in dXv, so the sample's product is exact for that
        dXv), compared over all surface points and along 5 random FFD
        directions."""
    import torch

    from idwarp_gb300 import USMesh
    from idwarp_gb300 import synthetic as S
    from idwarp_gb300.autograd import warp
    from idwarp_gb300.ffd import FFDBox, ffd_loop, inverse_volume_objective

    t0 = time.perf_counter()
    m = S.multibody()
    gen_s = time.perf_counter() - t0
    res = {"row": "D_multibody_20M", "volume_nodes": len(m["xv0"]), "surface_points": len(m["pts"]),
           "cells": len(m["cells"]), "ffd_vars": 48, "steps": steps, "generate_s": gen_s}
    o = mesh_options(m, "mixed")
    t0 = time.perf_counter()
    with contextlib.redirect_stdout(io.StringIO()):
        g = USMesh(options=o)
        g.createCommonGrid(m["xv0"])
        g.setSurfaceDefinition(m["pts"], m["conn"], m["faceSizes"])
    torch.cuda.synchronize()
    res["setup_s"] = time.perf_counter() - t0
    ffd = FFDBox(m["pts"], select=np.arange(m["nWingPts"]))
    xs0 = torch.tensor(m["pts"], device="cuda")
    cells = torch.tensor(m["cells"], device="cuda")
    out = ffd_loop(g, xs0, cells, ffd, steps=steps, lr=1e-3, check_directions=directions)
    res.update({"objective_initial": out["initial"], "objective_final": out["objective"][-1],
                "seconds": out["seconds"], "seconds_per_step": out["seconds_per_step"],
                "gradient_check_rotations": out["gradient_check"]})
    coef = torch.tensor(out["coef"], device="cuda")
    res["coef_max_abs"] = float(coef.abs().max())
    # FD at the deformed state (rotations on), starting the check there, with
    # the differences of the FP64 form (the mixed forward's rounding is of the
    # order of a 1e-6 step's effect)
    o64 = mesh_options(m, "fp64")
    with contextlib.redirect_stdout(io.StringIO()):
        g64 = USMesh(options=o64)
        g64.createCommonGrid(m["xv0"])
        g64.setSurfaceDefinition(m["pts"], m["conn"], m["faceSizes"])
    chk = ffd_loop(g, xs0, cells, ffd, steps=0, check_directions=directions, coef0=coef, fd_mesh=g64)
    res["gradient_check_rotations_deformed_fd64"] = chk["gradient_check"]
    # the same with the gradient of the FP64 form too (FP64 forward and
    # adjoint): the derivative itself, without the mixed forward's rounding
    # in the objective's 1/V of the wall cells
    chk = ffd_loop(g64, xs0, cells, ffd, steps=0, check_directions=directions, coef0=coef)
    res["gradient_check_rotations_deformed_fp64"] = chk["gradient_check"]
    chk = ffd_loop(g, xs0, cells, ffd, steps=0, check_directions=directions, coef0=coef)
    res["gradient_check_rotations_deformed"] = chk["gradient_check"]
    del g64
    g.setOption("useRotations", False)
    out2 = ffd_loop(g, xs0, cells, ffd, steps=0, check_directions=directions)
    res["gradient_check_no_rotations"] = out2["gradient_check"]
    g.setOption("useRotations", True)
    # the reverse product against the oracle on a volume sample, at the deformed state
    B, sel = ffd.torch_operator(xs0.device)
    xs = ffd.apply(xs0, coef, B, sel).detach()
    xv = warp(xs, g).detach().requires_grad_(True)
    f = inverse_volume_objective(xv, cells, 1e-12)
    (gxv,) = torch.autograd.grad(f, xv)
    rng = np.random.default_rng(301)
    idx = np.sort(rng.choice(len(m["xv0"]), min(sample, len(m["xv0"])), replace=False))
    gs = np.zeros(gxv.shape)
    gs[idx] = gxv.cpu().numpy()[idx]
    g.setSurfaceCoordinates(xs)
    g.warpMesh()
    g.warpDeriv(torch.tensor(gs.ravel(), device="cuda"), solverVec=False)
    dxs_gpu = g.getdXs()
    t0 = time.perf_counter()
    smp = dict(m)
    smp["xs"] = xs.cpu().numpy()
    ors = OracleSample(smp, idx, tree=TREE_BUILD)
    ors.step()
    dxs_or = ors.om.warp_deriv(gs[idx])
    res["oracle_seconds"] = time.perf_counter() - t0
    scale = float(np.abs(dxs_or).max())
    dirs = []
    Bn = B.cpu().numpy()
    for _ in range(directions):
        d = rng.normal(size=ffd.nVars)
        v = np.zeros(m["pts"].shape)
        v[ffd.sel, 2] = Bn @ d
        a, b = float(np.sum(dxs_gpu * v)), float(np.sum(dxs_or * v))
        dirs.append({"gpu": a, "oracle": b, "rel": abs(a - b) / max(abs(b), 1e-300)})
    res["adjoint_vs_oracle"] = {"sample_nodes": int(len(idx)), "max_rel_over_max_dXs":
                                float(np.abs(dxs_gpu - dxs_or).max() / scale), "directions": dirs}
    res["peak_memory_GB"] = torch.cuda.max_memory_allocated() / 1e9
    print(json.dumps(res), flush=True)
    return 0


def run_case(case, cfg, reps):
    """One operation on a config's mesh, repeated: the small cases the ncu
    captures profile (warp: warpMesh; deriv1: warpDeriv of one seed, double-float
    form; deriv1fast: the FP32 form; deriv16 / deriv16fast: 16 seeds in one
    call; batch: 8 surfaces through warpMeshBatch; setup: the surface
    definition, tree included, with the tree of --tree-build)."""
    import torch

    from idwarp_gb300 import _lib
    from idwarp_gb300 import synthetic as S

    m = make_workload(cfg)
    if case == "setup":
        out = []
        for _ in range(reps):
            t0 = time.perf_counter()
            mesh = build_mesh(m, "mixed")
            torch.cuda.synchronize()
            out.append({"setup_s": time.perf_counter() - t0, "treeBuildMs": mesh.getStats()["treeBuildMs"]})
            del mesh
        print(json.dumps({"case": case, "config": cfg, "reps": reps, "tree": TREE_BUILD, "runs": out}))
        return 0
    mesh = build_mesh(m, "mixed")
    L = mesh.lib
    L.idw_set_stream(mesh.ctx, C.c_void_p(torch.cuda.current_stream().cuda_stream))
    mesh.setSurfaceCoordinates(m["xs"])
    mesh.warpMesh()
    nvol = len(m["xv0"])
    if case.startswith("deriv"):
        if case.endswith("fast"):
            mesh.setOption("adjointPrecision", "fast")
            mesh._setMeshOptions()
        ns = 16 if case.startswith("deriv16") else 1
        sd = torch.tensor(np.random.default_rng(100).normal(size=(ns, nvol, 3)), device="cuda")
        npts = len(m["xs"])
        out = torch.zeros((ns, npts, 3), dtype=torch.float64, device="cuda")

        def deriv():
            if ns == 1:
                rc = L.idw_warp_deriv(mesh.ctx, C.c_void_p(sd.data_ptr()), 3 * nvol, _lib.IDW_DEVICE)
            else:
                rc = L.idw_warp_deriv_batch(mesh.ctx, C.c_void_p(sd.data_ptr()), ns, C.c_void_p(out.data_ptr()),
                                            _lib.IDW_DEVICE)
            _lib.check(L, mesh.ctx, rc, "warpDeriv")
            return (mesh.getdXs().copy() if ns == 1 else out.cpu().numpy().copy())

        stream = torch.cuda.current_stream()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        first = deriv()
        torch.cuda.synchronize()
        e0.record(stream)
        for _ in range(reps):
            deriv()
        e1.record(stream)
        torch.cuda.synchronize()
        again = deriv()
        scale = float(np.abs(first).max())
        extra = {"ms_per_call": e0.elapsed_time(e1) / max(reps, 1), "deterministic": DETERMINISTIC,
                 "repeat_bitwise_equal": bool(np.array_equal(first, again)),
                 "repeat_max_diff_over_max_dXs": float(np.abs(first - again).max() / scale)}
    else:
        extra = {}
    if case == "batch":
        sb = torch.tensor(np.stack([S.wing_perturbation(m["pts"], seed=200 + i) for i in range(8)]), device="cuda")
        ob = torch.empty((8, nvol, 3), dtype=torch.float64, device="cuda")
        for _ in range(reps):
            _lib.check(L, mesh.ctx, L.idw_warp_mesh_batch(mesh.ctx, C.c_void_p(sb.data_ptr()), 8,
                                                          C.c_void_p(ob.data_ptr()), _lib.IDW_DEVICE),
                       "warpMeshBatch")
    elif case == "warp":
        for _ in range(reps):
            mesh.warpMesh()
    torch.cuda.synchronize()
    st = mesh.getStats()
    line = {"case": case, "config": cfg, "reps": reps, "lastKernelMs": st["lastKernelMs"],
            "walkListEntries": st["walkListEntries"]}
    line.update(extra)
    print(json.dumps(line))
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="gb300", choices=["gb300", "reference"])
    ap.add_argument("--config", default="P", choices=sorted(CONFIGS))
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-extras", action="store_true")
    ap.add_argument("--mode", default="fast", choices=["fast", "exact"],
                    help="evalMode of the timed warp; the extra measurements and the CPU baseline are fast-mode only")
    ap.add_argument("--suite", action="store_true", help="measurement table rows (S1, W, P errTol sweep)")
    ap.add_argument("--suite-d", action="store_true", help="the 20M-node two-body FFD loop")
    ap.add_argument("--suite-tree", action="store_true",
                    help="error report of the GPU-built Morton tree against the kd tree (S1, W errTol sweep, P)")
    ap.add_argument("--deterministic", action="store_true",
                    help="reverse products with order-independent sums (bitwise repeatable dXs)")
    ap.add_argument("--tree-build", default="kd", choices=["kd", "morton"],
                    help="surface tree: the reference's kd tree (host) or the Morton tree (GPU)")
    ap.add_argument("--walk-lists", default="auto", choices=["auto", "off"],
                    help="mixed fast mode: replay recorded walk decisions (auto) or decide in every walk (off)")
    ap.add_argument("--case", choices=["warp", "deriv1", "deriv1fast", "deriv16", "deriv16fast", "batch", "setup"],
                    help="run one operation --steps times on --config's mesh (the small profiling cases)")
    args = ap.parse_args()
    global WALK_LISTS, TREE_BUILD, DETERMINISTIC
    WALK_LISTS = args.walk_lists
    TREE_BUILD = args.tree_build
    DETERMINISTIC = args.deterministic
    if args.case:
        import torch

        torch.cuda.set_device(_env_int("LOCAL_RANK", 0))
        return run_case(args.case, args.config, args.steps)
    if args.suite or args.suite_d or args.suite_tree:
        import torch

        torch.cuda.set_device(_env_int("LOCAL_RANK", 0))
        if args.suite_tree:
            return run_suite_tree()
        return run_suite() if args.suite else run_suite_d()

    rank = _env_int("RANK", 0)
    world = _env_int("WORLD_SIZE", 1)
    local_rank = _env_int("LOCAL_RANK", 0)
    metric = "volume nodes warped/s (mixed-precision %s warpMesh)" % args.mode
    unit = "volume nodes/s"

    if args.impl == "reference":
        if rank != 0:
            return 0
        from oracle.build import timing_flags
        from oracle.pyoracle import max_threads, timing_library

        m = make_workload(args.config)
        L = timing_library()
        nthr = max_threads(L)
        nvol = len(m["xv0"])
        rng = np.random.default_rng(100)
        # one step = setSurfaceCoordinates + warpMesh over a seeded sample of
        # the workload's volume nodes, sized to about 1.5 s on every core
        idx = np.sort(rng.choice(nvol, min(nvol, 20000), replace=False))
        cal = OracleSample(m, idx, L)
        cal.step()
        t0 = time.perf_counter()
        cal.step()
        rate = len(idx) / (time.perf_counter() - t0)
        nunique = cal.om.sizes()["nUnique"]
        del cal
        n = int(min(nvol, max(20000, 1.5 * rate)))
        smp = OracleSample(m, np.sort(rng.choice(nvol, n, replace=False)), L)
        per_step = []
        for st in range(args.warmup + args.steps):
            t0 = time.perf_counter()
            smp.step()
            dt = time.perf_counter() - t0
            if st >= args.warmup:
                per_step.append(n / dt)
        v = float(np.median(per_step))
        cpu = {"value": v, "unit": unit, "cores": nthr, "kind": "port",
               "sample": "%d of %d volume nodes (seeded uniform sample) per step, fast mode errTol %g, FP64; "
                         "median of %d steps" % (n, nvol, ERR_TOL, args.steps),
               "build": "oracle/idw_oracle.cpp timing build: g++ " + timing_flags()}
        cpu.update(cpu_info())
        line = {"impl": "reference", "metric": metric, "value": v, "unit": unit, "n_gpus": args.gpus,
                "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * n / v, "higher_is_better": True,
                "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
                "config": workload_config(args.config, m, args.mode, nunique, world),
                "cpu_baseline": cpu,
                "e2e": {"value": v, "unit": unit, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
                "note": "CPU restatement of the reference algorithm (oracle/idw_oracle.cpp); the Fortran/PETSc "
                        "reference cannot be built on this image"}
        print(json.dumps(line))
        return 0

    import torch

    torch.cuda.set_device(local_rank)
    dist_on = world > 1
    if dist_on:
        import torch.distributed as dist

        dist.init_process_group("nccl")

    def barrier():
        if dist_on:
            torch.distributed.barrier()
        torch.cuda.synchronize()

    from idwarp_gb300 import _lib

    m = make_workload(args.config)
    nvol, npts = len(m["xv0"]), len(m["pts"])
    t_setup = time.perf_counter()
    mesh = build_mesh(m, "mixed", args.mode)
    setup_s = time.perf_counter() - t_setup
    L = mesh.lib
    stream = torch.cuda.current_stream()
    L.idw_set_stream(mesh.ctx, C.c_void_p(stream.cuda_stream))
    xs_dev = torch.tensor(m["xs"], dtype=torch.float64, device="cuda")
    xs_ptr = C.c_void_p(xs_dev.data_ptr())

    def step():
        rc = L.idw_set_surface_coordinates(mesh.ctx, xs_ptr, 3 * npts, _lib.IDW_DEVICE)
        if rc != 0:
            _lib.check(L, mesh.ctx, rc, "setSurfaceCoordinates")
        rc = L.idw_warp_mesh(mesh.ctx)
        if rc != 0:
            _lib.check(L, mesh.ctx, rc, "warpMesh")

    # the first warp records the walk's decisions (walk lists) and the
    # precision gate's denominators: set-up work, timed apart from the steps
    barrier()
    t_first = time.perf_counter()
    step()
    barrier()
    first_warp_s = time.perf_counter() - t_first
    for _ in range(max(0, args.warmup - 1)):
        step()
    barrier()
    clocks = ClockSampler(local_rank)
    clocks.start()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    barrier()
    ev0.record(stream)
    for _ in range(args.steps):
        step()
    ev1.record(stream)
    barrier()
    clk = clocks.stop()
    ms_total = ev0.elapsed_time(ev1)
    st = mesh.getStats()
    kernel_ms = st["lastKernelMs"]
    ms_step = ms_total / args.steps
    ms_step_max, value = replica_throughput(ms_step, nvol, world, "cuda")

    # end-to-end through the public API with host buffers in pinned memory:
    # surface in, the whole warped grid out, every step; each step's grid is
    # read asynchronously into one of two pinned buffers, so the read of step
    # k overlaps the warp of step k + 1 (the library writes that warp into a
    # second device buffer)
    xs_host = torch.empty(m["xs"].shape, dtype=torch.float64, pin_memory=True).numpy()
    xs_host[...] = m["xs"]
    grids = [torch.empty(3 * nvol, dtype=torch.float64, pin_memory=True).numpy() for _ in range(2)]

    def e2e_steps(n):
        for k in range(n):
            mesh.setSurfaceCoordinates(xs_host)
            mesh.warpMesh()
            mesh.getWarpGrid(out=grids[k % 2], wait=False)
        mesh.synchronize()

    e2e_steps(2)
    barrier()
    t0 = time.perf_counter()
    e2e_steps(args.steps)
    torch.cuda.synchronize()
    e2e_s = (time.perf_counter() - t0) / args.steps
    grid = grids[(args.steps - 1) % 2]
    e2e_check = float(np.abs(grids[0] - grids[1]).max())
    _, e2e_value = replica_throughput(e2e_s * 1e3, nvol, world, "cuda")

    out = {
        "metric": metric, "value": value, "unit": unit, "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms_step_max, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32+f64", "data": "synthetic",
        "config": workload_config(args.config, m, args.mode, st["nUnique"], world),
        "e2e": {"value": e2e_value, "unit": unit, "h2d_bytes_per_step": int(xs_host.nbytes),
                "d2h_bytes_per_step": int(grid.nbytes),
                "note": "USMesh.setSurfaceCoordinates (host) + warpMesh + getWarpGrid(out=pinned, wait=False) per "
                        "step, synchronize at the end; the grid read of step k overlaps the warp of step k + 1",
                "max_diff_between_step_outputs": e2e_check},
        "clocks": clk,
        # per step: gather_xu, face_props, nodal, chunk_sums, node_means,
        # tile_max, tile_mot, counter add, tile_walk, tile_finalize (8 for the
        # gated walks)
        "gpu_launches": (10 if st["walkListEntries"] > 0 else 8) * args.steps,
        "setup_s": setup_s,
        "first_warp_s": first_warp_s,
        "walk_lists": {"entries": st["walkListEntries"], "bytes": 8 * max(0, st["walkListEntries"]),
                       "note": "decisions and weights recorded by the first warp (first_warp_s) and used by every step"},
        "work": {"leafPairs": st["leafPairs"], "approx": st["approx"], "visited": st["visited"],
                 "fp64Fallback": st["fp64Fallback"]},
    }
    # roofline of the walk's kernels (the tile walk and its finalisation): bytes against
    # the measured copy rate for the tile walk, FP32 operations against the FFMA probe
    # for the others; the other figure beside it
    flops = 42.0 * (st["leafPairs"] + st["approx"])
    peak = fp32_peak_tflops() if not args.no_extras else None
    kernel_s = kernel_ms * 1e-3 if kernel_ms > 0 else None
    # DRAM traffic of the walk.  The tile walk streams four FP16 digits of 32
    # weights and a term index per list entry and keeps 64 bytes of sums per
    # node and mirror; k_walk_mixed: ncu on the 2M-node wing, 148.4 + 42.0 MB
    # for 2,025,050 nodes, scaled by volume nodes.  The tree stays in L2.
    tile = args.mode == "fast" and st["walkListEntries"] > 0
    traffic = 260.0 * st["walkListEntries"] + 64.0 * st["nLoop"] * nvol if tile else 94.0 * nvol

    def rate(amount, most, unit, source):
        a = amount / kernel_s if kernel_s else None
        return {"achieved": a, "unit": unit, "peak": most, "peak_source": source,
                "frac": a / most if a and most else None}

    hbm = rate(traffic / 1e9, _measured_peak("hbm_gbs"), "GB/s", "MEASURED_PEAKS.json")
    fp32 = rate(flops / 1e12, peak, "TFLOP/s", "measured FFMA probe (idw_probe_ffma) in this run")
    out["roofline"] = {"bound": "hbm" if tile else "fp32",
                       "kernel": "k_exact_mixed" if args.mode == "exact" else ("k_tile_walk" if tile else "k_walk_mixed"),
                       **(hbm if tile else fp32), "fp32" if tile else "hbm": fp32 if tile else hbm,
                       "flops_per_launch": flops, "kernel_ms": kernel_ms, "traffic": traffic,
                       "traffic_note": "bytes per launch: the tile walk's digits, indices and sums, or ncu on the 2M-node wing "
                                       "scaled by volume nodes"}

    if args.mode == "exact":
        args.no_extras = args.no_cpu_baseline = True
    if not args.no_extras:
        # FP64 plain GPU form on the same workload, and the precision of the mixed form against it
        xm = grid.reshape(-1, 3).copy()
        m64 = build_mesh(m, "fp64")
        L.idw_set_stream(m64.ctx, C.c_void_p(stream.cuda_stream))
        m64.setSurfaceCoordinates(xs_host)
        m64.warpMesh()
        barrier()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        n64 = 2
        for _ in range(n64):
            L.idw_set_surface_coordinates(m64.ctx, xs_ptr, 3 * npts, _lib.IDW_DEVICE)
            L.idw_warp_mesh(m64.ctx)
        e1.record(stream)
        barrier()
        ms64 = e0.elapsed_time(e1) / n64
        x64 = m64.getWarpGrid().reshape(-1, 3)
        s64 = m64.getStats()
        Ldef = st["Ldef0"]
        errv = np.abs(xm - x64).max(axis=1) / Ldef
        out["fp64"] = {"value": nvol / (ms64 * 1e-3), "ms_per_step": ms64,
                       "speedup_mixed_over_fp64": ms64 / ms_step,
                       "same_decisions": bool(s64["leafPairs"] == st["leafPairs"] and s64["approx"] == st["approx"]),
                       "max_err_over_Ldef": float(errv.max()), "rms_err_over_Ldef": float(np.sqrt(np.mean(errv ** 2)))}
        # run-time launch shapes (surfaces per batched walk, seeds per adjoint
        # walk) tuned on this mesh before the batched timings below
        out["autotune"] = mesh.autotune(nSurfaces=8, nSeeds=16)
        L.idw_set_stream(mesh.ctx, C.c_void_p(stream.cuda_stream))
        mesh.setSurfaceCoordinates(xs_host)
        mesh.warpMesh()
        # 16-seed reverse derivative sharing one walk: mixed (product) and FP64 plain form
        rng = np.random.default_rng(100)
        seeds = rng.normal(size=(16, nvol, 3))
        sd = torch.tensor(seeds, dtype=torch.float64, device="cuda")
        del seeds
        dxs = torch.zeros((16, npts, 3), dtype=torch.float64, device="cuda")
        dxs64 = torch.zeros((16, npts, 3), dtype=torch.float64, device="cuda")

        def deriv(msh, out):
            rc = L.idw_warp_deriv_batch(msh.ctx, C.c_void_p(sd.data_ptr()), 16, C.c_void_p(out.data_ptr()),
                                        _lib.IDW_DEVICE)
            if rc != 0:
                _lib.check(L, msh.ctx, rc, "warpDerivBatch")

        # FP64 plain form (one launch of 16 seeds)
        barrier()
        e0.record(stream)
        deriv(m64, dxs64)
        e1.record(stream)
        barrier()
        msd64 = e0.elapsed_time(e1)
        dref = dxs64.abs().max().item()
        d1ref = dxs64[0].abs().max().item()

        # one seed (the solver-adjoint call pattern): idw_warp_deriv on the device
        def deriv1():
            rc = L.idw_warp_deriv(mesh.ctx, C.c_void_p(sd.data_ptr()), 3 * nvol, _lib.IDW_DEVICE)
            if rc != 0:
                _lib.check(L, mesh.ctx, rc, "warpDeriv")

        # the mixed adjoint in both forms: double-float (default) and FP32
        res16, res1 = {}, {}
        for adj in ("precise", "fast"):
            mesh.setOption("adjointPrecision", adj)
            mesh._setMeshOptions()
            deriv(mesh, dxs)  # warm-up (the precise form's denominator walk runs once here)
            barrier()
            e0.record(stream)
            for _ in range(3):
                deriv(mesh, dxs)
            e1.record(stream)
            barrier()
            msd = e0.elapsed_time(e1) / 3
            res16[adj] = {"seeds": 16, "value": 16 * nvol / (msd * 1e-3), "unit": "seeds*nodes/s", "ms": msd,
                          "adjointPrecision": adj, "speedup_mixed_over_fp64": msd64 / msd,
                          "max_rel_diff_vs_fp64": float((dxs - dxs64).abs().max().item() / dref)}
            deriv1()
            barrier()
            e0.record(stream)
            for _ in range(5):
                deriv1()
            e1.record(stream)
            barrier()
            ms1 = e0.elapsed_time(e1) / 5
            d1 = torch.tensor(mesh.getdXs(), device="cuda")
            res1[adj] = {"seeds": 1, "value": nvol / (ms1 * 1e-3), "unit": "seeds*nodes/s", "ms": ms1,
                         "adjointPrecision": adj,
                         "max_rel_diff_vs_fp64": float((d1 - dxs64[0]).abs().max().item() / d1ref)}
        mesh.setOption("adjointPrecision", "precise")
        mesh._setMeshOptions()
        out["warpDeriv"] = dict(res16["precise"], fp64_value=16 * nvol / (msd64 * 1e-3), fp64_ms=msd64,
                                fast=res16["fast"])
        out["warpDeriv1"] = dict(res1["precise"], fast=res1["fast"])
        del sd, dxs, dxs64, d1
        # 8 independent surface perturbations (seeds 200-207) through the batched
        # walk (four surfaces share one tree walk) against one warpMesh each
        from idwarp_gb300 import synthetic as S

        surf = np.stack([S.wing_perturbation(m["pts"], seed=200 + i) for i in range(8)])
        sb = torch.tensor(surf, dtype=torch.float64, device="cuda")
        ob = torch.empty((8, nvol, 3), dtype=torch.float64, device="cuda")

        def batch():
            rc = L.idw_warp_mesh_batch(mesh.ctx, C.c_void_p(sb.data_ptr()), 8, C.c_void_p(ob.data_ptr()),
                                       _lib.IDW_DEVICE)
            if rc != 0:
                _lib.check(L, mesh.ctx, rc, "warpMeshBatch")

        batch()  # warm-up
        barrier()
        e0.record(stream)
        for _ in range(2):
            batch()
        e1.record(stream)
        barrier()
        msb = e0.elapsed_time(e1) / 2
        m64.setSurfaceCoordinates(surf[7])
        m64.warpMesh()
        errb = np.abs(ob[7].cpu().numpy() - m64.getWarpGrid().reshape(-1, 3)).max() / Ldef
        out["warpMeshBatch"] = {"surfaces": 8, "value": 8 * nvol / (msb * 1e-3), "unit": "volume nodes/s",
                                "ms": msb, "ms_per_surface": msb / 8, "speedup_per_surface_over_single": ms_step * 8 / msb,
                                "max_err_over_Ldef_vs_fp64": float(errb)}
        del sb, ob
        # set-up with a restart file: the first build computes the estimate
        # and the dryRun costs and saves them, the next one loads and checks
        import tempfile

        with tempfile.TemporaryDirectory() as td:
            rf = os.path.join(td, "wing.restart")
            t0 = time.perf_counter()
            mr = build_mesh(m, "mixed", restartFile=rf)
            t_first = time.perf_counter() - t0
            first = mr.restartStatus
            del mr
            t0 = time.perf_counter()
            mr = build_mesh(m, "mixed", restartFile=rf)
            t_loaded = time.perf_counter() - t0
            out["restart"] = {"setup_s_without": setup_s, "setup_s_first": t_first, "first": first,
                              "setup_s_loaded": t_loaded, "loaded": mr.restartStatus,
                              "file_bytes": os.path.getsize(rf)}
            del mr
        # the GPU-built Morton tree (option treeBuild "morton"; the reference
        # builds the kd tree) on the same workload: set-up, the replayed warp,
        # its work, and its fast-mode grid against the kd tree's
        if TREE_BUILD == "kd":
            t0 = time.perf_counter()
            mm = build_mesh(m, "mixed", args.mode, tree="morton")
            torch.cuda.synchronize()
            t_m = time.perf_counter() - t0
            Lm = mm.lib
            Lm.idw_set_stream(mm.ctx, C.c_void_p(stream.cuda_stream))

            def step_m():
                _lib.check(Lm, mm.ctx, Lm.idw_set_surface_coordinates(mm.ctx, xs_ptr, 3 * npts, _lib.IDW_DEVICE),
                           "setSurfaceCoordinates")
                _lib.check(Lm, mm.ctx, Lm.idw_warp_mesh(mm.ctx), "warpMesh")

            t0 = time.perf_counter()
            step_m()
            torch.cuda.synchronize()
            first_m = time.perf_counter() - t0
            step_m()
            m0, m1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            m0.record(stream)
            for _ in range(5):
                step_m()
            m1.record(stream)
            torch.cuda.synchronize()
            ms_m = m0.elapsed_time(m1) / 5
            stm = mm.getStats()
            dk = np.abs(mm.getWarpGrid().reshape(-1, 3) - grid.reshape(-1, 3)).max(axis=1) / Ldef
            out["morton_tree"] = {"setup_s": t_m, "setup_s_kd": setup_s, "tree_build_ms": stm["treeBuildMs"],
                                  "tree_build_ms_kd": st["treeBuildMs"], "first_warp_s": first_m,
                                  "ms_per_step": ms_m, "value": nvol / (ms_m * 1e-3), "unit": "volume nodes/s",
                                  "leafPairs": stm["leafPairs"], "approx": stm["approx"],
                                  "max_diff_vs_kd_over_Ldef": float(dk.max()),
                                  "rms_diff_vs_kd_over_Ldef": float(np.sqrt(np.mean(dk ** 2))),
                                  "note": "other clusters than the reference's kd tree: fast-mode grids differ by "
                                          "what errTol allows (error against exact mode: bench.py --suite-tree)"}
            del mm

    if rank == 0 and not args.no_cpu_baseline:
        out["cpu_baseline"], idx, xv_cpu = run_cpu_baseline(m)
        # parity at this workload: the oracle's checker build on the same sample
        grids = {"mixed": grid.reshape(-1, 3)}
        if not args.no_extras:
            grids["fp64"] = x64

        def sample_run(prec, idx):
            ms = dict(m)
            ms["xv0"] = m["xv0"][idx]
            g = build_mesh(ms, prec)
            g.setSurfaceCoordinates(m["xs"])
            g.warpMesh()
            r = g.getStats()
            r["xv"] = g.getWarpGrid().reshape(-1, 3)
            del g
            return r

        out["parity"] = run_parity(m, idx, xv_cpu, grids, sample_run)
    if rank == 0:
        print(json.dumps(out))
    if dist_on:
        torch.distributed.destroy_process_group()
    return 0


if __name__ == "__main__":
    sys.exit(main())
