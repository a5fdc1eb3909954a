"""The work a user of this library has it do, as cases that can be timed.

A case goes through a public entry point with host arrays, the way the
reference's callers pass them (``TomoSh_CUDA`` through ``native.sweep``,
``tomoSweepStatic``, the multi-mesh batch, the proposal search, the network's
own functions), and returns everything that call computes.  Meshes are the
repository's seeded generators (closed perturbed spheres from a few hundred
triangles to 120k, the thin open manikin-like shell), orientation lists are
yaw x pitch grids.

The sweep's results are defined by one fixed sequence of single-precision
operations (integers and bits, compared exactly), so they have no 64-bit
counterpart; the network's have one, computed here with numpy.
"""
from __future__ import annotations

import math

import numpy as np

from tomo_shell2026_b200 import meshgen, native, surrogate
from tomo_shell2026_b200.options import BED_BRIM, BED_NONE, BED_RAFT, BED_SKIRT, PrintOptions

HIDDEN = 128
LAYERS = ((4, HIDDEN), (HIDDEN, HIDDEN), (HIDDEN, HIDDEN), (HIDDEN, 1))


# kind "sweep": native.sweep (TomoSh_CUDA).  mesh "sphere": perturbed closed
# sphere of about `tri` triangles, radius in mm, `scale` voxels per mm, fine
# surface detail or smooth; mesh "shell": manikin-like open shell triangulated
# at `spacing` mm, run in shell mode.  n_yaw x n_pitch orientations with
# yaw_step / pitch_step degrees between them.
def _sweep(mesh="sphere", tri=5120, radius=50.0, scale=1.0, detail=False, spacing=6.5, n_yaw=360, n_pitch=61,
           yaw_step=1.0, pitch_step=1.0, explicit=True, bed=BED_NONE, kind="sweep"):
    return {"kind": kind, "mesh": mesh, "tri": tri, "radius": radius, "scale": scale, "detail": detail,
            "spacing": spacing, "n_yaw": n_yaw, "n_pitch": n_pitch, "yaw_step": yaw_step, "pitch_step": pitch_step,
            "explicit": explicit, "bed": bed}


def _named(name, **kw):
    return {"name": name, **_sweep(**kw)}


def listed():
    return [
        # One known orientation re-evaluated for its masses, matrix and render
        # pixels (what a slicer preview asks for): one launch sequence.
        _named("one_orientation", n_yaw=1, n_pitch=1),
        # The reference front-end's default search (10-degree steps, both end
        # points, yaw and pitch over the full turn) on a part that gets a raft.
        _named("part_10deg_raft", n_yaw=37, n_pitch=37, yaw_step=10.0, pitch_step=10.0, bed=BED_RAFT),
        # A low-polygon part (large triangles), 5-degree steps, implicit
        # support volume, skirt.
        _named("lowpoly_5deg_implicit", tri=500, radius=70.0, n_yaw=72, n_pitch=13, yaw_step=5.0, pitch_step=5.0,
               explicit=False, bed=BED_SKIRT),
        # The small solid over the whole 1-degree grid.
        _named("solid5k_1deg"),
        # A 20k-triangle part with an odd number of orientations, implicit.
        _named("part20k_odd_implicit", tri=20000, radius=60.0, detail=True, n_yaw=121, n_pitch=37, yaw_step=2.97,
               pitch_step=1.63, explicit=False),
        # The headline: 82k-triangle solid, 0.5 mm voxels, 1-degree grid.
        _named("solid82k_1deg", tri=81920, radius=80.0, scale=2.0, detail=True),
        # The thin open shell in shell mode (the front-end's choice for meshes
        # that are not watertight), 2-degree grid.
        _named("shell87k_2deg", mesh="shell", n_yaw=180, n_pitch=31, yaw_step=2.0, pitch_step=2.0),
        # The allocation-free call on a small part, 10-degree grid.
        _named("static_10deg", kind="static", n_yaw=36, n_pitch=19, yaw_step=10.0, pitch_step=10.0),
        # Several uneven parts of one object in one batched launch.
        {"name": "batch_uneven", "kind": "batch", "meshes": 6, "tri_min": 1000, "tri_max": 40000, "n_yaw": 120,
         "n_pitch": 21, "yaw_step": 3.0, "pitch_step": 3.0},
        # The proposal search over the 0.5-degree grid, ranked by the trained
        # network and by interpolation of the coarse values.
        {"name": "search_network", "kind": "search", "tri": 5120, "radius": 50.0, "n_yaw": 720, "n_pitch": 121,
         "step": 0.5, "stride": 10, "proposal": "network"},
        {"name": "search_interpolation", "kind": "search", "tri": 5120, "radius": 50.0, "n_yaw": 720, "n_pitch": 121,
         "step": 0.5, "stride": 10, "proposal": "interpolation"},
        # The network alone: trained on a 5-degree coarse grid's points, then
        # evaluated on every point of the 0.5-degree grid.
        {"name": "network_fit_predict", "kind": "network", "samples": 936, "steps": 300, "points": 87120},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["sweep", "sweep", "sweep", "sweep", "shell", "static", "batch", "search", "network"])
    if kind == "sweep":
        tri = int(_log(rng, 300, 120000))
        # as many orientations as keep triangles x orientations within the headline's
        n = _log(rng, 1, min(21960.0, 81920.0 * 21960.0 / (1.5 * tri)))
        n_pitch = max(1, int(math.sqrt(n / 6.0)))
        n_yaw = max(1, int(n / n_pitch))
        bed = rng.choice([BED_NONE, BED_NONE, BED_BRIM, BED_RAFT, BED_SKIRT])
        fine = tri > 15000
        return _sweep(tri=tri, radius=round(rng.uniform(40.0, 80.0), 1), scale=rng.choice([1.0, 2.0]) if fine else 1.0,
                      detail=fine, n_yaw=n_yaw, n_pitch=n_pitch, yaw_step=360.0 / n_yaw,
                      pitch_step=round(rng.uniform(1.0, 60.0), 2) / n_pitch, explicit=rng.random() < 0.6, bed=bed)
    if kind == "shell":
        return _sweep(mesh="shell", spacing=round(rng.uniform(6.5, 16.0), 1), n_yaw=int(_log(rng, 5, 150)),
                      n_pitch=rng.randint(1, 21), yaw_step=2.3, pitch_step=2.9, explicit=rng.random() < 0.6)
    if kind == "static":
        return _sweep(kind="static", tri=int(_log(rng, 300, 16000)), radius=round(rng.uniform(30.0, 60.0), 1),
                      n_yaw=rng.randint(1, 40), n_pitch=rng.randint(1, 13), yaw_step=9.0, pitch_step=7.0,
                      explicit=rng.random() < 0.6, bed=rng.choice([BED_NONE, BED_RAFT]))
    if kind == "batch":
        return {"kind": "batch", "meshes": rng.randint(2, 7), "tri_min": 1000, "tri_max": int(_log(rng, 5000, 80000)),
                "n_yaw": rng.randint(31, 150), "n_pitch": rng.randint(3, 15), "yaw_step": 2.4, "pitch_step": 3.1}
    if kind == "search":
        return {"kind": "search", "tri": int(_log(rng, 2000, 20000)), "radius": round(rng.uniform(40.0, 55.0), 1),
                "n_yaw": 360, "n_pitch": 10 * rng.randint(3, 6) + 1, "step": 1.0, "stride": rng.choice([5, 10]),
                "proposal": rng.choice(["network", "interpolation"])}
    return {"kind": "network", "samples": int(_log(rng, 100, 2500)), "steps": rng.randint(20, 300),
            "points": int(_log(rng, 100, 87120))}


# ------------------------------------------------------------------ inputs

def _sphere(tri, radius, scale, detail, seed):
    if detail:
        return meshgen.perturbed_sphere(tri, radius, seed, n_harmonics=12, max_degree=8, amplitude=0.25, n_bumps=4,
                                        scale=scale, with_hull=False)
    return meshgen.perturbed_sphere(tri, radius, seed, scale=scale, with_hull=False)


def _grid(case):
    return meshgen.ypr_grid(case["yaw_step"] * np.arange(case["n_yaw"]), case["pitch_step"] * np.arange(case["n_pitch"]))


def _options(case):
    bed = case["bed"]
    inner, outer = {BED_NONE: (0.0, 0.0), BED_BRIM: (0.0, 3.0), BED_RAFT: (0.0, 2.0), BED_SKIRT: (1.0, 3.0)}[bed]
    shell = case["mesh"] == "shell"
    return PrintOptions(explicit_ss=case["explicit"], bed_type=bed, bed_inner=inner, bed_outer=outer,
                        bed_thickness=0.97 if bed != BED_NONE else 0.0, shell_mesh=shell)


def _pixel_rows(case):
    """Room for the best orientation's render pixels: several types per
    surface pixel, plus one row per voxel of explicit support."""
    if case["mesh"] == "shell":
        return 5_000_000
    r = case["radius"] * case["scale"]
    return int(40.0 * r * r + 0.8 * r ** 3)


def _store_pixels(state, pixels):
    """Append the pixel arrays in the caller's buffer; returns (counts, buffer)."""
    buf, at = state["pixels"], 0
    counts = np.array([p.shape[0] for p in pixels], np.int64)
    for p in pixels:
        buf[at:at + p.shape[0]] = p
        at += p.shape[0]
    if at < state["rows"]:
        buf[at:state["rows"]] = 0
    state["rows"] = at
    return counts, buf


def _network_arrays(case, seed):
    """Initial parameters (uniform, fan-in/fan-out scaled, zero biases), the
    training set (features of coarse directions, a smooth standardised target
    with a little noise) and the points to predict."""
    rng = np.random.default_rng(seed)
    parts = []
    for i, o in LAYERS:
        r = math.sqrt(6.0 / (i + o))
        parts += [rng.uniform(-r, r, i * o), np.zeros(o)]
    p0 = np.concatenate(parts).astype(np.float32)

    def features(n):
        y, p = rng.uniform(0, 2 * np.pi, n), rng.uniform(0, np.pi / 3, n)
        return np.stack([np.sin(y), np.cos(y), np.sin(p), np.cos(p)], 1).astype(np.float32)

    x, q = features(case["samples"]), features(case["points"])
    k = rng.normal(size=(4, 5))
    t = np.sin(x.astype(np.float64) @ k * 2.0).sum(1) + 0.05 * rng.normal(size=x.shape[0])
    y = ((t - t.mean()) / max(t.std(), 1e-9)).astype(np.float32)
    return p0, x, y, q


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("sweep", "static"):
        if case["mesh"] == "shell":
            mesh = meshgen.manikin_shell(seed, spacing=case["spacing"])
        else:
            mesh = _sphere(case["tri"], case["radius"], case["scale"], case["detail"], seed)
        ypr = _grid(case)
        if ypr.shape[0] == 1:   # a single orientation: any direction
            rng = np.random.default_rng(seed)
            ypr = rng.uniform(0.0, 2.0 * np.pi, (1, 3)).astype(np.float32)
            ypr[0, 2] = 0.0
        state = {"kind": kind, "mesh": mesh, "ypr": ypr, "opts": _options(case)}
        if kind == "sweep":
            # the caller's pixel buffer: rows of all 11 types one after another
            # (their number depends on the mesh), zero past the last
            state["pixels"] = np.zeros((_pixel_rows(case), 6), np.int16)
            state["rows"] = 0
        return state
    if kind == "batch":
        rng = np.random.default_rng(seed)
        lo, hi = math.log(case["tri_min"]), math.log(case["tri_max"])
        meshes = []
        for k in range(case["meshes"]):
            # spread over the range (the parts of one object differ in size)
            t = int(math.exp(lo + (hi - lo) * (k + rng.uniform(0.0, 1.0)) / case["meshes"]))
            fine = k % 2 == 1
            meshes.append(_sphere(t, 80.0 if fine else 50.0, 2.0 if fine else 1.0, fine, int(rng.integers(1 << 30))))
        return {"kind": kind, "meshes": meshes, "ypr": _grid(case), "opts": PrintOptions(explicit_ss=True)}
    if kind == "search":
        ypr = meshgen.ypr_grid(case["step"] * np.arange(case["n_yaw"]), case["step"] * np.arange(case["n_pitch"]))
        return {"kind": kind, "mesh": _sphere(case["tri"], case["radius"], 1.0, False, seed), "ypr": ypr,
                "opts": PrintOptions(explicit_ss=True), "n_yaw": case["n_yaw"], "n_pitch": case["n_pitch"],
                "stride": case["stride"], "proposal": case["proposal"]}
    p0, x, y, q = _network_arrays(case, seed)
    surrogate.mlp_init(0)
    return {"kind": kind, "p0": p0, "x": x, "y": y, "q": q, "steps": case["steps"]}


# ------------------------------------------------------------------ one pass

def run(state):
    kind = state["kind"]
    if kind == "sweep":
        r = native.sweep(state["mesh"], state["ypr"], state["opts"])
        return {"optID": r.optID, "Mo": r.Mo, "Mss": r.Mss, "Vtc": r.Vtc, "Vo64": r.Vo64, "Vss64": r.Vss64,
                "Vtc64": r.Vtc64, "VoF": r.VoF, "VssF": r.VssF, "VtcF": r.VtcF, "n_bed": r.n_bed, "flags": r.flags,
                "entries": r.entries, "columns": r.columns, "volmass": r.volmass, "mat4x4": r.mat4x4,
                "pixels": _store_pixels(state, r.pixels)}
    if kind == "static":
        opt, mo, mss, vtc = native.sweep_static(state["mesh"], state["ypr"], state["opts"])
        return {"optID": opt, "Mo": mo, "Mss": mss, "Vtc": vtc}
    if kind == "batch":
        b = native.Batch(state["meshes"], [state["ypr"]] * len(state["meshes"]), state["opts"])
        b.run()
        return [b.results(m) for m in range(len(state["meshes"]))]
    if kind == "search":
        r = surrogate.search(state["mesh"], state["ypr"], state["n_yaw"], state["n_pitch"], state["opts"],
                             stride=state["stride"], proposal=state["proposal"])
        return {"optID": r.optID, "Mss": r.Mss, "pred_vss": r.pred_vss, "evaluated": r.evaluated,
                "fallback": r.fallback, "cells_refined": r.cells_refined, "rounds": r.rounds, "coarse": r.coarse}
    surrogate.mlp_params(set_to=state["p0"])
    loss = surrogate.mlp_fit(state["x"], state["y"], state["steps"], 3e-3)
    return {"loss": loss, "params": surrogate.mlp_params(), "pred": surrogate.mlp_predict(state["q"])}


# ------------------------------------------------------------------ floors

def _sweep_work(tri, radius, scale, n, twin=1):
    """One sweep: the mesh and orientations in, per-orientation results out;
    per orientation the rotation of every vertex and its normal's z (20), the
    box and barycentric constants of every triangle (40), and per accepted
    pixel the barycentric coordinates, three interpolations and the column's
    pairing (60).  Accepted pixels of a closed surface: half its area in
    square voxels (mean projected footprint, both sides)."""
    vtx = tri / 2 + 2
    pixels = 2.0 * math.pi * (radius * scale) ** 2 * 1.1 * twin
    return {"bytes": 24.0 * vtx + 12.0 * tri + n * (12.0 + 68.0), "flops": n * (20.0 * vtx + 40.0 * tri + 60.0 * pixels)}


def work(case):
    kind = case["kind"]
    if kind in ("sweep", "static"):
        n = case["n_yaw"] * case["n_pitch"]
        if case["mesh"] == "shell":
            # two sheets, each with its offset twin: about 1.27M pixels an orientation
            tri = 87738.0 * (6.5 / case["spacing"]) ** 2
            return _sweep_work(tri, 214.0, 1.0, n, twin=4)
        return _sweep_work(case["tri"], case["radius"], case["scale"], n)
    if kind == "batch":
        lo, hi = math.log(case["tri_min"]), math.log(case["tri_max"])
        n = case["n_yaw"] * case["n_pitch"]
        parts = [_sweep_work(math.exp(lo + (hi - lo) * (k + 0.5) / case["meshes"]), 80.0 if k % 2 else 50.0,
                             2.0 if k % 2 else 1.0, n) for k in range(case["meshes"])]
        return {key: sum(p[key] for p in parts) for key in ("bytes", "flops")}
    params = sum(i * o + o for i, o in LAYERS)
    if kind == "search":
        # the coarse points and 64 blocks of 5 x 5 points exactly; the network
        # trained for 300 steps on the coarse points and read on the whole grid
        n = case["n_yaw"] * case["n_pitch"]
        coarse = math.ceil(case["n_yaw"] / case["stride"]) * math.ceil(case["n_pitch"] / case["stride"])
        w = _sweep_work(case["tri"], case["radius"], 1.0, min(n, coarse + 64 * 25))
        if case["proposal"] == "network":
            w["flops"] += 6.0 * params * coarse * 300 + 2.0 * params * n
        w["bytes"] += 20.0 * n
        return w
    return {"bytes": 4.0 * (2 * params + 5 * case["samples"] + 5 * case["points"]),
            "flops": 6.0 * params * case["samples"] * case["steps"] + 2.0 * params * case["points"]}


# ------------------------------------------------------------------ 64-bit values

def exact(case, seed):
    """The network's training and prediction in float64 (full-batch mean
    squared error, Adam with 0.9 / 0.999 / 1e-8 and bias correction)."""
    if case["kind"] != "network":
        return None
    p0, x, y, q = _network_arrays(case, seed)
    x, y, q = x.astype(np.float64), y.astype(np.float64), q.astype(np.float64)
    p = p0.astype(np.float64)
    lr = float(np.float32(3e-3))

    def split(v):
        out, at = [], 0
        for i, o in LAYERS:
            out.append((v[at:at + i * o].reshape(i, o), v[at + i * o:at + i * o + o]))
            at += i * o + o
        return out

    def forward(v, inp):
        acts = [inp]
        for k, (w, b) in enumerate(split(v)):
            z = acts[-1] @ w + b
            acts.append(np.tanh(z) if k < len(LAYERS) - 1 else z)
        return acts

    m, s = np.zeros_like(p), np.zeros_like(p)
    n = x.shape[0]
    loss = 0.0
    for step in range(1, case["steps"] + 1):
        acts = forward(p, x)
        d = acts[-1][:, 0] - y
        loss = float(np.mean(d * d))
        dz = (2.0 * d / n)[:, None]
        grads = []
        for k in range(len(LAYERS) - 1, -1, -1):
            w, _ = split(p)[k]
            grads.append(np.concatenate([(acts[k].T @ dz).ravel(), dz.sum(0)]))
            if k:
                dz = (dz @ w.T) * (1.0 - acts[k] ** 2)
        g = np.concatenate(grads[::-1])
        m = 0.9 * m + 0.1 * g
        s = 0.999 * s + 0.001 * g * g
        p = p - lr * (m / (1.0 - 0.9 ** step)) / (np.sqrt(s / (1.0 - 0.999 ** step)) + 1e-8)
    return {"loss": loss, "params": p, "pred": forward(p, q)[-1][:, 0]}
