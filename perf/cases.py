"""The work that users of this library have it do, as cases that can be timed.

Each case is a dict of plain values; `prepare` builds what a program holds
before the call (mesh, case handle, particles on the device, host arrays),
`run` is one pass through the public entry points of ``pydsmc.gpu``, and
`work` counts the bytes and operations such a pass cannot do without.

The kinds of pass (`do`):

- ``window``: the production loop between two hand-offs to the host's GSIS
  solver: `steps` fused steps (one call each), then the window-averaged
  fields and the particle count read back.
- ``stages``: the same loop by a host that makes the reference's five stage
  calls one after another.
- ``batch``: several independent cases advanced together, each one's local
  fields read at the end.
- ``gsis``: the update of the particles from the NS solution between two
  windows, and the fields that the host reads right after it.
- ``restart``: host particles uploaded (a checkpoint or another program's
  fill), their fields sampled, and a checkpoint read back.
- ``trace``: the tracing check of given particles.

Cells, particles per cell, Mach and Knudsen numbers, angles of attack and
sampling controls are those of the block, capsule, batched and served
workloads and of the tests.
"""
from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "dig-appolo_b200"))

from pydsmc import capsule  # noqa: E402
from pydsmc import case as C  # noqa: E402
from pydsmc import gpu  # noqa: E402
from pydsmc import mesh as M  # noqa: E402
from pydsmc import workload as W  # noqa: E402

CAPSULE_ZONES = [(3, 1, 0), (4, 2, 1), (5, 3, 0), (6, 4, 0)]
BOX_ZONES = CAPSULE_ZONES + [(7, 5, 0)]      # the box's other sides are specular


def listed():
    return [
        # the smallest case (the tests' 760-cell box): launches and latency
        {"name": "window_box_tiny", "do": "window", "mesh": "box", "size": 4, "ppc": 20.0, "precision": "mixed",
         "steps": 20, "Ma": 5.0, "Kn": 0.1, "aoa": 30.0, "walls": False},
        # a small case of the batched workload, stepped alone
        {"name": "window_box_small", "do": "window", "mesh": "box", "size": 8, "ppc": 85.0, "precision": "mixed",
         "steps": 100, "Ma": 7.5, "Kn": 0.03, "aoa": 12.0, "walls": False},
        # the block case in FP64, the reference's own precision, walls tallied
        {"name": "window_block_fp64", "do": "window", "mesh": "box", "size": 16, "ppc": 50.0, "precision": "fp64",
         "steps": 50, "Ma": 5.0, "Kn": 0.1, "aoa": 0.0, "walls": True},
        # cells with triangles and quads (wedges, an odd count), nothing regular
        {"name": "window_wedges", "do": "window", "mesh": "prism", "size": 23, "ppc": 61.0, "precision": "mixed",
         "steps": 50, "Ma": 4.0, "Kn": 0.2, "aoa": 5.0, "walls": False},
        # a served capsule request, coarse tetrahedra
        {"name": "window_capsule_served", "do": "window", "mesh": "capsule", "size": 2.65, "ppc": 55.0,
         "precision": "mixed", "steps": 100, "Ma": 5.0, "Kn": 0.01, "aoa": 30.0, "walls": False},
        # a capsule of middle size in FP64
        {"name": "window_capsule_fp64", "do": "window", "mesh": "capsule", "size": 1.8, "ppc": 100.0,
         "precision": "fp64", "steps": 20, "Ma": 5.0, "Kn": 0.01, "aoa": 30.0, "walls": False},
        # the headline case: 372,500 tetrahedra, 37M particles
        {"name": "window_capsule_full", "do": "window", "mesh": "capsule", "size": 1.0, "ppc": 100.0,
         "precision": "mixed", "steps": 50, "Ma": 5.0, "Kn": 0.01, "aoa": 30.0, "walls": True},
        # a host that calls the five stages itself
        {"name": "stages_box", "do": "stages", "mesh": "box", "size": 12, "ppc": 50.0, "precision": "mixed",
         "steps": 20, "Ma": 5.0, "Kn": 0.1, "aoa": 30.0, "walls": False},
        # eight cases of uneven size together
        {"name": "batch_boxes", "do": "batch", "mesh": "box", "cases": 8, "size": 14, "ppc": 70.0,
         "precision": "mixed", "steps": 20, "Ma": 6.0, "Kn": 0.1, "aoa": 20.0},
        # the GSIS exchange on a capsule
        {"name": "gsis_capsule", "do": "gsis", "mesh": "capsule", "size": 1.4, "ppc": 100.0, "precision": "mixed",
         "Ma": 5.0, "Kn": 0.01, "aoa": 30.0, "gate": 0.95},
        # a restart of the block case from host arrays
        {"name": "restart_block", "do": "restart", "mesh": "box", "size": 16, "ppc": 50.0, "precision": "mixed",
         "Ma": 5.0, "Kn": 0.1, "aoa": 0.0, "ordered": True},
        # the tracing check on the block mesh
        {"name": "trace_block", "do": "trace", "mesh": "box", "size": 16, "count": 200000, "precision": "mixed",
         "Ma": 5.0, "Kn": 0.1, "aoa": 0.0},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    do = rng.choice(["window"] * 6 + ["stages", "batch", "gsis", "restart", "trace"])
    kind = rng.choice(["box", "box", "capsule", "capsule", "prism", "pyramid"])
    if do in ("batch", "restart", "trace") and kind in ("prism", "pyramid"):
        kind = "box"
    if do == "trace":
        kind = "box"
    size = {"box": 2 * int(round(_log(rng, 4, 24) / 2)), "capsule": round(_log(rng, 1.3, 2.65), 2),
            "prism": int(round(_log(rng, 7, 36))), "pyramid": int(round(_log(rng, 5, 25)))}[kind]
    c = {"do": do, "mesh": kind, "size": size, "ppc": round(_log(rng, 11, 200), 1),
         "precision": rng.choice(["mixed", "mixed", "fp64"]),
         "Ma": round(rng.uniform(3, 10), 2), "Kn": round(_log(rng, 0.01, 1.0), 4), "aoa": round(rng.uniform(0, 40), 1)}
    if kind == "capsule":
        # the capsule is flown as served: Ma 5, Kn 0.01, 30 degrees
        c.update(Ma=5.0, Kn=0.01, aoa=30.0, ppc=round(_log(rng, 11, 100), 1))
    if do in ("window", "stages"):
        c["steps"] = int(round(_log(rng, 5, 50)))
        c["walls"] = rng.random() < 0.3
    elif do == "batch":
        c.update(cases=rng.randint(2, 10), size=min(size, 16) if kind == "box" else 2.65, steps=rng.randint(5, 30))
    elif do == "gsis":
        c["gate"] = round(rng.uniform(0.5, 1.0), 2)
    elif do == "restart":
        c["ordered"] = rng.random() < 0.7
        c["ppc"] = min(c["ppc"], round(2.5e6 / cells_of(c), 1))
    elif do == "trace":
        c.pop("ppc")
        c["count"] = int(_log(rng, 5e3, 4e5))
    if "ppc" in c:
        # a drawn case stays well below the headline case's particles
        c["ppc"] = round(max(5.0, min(c["ppc"], 1.2e7 / cells_of(c))), 1)
    return c


def cells_of(c):
    """The number of cells, about."""
    s = c["size"]
    return {"box": 12 * s ** 3 - (s // 2) ** 3, "capsule": int(372500 / s ** 3), "prism": 2 * s ** 3,
            "pyramid": 6 * s ** 3}[c["mesh"]]


# ---------------------------------------------------------------------------
# meshes (the same for every seed: a program has its mesh)
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def mesh(kind, size):
    """The mesh, and the length its Knudsen number is based on."""
    if kind == "box":
        # the block case's family: 3k x 2k x 2k hexahedra, the central (k/2)^3 block out
        k, h = int(size), int(size) // 2
        nx, ny = 3 * k, 2 * k
        i0, j0 = (nx - h) // 2, (ny - h) // 2
        raw = M.hex_box(nx, ny, ny, 1.0, 0.5, 0.5, (i0, i0 + h, j0, j0 + h, j0, j0 + h))
        return M.build_dsmc_mesh(raw), h * 0.5 / ny
    if kind == "capsule":
        if size == 1.0:
            raw = capsule.capsule_mesh(seed=0, target_cells=capsule.CAP_CELLS, morton=True)
        else:
            raw = capsule.capsule_mesh(h_fine=0.215 * size, h_coarse=0.60 * size, seed=0)
        return M.build_dsmc_mesh(raw), capsule.L0
    n = int(size)
    build = M.prism_box if kind == "prism" else M.pyramid_box
    return M.build_dsmc_mesh(build(n, n, n, 1.0, 1.0, 1.0)), 0.25


def zones_of(kind):
    return CAPSULE_ZONES if kind == "capsule" else BOX_ZONES


def constants(c, ppc=None):
    dm, l0 = mesh(c["mesh"], c["size"])
    ppc = c.get("ppc", 100.0) if ppc is None else ppc
    return dm, C.mesh_message(dm, c["Ma"], c["Kn"], ppc=max(1, int(round(ppc))), L0=l0)


def make_case(c, dm, mess, seed, aoa=None, **params):
    p = gpu.default_params(
        precision=gpu.PRECISION_MIXED if c["precision"] == "mixed" else gpu.PRECISION_FP64, seed=seed,
        zones=zones_of(c["mesh"]), inflow_dir=C.inflow_direction(c["aoa"] if aoa is None else aoa), **params)
    return gpu.Case(dm, mess, p, device=torch.cuda.current_device())


def host_particles(c, dm, mess, seed):
    """Particles as another program would hand them over: freestream
    velocities, uniform positions, counts in proportion to the volumes (the
    same counts for every seed), in the cells' order or in none."""
    rng = np.random.default_rng(seed)
    count = W.proportional_counts(dm, c["ppc"], np.random.default_rng(4))
    cell = np.repeat(np.arange(dm.ncell, dtype=np.int32), count)
    if not c["ordered"]:
        cell = rng.permutation(cell)
    u, sig, tN = W.freestream(mess, C.inflow_direction(c["aoa"]))
    return {"x": W.uniform_positions(dm, cell, rng), "v": u + sig * rng.standard_normal((cell.shape[0], 3)),
            "ir": -np.log(1.0 - rng.random(cell.shape[0])) * tN * 0.5, "cell": cell}


def prepare(case, seed):
    c = dict(case)
    torch.cuda.current_device()
    s = {"c": c, "i": 0}
    if c["do"] == "batch":
        rs = np.random.default_rng(977 + c["cases"])   # the cases' own sizes do not depend on the seed
        s.update(batch=None, cases=[])                 # the batch goes before its cases
        for j in range(c["cases"]):
            k = dict(c)
            if c["mesh"] == "box":
                k["size"] = 2 * int(rs.integers(2, max(3, int(c["size"]) // 2 + 1)))
            ppc = c["ppc"] * float(rs.uniform(0.3, 1.7))
            k["Ma"], k["aoa"] = c["Ma"] * float(rs.uniform(0.6, 1.5)), float(rs.uniform(0.0, 40.0))
            dm, mess = constants(k, ppc)
            one = make_case(k, dm, mess, 7000 + 64 * seed + j, nss=10 ** 9, nscheme=50, nrepeat=100)
            one.fill_freestream(ppc, 9000 + 64 * seed + j)
            one.statistic_macroPre()
            one.sync()
            s["cases"].append(one)
        s["batch"] = gpu.Batch(s["cases"])
        return s
    dm, mess = constants(c)
    if c["do"] == "trace":
        s["case"] = make_case(c, dm, mess, seed)
        p = W.trace_particles(dm, mess, c["count"], seed, C.inflow_direction(c["aoa"]))
        s["particles"] = (p["x"], p["v"], p["dt"], p["cell"])
        return s
    if c["do"] == "restart":
        s["case"] = make_case(c, dm, mess, seed)
        p = host_particles(c, dm, mess, seed)
        s["columns"] = [np.ascontiguousarray(p["x"][:, k]) for k in range(3)] + \
                       [np.ascontiguousarray(p["v"][:, k]) for k in range(3)] + [p["ir"], p["cell"]]
        return s
    if c["do"] == "gsis":
        one = make_case(c, dm, mess, seed)
        one.fill_freestream(c["ppc"], seed + 17)
        one.sync()
        rs = np.random.default_rng(seed)
        u, _, tN = W.freestream(mess, C.inflow_direction(c["aoa"]))
        vol = dm.cells["area"].astype(float)
        free = c["ppc"] * dm.ncell / vol.sum() * float(mess["Neff"]) / float(mess["n_ref"])
        s["ns"] = []
        for _ in range(2):      # two successive NS solutions, taken in turn
            ns = np.empty((dm.ncell, 6))
            ns[:, 0] = free * rs.uniform(0.9, 1.1, dm.ncell)
            ns[:, 1:4] = u + 0.05 * rs.standard_normal((dm.ncell, 3))
            ns[:, 4:6] = tN * rs.uniform(0.95, 1.05, (dm.ncell, 2))
            s["ns"].append(ns)
        s["accepted"] = (rs.random(dm.ncell) < c["gate"]).astype(np.int8)
        s["case"] = one
        return s
    # every sampler runs, as in the second half of a run
    one = make_case(c, dm, mess, seed, nss=0, nscheme=400, nrepeat=c["steps"], wall_stats=int(c["walls"]))
    one.fill_freestream(c["ppc"], 1000 + seed)
    one.statistic_macroPre()
    one.sync()
    s["case"] = one
    return s


def run(s):
    c = s["c"]
    if c["do"] == "batch":
        s["batch"].step(c["steps"])
        s["batch"].sync()
        return [k.macro(gpu.MACRO_LOCAL) for k in s["cases"]]
    one = s["case"]
    if c["do"] == "window":
        for _ in range(c["steps"]):
            s["i"] += 1
            one.step(s["i"])
        out = {"record": one.macro(gpu.MACRO_RECORD), "particles": one.particle_count()}
        if c["walls"]:
            out["wall"] = one.wall()
        return out
    if c["do"] == "stages":
        for _ in range(c["steps"]):
            s["i"] += 1
            one.preprocesseffquad(s["i"])
            one.advection(s["i"])
            one.cache2chain()
            one.collisionDSMC()
            one.statistic_macro(s["i"])
        return {"record": one.macro(gpu.MACRO_RECORD), "counts": one.counts(), "state": one.cell_state()}
    if c["do"] == "gsis":
        s["i"] += 1
        report = one.molecular_velocity_change(s["ns"][s["i"] % 2], s["accepted"])
        one.statistic_macroPre()
        return {"report": report, "local": one.macro(gpu.MACRO_LOCAL)}
    if c["do"] == "restart":
        one.upload_columns(*s["columns"])
        one.statistic_macroPre()
        x, v, ir, cell = one.download_particles()
        return {"local": one.macro(gpu.MACRO_LOCAL), "x": x, "v": v, "ir": ir, "cell": cell}
    return one.trace(*s["particles"], stop_at_wall=True)


def work(case):
    c = case
    n = cells_of(c)
    real = 4 if c["precision"] == "mixed" else 8
    state = 7 * real + 4                      # position, velocity, Ir, cell
    if c["do"] in ("window", "stages", "batch"):
        # a step reads and writes the particles, reads the cells' face planes
        # and neighbours, and updates the cells' 54 sums
        m = c.get("cases", 1)
        if m > 1 and c["mesh"] == "box":
            n = n * 0.4                       # the batch's sizes are spread below the largest
        parts = n * c["ppc"] * m
        faces = {"box": 6, "capsule": 4, "prism": 5, "pyramid": 5}[c["mesh"]]
        per_cell = faces * (4 * real + 16) + 24 + 2 * 54 * 8 + 44
        # move: two dot products per face; sampling: the 18 moments; a
        # collision partner's draw and test per particle and step
        flops = parts * (faces * 12 + 50 + 60)
        return {"bytes": c["steps"] * (2.0 * parts * state + n * m * per_cell) + n * m * 18 * 8, "flops": c["steps"] * flops}
    if c["do"] == "gsis":
        parts = n * c["ppc"]
        return {"bytes": 2.0 * parts * state + n * (6 * 8 + 1 + 2 * 18 * 8 + 8), "flops": parts * 40.0}
    if c["do"] == "restart":
        parts = n * c["ppc"]
        return {"bytes": parts * (2.0 * (7 * 8 + 4) + 2.0 * state) + n * 18 * 8 * 2, "flops": parts * 60.0}
    # the inputs, the outputs, and about two cells' faces a particle
    return {"bytes": c["count"] * (8.0 * 7 + 4 + 8 * 7 + 4 * 5), "flops": c["count"] * 2.0 * 6 * 60}


# ---------------------------------------------------------------------------
# what plain numpy gives in 64 bits
# ---------------------------------------------------------------------------
def exact(case, seed):
    """Fields and particles of a restart, and the traced particles. The other
    kinds are Monte Carlo runs on the library's own random streams: nothing
    that plain numpy computes has their values."""
    c = dict(case)
    if c["do"] == "restart":
        dm, mess = constants(c)
        p = host_particles(c, dm, mess, seed)
        o = np.argsort(p["cell"], kind="stable")
        return {"local": macro_fields(dm, mess, p), "x": p["x"][o], "v": p["v"][o], "ir": p["ir"][o],
                "cell": p["cell"][o]}
    if c["do"] == "trace":
        dm, mess = constants(c)
        p = W.trace_particles(dm, mess, c["count"], seed, C.inflow_direction(c["aoa"]))
        return traced(dm, p, {tag: role for tag, role, _ in zones_of(c["mesh"])})
    return None


def macro_fields(dm, mess, p):
    """[cell][18]: density, velocity, T, stress, heat flux, Tr and rotational
    heat flux from the particles of each cell."""
    nc, cell = dm.ncell, p["cell"]
    add = lambda w: np.bincount(cell, weights=w, minlength=nc)  # noqa: E731
    n = np.bincount(cell, minlength=nc).astype(float)
    nn = np.maximum(n, 1.0)
    u = np.stack([add(p["v"][:, k]) / nn for k in range(3)], 1)
    w = p["v"] - u[cell]
    w2 = (w ** 2).sum(1)
    rho = float(mess["Neff"]) / dm.cells["area"] * n / float(mess["n_ref"])
    f = 2.0 * rho / nn
    s = {(i, j): add(w[:, i] * w[:, j]) for i in range(3) for j in range(i, 3)}
    tr = (s[0, 0] + s[1, 1] + s[2, 2]) / 3.0
    q = np.zeros((nc, 18))
    q[:, 0], q[:, 1:4], q[:, 4] = rho, u, 2.0 / (3.0 * nn) * add(w2)
    q[:, 5], q[:, 7], q[:, 9] = f * (s[0, 0] - tr), f * (s[1, 1] - tr), f * (s[2, 2] - tr)
    q[:, 6], q[:, 8], q[:, 10] = f * s[0, 1], f * s[1, 2], f * s[0, 2]
    for k in range(3):
        q[:, 11 + k] = rho / nn * add(w[:, k] * w2)
        q[:, 15 + k] = f * add(w[:, k] * p["ir"])
    q[:, 14] = 4.0 / float(mess["dr"]) / nn * add(p["ir"])
    q[n == 0] = 0.0
    return q


def triangles(dm):
    """[cell][12] triangles of hexahedral cells: corner, two edges, face, half."""
    ends = {0: ((0, 1, 2), (0, 2, 3)), 1: ((0, 1, 3), (1, 2, 3))}
    pts = dm.points.reshape(-1, 3)
    nodes, split = dm.edges["faceMap"][:, :4], np.where(dm.split == 1, 1, 0)
    pick = np.array([ends[0], ends[1]])                                  # [split][half][corner]
    tri = np.take_along_axis(nodes[:, None, :].repeat(2, 1), pick[split], 2)   # [face][half][corner]
    faces = dm.cells["cell2face"]                                        # [cell][6]
    t = pts[tri[faces]].reshape(dm.ncell, 12, 3, 3)
    return t[:, :, 0], t[:, :, 1] - t[:, :, 0], t[:, :, 2] - t[:, :, 0], faces.repeat(2, 1), np.tile([1, 2], 6)


def traced(dm, p, role_of):
    a, e1, e2, face_of, half_of = triangles(dm)
    role = np.array([role_of.get(int(t), 0) for t in dm.edges["faceTag"]])
    ends = dm.edges["faceMap"][:, 4:6]
    n = p["cell"].shape[0]
    x, v, dt, cell = p["x"].copy(), p["v"].copy(), p["dt"].copy(), p["cell"].astype(np.int64)
    out_cell, ifout = cell.copy(), np.zeros(n, np.int64)
    hit, half, cross = np.full(n, -1), np.zeros(n, np.int64), np.zeros(n, np.int64)
    last_face, last_half = np.full(n, -1), np.full(n, -1)
    act = np.arange(n)
    for _ in range(400):
        if not act.size:
            break
        c, d, o = cell[act], v[act][:, None, :], x[act][:, None, :]
        h = np.cross(d, e2[c])
        det = (e1[c] * h).sum(-1)
        with np.errstate(divide="ignore", invalid="ignore"):
            s = o - a[c]
            b1 = (s * h).sum(-1) / det
            g = np.cross(s, e1[c])
            b2 = (d * g).sum(-1) / det
            t = (e2[c] * g).sum(-1) / det
        ok = (np.abs(det) >= 1e-14) & (b1 >= 0) & (b1 <= 1) & (b2 >= 0) & (b1 + b2 <= 1) & (t > 1e-14)
        same = face_of[c] == last_face[act][:, None]
        ok &= ~(same & ((last_half[act] < 1)[:, None] | (half_of == last_half[act][:, None])))
        t = np.where(ok, t, np.inf)
        k = t.argmin(1)
        t = t[np.arange(act.size), k]
        f, hf = face_of[c, k], half_of[k]
        none = ~np.isfinite(t)
        stay = ~none & (t >= dt[act])
        x[act[stay]] += v[act[stay]] * dt[act[stay]][:, None]
        dt[act[stay | none]] = 0.0
        out_cell[act[stay]] = cell[act[stay]]
        out_cell[act[none]], ifout[act[none]] = c[none], -1
        go = ~none & ~stay
        act, t, f, hf, c = act[go], t[go], f[go], hf[go], c[go]
        r = role[f]
        first = (r != 1) & (hit[act] < 0)
        hit[act[first]], half[act[first]] = f[first], hf[first]
        x[act] += v[act] * t[:, None]
        dt[act] -= t
        wall = r == 4
        cross[act[~wall]] += 1
        last_face[act], last_half[act] = f, hf
        left = (r == 2) | (r == 3)
        dt[act[left]] = 0.0
        out_cell[act[left]], ifout[act[left]] = -1, -1
        out_cell[act[wall]] = c[wall]
        inner = r == 1
        i = act[inner]
        other = ends[f[inner]]
        cell[i] = np.where(other[:, 0] == c[inner], other[:, 1], other[:, 0])
        ifout[i] = 1
        mirror = act[r == 5]
        nrm = dm.edges["edgeNormal"][f[r == 5]]
        v[mirror] -= 2.0 * (v[mirror] * nrm).sum(1)[:, None] * nrm
        act = act[inner | (r == 5)]
    whole = lambda q: q.astype(np.int32)  # noqa: E731
    return {"cell": whole(out_cell), "ifout": whole(ifout), "face": whole(hit), "tri": whole(half),
            "ncross": whole(cross), "x": x, "v": v, "dt": dt}
