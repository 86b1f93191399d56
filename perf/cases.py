"""The work that programs of this library have it do, as measurable cases.

A case is one simulation (or, for ``kind`` "serve", a handful of them in one
batch): a lattice with its walls and body force, blood cells placed in it, the
precision form and launch mode of its handle.  A pass steps it by ``steps``
iterations the way a case program does and reads the state it writes out.
Sizes come from the repository's workloads (``hemocell_gb300/cases.py``,
``hemocell_gb300/serving.py``, the C++ example, the tests) and odd or ragged
sizes between them.

Step counts are even: ``read_fluid`` reports half the last force on wall nodes,
and the force field holds nothing there after an even number of steps.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from hemocell_gb300 import _lib as L
from hemocell_gb300 import cases as workloads
from hemocell_gb300.hemocell import Batch, HemoCell, Material

DX, DT, RHO_P, KBT = workloads.DX, workloads.DT, workloads.RHO_P, workloads.KBT

# every field of a case and what it is when a case does not name it
DEFAULTS = {
    "kind": "box",          # "box", "pipe" (cylinder along z) or "serve" (a batch of sheared boxes)
    "nx": 32, "ny": 32, "nz": 32,
    "walls": "shear",       # box: "shear" (moving z walls), "periodic", "closed", "obstacles" (spheres in a periodic box)
    "form": "f64",          # "f64" (the plain form) or "f32" (the mixed form)
    "batched": True,        # one launch per stage over all cell types, graph replay; False: one per stage and type
    "steps": 100,           # iterations of a pass
    "calls": "whole",       # iterate(steps); "single": iterate(1) in a loop; "stream": with body force and positions each step
    "rbc": 0, "plt": 0, "wbc": 0,   # cells of each type at most (as many as have room)
    "triangles": 600,       # least faces of an RBC mesh (600 -> 642 vertices, 320 -> 162)
    "material_every": 1, "velocity_every": 1,   # timescale separation
    "repulsion": False,     # cell-cell and wall repulsion, every step
    "stretch": False,       # external forces on the outermost vertices of the first cell
    "autotune": False,      # the program lets the library time its launch shapes once
    "tau": 1.0,
    "solves": 0,            # serve: how many boxes, edges from nx to nz
}


def _full(case):
    c = dict(DEFAULTS)
    c.update(case)
    return c


def listed():
    return [
        # the smoke run and the smallest example: a coarse cell in a small Couette
        # box, the default handle, iterate() called once per step
        {"name": "cell_24_f64_single", "nx": 24, "ny": 24, "nz": 24, "batched": False, "steps": 20,
         "calls": "single", "rbc": 1, "triangles": 320},
        # oneCellShear: one RBC in a 50^3 Couette box with the default handle
        {"name": "shear_50_f64", "nx": 50, "ny": 50, "nz": 50, "batched": False, "steps": 100, "rbc": 1},
        # the optical-tweezer validation: closed box, static walls, forced vertices
        {"name": "stretch_f64", "nx": 52, "ny": 26, "nz": 26, "walls": "closed", "batched": False, "steps": 100,
         "rbc": 1, "stretch": True, "tau": 1.82},
        # continuous batching of small independent solves (the serving mix)
        {"name": "serve_8_f32", "kind": "serve", "form": "f32", "nx": 32, "nz": 96, "rbc": 8, "steps": 200, "solves": 8},
        # the benchmark's pipe at 25% haematocrit, launch shapes tuned once
        {"name": "pipe_f32_tuned", "kind": "pipe", "nx": 64, "ny": 64, "nz": 256, "form": "f32", "steps": 800,
         "rbc": 280, "autotune": True},
        # the same pipe in the reference's arithmetic
        {"name": "pipe_f64", "kind": "pipe", "nx": 64, "ny": 64, "nz": 256, "form": "f64", "steps": 100, "rbc": 280},
        # the suspension of all three cell types in a periodic cube (Kolmogorov flow)
        {"name": "suspension_128_f32", "nx": 128, "ny": 128, "nz": 128, "walls": "periodic", "form": "f32",
         "steps": 300, "rbc": 960, "plt": 96, "wbc": 2},
        # a smaller, ragged suspension in FP64
        {"name": "suspension_f64", "nx": 67, "ny": 81, "nz": 50, "walls": "periodic", "form": "f64", "steps": 60,
         "rbc": 110, "plt": 11, "wbc": 1},
        # plasma through a bed of obstacles on a ragged lattice, no cells (warm-up of every porous or vessel run)
        {"name": "channel_f32", "nx": 181, "ny": 117, "nz": 93, "walls": "obstacles", "form": "f32", "steps": 600},
        # fluid alone in FP64, moving walls
        {"name": "couette_f64", "nx": 150, "ny": 150, "nz": 150, "walls": "shear", "form": "f64", "steps": 60},
        # the reference's performance-testing timescales (material every 20, velocity every 5 steps), ragged pipe,
        # with repulsion between cells and from the wall
        {"name": "pipe_every_f32", "kind": "pipe", "nx": 61, "ny": 59, "nz": 131, "form": "f32", "steps": 400,
         "rbc": 120, "material_every": 20, "velocity_every": 5, "repulsion": True},
        # a program that sets the body force and takes the positions every step
        {"name": "pipe_stream_f32", "kind": "pipe", "nx": 49, "ny": 53, "nz": 160, "form": "f32", "steps": 400,
         "rbc": 60, "calls": "stream"},
    ]


def draw(rng):
    """A case of the listed ones' ranges: sizes spread over their logarithm."""
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["box", "box", "box", "pipe", "pipe", "serve"])
    form = rng.choice(["f32", "f64"])
    c = {"kind": kind, "form": form}
    if kind == "serve":
        lo = logint(32, 48)
        c.update(nx=lo, nz=logint(lo, 96), rbc=rng.randint(1, 8), solves=rng.randint(2, 10 if form == "f32" else 4),
                 steps=2 * rng.randint(25, 100))
    elif kind == "pipe":
        d = logint(36, 72)
        c.update(nx=d, ny=d + rng.randint(-3, 3), nz=logint(40, 256), rbc=logint(8, 280),
                 steps=2 * rng.randint(20, 50) if form == "f64" else 2 * rng.randint(50, 200),
                 calls=rng.choice(["whole", "whole", "single", "stream"]))
        if rng.random() < 0.3:
            c.update(material_every=20, velocity_every=rng.choice([1, 5]))
        if rng.random() < 0.3:
            c.update(repulsion=True)
    else:
        walls = rng.choice(["shear", "periodic", "obstacles", "closed"])
        c.update(walls=walls, nx=logint(24, 140), ny=logint(24, 140), nz=logint(24, 140),
                 tau=rng.choice([1.0, 1.0, round(rng.uniform(0.6, 1.8), 2)]),
                 batched=rng.random() < 0.7, steps=2 * rng.randint(15, 40) if form == "f64" else 2 * rng.randint(40, 150))
        if walls != "obstacles" and rng.random() < 0.75:
            c.update(rbc=logint(1, 700), triangles=rng.choice([320, 600, 600]))
            if min(c["nx"], c["ny"], c["nz"]) >= 40:
                c.update(plt=logint(1, 60), wbc=rng.randint(0, 2))
    return c


# --- placement ------------------------------------------------------------
def _rotation(rng, axis, tilt):
    """A rotation taking the discs' template axis (y) to `axis`, turned about
    it by a random angle and tilted by up to `tilt` radians."""
    a = rng.uniform(0, 2 * math.pi)
    turn = np.array([[math.cos(a), 0, math.sin(a)], [0, 1, 0], [-math.sin(a), 0, math.cos(a)]])
    t, p = rng.uniform(-tilt, tilt), rng.uniform(-tilt, tilt)
    tx = np.array([[1, 0, 0], [0, math.cos(t), -math.sin(t)], [0, math.sin(t), math.cos(t)]])
    tz = np.array([[math.cos(p), -math.sin(p), 0], [math.sin(p), math.cos(p), 0], [0, 0, 1]])
    perm = np.roll(np.eye(3), axis - 1, axis=0)  # a cyclic permutation: y goes to `axis`
    return perm @ tx @ tz @ turn


def _place(rng, mesh, rot, centre):
    """A cell as a flow has it: its rest shape strained by up to two percent per
    axis at constant volume (the membrane forces of an undeformed cell are nothing
    but rounding), rotated and moved to its place."""
    e = rng.uniform(-0.02, 0.02, 2)
    strain = np.exp(np.array([e[0], e[1], -e[0] - e[1]]))
    return (mesh.xyz * strain) @ rot.T + np.asarray(centre)


def _pipe_cells(rng, c, types, radius):
    """Discs stacked along the pipe, in hexagonal layers 6.4 nodes apart."""
    room = radius - 1.0 - 7.9
    best = []
    for ox, oy in ((0.0, 0.0), (8.0, 8.0 / math.sqrt(3.0)), (8.0, 0.0)):
        pts = [(16 * i + 8 * j + ox, 8 * math.sqrt(3.0) * j + oy) for i in range(-6, 7) for j in range(-6, 7)]
        pts = [p for p in pts if math.hypot(*p) <= room]
        best = pts if len(pts) > len(best) else best
    layers = max(1, int(c["nz"] / 6.4))
    dz = c["nz"] / layers
    slots = []
    for k in range(layers):
        a = rng.uniform(0, 2 * math.pi)
        for x, y in best:
            slots.append(((c["nx"] - 1) / 2 + math.cos(a) * x - math.sin(a) * y,
                          (c["ny"] - 1) / 2 + math.sin(a) * x + math.cos(a) * y, (k + 0.5) * dz + rng.uniform(-0.05, 0.05)))
    keep = sorted(rng.permutation(len(slots))[: c["rbc"]])
    return [(0, _place(rng, types[0].mesh, _rotation(rng, 2, 0.05), slots[k])) for k in keep]


def _box_cells(rng, c, types):
    """Blocks of 16^3 nodes, each with two stacked RBCs, eight platelets or a WBC."""
    lo = np.array([0.0, 0.0, 0.0])
    hi = np.array([c["nx"], c["ny"], c["nz"]], float)
    if c["walls"] == "closed":
        lo += 1.5
        hi -= 2.5
    elif c["walls"] == "shear":
        lo[2], hi[2] = 1.5, c["nz"] - 2.5
    size = hi - lo
    n = np.maximum(1, (size / 16.0).astype(int))
    step = size / n
    blocks = [lo + (np.array([i, j, k]) + 0.5) * step for i in range(n[0]) for j in range(n[1]) for k in range(n[2])]
    blocks = [blocks[k] for k in rng.permutation(len(blocks))]
    two = min(step) >= 16.0
    cells = []
    for _ in range(min(c["wbc"], len(blocks) - 1 if c["rbc"] else len(blocks)) if two else 0):
        cells.append((2, _place(rng, types[2].mesh, _rotation(rng, 1, 0.5), blocks.pop())))
    left = c["plt"] if two else 0
    while left > 0 and len(blocks) > 1:
        b = blocks.pop()
        for s in range(min(8, left)):
            off = np.array([(s & 1) - 0.5, (s >> 1 & 1) - 0.5, (s >> 2) - 0.5]) * 8.0 + rng.uniform(-0.8, 0.8, 3)
            cells.append((1, _place(rng, types[1].mesh, _rotation(rng, int(rng.integers(3)), 0.5), b + off)))
        left -= 8
    left = c["rbc"]
    per_block = 2 if two and left > 1 else 1
    for b in blocks:
        axis = int(rng.integers(3))
        for s in range(min(per_block, left)):
            off = np.zeros(3)
            off[axis] = (s - 0.5) * 8.0 if per_block == 2 else 0.0
            cells.append((0, _place(rng, types[0].mesh, _rotation(rng, axis, 0.05), b + off + rng.uniform(-0.08, 0.08, 3))))
        left -= per_block
        if left <= 0:
            break
    return sorted(cells, key=lambda t: t[0])


def _scene(case, seed):
    """Everything of one simulation as plain arrays: what both a handle and a
    64-bit restatement start from."""
    c = _full(case)
    rng = np.random.default_rng([int(seed), 20, c["nx"], c["ny"], c["nz"]])
    dims = (c["nx"], c["ny"], c["nz"])
    nx, ny, nz = dims
    s = {"case": c, "dims": dims, "periodic": (1, 1, 1), "flags": None, "walls": {}, "mode": L.HC_BODY_NONE,
         "body": (0.0, 0.0, 0.0), "u0": (0.0, 0.0, 0.0), "tau": float(c["tau"]), "types": [], "cells": [], "ext": None}
    stiff = math.exp(rng.uniform(math.log(0.7), math.log(2.0)))
    rate = rng.uniform(100.0, 500.0)
    if c["rbc"] or c["plt"] or c["wbc"]:
        s["types"] = [workloads.rbc_type(c["triangles"])]
        if c["plt"] or c["wbc"]:
            s["types"] += [workloads.plt_type(320), workloads.wbc_type(5120)]
        m = s["types"][0].material
        s["types"][0].material = Material(**{**m.__dict__, "kLink": m.kLink * stiff, "kBend": m.kBend * stiff})
    nu = (c["tau"] - 0.5) / 3.0
    if c["kind"] == "pipe":
        radius = (min(nx, ny) - 1) / 2.0 - 1.5
        s["flags"] = workloads.cylinder_flags(nx, ny, nz, radius)
        u_max = rng.uniform(0.5, 2.0) * 1e-3 * DT / DX
        s["mode"], s["body"] = L.HC_BODY_UNIFORM, (0.0, 0.0, 4.0 * nu * u_max / radius ** 2)
        s["cells"] = _pipe_cells(rng, c, s["types"], radius)
        return s
    if c["walls"] == "shear":
        s["flags"], s["walls"] = workloads.shear_walls(dims, rate)
        s["periodic"] = (1, 1, 0)
    elif c["walls"] == "closed":
        f = np.ones((nz, ny, nx), np.uint8)
        f[1:-1, 1:-1, 1:-1] = 0
        s["flags"], s["walls"], s["periodic"] = f.reshape(-1), {1: (0.0, 0.0, 0.0)}, (0, 0, 0)
        s["mode"], s["body"] = L.HC_BODY_UNIFORM, tuple(rng.uniform(-1e-6, 1e-6, 3))
    elif c["walls"] == "obstacles":
        Z, Y, X = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij", sparse=True)
        f = np.zeros((nz, ny, nx), np.uint8)
        for _ in range(max(1, nx * ny * nz // 30000)):
            r, q = rng.uniform(4.0, 9.0), rng.uniform(0, 1, 3) * dims
            d = [np.abs(A - q[a]) for a, A in enumerate((X, Y, Z))]
            d = [np.minimum(v, dims[a] - v) for a, v in enumerate(d)]
            f[d[0] ** 2 + d[1] ** 2 + d[2] ** 2 <= r * r] = 1
        s["flags"] = f.reshape(-1)
        s["mode"], s["body"] = L.HC_BODY_UNIFORM, (2e-6 * rng.uniform(0.5, 2.0), 0.0, 0.0)
    else:
        s["mode"] = L.HC_BODY_KOLMOGOROV
        s["body"] = (rng.uniform(2e-3, 5e-3) * nu * (2 * math.pi / nz) ** 2, 0.0, 0.0)
    if s["types"]:
        s["cells"] = _box_cells(rng, c, s["types"])
    elif c["walls"] in ("periodic", "obstacles"):
        s["u0"] = tuple(rng.uniform(-2e-3, 2e-3, 3))
    if c["stretch"] and s["cells"]:
        s["ext"] = workloads.stretch_forces(s["cells"][0][1], rng.uniform(25.0, 125.0))
    return s


def _scenes(case, seed):
    """The simulations of a case: one, or a batch of sheared boxes."""
    c = _full(case)
    if c["kind"] != "serve":
        return [_scene(c, seed)]
    out = []
    for k in range(c["solves"]):
        edge = int(round(c["nx"] * (c["nz"] / c["nx"]) ** (k / max(1, c["solves"] - 1))))
        out.append(_scene({**c, "kind": "box", "walls": "shear", "nx": edge, "ny": edge, "nz": edge,
                           "rbc": 1 + (k * 3) % c["rbc"]}, int(seed) * 1000 + k))
    return out


def _build(s):
    c = s["case"]
    hc = HemoCell(*s["dims"], periodic=s["periodic"], dx=DX, dt=DT, rho_p=RHO_P, kBT_p=KBT, tau=s["tau"],
                  form=L.HC_FORM_MIXED_F32 if c["form"] == "f32" else L.HC_FORM_PLAIN_F64,
                  launch=L.HC_LAUNCH_BATCHED if c["batched"] else L.HC_LAUNCH_PER_STAGE)
    if s["flags"] is not None:
        hc.set_flags(s["flags"])
    for cls, u in s["walls"].items():
        hc.set_wall_velocity(cls, u)
    hc.latticeEquilibrium(1.0, s["u0"])
    hc.setExternalVector(s["mode"], s["body"])
    for t in s["types"]:
        hc.addCellType(t.name, t.model, t.material, t.mesh)
    for t in range(len(s["types"])):
        xyz = [x for k, x in s["cells"] if k == t]
        if xyz:
            hc.add_cells_xyz(t, np.concatenate(xyz))
    if c["material_every"] > 1 or c["velocity_every"] > 1:
        hc.setMaterialTimeScaleSeparation([c["material_every"]] * len(s["types"]), c["velocity_every"])
    if c["repulsion"]:
        hc.setRepulsion(*REPULSION)
        hc.enableBoundaryParticles(*WALL_REPULSION)
    if s["ext"] is not None:
        hc.set_vertex_forces(*s["ext"])
    if c["autotune"]:
        hc.autotune()
    return hc


REPULSION = (1e-6, 0.5)         # constant, cutoff in micrometres
WALL_REPULSION = (5e-7, 0.5)


def prepare(case, seed):
    c = _full(case)
    scenes = _scenes(case, seed)
    state = {"case": c, "hc": [_build(s) for s in scenes], "scenes": [(s["mode"], s["body"]) for s in scenes]}
    if c["kind"] == "serve":
        state["batch"] = Batch(64 << 30, max_slots=64, chunk_steps=50)
    if c["calls"] == "stream":
        n = state["hc"][0].stats().vertices
        state["pinned"] = [torch.empty((n, 3), dtype=torch.float64, pin_memory=True).numpy() for _ in range(2)]
    return state


def _kept(c, a):
    """The mixed form's velocities are 32-bit numbers that the API hands out as
    doubles: a program keeps them as what they are."""
    a = torch.from_numpy(a)
    return a.float() if c["form"] == "f32" else a


def _vertices(c, hc):
    """Positions and velocities, and the plain form's forces.  The mixed form's
    vertex forces are differences of nearly equal 32-bit lengths, 1e-4 off by
    themselves and assembled anew from the positions in the next step; what they
    did is in the velocities."""
    x, v, f = hc.read_vertices()
    out = {"x": torch.from_numpy(x), "v": _kept(c, v)}
    if c["form"] == "f64":
        out["f"] = torch.from_numpy(f)
    return out


def run(state):
    c, hc = state["case"], state["hc"][0]
    n = c["steps"]
    if c["kind"] == "serve":
        b = state["batch"]
        for k, h in enumerate(state["hc"]):
            if not b.admit(h, n, k):
                raise RuntimeError("the batch refused a solve")
        out, left = {}, len(state["hc"])
        while left:
            b.pump(2.0)
            while (got := b.pop()) is not None:
                tag, h, status = got
                if status != L.HC_OK:
                    raise RuntimeError("a solve failed")
                out[str(tag)] = _vertices(c, h)
                b.release(h, destroy=False)
                left -= 1
        return out
    if c["calls"] == "single":
        for _ in range(n):
            hc.iterate()
    elif c["calls"] == "stream":
        pos = state["pinned"]
        mode, body = state["scenes"][0]
        for k in range(n):
            hc.setExternalVector(mode, body)
            hc.iterate(1)
            hc.read_positions_async(pos[k & 1], k & 1)
            if k:
                hc.wait_positions((k - 1) & 1)
        hc.wait_positions((n - 1) & 1)
        return {"streamed": torch.from_numpy(pos[(n - 1) & 1].copy()), **_vertices(c, hc)}
    else:
        hc.iterate(n)
    out = _vertices(c, hc) if state["hc"][0].cell_types else {}
    rho, u = hc.read_fluid()
    out["rho"], out["u"] = torch.from_numpy(rho), _kept(c, u)
    return out


def work(case):
    """Each step reads and writes the populations and the force of every fluid
    node and the position, velocity and force of every vertex."""
    total_b = total_f = 0.0
    c = _full(case)
    s = 4 if c["form"] == "f32" else 8
    for sc in _scenes(case, 1):
        N = int(np.prod(sc["dims"]))
        fluid = N if sc["flags"] is None else int((sc["flags"] == 0).sum())
        V = sum(x.shape[0] for _, x in sc["cells"])
        total_b += c["steps"] * (fluid * (38 * s + 6 * s) + V * (2 * 24 + 12 * s)) + V * 72
        total_b += 0 if c["kind"] == "serve" or c["calls"] == "stream" else 32 * N
        total_b += c["steps"] * 24 * V if c["calls"] == "stream" else 0
        total_f += c["steps"] * (fluid * 250.0 + V * 800.0)
    return {"bytes": total_b, "flops": total_f}


# --- the same step in 64 bits, in plain torch ------------------------------
C3 = np.array([(0, 0, 0), (-1, 0, 0), (0, -1, 0), (0, 0, -1), (-1, -1, 0), (-1, 1, 0), (-1, 0, -1), (-1, 0, 1),
               (0, -1, -1), (0, -1, 1), (1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, -1, 0), (1, 0, 1), (1, 0, -1),
               (0, 1, 1), (0, 1, -1)])
W = np.array([1 / 3] + [1 / 18 if abs(v).sum() == 1 else 1 / 36 for v in C3[1:]])
OPP = [0] + [i + 9 if i <= 9 else i - 9 for i in range(1, 19)]


class _Type:
    """Rest state and lattice-unit constants of one cell type."""

    def __init__(self, spec, dev):
        m, mat = spec.mesh, spec.material
        self.model = spec.model
        t = torch.as_tensor(np.asarray(m.tris, np.int64), device=dev)
        P = torch.as_tensor(m.xyz, dtype=torch.float64, device=dev)
        self.tris, self.nv = t, P.shape[0]
        a = torch.cat([t[:, 0], t[:, 1], t[:, 2]])
        b = torch.cat([t[:, 1], t[:, 2], t[:, 0]])
        third = torch.cat([t[:, 2], t[:, 0], t[:, 1]])
        face = torch.arange(t.shape[0], device=dev).repeat(3)
        key = a * self.nv + b
        order = torch.argsort(key)
        e = a < b
        self.ea, self.eb = a[e], b[e]
        fwd = face[e], third[e]
        back = order[torch.searchsorted(key[order], self.eb * self.nv + self.ea)]
        self.t0, self.t1 = face[back], fwd[0]          # the triangle with the edge b->a, then a->b
        self.o0, self.o1 = third[back], fwd[1]
        self.valence = torch.zeros(self.nv, dtype=torch.float64, device=dev).index_add_(
            0, torch.cat([self.ea, self.eb]), torch.ones(2 * len(self.ea), dtype=torch.float64, device=dev))
        inner = torch.as_tensor(np.asarray(m.inner, np.int64).reshape(-1, 2), device=dev)
        self.ia, self.ib = inner[:, 0], inner[:, 1]
        df = RHO_P * DX ** 4 / DT ** 2
        kbt, nfs = KBT / (df * DX), 1280.0 / t.shape[0]
        self.k_link = mat.kLink * kbt / (7.5e-9 / DX)
        self.k_bend = mat.kBend * kbt / (5e-7 / DX)
        self.k_volume = mat.kVolume * nfs * kbt / (5e-7 / DX)
        self.k_area = mat.kArea * nfs * kbt / (5e-7 / DX)
        self.eta = mat.eta_m * DX / DT / df
        self.k_rigid, self.k_cyto = mat.kInnerRigid / df, mat.kCytoskeleton / df
        self.core, self.radius = mat.coreRadius / DX, mat.radius / DX
        X = P[None]
        n, area, _ = self.faces(X)
        self.a0, self.l0 = area[0], (P[self.eb] - P[self.ea]).norm(dim=1)
        self.area_mean, self.edge_mean = self.a0.mean(), self.l0.mean()
        self.v_eq = self.volume(X)[0]
        self.angle0 = self.angle(X, n)[0]
        self.d0 = self.patch(X, n)[1][0]
        self.i0 = (P[self.ib] - P[self.ia]).norm(dim=1)

    def faces(self, X):
        v0, v1, v2 = (X[:, self.tris[:, k]] for k in range(3))
        n = torch.linalg.cross(v1 - v0, v2 - v0)
        l = n.norm(dim=-1)
        return n / l[..., None], 0.5 * l, (v0 + v1 + v2) / 3.0

    def volume(self, X):
        Y = X - X[:, :1]
        v0, v1, v2 = (Y[:, self.tris[:, k]] for k in range(3))
        return (v0 * torch.linalg.cross(v1, v2)).sum(dim=(-1, -2)) / 6.0

    def angle(self, X, n):
        uv = X[:, self.eb] - X[:, self.ea]
        uv = uv / uv.norm(dim=-1, keepdim=True)
        n1, n2 = n[:, self.t0], n[:, self.t1]
        return torch.atan2((torch.linalg.cross(n1, n2) * uv).sum(-1), (n1 * n2).sum(-1))

    def patch(self, X, n):
        pn = torch.zeros_like(X)
        for k in range(3):
            pn.index_add_(1, self.tris[:, k], n)
        pn = pn / pn.norm(dim=-1, keepdim=True)
        s = torch.zeros_like(X).index_add_(1, self.ea, X[:, self.eb]).index_add_(1, self.eb, X[:, self.ea])
        return pn, (pn * (s / self.valence[:, None] - X)).sum(-1)

    def forces(self, X, vel):
        X = X - X[:, :1]
        f = torch.zeros_like(X)
        n, area, cen = self.faces(X)
        ar = (area - self.a0) / self.a0
        af = (self.k_area * (ar + ar / (0.09 - ar * ar).abs()))[..., None]
        vf = (self.volume(X) - self.v_eq) / self.v_eq
        vf = -self.k_volume * vf / (0.01 - vf * vf).abs()
        push = n * (vf[:, None] * (area / self.area_mean))[..., None]
        for k in range(3):
            f.index_add_(1, self.tris[:, k], (cen - X[:, self.tris[:, k]]) * af + push)
        ev = X[:, self.eb] - X[:, self.ea]
        l = ev.norm(dim=-1)
        uv = ev / l[..., None]
        ef = (l - self.l0) / self.l0
        fe = uv * (self.k_link * (ef + ef / (9.0 - ef * ef).abs()))[..., None]
        if self.model != 0 or self.eta != 0.0:
            fv = uv * (((vel[:, self.eb] - vel[:, self.ea]) * uv).sum(-1) * self.eta)[..., None]
            mm = fv.norm(dim=-1, keepdim=True)
            fe = fe + torch.where(mm > 12.5, fv * (12.5 / mm.clamp_min(1e-300)), fv)
        f.index_add_(1, self.ea, fe).index_add_(1, self.eb, -fe)
        if self.model == 1:
            d = self.angle(X, n) - self.angle0
            b = (n[:, self.t0] + n[:, self.t1]) * (0.5 * self.k_bend * (d + d / (2.467 - d * d).abs()))[..., None]
            f.index_add_(1, self.ea, b).index_add_(1, self.eb, b)
            f.index_add_(1, self.o0, -b).index_add_(1, self.o1, -b)
        else:
            pn, dist = self.patch(X, n)
            d = (dist - self.d0) / self.edge_mean
            b = pn * (self.k_bend * (d + d / (0.0555 - d * d).abs()))[..., None]
            f = f + b
            r = b / self.valence[:, None]
            f.index_add_(1, self.ea, -r[:, self.eb]).index_add_(1, self.eb, -r[:, self.ea])
        if len(self.ia):
            ev = X[:, self.ib] - X[:, self.ia]
            l = ev.norm(dim=-1)
            uv = ev / l[..., None]
            if self.model == 1:
                fi = uv * (self.k_link * 5.0 * (l - self.i0) / self.i0)[..., None]
            else:
                s = torch.zeros_like(l)
                if self.model == 2:
                    s = torch.where(l < 2 * self.radius, -(1 - l / (2 * self.radius)) * self.k_cyto, s)
                    s = s + torch.where(l < 2 * self.core, -(1 - l / (2 * self.core)) * self.k_rigid, torch.zeros_like(l))
                fi = uv * s[..., None]
            f.index_add_(1, self.ia, fi).index_add_(1, self.ib, -fi)
        return f


class _Exact:
    def __init__(self, s):
        self.s, self.c = s, s["case"]
        self.dev = dev = "cuda" if torch.cuda.is_available() else "cpu"
        nx, ny, nz = self.dims = s["dims"]
        D = torch.float64
        flags = np.zeros(nx * ny * nz, np.uint8) if s["flags"] is None else s["flags"]
        fl = torch.as_tensor(flags.astype(np.int64), device=dev).reshape(nz, ny, nx)
        self.solid = fl != 0
        self.om = 1.0 / s["tau"]
        uw = torch.zeros((256, 3), dtype=D, device=dev)
        for k, u in s["walls"].items():
            uw[k] = torch.as_tensor(u, dtype=D)
        # bounce-back links and their moving-wall term, of population j pulled from x - c_j
        self.bounce, self.term = [None], [None]
        for j in range(1, 19):
            sh = tuple(int(v) for v in C3[j][::-1])
            src = torch.roll(fl, sh, (0, 1, 2))
            for a in range(3):
                if not s["periodic"][a] and C3[j][a]:
                    ix = [slice(None)] * 3
                    ix[2 - a] = 0 if C3[j][a] > 0 else -1
                    src[tuple(ix)] = 255
            self.bounce.append(src != 0)
            ci = torch.as_tensor(-C3[j], dtype=D, device=dev)
            self.term.append(6.0 * float(W[j]) * (uw[src] @ ci) if s["walls"] else 0.0)
        body = torch.zeros((3, nz), dtype=D, device=dev)
        if s["mode"] == L.HC_BODY_UNIFORM:
            body[:] = torch.as_tensor(s["body"], dtype=D, device=dev)[:, None]
        elif s["mode"] == L.HC_BODY_KOLMOGOROV:
            body[0] = s["body"][0] * torch.sin(2 * math.pi * torch.arange(nz, dtype=D, device=dev) / nz)
        self.body = body[:, :, None, None].expand(3, nz, ny, nx) * (~self.solid)
        u0 = torch.as_tensor(s["u0"], dtype=D, device=dev)
        self.f = torch.zeros((19, nz, ny, nx), dtype=D, device=dev)
        for j in range(19):
            cu = float((torch.as_tensor(C3[j], dtype=D, device=dev) * u0).sum())
            self.f[j] = float(W[j]) * (3 * cu + 4.5 * cu * cu - 1.5 * float((u0 * u0).sum()))
        self.f[:, self.solid] = 0.0
        self.F = self.body.clone()
        self.types = [_Type(t, dev) for t in s["types"]]
        self.x = [torch.as_tensor(np.stack([x for k, x in s["cells"] if k == t]), dtype=D, device=dev)
                  if any(k == t for k, _ in s["cells"]) else torch.zeros((0, ty.nv, 3), dtype=D, device=dev)
                  for t, ty in enumerate(self.types)]
        self.v = [torch.zeros_like(x) for x in self.x]
        self.fv = [torch.zeros_like(x) for x in self.x]
        df = RHO_P * DX ** 4 / DT ** 2
        self.f_limit = 50.0 / 1e12 / df
        self.it = 0
        if self.c["repulsion"]:
            near = torch.zeros_like(self.solid)
            for dz in (-1, 0, 1):
                for dy in (-1, 0, 1):
                    for dx in (-1, 0, 1):
                        near |= torch.roll(~self.solid, (dz, dy, dx), (0, 1, 2))
            self.wall = (near & self.solid).reshape(-1)

    def flat(self, parts):
        return torch.cat([p.reshape(-1, 3) for p in parts]) if parts else torch.zeros((0, 3), dtype=torch.float64, device=self.dev)

    def unflat(self, v):
        out, k = [], 0
        for x in self.x:
            n = x.shape[0] * x.shape[1]
            out.append(v[k:k + n].reshape(x.shape))
            k += n
        return out

    def stencil(self, x):
        q = torch.floor(x)
        fr = x - q
        nodes, w = [], []
        for s in range(8):
            o = torch.tensor([s >> 2, s >> 1 & 1, s & 1], device=self.dev)
            i = q.long() + o
            ok = torch.ones(len(x), dtype=torch.bool, device=self.dev)
            for a in range(3):
                if not self.s["periodic"][a]:
                    ok &= (i[:, a] >= 0) & (i[:, a] < self.dims[a])
                i[:, a] %= self.dims[a]
            n = i[:, 0] + self.dims[0] * (i[:, 1] + self.dims[1] * i[:, 2])
            wt = torch.where(o.bool(), fr, 1.0 - fr).prod(dim=1)
            w.append(torch.where(ok & ~self.solid.reshape(-1)[n], wt, torch.zeros_like(wt)))
            nodes.append(n)
        w = torch.stack(w)
        return torch.stack(nodes), w / w.sum(0).clamp_min(1e-300)

    def repel(self, x):
        cell, k = [], 0
        for p in self.x:
            cell.append(torch.arange(p.shape[0], device=self.dev).repeat_interleave(p.shape[1]) + k)
            k += p.shape[0]
        cell = torch.cat(cell)
        b = torch.floor(x + 0.5)
        r, i = x - b, b.long()
        dims = torch.tensor(self.dims, device=self.dev)
        i = i % dims
        key = i[:, 0] + self.dims[0] * (i[:, 1] + self.dims[1] * i[:, 2])
        order = torch.argsort(key, stable=True)
        sk = key[order]
        at = torch.arange(len(sk), device=self.dev) - torch.searchsorted(sk, sk)
        slots = torch.full((self.solid.numel(), 10), -1, dtype=torch.long, device=self.dev)
        fits = at < 10
        slots[sk[fits], at[fits]] = order[fits]
        f = torch.zeros_like(x)
        kc, rc = REPULSION[0], REPULSION[1] * 1e-6 / DX
        kw, rw = WALL_REPULSION[0], WALL_REPULSION[1] * 1e-6 / DX
        for s in range(27):
            d = torch.tensor([s % 3 - 1, s // 3 % 3 - 1, s // 9 - 1], device=self.dev)
            j = (i + d) % dims
            n = j[:, 0] + self.dims[0] * (j[:, 1] + self.dims[1] * j[:, 2])
            o = slots[n]
            dv = (r[:, None] - r[o]) - d.double()
            l = dv.norm(dim=-1)
            hit = (o >= 0) & (cell[o] != cell[:, None]) & (l < rc)
            sc = torch.where(hit, (2.0 if s == 13 else 1.0) * kc * rc / (l * l).clamp_min(1e-300), torch.zeros_like(l))
            f += (dv * sc[..., None]).sum(1)
            dv = r - d.double()
            l = dv.norm(dim=-1)
            sc = torch.where(self.wall[n] & (l < rw), kw * rw / (l * l).clamp_min(1e-300), torch.zeros_like(l))
            f += dv * sc[:, None]
        return f

    def moments(self, F):
        f = self.f
        rb = f.sum(0)
        j = [sum(float(C3[i][a]) * f[i] for i in range(1, 19) if C3[i][a]) for a in range(3)]
        return rb, torch.stack([(j[a] + 0.5 * F[a]) / (1.0 + rb) for a in range(3)])

    def step(self):
        c, x = self.c, self.flat(self.x)
        F = self.body.clone()
        if len(x):
            if self.s["ext"] is not None:
                g = self.flat(self.fv)
                ids, fo = self.s["ext"]
                g = g.index_add(0, torch.as_tensor(np.asarray(ids, np.int64), device=self.dev),
                                torch.as_tensor(fo, dtype=torch.float64, device=self.dev))
                self.fv = self.unflat(g)
            g = self.flat(self.fv)
            mag = g.norm(dim=1, keepdim=True)
            g = torch.where(mag > self.f_limit, g * (self.f_limit / mag.clamp_min(1e-300)), g)
            if c["repulsion"]:
                g = g + self.repel(x)
            nodes, w = self.stencil(x)
            Ff = F.reshape(3, -1)
            for k in range(8):
                Ff.index_add_(1, nodes[k], (g * w[k][:, None]).T)
        rb, u = self.moments(F)
        rho, uu, uF = 1.0 + rb, (u * u).sum(0), (u * F).sum(0)
        post = torch.empty_like(self.f)
        for j in range(19):
            cx = [float(v) for v in C3[j]]
            cu = sum((cx[a] * u[a] for a in range(3) if cx[a]), torch.zeros_like(rb))
            cF = sum((cx[a] * F[a] for a in range(3) if cx[a]), torch.zeros_like(rb))
            eq = float(W[j]) * (rb + rho * (3 * cu + 4.5 * cu * cu - 1.5 * uu))
            src = (1 - 0.5 * self.om) * float(W[j]) * (3 * (cF - uF) + 9 * cu * cF)
            post[j] = self.f[j] + self.om * (eq - self.f[j]) + src
        new = torch.empty_like(post)
        new[0] = post[0]
        for j in range(1, 19):
            new[j] = torch.roll(post[j], tuple(int(v) for v in C3[j][::-1]), (0, 1, 2))
            new[j] = torch.where(self.bounce[j], post[OPP[j]] - self.term[j], new[j])
        new[:, self.solid] = 0.0
        self.f, self.F = new, F
        if len(x):
            if self.it % c["velocity_every"] == 0:
                _, u = self.moments(F)
                u = u.reshape(3, -1)
                self.v = self.unflat(sum((u[:, nodes[k]] * w[k]).T for k in range(8)))
            self.x = [a + b for a, b in zip(self.x, self.v)]
            if self.it % c["material_every"] == 0:
                self.fv = [t.forces(a, b) if len(a) else a for t, a, b in zip(self.types, self.x, self.v)]
        self.it += 1

    def outputs(self, fluid):
        out = {}
        if self.types:
            out = {"x": self.flat(self.x), "v": self.flat(self.v)}
            if self.c["form"] == "f64":
                out["f"] = self.flat(self.fv)
        if fluid:
            rb, u = self.moments(self.F)
            u = u * (~self.solid)
            out["rho"], out["u"] = 1.0 + rb.reshape(-1), u.reshape(3, -1)
        return {k: v.cpu() for k, v in out.items()}


def exact(case, seed):
    c = _full(case)
    outs = []
    for s in _scenes(case, seed):
        e = _Exact(s)
        for _ in range(c["steps"]):
            e.step()
        outs.append(e.outputs(c["kind"] != "serve" and c["calls"] != "stream"))
    if c["kind"] == "serve":
        return {str(k): o for k, o in enumerate(outs)}
    if c["calls"] == "stream":
        return {"streamed": outs[0]["x"], **outs[0]}
    return outs[0]
