"""Workloads of the SPH engine at the sizes and options it is used at, each a
call (or the few calls of one main-loop step) through the public entry points
of reyn_b200.

Kinds of case:

* "step": load a device-resident checkpoint into the particle state, then one
  main-loop step: Grid.construct_and_reorder, Solver.step with the hard
  bounds. One scene, every scheme and precision.
* "graph": the same step of a small scene as a captured step (StepGraph).
* "batch": the same step of many independent scenes at once.
* "grid": Grid.construct_and_reorder of a state in arbitrary order.
* "density": Grid.neighbour_stats over an unordered point cloud whose grid is
  built (counts, squared distances and densities).
* "boundary": Boundary over wall samples with the Akinci mass refinement.
* "project": Mesh.project of points near a triangle mesh.

Scenes: a fluid block with seeded jitter in a closed box, with a smooth
velocity field, its particles in the order the grid of the step before would
have left them. "flow" 1 shears the block (volume preserving), so that it no
longer lines up with the grid's cells, as in a developed flow; 0 leaves it on
its lattice, as in the first steps of a dam break.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import reyn_b200 as rb
from reyn_b200 import meshes

RHO0 = 1000.0
GRAVITY = (0.0, -9.81, 0.0)
KERNELS = {"C2": rb.C2, "B3": rb.B3, "W6": rb.W6, "COS": rb.COS}
SCHEMES = {"SESPH": rb.SESPH, "PCISPH": rb.PCISPH, "IISPH": rb.IISPH}
PRECISIONS = {"FP32": rb.PRECISION_FP32, "MIXED": rb.PRECISION_MIXED,
              "POS16": rb.PRECISION_MIXED_POS16}
# spacing, viscosity, time step and average density tolerance of the schemes' scenes
SPACING = {"SESPH": 0.02, "PCISPH": 0.01, "IISPH": 0.005}
NU = 0.01
DT = {"SESPH": 5e-4, "PCISPH": 2e-4, "IISPH": 2e-4}
ETA = {"SESPH": 0.01, "PCISPH": 0.01, "IISPH": 0.005}
SWEEP_LIMIT = 200
JITTER = 0.07
# density of the unit cubic lattice at support two spacings, in units of rho0
LATTICE = {"C2": 1.0340, "B3": 1.0, "W6": 1.1692, "COS": 0.9880}


def listed():
    def step(name, scheme, kernel, precision, nx, ny, nz, flow):
        return {"name": name, "kind": "step", "scheme": scheme, "kernel": kernel,
                "precision": precision, "nx": nx, "ny": ny, "nz": nz, "flow": flow}

    return [
        # the small state-equation dam break: a step of a few launches
        step("sesph_32k", "SESPH", "B3", "FP32", 32, 32, 32, 1),
        # a small interactive scene as a captured step, where launches count
        {"name": "graph_pcisph_8k", "kind": "graph", "scheme": "PCISPH", "kernel": "B3",
         "precision": "FP32", "nx": 21, "ny": 20, "nz": 19, "flow": 1},
        # mid-sized scene with odd edges, FP16 neighbour values, Wendland C6
        step("iisph_mixed_w6_310k", "IISPH", "W6", "MIXED", 77, 61, 67, 1),
        # a million particles in the reference's arithmetic, developed flow
        step("iisph_fp32_1m", "IISPH", "C2", "FP32", 131, 97, 83, 1),
        # the headline dam break, in the fastest mode, from rest
        step("iisph_pos16_4m", "IISPH", "C2", "POS16", 256, 128, 128, 0),
        # the large column collapse
        step("iisph_pos16_w6_16m", "IISPH", "W6", "POS16", 256, 256, 256, 0),
        # many small independent scenes at once: PCISPH, and mixed IISPH
        {"name": "batch_pcisph_64", "kind": "batch", "scheme": "PCISPH", "kernel": "B3",
         "precision": "FP32", "scenes": 64, "nmin": 2000, "nmax": 200000, "flow": 1},
        {"name": "batch_iisph_pos16_96", "kind": "batch", "scheme": "IISPH", "kernel": "C2",
         "precision": "POS16", "scenes": 96, "nmin": 2000, "nmax": 200000, "flow": 1},
        # the reference's grid benchmark: build and reorder a million shuffled particles
        {"name": "grid_1m", "kind": "grid", "n": 1000000, "ratio": 0.5},
        # the neighbour-search microbenchmark: a uniform cloud, cell size = support radius
        {"name": "density_1m", "kind": "density", "n": 1048576, "kernel": "C2", "ratio": 1.0},
        # set-up: the walls of a box with their boundary masses
        {"name": "boundary_400k", "kind": "boundary", "nx": 400, "ny": 200, "nz": 200},
        # set-up: projections of surface samples onto a mesh
        {"name": "project_300k", "kind": "project", "n": 300001, "subdivisions": 6},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _edges(rng, n):
    """Three edges of a block of about n particles, no two alike as a rule."""
    a, b = rng.uniform(0.6, 1.7), rng.uniform(0.6, 1.7)
    e = n ** (1.0 / 3.0)
    return [max(4, round(e * f)) for f in (a, b, 1.0 / (a * b))]


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "batch", "batch", "graph", "grid",
                       "density", "boundary", "project"])
    if kind in ("step", "graph"):
        scheme = rng.choice(["SESPH", "PCISPH", "IISPH", "IISPH"])
        if kind == "graph":
            scheme = rng.choice(["SESPH", "PCISPH"])
        precision = rng.choice(["FP32", "MIXED", "POS16"]) if scheme == "IISPH" else "FP32"
        top = 60000 if kind == "graph" else (4000000 if scheme == "IISPH" else 1000000)
        nx, ny, nz = _edges(rng, _log(rng, 8000, top))
        return {"kind": kind, "scheme": scheme, "kernel": rng.choice(["C2", "B3", "W6", "C2"]),
                "precision": precision, "nx": nx, "ny": ny, "nz": nz,
                "flow": rng.choice([0, 1])}
    if kind == "batch":
        scheme = rng.choice(["SESPH", "PCISPH", "IISPH"])
        precision = rng.choice(["FP32", "MIXED", "POS16"]) if scheme == "IISPH" else "FP32"
        return {"kind": "batch", "scheme": scheme, "kernel": rng.choice(["C2", "B3"]),
                "precision": precision, "scenes": round(_log(rng, 4, 128)), "nmin": 2000,
                "nmax": round(_log(rng, 10000, 200000)), "flow": rng.choice([0, 1])}
    if kind == "grid":
        return {"kind": "grid", "n": round(_log(rng, 20000, 8000000)),
                "ratio": rng.choice([0.5, 0.5, 1.0])}
    if kind == "density":
        return {"kind": "density", "n": round(_log(rng, 20000, 4000000)),
                "kernel": rng.choice(["C2", "B3", "W6", "COS"]),
                "ratio": rng.choice([0.5, 1.0])}
    if kind == "boundary":
        nx, ny, nz = _edges(rng, _log(rng, 27000, 20000000))
        return {"kind": "boundary", "nx": nx, "ny": ny, "nz": nz}
    return {"kind": "project", "n": round(_log(rng, 5000, 1000000)),
            "subdivisions": rng.choice([4, 5, 6])}


# ---- scenes -----------------------------------------------------------------------


def _rand(gen, n):
    """n uniform float64 in [-1, 1)."""
    return torch.rand(n, generator=gen, device="cuda", dtype=torch.float64) * 2.0 - 1.0


def _block(counts, h, flow, speed, gen):
    """Positions (n, 3) and velocities (n, 3) in float64 and the box of one scene."""
    nx, ny, nz = counts
    dev = "cuda"
    k, j, i = torch.meshgrid(torch.arange(nz, device=dev), torch.arange(ny, device=dev),
                             torch.arange(nx, device=dev), indexing="ij")
    n = nx * ny * nz
    ext = np.array([nx, ny, nz]) * h
    amp = 2.5 * h if flow else 0.0
    gap = 1.5 * h + amp
    x = torch.stack([i.reshape(-1), j.reshape(-1), k.reshape(-1)], 1).double() * h
    for a in range(3):
        x[:, a] += JITTER * h * _rand(gen, n)
    if flow:
        # three shears, each volume preserving
        w = 2.0 * math.pi / (40.0 * h)
        x[:, 0] += amp * torch.sin(w * x[:, 1])
        x[:, 1] += amp * torch.sin(w * x[:, 2])
        x[:, 2] += amp * torch.sin(w * x[:, 0])
    x += gap
    w = 2.0 * math.pi / (60.0 * h)
    v = torch.stack([torch.sin(w * x[:, 0]) * torch.cos(w * x[:, 1]),
                     -torch.cos(w * x[:, 0]) * torch.sin(w * x[:, 1]),
                     0.3 * torch.sin(w * x[:, 0])], 1) * speed
    for a in range(3):
        v[:, a] += 0.05 * speed * _rand(gen, n)
    box = np.float32(np.array([2.0, 1.5, 1.5]) * ext + 2.0 * gap)
    return x, v, np.zeros(3, np.float32), box


def _geometry(lo, hi, r, ratio):
    """Lower bound and cell counts of the grid over a box, in float32."""
    r = np.float32(r)
    cell = np.float32(r / np.float32(2)) if ratio == 0.5 else r
    m = np.float32(r * 2.0)
    low = np.float32(lo) - m
    n = np.ceil(((np.float32(hi) + m) - low) / cell).astype(np.int64)
    return low, n, cell


def _order(x, lo, hi, r, ratio, sid=None):
    """The grid's order of the points x (n, 3): by cell, ties by index. lo, hi: (scenes, 3)."""
    geo = [_geometry(a, b, r, ratio) for a, b in zip(np.atleast_2d(lo), np.atleast_2d(hi))]
    dev = x.device
    low = torch.tensor(np.stack([g[0] for g in geo]), device=dev)
    cnt = torch.tensor(np.stack([g[1] for g in geo]), device=dev)
    base = torch.cumsum(cnt.prod(1), 0) - cnt.prod(1)
    s = torch.zeros(x.shape[0], dtype=torch.long, device=dev) if sid is None else sid
    cell = torch.tensor(geo[0][2], device=dev)
    c = torch.floor((x.float() - low[s]) / cell).long()
    key = (c[:, 2] * cnt[s, 1] + c[:, 1]) * cnt[s, 0] + c[:, 0] + base[s]
    return torch.argsort(key, stable=True)


def _scene_counts(case, seed):
    """Edges of each scene of a batch; the sizes belong to the case, not to the seed."""
    rng = np.random.Generator(np.random.PCG64(case["scenes"] * 1000003 + case["nmax"]))
    n = np.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"]), case["scenes"]))
    e = np.maximum(3, np.rint(np.cbrt(n))).astype(int)
    return [(int(v), int(v), int(v)) for v in e]


def _scene(case, seed):
    """Inputs of a step: state arrays in the order of the step before, boxes, walls."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    h = SPACING[case["scheme"]]
    speed = {"SESPH": 0.5, "PCISPH": 0.5, "IISPH": 1.0}[case["scheme"]]
    batch = case["kind"] == "batch"
    counts = _scene_counts(case, seed) if batch else [(case["nx"], case["ny"], case["nz"])]
    parts = [_block(c, h, case["flow"], speed, gen) for c in counts]
    x = torch.cat([p[0] for p in parts])
    v = torch.cat([p[1] for p in parts])
    lo = np.stack([p[2] for p in parts])
    hi = np.stack([p[3] for p in parts])
    size = torch.tensor([p[0].shape[0] for p in parts], device="cuda")
    sid = torch.repeat_interleave(torch.arange(len(parts), device="cuda"), size)
    # the order the step before left: by the cells the particles came from
    before = torch.clamp_min(x - DT[case["scheme"]] * v, 0.0)
    o = _order(before, lo, hi, 2.0 * h, 0.5, sid)
    x, v = x[o].float(), v[o].float()
    m = np.float32(RHO0 * h ** 3)
    if case["scheme"] == "IISPH":  # the unperturbed lattice at rest density
        m = np.float32(m / LATTICE[case["kernel"]])
    state = [x[:, 0].contiguous(), x[:, 1].contiguous(), x[:, 2].contiguous(),
             v[:, 0].contiguous(), v[:, 1].contiguous(), v[:, 2].contiguous(),
             torch.full((x.shape[0],), float(m), device="cuda")]
    walls = [rb.scene_box_walls(a, b, h) for a, b in zip(lo, hi)]
    first = np.concatenate([[0], np.cumsum([p[0].shape[0] for p in parts])]).astype(np.uint32)
    bfirst = np.concatenate([[0], np.cumsum([w[0].numel() for w in walls])]).astype(np.uint32)
    walls = [torch.cat([w[a] for w in walls]) for a in range(3)]
    return {"h": h, "state": state, "lo": lo, "hi": hi, "sid": sid, "walls": walls,
            "first": first, "bfirst": bfirst}


def _params(case, h):
    p = rb.reference_params(SCHEMES[case["scheme"]], KERNELS[case["kernel"]], h, RHO0, NU)
    p.k_sesph = 1000.0
    p.eta = ETA[case["scheme"]]
    p.max_iter = SWEEP_LIMIT
    p.convergence = rb.CONV_AVERAGE
    p.precision = PRECISIONS[case["precision"]]
    return p


class _Views:
    """torch views of engine arrays, made once per array; each keeps the
    engine's handles alive."""

    def __init__(self, *handles):
        self.seen = {}
        self.handles = handles

    def __call__(self, ptr, n, dtype=np.float32):
        t = self.seen.get((ptr, n))
        if t is None:
            t = self.seen[(ptr, n)] = rb.device_tensor(ptr, n, dtype)
            t.handles = self.handles
        return t

    def state(self, st):
        s = st.soa()
        return [self(p, st.n) for p in (s.xx, s.xy, s.xz, s.vx, s.vy, s.vz, s.m)]


def _prepare_step(case, seed):
    sc = _scene(case, seed)
    n = sc["state"][0].numel()
    batch = case["kind"] == "batch"
    h = sc["h"]
    scenes = {"scene_first": sc["first"], "scene_min": sc["lo"], "scene_max": sc["hi"]}
    s = {"init": sc["state"], "turn": 0, "dt": DT[case["scheme"]],
         "bounds": (sc["lo"][0], sc["hi"][0]), "iisph": case["scheme"] == "IISPH"}
    s["grid"] = rb.Grid(sc["lo"].min(0), sc["hi"].max(0), 2.0 * h, 0.5,
                        **(scenes if batch else {}))
    s["bdy"] = rb.Boundary(*sc["walls"], None, h=h, rho0=RHO0, mass_iters=5,
                           **({"scene_first": sc["bfirst"]} if batch else {}))
    s["solver"] = rb.Solver(SCHEMES[case["scheme"]], _params(case, h), n)
    # two states share the solver and take turns: IISPH carries its pressure
    # from step to step of one state and starts cold on the other
    s["states"] = [rb.Particles(n, RHO0) for _ in range(2 if s["iisph"] else 1)]
    s["views"] = _Views(s["states"], s["solver"], s["grid"])
    for st in s["states"]:
        torch._foreach_copy_(s["views"].state(st), sc["state"])
    if case["kind"] == "graph":
        s["graph"] = rb.StepGraph(s["solver"], s["states"][0], s["grid"], s["bdy"], s["dt"],
                                  bounds=s["bounds"])
    return s


def _run_step(s, kind):
    st = s["states"][s["turn"]]
    s["turn"] = (s["turn"] + 1) % len(s["states"])
    views = s["views"]
    torch._foreach_copy_(views.state(st), s["init"])  # the checkpoint, on the device
    if kind == "graph":
        s["graph"].launch()
        iters = None
    else:
        s["grid"].construct_and_reorder(st)
        if kind == "batch":
            iters = s["solver"].step_batched(st, s["grid"], s["bdy"], s["dt"])
        else:
            iters = s["solver"].step(st, s["grid"], s["bdy"], s["dt"], bounds=s["bounds"])
    out = dict(zip(("x", "y", "z", "vx", "vy", "vz"), views.state(st)))
    b = s["solver"].buffers()
    for k in ("rho", "ax", "ay", "az") + (("p", "aii", "sii") if s["iisph"] else ()):
        out[k] = views(getattr(b, k), b.n)
    out["iters"] = iters
    return out


# ---- the calls ---------------------------------------------------------------------


@functools.lru_cache(maxsize=None)
def _icosphere(subdivisions):
    return meshes.icosphere(subdivisions, 0.5)


def _mesh_inputs(case, seed):
    v, f = _icosphere(case["subdivisions"])
    edge = 0.6 / 2 ** case["subdivisions"]
    v = meshes.perturb(v, 0.1 * edge, seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    p = torch.stack([_rand(gen, case["n"]) for _ in range(3)], 1)
    p = p / p.norm(dim=1, keepdim=True).clamp_min(1e-3) * 0.5
    p = p + torch.stack([_rand(gen, case["n"]) for _ in range(3)], 1) * edge
    return v, f, p.float(), edge


def _cloud(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    n = case["n"]
    x = torch.rand((3, n), generator=gen, device="cuda", dtype=torch.float32)
    r = 2.0 * n ** (-1.0 / 3.0)
    return x, r


def _lattice(case, seed):
    """The reference's grid benchmark: a half-jittered lattice, shuffled."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    n = case["n"]
    e = math.ceil(n ** (1.0 / 3.0))
    q = torch.randperm(e ** 3, generator=gen, device="cuda")[:n]
    x = torch.stack([q % e, (q // e) % e, q // (e * e)], 0).double()
    for a in range(3):
        x[a] += 0.25 * _rand(gen, n)
    rest = [_rand(gen, n).float() for _ in range(3)] + [torch.ones(n, device="cuda")]
    return [x[a].float().contiguous() for a in range(3)] + rest, float(e)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step", "graph", "batch"):
        s = _prepare_step(case, seed)
    elif kind == "grid":
        init, e = _lattice(case, seed)
        s = {"init": init, "state": rb.Particles(case["n"], 1.0),
             "ids": torch.arange(case["n"], device="cuda", dtype=torch.float32)}
        s["id_init"] = s["ids"].clone()
        s["grid"] = rb.Grid((-1.0,) * 3, (e,) * 3, 2.2, case["ratio"])
        s["views"] = _Views(s["state"], s["grid"])
        torch._foreach_copy_(s["views"].state(s["state"]), init)
    elif kind == "density":
        x, r = _cloud(case, seed)
        s = {"x": x, "grid": rb.Grid((0.0,) * 3, (1.0,) * 3, r, case["ratio"]),
             "m": torch.full((case["n"],), RHO0 / case["n"], device="cuda"),
             "kernel": KERNELS[case["kernel"]]}
        s["grid"].construct(x[0], x[1], x[2])
    elif kind == "boundary":
        h = 0.005
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        w = rb.scene_box_walls((0.0,) * 3, [h * case[k] for k in ("nx", "ny", "nz")], h)
        s = {"h": h,
             "walls": [(t.double() + 0.1 * h * _rand(gen, t.numel())).float() for t in w]}
    else:
        v, f, p, _ = _mesh_inputs(case, seed)
        s = {"mesh": rb.Mesh(v, f), "points": [p[:, a].contiguous() for a in range(3)],
             "out": [torch.empty(case["n"], device="cuda") for _ in range(3)]}
    s["kind"] = kind
    return s


def run(s):
    kind = s["kind"]
    if kind in ("step", "graph", "batch"):
        return _run_step(s, kind)
    if kind == "grid":
        views, st = s["views"], s["state"]
        torch._foreach_copy_(views.state(st) + [s["ids"]], s["init"] + [s["id_init"]])
        s["grid"].construct_and_reorder(st, [s["ids"]])
        g = s["grid"].info()
        return {"state": views.state(st), "ids": s["ids"],
                "prefix": views(g.prefix, g.n_keys + 1, np.int32)}
    if kind == "density":
        x = s["x"]
        return s["grid"].neighbour_stats(x[0], x[1], x[2], s["m"], s["kernel"])
    if kind == "boundary":
        b = rb.Boundary(*s["walls"], None, h=s["h"], rho0=RHO0, mass_iters=5)
        ptrs, nb = b.arrays()
        out = {k: rb.device_tensor(p, nb).clone() for k, p in zip("xyzm", ptrs)}
        b.close()
        return out
    torch._foreach_copy_(s["out"], s["points"])
    s["mesh"].project(*s["out"])
    return s["out"]


def work(case):
    kind = case["kind"]
    if kind in ("step", "graph", "batch"):
        if kind == "batch":
            n = sum(a * b * c for a, b, c in _scene_counts(case, 0))
        else:
            n = case["nx"] * case["ny"] * case["nz"]
        # the state in and out, densities, accelerations (and p, a_ii, s_i);
        # about 30 neighbours and 30 operations a pair and pass
        iisph = case["scheme"] == "IISPH"
        passes = {"SESPH": 2, "PCISPH": 8, "IISPH": 9}[case["scheme"]]
        return {"bytes": 4.0 * n * (7 + 6 + 4 + (3 if iisph else 0)),
                "flops": 30.0 * 30.0 * passes * n}
    if kind == "grid":
        e = math.ceil(case["n"] ** (1.0 / 3.0))
        cell = 1.1 if case["ratio"] == 0.5 else 2.2
        cells = ((e + 9.8) / cell) ** 3
        return {"bytes": 4.0 * (16 * case["n"] + cells), "flops": 0.0}
    if kind == "density":
        return {"bytes": 4.0 * 7 * case["n"], "flops": 34.0 * 30.0 * case["n"]}
    if kind == "boundary":
        a, b, c = case["nx"], case["ny"], case["nz"]
        n = 2.0 * (a * b + b * c + a * c)
        return {"bytes": 4.0 * 7 * n, "flops": 6 * 13.0 * 25.0 * n}
    faces = 20.0 * 4 ** case["subdivisions"]
    return {"bytes": 24.0 * case["n"] + 36.0 * faces, "flops": 2000.0 * case["n"]}


# ---- the same results in 64 bits ------------------------------------------------------


def _w(kernel, q):
    t = torch.clamp_min(1.0 - q, 0.0)
    if kernel == "C2":
        return 21.0 / (2.0 * math.pi) * t ** 4 * (4.0 * q + 1.0)
    if kernel == "B3":
        return 16.0 / math.pi * (t ** 3 - 4.0 * torch.clamp_min(0.5 - q, 0.0) ** 3)
    if kernel == "W6":
        return 1365.0 / (64.0 * math.pi) * t ** 8 * (((32.0 * q + 25.0) * q + 8.0) * q + 1.0)
    s = math.pi * torch.clamp_max(q, 1.0)
    return math.pi / (4.0 * math.pi ** 2 - 30.0) * (4.0 * torch.cos(s) + torch.cos(2.0 * s) + 3.0)


def _dw(kernel, q):
    t = torch.clamp_min(1.0 - q, 0.0)
    if kernel == "C2":
        return 21.0 / (2.0 * math.pi) * t ** 3 * (-20.0 * q)
    if kernel == "B3":
        return 16.0 / math.pi * (-3.0 * t * t + 12.0 * torch.clamp_min(0.5 - q, 0.0) ** 2)
    if kernel == "W6":
        return 1365.0 / (64.0 * math.pi) * t ** 7 * ((16.0 * q + 7.0) * q + 1.0) * (-22.0 * q)
    s = math.pi * torch.clamp_max(q, 1.0)
    return -2.0 * math.pi ** 2 / (4.0 * math.pi ** 2 - 30.0) * (2.0 * torch.sin(s)
                                                                + torch.sin(2.0 * s))


def _pairs(a, b, r, sa=None, sb=None, chunk=1 << 18):
    """(i, j) with |a_i - b_j| <= r (and of one scene), by cubes of edge r."""
    lo = torch.minimum(a.min(0).values, b.min(0).values) - r
    hi = torch.maximum(a.max(0).values, b.max(0).values) + r
    nx, ny, nz = [int(v) + 3 for v in ((hi - lo) / r).floor()]

    def key(p, s):
        c = ((p - lo) / r).floor().long()
        z = c[:, 2] if s is None else c[:, 2] + s * (nz + 2)
        return (z * ny + c[:, 1]) * nx + c[:, 0]

    kb, order = torch.sort(key(b, sb))
    ka = key(a, sa)
    rows = torch.tensor([(dz * ny + dy) * nx for dz in (-1, 0, 1) for dy in (-1, 0, 1)],
                        device=a.device)
    ii, jj = [], []
    for c0 in range(0, a.shape[0], chunk):
        k = (ka[c0:c0 + chunk, None] + rows).reshape(-1)
        st = torch.searchsorted(kb, k - 1)
        cnt = torch.searchsorted(kb, k + 1, right=True) - st
        total = int(cnt.sum())
        if not total:
            continue
        seg = torch.repeat_interleave(torch.arange(k.numel(), device=a.device), cnt,
                                      output_size=total)
        pos = torch.arange(total, device=a.device) - (torch.cumsum(cnt, 0) - cnt - st)[seg]
        i, j = seg // 9 + c0, order[pos]
        keep = ((a[i] - b[j]) ** 2).sum(1) <= r * r
        ii.append(i[keep])
        jj.append(j[keep])
    if not ii:
        z = torch.zeros(0, dtype=torch.long, device=a.device)
        return z, z
    return torch.cat(ii), torch.cat(jj)


class _Sums:
    """Pairs of points a and b within the support, with W and the factor g of
    the gradient g x_ij; add(v) sums a value per pair into the points a."""

    def __init__(self, kernel, r, a, b, sa=None, sb=None):
        self.n = a.shape[0]
        self.i, self.j = _pairs(a, b, r, sa, sb)
        self.x = a[self.i] - b[self.j]
        self.r2 = (self.x * self.x).sum(1)
        d = self.r2.sqrt()
        self.w = _w(kernel, d / r) / r ** 3
        g = _dw(kernel, d / r) / r ** 4 / d
        self.g = torch.where(d > 0, g, torch.zeros_like(g))

    def add(self, v):
        out = torch.zeros((self.n,) + v.shape[1:], dtype=v.dtype, device=v.device)
        return out.index_add_(0, self.i, v)


def _masses(walls, h, sb=None):
    """Akinci masses after five refinements, cubic B-spline at support 2h."""
    B = _Sums("B3", 2.0 * h, walls, walls, sb, sb)
    m = torch.ones(walls.shape[0], dtype=torch.float64, device="cuda")
    for _ in range(5):
        m = RHO0 * m / B.add(m[B.j] * B.w)
    return m


def _pcisph_stiffness(kernel, h, dt):
    r = torch.arange(-2, 3, device="cuda").double() * h
    x = torch.stack(torch.meshgrid(r, r, r, indexing="ij"), -1).reshape(-1, 3)
    d = x.norm(dim=1)
    g = torch.where(d > 0, _dw(kernel, torch.clamp_max(d / (2 * h), 1.0)) / (2 * h) ** 4 / d,
                    torch.zeros_like(d))[:, None] * x
    s = g.sum(0)
    beta = 2.0 * h ** 6 * dt * dt
    return 1.0 / (beta * float((s * s).sum() + (g * g).sum()))


def _exact_step(case, seed):
    sc = _scene(case, seed)
    batch = case["kind"] == "batch"
    kernel, scheme = case["kernel"], case["scheme"]
    f32 = lambda v: float(np.float32(v))  # noqa: E731
    h, dt = f32(sc["h"]), f32(DT[scheme])
    eta, r0 = f32(ETA[scheme]), RHO0
    sid = sc["sid"]
    o = _order(torch.stack(sc["state"][:3], 1), sc["lo"], sc["hi"], 2.0 * sc["h"], 0.5, sid)
    sid = sid[o]
    ns = len(sc["lo"])
    X = torch.stack(sc["state"][:3], 1)[o].double()
    V = torch.stack(sc["state"][3:6], 1)[o].double()
    m = sc["state"][6][o].double()
    wsid = torch.repeat_interleave(torch.arange(ns, device="cuda"),
                                   torch.tensor(np.diff(sc["bfirst"].astype(np.int64)), device="cuda"))
    W = torch.stack(sc["walls"], 1).double()
    two = (sid, sid) if batch else ()
    mb = _masses(W, h, wsid if batch else None)
    F = _Sums(kernel, 2.0 * h, X, X, *two)
    B = _Sums(kernel, 2.0 * h, X, W, *((sid, wsid) if batch else ()))
    mj = m[F.j]
    wb = B.add(mb[B.j] * B.w)
    gb = B.add((mb[B.j] * B.g)[:, None] * B.x)
    del B
    rho = F.add(mj * F.w) + wb
    grav = torch.tensor([f32(v) for v in GRAVITY], device="cuda", dtype=torch.float64)
    dot = lambda a, b: (a * b).sum(1)  # noqa: E731

    def viscosity():
        s = 10.0 * f32(NU) * mj * dot(V[F.i] - V[F.j], F.x) * F.g
        s = s / (rho[F.j] * (F.r2 + 0.01 * h * h))
        return grav + F.add(s[:, None] * F.x)

    size = torch.bincount(sid, minlength=ns).double()
    live = torch.ones(ns, dtype=torch.bool, device="cuda")
    iters = np.zeros(ns, np.int64)

    def mean(v):  # of each scene
        return torch.zeros(ns, dtype=torch.float64, device="cuda").index_add_(0, sid, v) / size

    def go_on(k, more):  # after sweep k + 1; scenes that met the tolerance stop
        nonlocal live
        iters[live.cpu().numpy()] = k + 1
        if k + 1 >= 3:
            live = live & more
        return bool(live.any())

    extra = {}
    if scheme == "SESPH":
        p = torch.clamp_min(1000.0 * (rho / r0 - 1.0), 0.0) / rho ** 2
        A = viscosity() - F.add((mj * (p[F.i] + p[F.j]) * F.g)[:, None] * F.x) - p[:, None] * gb
        V = V + dt * A
        iters[:] = 1
    elif scheme == "PCISPH":
        kp = _pcisph_stiffness(kernel, h, dt)
        V = V + dt * viscosity()
        A = torch.zeros_like(V)
        for k in range(SWEEP_LIMIT):
            on = live[sid]
            new = F.add(mj * (F.w + dt * F.g * dot(V[F.i] - V[F.j], F.x))) + wb + dt * dot(gb, V)
            rho = torch.where(on, new, rho)
            p = torch.clamp_min(kp * (rho - r0), 0.0)
            q = p / rho ** 2
            acc = -F.add((mj * (q[F.i] + q[F.j]) * F.g)[:, None] * F.x) \
                - (0.5 * (q + p / r0 ** 2))[:, None] * gb
            A = torch.where(on[:, None], acc, A)
            V = V + dt * torch.where(on[:, None], acc, torch.zeros_like(acc))
            if not go_on(k, mean(rho) > (1.0 + eta) * r0):
                break
    else:
        V = V + dt * viscosity()
        mg = (mj * F.g)[:, None] * F.x
        G = F.add(mg) + gb
        a = -dt * (dot(G, G) + m * F.add(mj * F.g * F.g * F.r2)) / r0 ** 2
        s = (r0 - rho) / dt - F.add(dot(mg, V[F.i] - V[F.j])) - dot(V, gb)
        p = torch.zeros_like(rho)

        def accelerations():
            return -(F.add(mg * (p[F.i] + p[F.j])[:, None]) + p[:, None] * gb) / r0 ** 2

        for k in range(SWEEP_LIMIT):
            on = live[sid]
            A = accelerations()
            Ap = dt * (F.add(dot(mg, A[F.i] - A[F.j])) + dot(A, gb))
            d = torch.where(a.abs() < 1e-6, torch.zeros_like(a), 0.5 * (s - Ap) / a)
            p = torch.where(on, p + torch.clamp_min(d, 0.0), p)
            if not go_on(k, mean(torch.clamp_min((Ap - s) * dt, 0.0)) > eta * r0):
                break
        A = accelerations()
        V = V + dt * A
        extra = {"p": p, "aii": a, "sii": s}
    X = X + dt * V
    lo, hi = (torch.tensor(sc[k], device="cuda").double()[sid] for k in ("lo", "hi"))
    hit = ((X <= lo) | (X >= hi)).any(1)
    V = torch.where(hit[:, None], V * f32(-0.1), V)
    X = torch.minimum(torch.maximum(X, lo), hi)
    out = {"x": X[:, 0], "y": X[:, 1], "z": X[:, 2], "vx": V[:, 0], "vy": V[:, 1], "vz": V[:, 2],
           "rho": rho, "ax": A[:, 0], "ay": A[:, 1], "az": A[:, 2], **extra}
    out["iters"] = None if case["kind"] == "graph" else iters if batch else int(iters[0])
    return out


def _closest(p, a, b, c):
    """Closest point of triangles (a, b, c) to points p, and its squared distance."""
    def segment(u, v):
        d = v - u
        t = (((p - u) * d).sum(1) / (d * d).sum(1).clamp_min(1e-300)).clamp(0.0, 1.0)
        return u + t[:, None] * d

    n = torch.linalg.cross(b - a, c - a)
    nn = (n * n).sum(1)
    q = p - (((p - a) * n).sum(1) / nn)[:, None] * n
    inside = torch.ones_like(nn, dtype=torch.bool)
    for u, v in ((a, b), (b, c), (c, a)):
        inside &= (torch.linalg.cross(v - u, q - u) * n).sum(1) >= 0
    best, d2 = q, torch.where(inside, ((p - q) ** 2).sum(1), torch.full_like(nn, math.inf))
    for u, v in ((a, b), (b, c), (c, a)):
        s = segment(u, v)
        e = ((p - s) ** 2).sum(1)
        best = torch.where((e < d2)[:, None], s, best)
        d2 = torch.minimum(d2, e)
    return best, d2


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "graph", "batch"):
        if work(case)["bytes"] > 4.0 * 20 * 6e6:  # the pairs of more particles take too long
            return None
        return _exact_step(case, seed)
    if kind == "grid":
        return None  # whole numbers, and copies of the inputs
    if kind == "density":
        x, r = _cloud(case, seed)
        r = float(np.float32(r))
        X = x.T.double().contiguous()
        n = case["n"]
        m = float(np.float32(RHO0 / n))
        rho = torch.zeros(n, dtype=torch.float64, device="cuda")
        l2 = torch.zeros_like(rho)
        S = _Sums(case["kernel"], r, X, X)
        l2, rho = S.add(S.r2), S.add(m * S.w)
        return (None, l2, rho)
    if kind == "boundary":
        s = prepare(case, seed)
        W = torch.stack(s["walls"], 1)
        lo, hi = W.min(0).values.cpu().numpy(), W.max(0).values.cpu().numpy()
        o = _order(W, lo, hi, float(np.float32(2) * np.float32(s["h"])), 0.5)
        W = W[o].double()
        return {"x": W[:, 0], "y": W[:, 1], "z": W[:, 2],
                "m": _masses(W, float(np.float32(s["h"])))}
    v, f, p, edge = _mesh_inputs(case, seed)
    tri = torch.tensor(np.float32(v), device="cuda").double()[torch.tensor(f.astype(np.int64),
                                                                          device="cuda")]
    P = p.double()
    center = tri.mean(1)
    # the surface lies within about two edges of every point, a face's points
    # within an edge and a half of its centre
    best = torch.empty_like(P)
    for c0 in range(0, P.shape[0], 1 << 17):
        q = P[c0:c0 + (1 << 17)]
        i, j = _pairs(q, center, 4.5 * edge)
        pt, d2 = _closest(q[i], tri[j, 0], tri[j, 1], tri[j, 2])
        low = torch.full((q.shape[0],), math.inf, dtype=torch.float64, device="cuda")
        low.scatter_reduce_(0, i, d2, "amin")
        hit = d2 == low[i]
        best[c0 + i[hit]] = pt[hit]
    return [best[:, a] for a in range(3)]
