"""The work that programs using this library have it do, as cases for measuring it.

listed() are twelve calls over the range a user meets, draw() gives more of the same ranges:

* the reference's own default cut scene (thousands of particles, where launches and latency count),
* the small adiabatic cut of a parameter study, driven one step at a time with the tool force
  recorded every step,
* the impact validation scene on an adaptive grid (SI units, the Green order, yielding),
* the ~23k-particle cut with the PSE heat solver in plain FP64,
* the ~177k-particle benchmark cut with thermal contact in FP64 and in mixed precision on
  neighbour lists, a ~46k-particle one in mixed precision sorted every step,
* the ~577k-particle high-resolution cut (PSE, mixed precision), the largest,
* a sweep of uneven small cuts stepped as one batch,
* the derivative of the mean cutting force, all six material parameters at once and one alone,
* the cell-list build by itself on an adaptive grid.

The cut scenes are the benchmark's (Ti6Al4V, 2.0 mm x 0.6 mm, seeded lattice jitter) in a state of
ongoing cutting rather than at rest: the tool has just entered the workpiece, and around its edge
the material is hot, compressed, strained and sheared to the yield stress, so that contact,
friction and the return map are at work as they are for nearly all of a real run.

Outputs are the particles' fields in the order of their numbers at creation. Mixed-precision runs
hand theirs out in float32, as a program does that keeps or dumps snapshots of a run whose rates
are FP32 sums.
"""
from __future__ import annotations

import ctypes as C
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

PKG = Path(__file__).resolve().parent.parent / "mfree_iwf-ul_cut_gpu_b200"


def _package():
    name = "mfree_b200"
    if name not in sys.modules:
        spec = importlib.util.spec_from_file_location(name, PKG / "__init__.py", submodule_search_locations=[str(PKG)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


# ---------------------------------------------------------------------------------------------
# the cases

def _cut(name, nx, steps, thermal="brookshaw", precision="fp64", lists=False, each=False):
    return {"name": name, "kind": "cut", "nx": nx, "steps": steps, "thermal": thermal, "precision": precision,
            "lists": lists, "each": each}


def listed():
    return [
        # the reference's default program: setup_ref_cut with 30 rows, plain FP64
        {"name": "ref_cut_7k_fp64", "kind": "ref_cut", "ny": 30, "steps": 40},
        # a 10,000-step force curve of a small cut: one call per step, its force to pinned memory
        _cut("cut_6k_mixed_lists_force", 143, 60, "none", "mixed", lists=True, each=True),
        # the validation scene of the plasticity model, whose bounding box and cells follow the body
        {"name": "impact_32k_fp64_adaptive", "kind": "impact", "nbox": 100, "steps": 20},
        # a mid-size cut with the other heat solver, in the reference's precision
        _cut("cut_23k_fp64_pse", 260, 10, "pse"),
        # the headline configuration in the reference's precision ...
        _cut("cut_177k_fp64", 714, 10),
        # ... and in the form production runs use
        _cut("cut_177k_mixed_lists", 714, 30, precision="mixed", lists=True),
        # mixed precision in the reference's particle order
        _cut("cut_46k_mixed_sorted", 361, 20, precision="mixed"),
        # the high-resolution stress run
        _cut("cut_577k_mixed_pse", 1290, 4, "pse", "mixed"),
        # a parameter sweep: uneven instances, one launch per 16 steps for all of them
        {"name": "sweep_24_mixed", "kind": "sweep", "instances": 24, "nx_min": 90, "nx_max": 330, "steps": 32},
        # material identification: every derivative of the mean cutting force over a window
        {"name": "gradient_six_23k", "kind": "gradient", "nx": 260, "skip": 2, "window": 8, "param": -1,
         "thermal": "brookshaw"},
        # friction identification: one derivative on a small adiabatic cut
        {"name": "gradient_mu_6k", "kind": "gradient", "nx": 143, "skip": 0, "window": 16, "param": 5,
         "thermal": "none"},
        # the neighbour search used by itself, once per call, box and cells from the particles
        {"name": "cells_577k_adaptive", "kind": "cells", "nx": 1290},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ref_cut", "impact", "cut", "cut", "cut", "cut", "sweep", "gradient", "cells"])
    if kind == "ref_cut":
        return {"kind": kind, "ny": _log_int(rng, 14, 90), "steps": rng.randint(10, 40)}
    if kind == "impact":
        return {"kind": kind, "nbox": _log_int(rng, 30, 200), "steps": rng.randint(5, 20)}
    if kind == "cut":
        thermal = rng.choice(["brookshaw", "brookshaw", "pse", "none"])
        precision = rng.choice(["fp64", "mixed"])
        lists = precision == "mixed" and thermal != "pse" and rng.random() < 0.6
        nx = _log_int(rng, 100, 1200)
        steps = rng.randint(2, 4) if nx > 700 else rng.randint(4, 16)
        return {"kind": kind, "nx": nx, "steps": steps, "thermal": thermal, "precision": precision, "lists": lists,
                "each": rng.random() < 0.25}
    if kind == "sweep":
        return {"kind": kind, "instances": rng.randint(3, 24), "nx_min": rng.randint(80, 120),
                "nx_max": rng.randint(140, 330), "steps": 16 * rng.randint(1, 2)}
    if kind == "gradient":
        return {"kind": kind, "nx": _log_int(rng, 100, 260), "skip": rng.randint(0, 3), "window": rng.randint(4, 8),
                "param": rng.choice([-1, 0, 2, 4, 5]), "thermal": rng.choice(["brookshaw", "none"])}
    return {"kind": "cells", "nx": _log_int(rng, 100, 1290)}


# ---------------------------------------------------------------------------------------------
# inputs

SCALAR = ("rho", "T", "h", "eps_pl", "eps_pl_dot")


def _cut_params(mf, nx, thermal, seed):
    """The benchmark's orthogonal cut on an nx-column lattice."""
    p = mf.reference_cut_params()
    dx = 2.8e-4 * 714 / nx
    p.nx_lattice, p.ny, p.dx = nx, max(8, int(round(0.3 * nx))), dx
    p.lo_x, p.lo_y = 0.0, 0.0
    p.jitter, p.seed = 0.005, 1 + seed
    p.rake, p.clear, p.chamfer = 0.0, 7.0, 5e-4
    p.feed, p.speed, p.mu_fric = 0.005, 70.0 * 100.0 / 60.0e6, 0.35
    p.tool_front_x = -0.1 * dx
    p.sample_tool = p.use_thermals = 0 if thermal == "none" else 1
    p.E, p.nu, p.rho0 = 1.1, 0.35, 4.43
    jc = p.joco
    jc.A, jc.B, jc.n, jc.C, jc.m = 0.01098, 0.01092, 0.93, 0.014, 1.1
    jc.eps_dot_ref, jc.Tref, jc.Tmelt = 1e-6, 300.0, 1878.0
    p.trml_wp.cp, p.trml_wp.k, p.trml_wp.tq, p.trml_wp.eta = 553e-8, 7.1e-13, 0.9, 0.9
    p.cfl = 0.3
    return p


def _fields(scene):
    st = {"scene": scene, "N": scene.N, "pos": scene.array("pos").copy(), "vel": np.zeros((scene.N, 2)),
          "rho": scene.array("rho").copy(), "T": scene.array("T").copy(), "h": scene.array("h").copy(),
          "fixed": scene.array("fixed").copy(), "tool_p": scene.array("tool_p").copy(),
          "S": np.zeros((scene.N, 4)), "eps_pl": np.zeros(scene.N), "eps_pl_dot": np.zeros(scene.N)}
    return st


def _in_cut(mf, scene, seed):
    """The scene's particles in ongoing cutting: tool just inside the workpiece, its edge's
    surroundings hot, compressed and at the yield stress."""
    s = scene.s
    st = _fields(scene)
    rng = np.random.default_rng(seed)
    wp = st["tool_p"] == 0.0
    n = int(wp.sum())
    spacing = s.grid_h / 1.5
    tool = mf.ToolState()
    C.memmove(C.byref(tool), C.byref(s.tool), C.sizeof(mf.ToolState))
    xs = [e for k in range(tool.num_seg) for e in (tool.seg[k].left[0], tool.seg[k].right[0])]
    front = max(max(xs), tool.fillet.p[0] + tool.fillet.r) if tool.has_fillet else max(xs)
    x0 = float(st["pos"][wp, 0].min())
    t = (x0 + 0.05 * spacing - front) / tool.vel[0]
    mf.tool_translate(tool, t)
    st["pos"][~wp] += t * np.array([tool.vel[0], tool.vel[1]])
    y0 = float(st["pos"][wp, 1].max()) - s.feed
    r = np.hypot(st["pos"][wp, 0] - x0, st["pos"][wp, 1] - y0)
    zone = np.exp(-np.maximum(r - 0.006, 0.0) ** 2 / 0.006**2)  # 60 um plateau, 60 um fall-off
    jc = s.joco
    eps = 0.3 * zone * rng.uniform(0.9, 1.1, n)
    rate = 1e-2 * zone * rng.uniform(0.5, 1.5, n)
    T = np.full(n, jc.Tref) + 250.0 * zone + rng.uniform(0.0, 5.0, n)
    theta = (T - jc.Tref) / (jc.Tmelt - jc.Tref)
    flow = (jc.A + jc.B * eps**jc.n) * (1 + jc.C * np.log(np.maximum(rate / jc.eps_dot_ref, 1.0))) * (1 - theta**jc.m)
    st["S"][wp, 1] = -1.02 * zone * flow / math.sqrt(3.0) * rng.uniform(0.995, 1.005, n)
    st["eps_pl"][wp], st["eps_pl_dot"][wp], st["T"][wp] = eps, rate, T
    st["T"][~wp] = jc.Tref + rng.uniform(0.0, 5.0, scene.N - n)
    st["rho"][wp] *= 1.0 + 2e-3 * zone + rng.uniform(0.0, 1e-5, n)
    st["vel"][wp] = rng.normal(0.0, 1e-7, (n, 2))
    st["tool"] = tool
    return st


def _impact(mf, case, seed):
    """The disc on its way into the wall, a smooth shear field of the first contact in it."""
    scene = mf.Scene.impact(case["nbox"])
    st = _fields(scene)
    rng = np.random.default_rng(seed)
    st["vel"] = scene.array("vel") * (1.0 + rng.uniform(-1e-4, 1e-4, (scene.N, 1)))
    move = st["fixed"] == 0.0
    lead = st["pos"][move]
    far = np.abs(lead - lead.mean(axis=0)).max()
    wave = np.cos(np.pi * (lead - lead.mean(axis=0)) / (2 * far)).prod(axis=1)
    st["S"][move, 1] = 0.62 * scene.s.joco.A * wave * rng.uniform(0.99, 1.01, len(lead))
    st["tool"] = None
    return st


def _inputs(mf, case, seed):
    if case["kind"] == "ref_cut":
        return [_in_cut(mf, mf.Scene.ref_cut(case["ny"]), seed)]
    if case["kind"] == "impact":
        return [_impact(mf, case, seed)]
    if case["kind"] == "sweep":
        # one instance per point of the sweep: speed, rake, depth of cut and the yield constants vary
        # (sizes and tool shapes are the sweep's plan; the seed gives the material and its state)
        plan, rng, out = np.random.default_rng(case["instances"]), np.random.default_rng(seed), []
        for k in range(case["instances"]):
            p = _cut_params(mf, int(plan.integers(case["nx_min"], case["nx_max"] + 1)), "brookshaw", seed + k)
            p.speed *= float(plan.uniform(30, 200)) / 70.0
            p.rake, p.feed = float(plan.uniform(-10, 15)), float(plan.uniform(20, 100)) * 1e-4
            p.joco.A *= float(rng.uniform(0.9, 1.1))
            p.joco.B *= float(rng.uniform(0.9, 1.1))
            out.append(_in_cut(mf, mf.Scene.from_params(p), seed + k))
        return out
    return [_in_cut(mf, mf.Scene.from_params(_cut_params(mf, case["nx"], case.get("thermal", "brookshaw"), seed)), seed)]


def _context(mf, case, st):
    s = st["scene"].s
    ctx = mf.Context(0)
    ctx.particles_create(st["pos"], st["vel"], st["rho"], st["h"], T=st["T"], fixed=st["fixed"], tool_p=st["tool_p"],
                         S=st["S"])
    ctx.set("eps_pl", st["eps_pl"])
    ctx.set("eps_pl_dot", st["eps_pl_dot"])
    if case["kind"] in ("impact", "cells"):
        ctx.grid_adaptive(mf.GRID_GREEN, s.grid_max_cell if case["kind"] == "impact" else 4 * st["N"])
    else:
        ctx.grid_locked(mf.GRID_GREEN, tuple(s.grid_bbmin), tuple(s.grid_bbmax), s.grid_h)
    ctx.set_constants(s.phys, s.corr, s.joco if s.has_joco else None, s.trml_wp, s.trml_tool)
    mixed = case.get("precision") == "mixed" or case["kind"] == "sweep"
    ctx.set_options(mf.THERMAL_PSE if case.get("thermal") == "pse" else mf.THERMAL_BROOKSHAW, mf.JC_JOHNSON_COOK,
                    mf.PRECISION_MIXED if mixed else mf.PRECISION_FP64)
    if case.get("lists"):
        ctx.set_flags(mf.OPT_NEIGHBOUR_LISTS)
    ctx.tool_set(st["tool"])
    ctx.set_dt(s.dt)
    return ctx


OUT = ("pos", "vel", "S", "rho", "T", "eps_pl", "fc", "ft")
WIDTH = {"pos": 2, "vel": 2, "S": 4, "fc": 2, "ft": 2}


class _State:
    """A program's contexts, and the device buffers it reads their fields into."""

    def __init__(self, case, seed):
        mf = _package()
        self.case, self.mf = case, mf
        self.inputs = _inputs(mf, case, seed)
        self.ctx = [_context(mf, case, st) for st in self.inputs]
        sizes = [st["N"] for st in self.inputs]
        for st in self.inputs:
            st.clear()
        n = sum(sizes)
        self.first = [sum(sizes[:k]) for k in range(len(sizes))]
        self.stream = torch.cuda.Stream()
        with torch.cuda.stream(self.stream):
            self.raw = {k: torch.zeros((n, WIDTH[k]) if k in WIDTH else (n,), dtype=torch.float64, device="cuda")
                        for k in OUT}
            self.id = torch.zeros(n, dtype=torch.int32, device="cuda")
            self.hash = torch.zeros(n, dtype=torch.int32, device="cuda")
            self.offset = torch.cat([torch.full((m,), f, dtype=torch.int64, device="cuda")
                                     for m, f in zip(sizes, self.first)])
            mixed = case.get("precision") == "mixed" or case["kind"] == "sweep"
            self.out = {k: torch.zeros_like(v, dtype=torch.float32 if mixed else torch.float64)
                        for k, v in self.raw.items()}
        self.force = torch.zeros((case.get("steps", 1), 2), dtype=torch.float64).pin_memory()
        self.batch = mf.Batch(self.ctx, steps_per_launch=16) if case["kind"] == "sweep" else None

    def __del__(self):
        if getattr(self, "batch", None) is not None:
            self.batch.close()
        for c in getattr(self, "ctx", []):
            c.close()


def prepare(case, seed):
    return _State(case, seed)


def _address(t, first):
    return t.data_ptr() + first * t.stride(0) * t.element_size()


def _read(s, names):
    """Every context's fields, by particle number."""
    handle = s.stream.cuda_stream
    for c, f in zip(s.ctx, s.first):
        c.get_device("id", _address(s.id, f), handle)
        for k in names:
            c.get_device(k, _address(s.raw[k], f), handle)
    with torch.cuda.stream(s.stream):
        at = s.id + s.offset
        for k in names:
            s.out[k].index_copy_(0, at, s.raw[k].to(s.out[k].dtype))
    # the program looks at what it has (writes it out, decides how to go on) before it steps again:
    # one simulation at a time, each waiting for its own result
    s.stream.synchronize()
    return {k: s.out[k] for k in names}


def run(s):
    case = s.case
    kind = case["kind"]
    if kind == "gradient":
        if case["param"] < 0:
            mean, dmean = s.ctx[0].tangent_mean_force_all(case["skip"], case["window"])
        else:
            mean, dmean = s.ctx[0].tangent_mean_force(case["skip"], case["window"], case["param"])
        return {"mean": mean, "dmean": dmean}
    if kind == "cells":
        c = s.ctx[0]
        c.grid_build()
        c.get_device("id", s.id.data_ptr(), s.stream.cuda_stream)
        c.get_device("hash", s.hash.data_ptr(), s.stream.cuda_stream)
        c.get_device("pos", s.raw["pos"].data_ptr(), s.stream.cuda_stream)
        return {"id": s.id, "hash": s.hash, "pos": s.raw["pos"]}
    if kind == "sweep":
        s.batch.step(case["steps"] // 16)
        return _read(s, OUT)
    c = s.ctx[0]
    if case.get("each"):  # the force curve: each step's tool force into pinned host memory
        for k in range(case["steps"]):
            c.step(1)
            c.force_last_async(s.force.data_ptr() + 16 * k)
        out = _read(s, OUT)
        return dict(out, force=s.force.to(s.out["fc"].dtype))
    c.step(case["steps"])
    return _read(s, OUT)


def _lattice(case):
    """(particles, particle-steps) of a case, near enough for its work."""
    kind = case["kind"]
    if kind == "ref_cut":
        n = 8.5 * case["ny"] ** 2
    elif kind == "impact":
        n = 3.25 * case["nbox"] ** 2
    elif kind == "sweep":
        m = [case["nx_min"] + (case["nx_max"] - case["nx_min"]) * (k + 0.5) / case["instances"]
             for k in range(case["instances"])]
        n = sum(0.347 * x * x for x in m)
    else:
        n = (0.3 if case.get("thermal") == "none" else 0.347) * case["nx"] ** 2
    steps = case["skip"] + case["window"] if kind == "gradient" else case.get("steps", 1)
    return n, n * steps


def work(case):
    """A particle-step reads and writes the 224 bytes of its changing FP64 state and reads 32 bytes of
    constants; its ~28 neighbours within the support cost ~110 floating-point operations each (the
    gradient carries the state's tangents too: one or six of them). The cell build moves the state
    (248 bytes) and reads the positions."""
    n, ns = _lattice(case)
    if case["kind"] == "cells":
        return {"bytes": n * (2 * 248 + 24), "flops": n * 8}
    w = 1 if case["kind"] != "gradient" else 7 if case["param"] < 0 else 2
    return {"bytes": ns * (w * 448 + 32), "flops": ns * 28 * 110 * w}


# ---------------------------------------------------------------------------------------------
# the step in plain torch, 64 bits: what run() returns

def _f32(x):
    """x rounded to float and back (the model's float functions), derivatives passed through."""
    return x + (x.float().double() - x).detach()


def _sqrtf(x):
    safe = torch.where(x > 0, x, torch.ones_like(x))
    root = torch.where(x > 0, torch.sqrt(safe), torch.zeros_like(x))
    return root + (torch.sqrt(x.float()).double() - root).detach()


class _Tool:
    def __init__(self, t):
        self.seg = [[e.left[0], e.left[1], e.right[0], e.right[1], e.a, e.b, bool(e.vertical), e.n[0], e.n[1]]
                    for e in t.seg[: t.num_seg]]
        self.fillet = [t.fillet.p[0], t.fillet.p[1]] if t.has_fillet else None
        self.r, self.t1, self.t2 = t.fillet.r, t.fillet.t1, t.fillet.t2
        self.vel = [t.vel[0], t.vel[1]]
        self.mu, self.alpha, self.mass = t.mu, t.contact_alpha, t.slave_mass

    def advance(self, dt):
        sx, sy = dt * self.vel[0], dt * self.vel[1]
        for e in self.seg:
            e[0] += sx; e[1] += sy; e[2] += sx; e[3] += sy
            det = e[0] - e[2]
            e[6] = abs(det) < 1e-12
            if not e[6]:
                e[4], e[5] = (e[1] - e[3]) / det, (e[3] * e[0] - e[2] * e[1]) / det
        if self.fillet:
            self.fillet[0] += sx
            self.fillet[1] += sy

    def contact(self, x, y):
        """inside, contact point and normal of the closest feature."""
        inside = torch.ones_like(x, dtype=torch.bool)
        for e in self.seg:
            inside &= (e[0] - x) * e[7] + (e[1] - y) * e[8] < 0
        round_ = len(self.seg) == 5
        if round_:
            dx, dy = self.fillet[0] - x, self.fillet[1] - y
            inside |= torch.sqrt(dx * dx + dy * dy) < self.r
        idx = torch.nonzero(inside.detach()).flatten()
        qx, qy = x[idx], y[idx]
        depth = torch.full_like(qx, 3.402823466e38).detach()
        cx, cy, nx, ny = (torch.zeros_like(qx) for _ in range(4))
        for k, e in enumerate(self.seg):
            if e[6]:
                d = (e[0] - qx).abs()
                px, py, mx, my = torch.full_like(qx, e[0]), qy, torch.sign(e[0] - qx), torch.zeros_like(qx)
            elif round_ and k == 2:
                vx, vy = qx - self.fillet[0], qy - self.fillet[1]
                inv = 1 / torch.sqrt(vx * vx + vy * vy)
                mx, my = vx * inv, vy * inv
                px, py = self.fillet[0] + mx * self.r, self.fillet[1] + my * self.r
                ang = torch.atan2(self.fillet[1] - py.detach(), self.fillet[0] - px.detach())
                ang = torch.where(ang > 0, ang, ang + 2 * math.pi)
                ok = (ang > min(self.t1, self.t2)) & (ang < max(self.t1, self.t2))
                d = torch.where(ok, torch.sqrt((px - qx) ** 2 + (py - qy) ** 2), torch.full_like(qx, 3.402823466e38))
            else:
                a, c = e[4], e[5]
                px, py = (qx + a * qy - a * c) / (a * a + 1), (a * (qx + a * qy) + c) / (a * a + 1)
                d = torch.sqrt((px - qx) ** 2 + (py - qy) ** 2)
                mx, my = torch.full_like(qx, -e[7]), torch.full_like(qx, -e[8])
            take = d.detach() < depth
            depth = torch.where(take, d.detach(), depth)
            cx, cy = torch.where(take, px, cx), torch.where(take, py, cy)
            nx, ny = torch.where(take, mx, nx), torch.where(take, my, ny)
        return inside.detach(), idx, cx, cy, nx, ny


class _Exact:
    """One particle system stepped in 64-bit torch, its particles in the library's order."""

    def __init__(self, case, st):
        s = st["scene"].s
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.dev, self.case, self.N, self.dt = dev, case, st["N"], s.dt
        d = lambda a: torch.as_tensor(np.array(a, dtype=np.float64), device=dev)  # noqa: E731
        self.f = {k: d(st[k]) for k in ("pos", "vel", "S", "rho", "T", "eps_pl", "eps_pl_dot", "h")}
        for k, w in (("fc", 2), ("ft", 2), ("pos_t", 2), ("vel_t", 2), ("S_t", 4), ("rho_t", 0), ("T_t", 0)):
            self.f[k] = torch.zeros((self.N, w) if w else (self.N,), dtype=torch.float64, device=dev)
        self.f["fixed"], self.f["tool"] = d(st["fixed"]) == 1, d(st["tool_p"]) == 1
        self.f["id"] = torch.arange(self.N, device=dev)
        self.n = torch.zeros((self.N, 2), dtype=torch.float64, device=dev)
        self.phys, self.corr, self.jc, self.wp, self.tl = s.phys, s.corr, s.joco, s.trml_wp, s.trml_tool
        self.plastic = bool(s.has_joco)
        self.par = {k: getattr(s.joco, k) for k in ("A", "B", "n", "C", "m")}
        self.tool = _Tool(st["tool"]) if st["tool"] is not None else None
        self.adaptive = case["kind"] in ("impact", "cells")
        if not self.adaptive:
            lo, hi, h = list(s.grid_bbmin), list(s.grid_bbmax), s.grid_h
            self.lo, self.hi = [v - 1e-6 for v in lo], [v + 1e-6 for v in hi]
            self.cell = h
        self.pse = case.get("thermal") == "pse"
        self.lists = bool(case.get("lists"))
        self.sort_now = True

    def sort(self):
        f = self.f
        pos = f["pos"].detach()
        if self.adaptive:
            self.lo = [float(pos[:, k].min()) - 1e-6 for k in (0, 1)]
            self.hi = [float(pos[:, k].max()) + 1e-6 for k in (0, 1)]
            self.cell = float(f["h"].max())
        self.nx, self.ny = (int(math.ceil((self.hi[k] - self.lo[k]) / self.cell)) for k in (0, 1))
        ix = ((pos[:, 0] - self.lo[0]) / self.cell).to(torch.int64)
        iy = ((pos[:, 1] - self.lo[1]) / self.cell).to(torch.int64)
        h = (ix * self.ny + iy).clamp(0, self.nx * self.ny - 1)
        order = torch.argsort(h, stable=True)
        self.f = {k: v[order] for k, v in f.items()}
        self.hash = h[order]
        self.off = torch.searchsorted(self.hash, torch.arange(self.nx * self.ny + 1, device=self.dev))

    def pairs(self, widen):
        """(i, j) of the candidates of each window column."""
        gi, gj = self.hash // self.ny, self.hash % self.ny
        r = 3 if widen else 2
        for a in range(-r, r + 1):
            ii = gi + a
            ok = (ii >= 0) & (ii < self.nx)
            ii = ii.clamp(0, self.nx - 1)
            j0 = self.off[ii * self.ny + (gj - r).clamp(min=0)]
            j1 = self.off[ii * self.ny + (gj + r + 1).clamp(max=self.ny)]
            cnt = torch.where(ok, j1 - j0, torch.zeros_like(j0))
            i = torch.repeat_interleave(torch.arange(self.N, device=self.dev), cnt)
            start = torch.cumsum(cnt, 0) - cnt
            yield i, torch.arange(i.numel(), device=self.dev) - start[i] + j0[i]

    def step(self):
        P, K, dt, wp, tl = self.phys, self.corr, self.dt, self.wp, self.tl
        if self.sort_now or not self.lists:
            self.sort()
        built = self.sort_now
        f = self.f
        z = torch.zeros(self.N, dtype=torch.float64, device=self.dev)
        half = {k: f[k] + 0.5 * dt * f[k + "_t"] for k in ("pos", "vel", "S", "rho", "T")}
        if built:
            self.built = half["pos"].detach()
        x, v, S, rho, T = (half[k] for k in ("pos", "vel", "S", "rho", "T"))
        tool, mech = f["tool"], ~f["tool"]
        c0 = float(np.sqrt(np.float32(P.K / P.rho0)))
        p = torch.where(tool, z, c0 * c0 * (rho - P.rho0))
        # artificial stress
        sxx, syy, sxy = S[:, 0] - p, S[:, 2] - p, S[:, 1]
        num, den = 2 * sxy, sxx - syy
        flat = (num == 0) & (den == 0)
        ang = torch.atan2(torch.where(flat, z, num), torch.where(flat, z + 1, den))
        ang = ang + (torch.atan2(num.float(), den.float()).double() - ang).detach()
        th = 0.5 * ang
        ct = torch.cos(th) + (torch.cos(th.float()).double() - torch.cos(th)).detach()
        sn = torch.sin(th) + (torch.sin(th.float()).double() - torch.sin(th)).detach()
        c2, s2, cs = ct * ct, sn * sn, ct * sn
        r21 = 1 / (rho * rho)
        rx, ry = c2 * sxx + 2 * cs * sxy + s2 * syy, s2 * sxx - 2 * cs * sxy + c2 * syy
        rx = torch.where((rx > 0) & mech, -K.stresseps * rx * r21, z)
        ry = torch.where((ry > 0) & mech, -K.stresseps * ry * r21, z)
        R = torch.stack([c2 * rx + s2 * ry, cs * (rx - ry), s2 * rx + c2 * ry], 1)
        s3 = torch.stack([sxx * r21, sxy * r21, syy * r21], 1)
        c = _sqrtf(P.K / rho)
        vol = P.mass / rho
        h = f["h"]
        heat = (torch.where(tool, z + tl.alpha, z + wp.alpha) if not self.pse else z)
        vd, sd, acc, lap, pse = z.new_zeros(self.N, 4), z.new_zeros(self.N, 4), z.new_zeros(self.N, 4), z.clone(), z.clone()
        xd = x.detach()
        for i, j in self.pairs(self.lists and not built):
            if self.pse and wp.alpha != 0:
                d = xd[i] - xd[j]
                h2 = h[i] ** 2
                w2 = 4.0 / (h2 * h2 * math.pi) * torch.exp(-(d * d).sum(1) / h2)
                pse = pse.index_add(0, i, (T[j] - T[i]) * w2 * vol[j])
            rr = ((xd[i] - xd[j]) ** 2).sum(1)
            keep = (rr < 4 * h[i] ** 2) & (rr >= 1e-8)
            if self.pse:
                keep &= mech[i]
            i, j = i[keep], j[keep]
            d = x[i] - x[j]
            rr = (d * d).sum(1)
            h1 = 1 / h[i]
            rad = _sqrtf(rr)
            q = rad * h1
            fac = 0.454728408833987 * h1 * h1
            t = 2 - q
            out = q.detach() > 1
            w = torch.where(out, 0.25 * t**6, 1 - 1.5 * q * q * (1 - 0.5 * q)) * fac
            dw = torch.where(out, -0.75 * t * t, -3.0 * q * (1 - 0.75 * q)) * h1 / rad * fac
            lap = lap.index_add(0, i, 2.0 * vol[j] * (T[i] - T[j]) * dw)
            both = mech[i] & mech[j]
            i, j, d, rr, w, dw = i[both], j[both], d[both], rr[both], w[both], dw[both]
            wx, wy = dw * d[:, 0], dw * d[:, 1]
            dv = (v[j] - v[i]) * vol[j][:, None]
            vd = vd.index_add(0, i, torch.stack([dv[:, 0] * wx, dv[:, 0] * wy, dv[:, 1] * wx, dv[:, 1] * wy], 1))
            fab = (w / K.wdeltap) ** 4
            st = P.mass * (s3[i] + s3[j] + fab[:, None] * (R[i] + R[j]))
            sd = sd.index_add(0, i, torch.stack([st[:, 0] * wx, st[:, 1] * wy, st[:, 1] * wx, st[:, 2] * wy], 1))
            u = v[i] - v[j]
            ur = (u * d).sum(1)
            ir = 1 / (0.5 * (rho[i] + rho[j]))
            hij = 0.5 * (h[i] + h[j])
            mu = hij * ur / (rr + K.eta**2 * hij * hij)
            pi = torch.where(ur.detach() < 0, (-K.alpha * 0.5 * (c[i] + c[j]) * mu + K.beta * mu * mu) * ir,
                             torch.zeros_like(mu))
            xs = -K.xspheps * P.mass * w * ir
            acc = acc.index_add(0, i, torch.stack([-P.mass * pi * wx, -P.mass * pi * wy, xs * u[:, 0], xs * u[:, 1]], 1))
        e01, w01 = 0.5 * (vd[:, 1] + vd[:, 2]), 0.5 * (vd[:, 2] - vd[:, 1])
        t3, g2 = (vd[:, 0] + vd[:, 3]) / 3, 2 * P.G
        S_t = torch.stack([g2 * (vd[:, 0] - t3) - 2 * w01 * S[:, 1], g2 * e01 + w01 * (S[:, 0] - S[:, 2]),
                           g2 * (vd[:, 3] - t3) + 2 * w01 * S[:, 1], -g2 * t3], 1)
        m1 = mech[:, None]
        vel_t = acc[:, :2] + torch.stack([sd[:, 0] + sd[:, 1], sd[:, 2] + sd[:, 3]], 1) + (f["fc"] + f["ft"]) / P.mass
        pos_t = acc[:, 2:] + v
        zero2 = torch.zeros_like(pos_t)
        keep2 = (f["pos_t"], f["vel_t"]) if self.pse else (zero2, zero2)
        g = dict(f)
        g["pos_t"], g["vel_t"] = torch.where(m1, pos_t, keep2[0]), torch.where(m1, vel_t, keep2[1])
        g["S_t"] = torch.where(m1, S_t, f["S_t"])
        g["rho_t"] = torch.where(mech, -rho * (vd[:, 0] + vd[:, 3]), f["rho_t"])
        if self.pse:
            if wp.alpha != 0:
                # the model's half-length reading of the tool mark: only the first half of the array
                first = torch.arange(self.N, device=self.dev) < (4 * self.N) // 8
                g["T_t"] = torch.where(tool & first, z + tl.alpha, z + wp.alpha) * pse
        else:
            g["T_t"] = torch.where(heat != 0, heat * lap, f["T_t"])
        self.finish(f, g, p)
        self.f = g
        self.sort_now = not self.lists
        if self.lists:
            skin = float(np.float32(0.1 * self.cell))
            away = g["pos"].detach() + 0.5 * dt * g["pos_t"].detach() - self.built
            self.sort_now = bool(((away * away).sum(1) > (0.45 * skin) ** 2).any())

    def flow(self, eps, rate, T):
        jc, a = self.jc, self.par
        theta = (T - jc.Tref) / (jc.Tmelt - jc.Tref)

        def power(b, e):
            safe = torch.where(b > 0, b, torch.ones_like(b))
            return torch.where(b > 0, torch.pow(safe, e), torch.zeros_like(b))
        r = rate / jc.eps_dot_ref
        fast = r.detach() > 1
        term = torch.where(fast, 1 + a["C"] * torch.log(torch.where(fast, r, torch.ones_like(r))), torch.pow(1 + torch.where(fast, torch.zeros_like(r), r), a["C"]))
        return (a["A"] + a["B"] * power(eps, a["n"])) * term * (1 - power(theta, a["m"]))

    def finish(self, f, g, p):
        P, dt, wp, tl, tool = self.phys, self.dt, self.wp, self.tl, f["tool"]
        mech = ~tool
        pos, vel = f["pos"] + dt * g["pos_t"], f["vel"] + dt * g["vel_t"]
        S, rho, T = f["S"] + dt * g["S_t"], f["rho"] + dt * g["rho_t"], f["T"] + dt * g["T_t"]
        fc, ft = f["fc"], f["ft"]
        if self.tool is not None:
            self.tool.advance(dt)
            tv = torch.tensor(self.tool.vel, dtype=torch.float64, device=self.dev)
            if wp.eta != 0:
                idx = torch.nonzero(mech & ((ft.detach() ** 2).sum(1) > 0)).flatten()
                mag = _sqrtf((ft[idx] ** 2).sum(1))
                u = vel[idx] - tv
                un = (u * self.n[idx]).sum(1)
                T = T.index_add(0, idx, wp.eta * dt * mag * _sqrtf(((u - un[:, None]) ** 2).sum(1)) / (wp.cp * P.mass))
        eps, epsd = f["eps_pl"], f["eps_pl_dot"]
        if self.plastic:
            svm = _sqrtf(S[:, 0] ** 2 + S[:, 2] ** 2 + S[:, 3] ** 2 - S[:, 0] * S[:, 2] - S[:, 0] * S[:, 3]
                         - S[:, 2] * S[:, 3] + 3.0 * S[:, 1] ** 2)
            y = torch.nonzero(mech & ~(svm.detach() < self.flow(eps, epsd, T).detach())).flatten()
            e0, Ty, Sy = eps[y], T[y], S[y]
            norm = _sqrtf((Sy * Sy).sum(1))
            s23 = math.sqrt(2.0 / 3.0)
            init = epsd[y] * dt * s23
            dl = torch.where(init.detach() > 1e-8, init, torch.full_like(init, 1e-8))
            open_ = torch.ones_like(dl, dtype=torch.bool)

            def residual(d):
                dp = torch.where(d.detach() > 0, d, torch.zeros_like(d))
                return norm - 2 * P.G * d - s23 * self.flow(e0 + s23 * dp, s23 * dp / dt, Ty)
            for _ in range(51):
                if not bool(open_.any()):
                    break
                d1 = dl * 1.01
                r0, r1 = residual(dl), residual(d1)
                new = dl - r0 / ((r0 - r1) / (dl - d1))
                new = torch.where(new.detach() < 0, -0.1 * new, new)
                new = torch.where(open_, new, dl)
                open_ = open_ & ~((new.detach() - dl.detach()).abs() < 1e-6)
                dl = new
            s23f = float(np.sqrt(np.float32(2.0 / 3.0)))
            inc = torch.where(dl.detach() > 0, dl, torch.zeros_like(dl)) * s23
            rounded = (np.float32(s23f) * torch.clamp(dl.detach().float(), min=0)).double()
            inc = inc + (rounded - inc).detach()
            en, rn = e0 + inc, inc / dt
            if wp.tq != 0:
                T = T.index_add(0, y, wp.tq / (wp.cp * rho[y]) * (en - e0) * self.flow(en, rn, Ty))
            S = S.index_copy(0, y, Sy - Sy / norm[:, None] * dl[:, None] * 2.0 * P.G)
            rate = torch.zeros_like(epsd).index_copy(0, y, rn)
            epsd = torch.where(mech, rate, epsd)
            eps = eps.index_copy(0, y, en)
        if self.tool is not None:
            pos = torch.where(tool[:, None], pos + dt * tv, pos)
            inside, idx, cx, cy, nx, ny = self.tool.contact(pos[:, 0], pos[:, 1])
            sel = mech[idx]
            idx, cx, cy, nx, ny = idx[sel], cx[sel], cy[sel], nx[sel], ny[sel]
            tl_ = self.tool
            fN = (-tl_.mass * ((pos[idx, 0] - cx) * nx + (pos[idx, 1] - cy) * ny))[:, None] * torch.stack([nx, ny], 1)
            fN = fN / (dt * dt) * tl_.alpha
            fT = torch.zeros_like(fN)
            mu = self.par.get("mu", tl_.mu)
            if float(mu) != 0:
                u = vel[idx] - tv
                nn = torch.stack([nx, ny], 1)
                k = tl_.alpha * tl_.mass * (u - u * nn) / dt
                lim = mu * torch.sqrt((fN * fN).sum(1))
                stick = ft[idx] - k
                ls = torch.sqrt((stick * stick).sum(1))
                fT = torch.where((ls.detach() > lim.detach())[:, None], lim[:, None] * stick / ls[:, None], stick)
            new_c, new_t, new_n = torch.zeros_like(fc), torch.zeros_like(ft), torch.zeros_like(self.n)
            new_c, new_t = new_c.index_copy(0, idx, fN), new_t.index_copy(0, idx, fT)
            new_n = new_n.index_copy(0, idx, torch.stack([nx, ny], 1))
            fc, ft = torch.where(tool[:, None], fc, new_c), torch.where(tool[:, None], ft, new_t)
            self.n = torch.where(tool[:, None], self.n, new_n)
        hold = (mech & f["fixed"])[:, None]
        zero = torch.zeros_like(pos)
        vel, fc = torch.where(hold, zero, vel), torch.where(hold, zero, fc)
        g["pos_t"], g["vel_t"] = torch.where(hold, zero, g["pos_t"]), torch.where(hold, zero, g["vel_t"])
        if tl.alpha != 0:
            T = torch.where(f["fixed"], torch.full_like(T, wp.T_init), T)
        g.update(pos=pos, vel=vel, S=S, rho=rho, T=T, eps_pl=eps, eps_pl_dot=epsd, fc=fc, ft=ft)

    def force(self):
        return (self.f["fc"] + self.f["ft"]).sum(0)

    def by_number(self, k):
        out = torch.empty_like(self.f[k])
        out[self.f["id"]] = self.f[k]
        return out


def _exact_gradient(case, st):
    steps, names = case["skip"] + case["window"], ("A", "B", "n", "C", "m", "mu")
    which = range(6) if case["param"] < 0 else [case["param"]]
    fw = torch.autograd.forward_ad
    mean, rows = None, []
    for k in which:
        with torch.no_grad(), fw.dual_level():
            e = _Exact(case, st)
            e.par["mu"] = e.tool.mu
            v = torch.tensor(e.par[names[k]], dtype=torch.float64, device=e.dev)
            e.par[names[k]] = fw.make_dual(v, torch.ones_like(v))
            total = torch.zeros(2, dtype=torch.float64, device=e.dev)
            for n in range(steps):
                e.step()
                if n >= case["skip"]:
                    total = total + e.force()
            value, tangent = fw.unpack_dual(total / case["window"])
            mean = value.cpu().numpy()
            rows.append(np.zeros(2) if tangent is None else tangent.cpu().numpy())
    return {"mean": mean, "dmean": np.stack(rows) if case["param"] < 0 else rows[0]}


def exact(case, seed):
    mf = _package()
    inputs = _inputs(mf, case, seed)
    if case["kind"] == "gradient":
        return _exact_gradient(case, inputs[0])
    got, force = [], []
    with torch.no_grad():
        for st in inputs:
            e = _Exact(case, st)
            if case["kind"] == "cells":
                e.sort()
                return {"id": e.f["id"].to(torch.int32), "hash": e.hash.to(torch.int32), "pos": e.f["pos"]}
            for _ in range(case["steps"]):
                e.step()
                if case.get("each"):
                    force.append(e.force())
            got.append({k: e.by_number(k) for k in OUT})
            del e
    out = {k: torch.cat([g[k] for g in got]) for k in OUT}
    return dict(out, force=torch.stack(force)) if case.get("each") else out
