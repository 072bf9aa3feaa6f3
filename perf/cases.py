"""The measured work: what a program built on `arphys` has it do, through its
public entry points.

A pass of a stepping case is one frame of such a program: the particle records
go in (`set_particles_async`, page-locked host memory), the simulation advances
(`update` or `step`), and the records come back (`particles_async`,
`synchronize`).  A pass of a gradient case records a few steps on a tape and
runs the reverse pass; a pass of a render case draws one frame into host
memory; a pass of a grid case builds a cell grid over device positions without
allocating.  Starting states are in motion (a smooth velocity field with some
noise, densities off their rest value by a fraction of a percent), as a
simulation meets them after its first few steps.  The sizes of a batch's scenes
come from its layout number, their states from the seed.

`exact` restates the step in double precision with torch: neighbor pairs from a
cell list, every pair term and the total-Lagrangian solids as index sums, the
integrators, and the gradients by automatic differentiation of that.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch
import torch.utils.checkpoint

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ar-physics_b200"))

from arphys import FluidSim, PARTICLE_DTYPE, load_library, scenes  # noqa: E402
from arphys.abi import ArpAABB, check  # noqa: E402


# ---- the cases -------------------------------------------------------------------

def listed():
    return [
        # an interactive 2D demo: a few hundred particles in a walled box, one
        # frame of 4 subticks by plain launches; launch latency is everything
        {"name": "frame_2d_small", "kind": "dam2d", "nx": 19, "ny": 17, "integrator": "rk4", "steps": 4,
         "graph": False, "update": True},
        # the 2D dam break benchmark configuration (128 x 128, RK4), steps replayed from graphs
        {"name": "dam_break_2d", "kind": "dam2d", "nx": 128, "ny": 128, "integrator": "rk4", "steps": 10,
         "graph": True, "update": False},
        # a 3D scene of a real-time demo's size, odd extents: fluid meeting an elastic bar over a floor
        # with friction, velocity Verlet (the integrator scene files get by default), plain launches
        {"name": "verlet_3d_demo", "kind": "bar3d", "fluid": 25, "bar": 7, "integrator": "verlet", "steps": 10,
         "graph": False, "friction": 0.1},
        # a mid-size 3D scene, RK4 (the integrator most scene files name), graphs
        {"name": "rk4_3d_mid", "kind": "bar3d", "fluid": 48, "bar": 16, "integrator": "rk4", "steps": 5,
         "graph": True, "friction": 0.0},
        # the 3D benchmark configuration: 1,048,576 particles, RK2, graphs
        {"name": "fluid_bar_3d_1m", "kind": "bar3d", "fluid": 96, "bar": 32, "integrator": "rk2", "steps": 10,
         "graph": True, "friction": 0.0},
        # many uneven 3D scenes stepped as one batch (2,048 to 65,536 particles each, h of 1.5 to 2.5 spacings)
        {"name": "batch_3d", "kind": "batch3d", "count": 48, "n_max": 65536, "layout": 3, "steps": 10,
         "graph": True},
        # a plastic solid under velocity Verlet, as the shipped plastic scenes are stepped
        {"name": "plastic_bar", "kind": "solid", "w": 12, "height": 65, "order": 2, "plastic": True,
         "integrator": "verlet", "steps": 10, "graph": True},
        # reverse mode through an elastic bar with per-particle stiffness
        {"name": "bar_gradient", "kind": "bargrad", "w": 16, "height": 128, "steps": 6, "every": 3},
        # reverse mode through a batch of 2D Rayleigh-Taylor scenes
        {"name": "rt_batch_gradient", "kind": "rtgrad", "count": 8, "n_max": 65536, "layout": 5, "steps": 4,
         "every": 2},
        # one recorded 1080p frame, density-ramp splats in draw order
        {"name": "render_splats_1080p", "kind": "render", "fluid": 64, "width": 1920, "height": 1080,
         "lighting": False},
        # the same with lit spheres
        {"name": "render_lit_1080p", "kind": "render", "fluid": 64, "width": 1920, "height": 1080, "lighting": True},
        # the allocation-free grid build of a host framework, at close to its particle maximum
        {"name": "grid_build_1m", "kind": "grid", "n": 1000000, "per_cell": 8.0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dam2d", "dam2d", "bar3d", "bar3d", "bar3d", "batch3d", "solid", "solid", "bargrad", "rtgrad",
                       "render", "grid"])
    rk = ["rk4", "rk2", "verlet", "heun2", "rk3", "euler"]
    if kind == "dam2d":
        return {"kind": kind, "nx": _log_int(rng, 12, 300), "ny": _log_int(rng, 12, 300),
                "integrator": rng.choice(rk), "steps": rng.randint(1, 10), "graph": rng.random() < 0.5,
                "update": rng.random() < 0.5}
    if kind == "bar3d":
        f = _log_int(rng, 10, 80)
        return {"kind": kind, "fluid": f, "bar": max(4, f // 3), "integrator": rng.choice(rk[:3]),
                "steps": rng.randint(1, 8), "graph": rng.random() < 0.5, "friction": rng.choice([0.0, 0.1])}
    if kind == "batch3d":
        return {"kind": kind, "count": rng.randint(3, 40), "n_max": _log_int(rng, 4096, 65536),
                "layout": rng.randint(0, 1 << 20), "steps": rng.randint(1, 8), "graph": rng.random() < 0.5}
    if kind == "solid":
        return {"kind": kind, "w": _log_int(rng, 4, 20), "height": _log_int(rng, 16, 120),
                "order": rng.choice([2, 2, 0, 1, -2]), "plastic": rng.random() < 0.4,
                "integrator": rng.choice(["verlet", "rk4", "rk2"]), "steps": rng.randint(1, 8),
                "graph": rng.random() < 0.5}
    if kind == "bargrad":
        return {"kind": kind, "w": _log_int(rng, 4, 16), "height": _log_int(rng, 16, 120), "steps": rng.randint(2, 6),
                "every": rng.randint(1, 4)}
    if kind == "rtgrad":
        return {"kind": kind, "count": rng.randint(1, 7), "n_max": _log_int(rng, 9000, 65536),
                "layout": rng.randint(0, 1 << 20), "steps": rng.randint(1, 4), "every": rng.randint(1, 3)}
    if kind == "render":
        w = _log_int(rng, 320, 1920)
        return {"kind": kind, "fluid": _log_int(rng, 12, 60), "width": w, "height": max(180, int(w * 0.5625)),
                "lighting": rng.random() < 0.5}
    return {"kind": kind, "n": _log_int(rng, 1000, 1000000), "per_cell": rng.choice([1.0, 4.0, 8.0, 20.0])}


# ---- scenes and starting states -----------------------------------------------------

def _in_motion(sc, seed, speed=0.5, noise=0.02, dens=0.002):
    """A state in motion for a scene: a smooth velocity field over the box plus
    noise, and densities off their rest value by up to `dens`."""
    rng = np.random.default_rng(1000003 + seed)
    p = sc.particles
    lo, d = np.asarray(sc.bounds_min[:3]), np.asarray(sc.bounds_dim[:3])
    flat = d[2] == 0.0
    x = (p["pos"][:, :3].astype(np.float64) - lo) / np.where(d > 0, d, 1.0)
    ph = rng.uniform(0, 2 * math.pi, size=(3, 3))
    v = np.stack([sum(np.sin(2 * math.pi * x[:, a] + ph[c, a]) for a in range(3)) for c in range(3)], axis=1)
    v = speed * v / math.sqrt(1.5) + rng.normal(0.0, noise, size=v.shape)
    if flat:
        v[:, 2] = 0.0
    p["vel"][:, :3] += v.astype(np.float32)
    p["den"] *= (1.0 + dens * rng.uniform(-1.0, 1.0, size=len(p))).astype(np.float32)
    return sc


def _scenes_of(case, seed):
    """The scene (or the batch's scenes) of a case."""
    k = case["kind"]
    if k == "dam2d":
        nx, ny = case["nx"], case["ny"]
        sc = scenes.dam_break_2d(nx=nx, ny=ny, seed=seed, integrator=case["integrator"],
                                 box=(round(0.01 * (2 * nx + 2), 6), round(0.01 * (ny + 20), 6)))
        if case["update"]:
            sc.subticks = case["steps"]
            sc.dt = 1e-4 * case["steps"]
        return [_in_motion(sc, seed)]
    if k == "bar3d":
        f, b = case["fluid"], case["bar"]
        bx = round(0.01 * max(int(2.6667 * f), f + b + 16), 6)
        by = round(0.01 * max(int(1.3334 * f), 4 * b), 6)
        bz = round(0.01 * max(int(1.3334 * f), b + 8, f + 4), 6)
        sc = scenes.fluid_bar_3d(fluid_n=(f, f, f), bar_n=(b, 4 * b, b),
                                 floor_n=(int(round(bx * 100)), int(round(bz * 100))), seed=seed,
                                 box=(bx, by, bz), integrator=case["integrator"])
        if case["friction"]:
            sc.materials["visc"][0] = case["friction"]  # an immobile material's friction
        return [_in_motion(sc, seed)]
    if k == "batch3d":
        scs = scenes.batched_scenes(count=case["count"], n_max=case["n_max"], seed=case["layout"])
        return [_in_motion(sc, seed + 17 * q) for q, sc in enumerate(scs)]
    if k == "solid":
        sc = scenes.cantilever_bar(n=(case["w"], case["height"], case["w"]), seed=seed,
                                   integrator=case["integrator"])
        sc.materials["strain_order"][1] = case["order"]
        sc.materials["normal_damp"][1] = -2.0
        sc.materials["shear_damp"][1] = -2.0
        if case["plastic"]:
            for key, v in dict(plastic=1, yield_strength=100.0, relaxation_time=1e4, work_hardening_exp=2.0).items():
                sc.materials[key][1] = v
        return [_in_motion(sc, seed)]
    if k == "bargrad":
        return [_in_motion(scenes.cantilever_bar(n=(case["w"], case["height"], case["w"]), seed=seed), seed, speed=1.0)]
    if k == "rtgrad":
        scs = scenes.rayleigh_taylor_batch(count=case["count"], n_max=case["n_max"], seed=case["layout"])
        return [_in_motion(sc, seed + 17 * q) for q, sc in enumerate(scs)]
    if k == "render":
        f = case["fluid"]
        return [_in_motion(scenes.fluid_bar_3d(fluid_n=(f, f, f), bar_n=(f // 3, 4 * (f // 3), f // 3), seed=seed,
                                               floor_n=(int(2.6667 * f), int(1.3334 * f)),
                                               box=(round(0.01 * int(2.6667 * f), 6), round(0.01 * int(1.34 * f), 6),
                                                    round(0.01 * int(1.3334 * f), 6))), seed, dens=0.5)]
    raise ValueError(k)


def _pinned(n):
    t = torch.empty(n * PARTICLE_DTYPE.itemsize, dtype=torch.uint8, pin_memory=torch.cuda.is_available())
    return t, t.numpy().view(PARTICLE_DTYPE)


def _grad_weights(n, seed, flat):
    """dL/d(state) of a loss over positions, velocities and densities."""
    g = np.random.default_rng(7 + seed).normal(size=(n, 8)).astype(np.float32)
    g[:, 3] *= 1e-3
    g[:, 7] = 0.0
    if flat:
        g[:, 2] = g[:, 6] = 0.0
    return g


def _grid_inputs(case, seed):
    n = case["n"]
    cells = max(1, int(round((n / case["per_cell"]) ** (1.0 / 3.0))))
    box = np.float32(0.02) * np.float32(cells)
    rng = np.random.default_rng(11 + seed)
    p = rng.uniform(0.0, 1.0, size=(n, 4)).astype(np.float32)
    p[:, :3] *= box
    order = np.lexsort((p[:, 0], (p[:, 1] / 0.02).astype(np.int32), (p[:, 2] / 0.02).astype(np.int32)))
    return p[order], float(box)  # in cell rows, as a simulation keeps its particles


# ---- prepare and run ------------------------------------------------------------------

def prepare(case, seed):
    k = case["kind"]
    if k == "grid":
        p, box = _grid_inputs(case, seed)
        b = ArpAABB()
        for a in range(3):
            b.dim[a] = box
        sub = int(max(np.float32(1.0), np.float32(box) / np.float32(0.02)))
        nc = sub ** 3
        return {"kind": k, "lib": load_library(), "pos": torch.from_numpy(p).cuda(), "bounds": b, "nc": nc,
                "start": torch.empty(nc + 2, dtype=torch.int32, device="cuda"),
                "perm": torch.empty(case["n"], dtype=torch.int32, device="cuda")}
    scs = _scenes_of(case, seed)
    sim = FluidSim(scs[0]) if len(scs) == 1 else FluidSim.batch(scs)
    sim.init()
    state = {"kind": k, "sim": sim, "case": case}
    if k == "render":
        f = case["fluid"]
        m = len(scs[0].materials)
        colors = np.zeros((m, 12), np.float32)
        colors[:, 0:4] = [[0.2 + 0.2 * q, 0.4, 1.0 - 0.2 * q, 0.9] for q in range(m)]
        colors[:, 4:8] = [0.1, 0.1, 0.4, 0.8]
        colors[:, 8:12] = [1.0, 0.9, 0.2, 1.0]
        state["view"] = dict(angle=0.3, pos=(0.0133 * f, -0.0066 * f), scale=1.0)
        state["style"] = dict(render_h=0.02 * 0.7, lighting=case["lighting"], light_pos=(-1.0, 1.0, -1.0),
                              ambient=0.6, diffuse=1.0, specular=0.2, colors=colors,
                              densities=scs[0].materials["start_den"].copy())
        return state
    state["keep"], state["in"] = _pinned(sim.n)
    state["in"][:] = np.concatenate([sc.particles for sc in scs])
    if k in ("bargrad", "rtgrad"):
        if k == "bargrad":
            sim.set_solid_stiffness(scs[0].meta["stiffness"])
        state["dl"] = _grad_weights(sim.n, seed, k == "rtgrad")
        return state
    state["keep_out"], state["out"] = _pinned(sim.n)
    sim.set_graph(case["graph"])
    return state


def run(state):
    k = state["kind"]
    if k == "grid":
        p, nc = state["pos"], state["nc"]
        check(state["lib"].arp_grid_build_noalloc(p.data_ptr(), p.shape[0], ctypes.byref(state["bounds"]), 0.02,
                                                  state["start"].data_ptr(), nc + 2, state["perm"].data_ptr(),
                                                  torch.cuda.current_stream().cuda_stream))
        return {"cell_start": state["start"], "perm": state["perm"]}
    sim, case = state["sim"], state["case"]
    if k == "render":
        return sim.render(case["width"], case["height"], state["view"], state["style"])
    if k in ("bargrad", "rtgrad"):
        sim.set_particles(state["in"])
        sim.tape_begin(case["every"])
        sim.step(case["steps"])
        g, gs = sim.backward(state["dl"])
        sim.tape_end()
        return {"state": g, "stiffness": gs} if k == "bargrad" else {"state": g}
    sim.set_particles_async(state["in"])
    if case.get("update"):
        sim.update()
    else:
        sim.step(case["steps"])
    sim.particles_async(state["out"])
    sim.synchronize()
    o = state["out"]
    return {"den": o["den"], "pos": o["pos"][:, :3], "vel": o["vel"][:, :3], "mat": o["mat"],
            "solid_id": o["solid_id"]}


# ---- what a pass cannot do without ---------------------------------------------------

_STAGES = {"euler": 1, "rk2": 2, "midpoint": 2, "heun2": 2, "rk3": 3, "rk4": 4, "verlet": 1}


def work(case):
    k = case["kind"]
    if k == "grid":
        cells = max(1, int(round((case["n"] / case["per_cell"]) ** (1.0 / 3.0)))) ** 3
        return {"bytes": 16 * case["n"] + 4 * case["n"] + 4 * cells, "flops": 12 * case["n"]}
    if k == "render":
        n = case["fluid"] ** 3 + 4 * (case["fluid"] // 3) ** 3 + int(3.5 * case["fluid"] ** 2)
        return {"bytes": 32 * n + 3 * case["width"] * case["height"], "flops": 60 * n}
    # particles, solids among them, neighbors within h per particle (bodies of finite size)
    if k == "dam2d":
        n, ns, nbr, st = case["nx"] * case["ny"], 0, 12, _STAGES[case["integrator"]]
    elif k == "bar3d":
        ns = 4 * case["bar"] ** 3
        n, nbr, st = case["fluid"] ** 3 + ns, 28, _STAGES[case["integrator"]]
    elif k == "batch3d":
        n = int(case["count"] * (case["n_max"] - 2048) / math.log(case["n_max"] / 2048.0) * 0.75)
        ns, nbr, st = n // 3, 28, 2
    elif k == "rtgrad":
        n, ns, nbr, st = case["count"] * (case["n_max"] + 8192) // 2, 0, 12, 2
    else:
        n = ns = case["w"] ** 2 * case["height"]
        nbr, st = 24, _STAGES[case.get("integrator", "rk2")]
    flops = case["steps"] * st * nbr * (45.0 * n + 150.0 * ns)
    if k in ("bargrad", "rtgrad"):  # the reverse pass evaluates both orientations of each pair's derivative
        return {"bytes": 48 * n + 32 * n + 32 * n + 8 * ns, "flops": 4.0 * flops}
    return {"bytes": 96 * n, "flops": flops}


# ---- the same in double precision -----------------------------------------------------

_TABLEAUS = {
    "euler": ([[]], [1.0]),
    "rk2": ([[], [0.5]], [0.0, 1.0]),
    "heun2": ([[], [1.0]], [0.5, 0.5]),
    "rk3": ([[], [0.5], [-1.0, 2.0]], [1 / 6, 2 / 3, 1 / 6]),
    "rk4": ([[], [0.5], [0.0, 0.5], [0.0, 0.0, 1.0]], [1 / 6, 1 / 3, 1 / 3, 1 / 6]),
}


def _norm_const(n, h):
    def vol(m):
        return 1.0 if m == 0 else 2.0 * h if m == 1 else 2.0 * math.pi * h * h * vol(m - 2) / m
    return math.pi ** 3 / (6.0 * vol(n + 6))


def _dot(a, b):
    return (a * b).sum(-1)


class _Step64:
    """One or several scenes in double precision: constants, reference lists, forces, integrators."""

    def __init__(self, scs, stiffness=None, slack=0.05):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        f8 = dict(dtype=torch.float64, device=dev)
        self.dev, self.dt = dev, float(np.float32(np.float32(scs[0].dt) / np.float32(scs[0].subticks)))
        self.integrator = {"midpoint": "rk2"}.get(scs[0].integrator, scs[0].integrator)
        self.scs = scs
        mats, base, inter = [], [], []
        for sc in scs:
            base.append(sum(len(m) for m in mats))
            mats.append(sc.materials)
        M = np.concatenate(mats)
        nm = len(M)
        it = np.zeros((nm, nm, 5))
        for sc, b in zip(scs, base):
            for i, a in enumerate(sc.materials):
                for j, c in enumerate(sc.materials):
                    if i != j and (a["state_eq"] == 0 or c["state_eq"] == 0):  # the default interaction: linear contact
                        it[b + i, b + j] = (2, 10000.0, np.float32(sc.h) * np.float32(2.0), 0.0,
                                            np.float32(a["visc"]) + np.float32(c["visc"]))
        self.it = torch.tensor(it, **f8)
        self.m = {k: torch.tensor(M[k].astype(np.float64), **f8) for k in M.dtype.names}

        def scene_t(vals):
            return torch.tensor([float(v) for v in vals], **f8)
        self.h = scene_t([np.float32(sc.h) for sc in scs])
        self.k = scene_t([_norm_const(sc.dim, float(np.float32(sc.h))) for sc in scs])
        self.g = scene_t([np.float32(sc.gravity) for sc in scs])
        self.dim = torch.tensor([sc.dim for sc in scs], device=dev)
        self.branch = torch.tensor([sc.n_solids() > 1 for sc in scs], device=dev)

        def cat(attr, field):
            return np.concatenate([getattr(sc, attr)[field] for sc in scs])
        mat = np.concatenate([sc.particles["mat"].astype(np.int64) + b for sc, b in zip(scs, base)])
        bmat = np.concatenate([sc.boundary["mat"].astype(np.int64) + b for sc, b in zip(scs, base)])
        self.n, self.nb = len(mat), len(bmat)
        self.mat = torch.tensor(np.concatenate([mat, bmat]), device=dev)  # boundary particles follow the mobile ones
        self.scene = torch.tensor(np.concatenate(
            [np.repeat(np.arange(len(scs)), [sc.n for sc in scs]),
             np.repeat(np.arange(len(scs)), [sc.nb for sc in scs])]).astype(np.int64), device=dev)
        self.x0 = torch.tensor(cat("particles", "pos")[:, :3].astype(np.float64), **f8)
        self.v0 = torch.tensor(cat("particles", "vel")[:, :3].astype(np.float64), **f8)
        self.r0 = torch.tensor(cat("particles", "den").astype(np.float64), **f8)
        self.bx = torch.tensor(cat("boundary", "pos")[:, :3].astype(np.float64), **f8)
        self.bv = torch.tensor(cat("boundary", "vel")[:, :3].astype(np.float64), **f8)
        self.br = torch.tensor(cat("boundary", "den").astype(np.float64), **f8)
        self.lo = torch.tensor(np.array([sc.bounds_min[:3] for sc in scs], np.float64), **f8)
        stiff = (self.m["normal_stiffness"] != 0) | (self.m["shear_stiffness"] != 0)
        self.stiff = stiff[self.mat]
        self.sol = torch.nonzero(self.stiff[:self.n] & self.branch[self.scene[:self.n]]).reshape(-1)
        self.plastic = bool((self.m["plastic"][self.mat[self.sol]] != 0).any())
        if len(self.sol):
            self._reference_lists(stiffness)
        self.pairs, self.pair_x, self.slack = None, None, slack

    # pairs (i mobile, j any) closer than (1 + slack) h
    def _search(self, x, n_self, scene, slack):
        h = self.h[scene]
        cell = torch.floor((x - self.lo[scene]) / (h * (1.0 + slack))[:, None]).to(torch.int64)
        cell -= cell.amin(0)
        span = cell.amax(0) + 3
        key = ((scene * span[2] + cell[:, 2] + 1) * span[1] + cell[:, 1] + 1) * span[0] + cell[:, 0] + 1
        order = torch.argsort(key, stable=True)
        skey = key[order]
        me = torch.arange(n_self, device=x.device)
        out_i, out_j = [], []
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                c = key[:n_self] + dz * span[1] * span[0] + dy * span[0]
                a = torch.searchsorted(skey, c - 1)
                b = torch.searchsorted(skey, c + 1, right=True)
                for part in torch.split(me, 1 << 18):  # rows of three cells at a time
                    cnt = b[part] - a[part]
                    i = torch.repeat_interleave(part, cnt)
                    first = torch.cumsum(cnt, 0) - cnt
                    j = order[torch.arange(len(i), device=x.device) - torch.repeat_interleave(first - a[part], cnt)]
                    d = x[j] - x[i]
                    ok = (_dot(d, d) < (h[i] * (1.0 + slack)) ** 2) & (j != i)
                    out_i.append(i[ok])
                    out_j.append(j[ok])
        return torch.cat(out_i), torch.cat(out_j)

    def _reference_lists(self, stiffness):
        X = self.x0[self.sol]
        sc = self.scene[self.sol]
        i, j = self._search(X, len(X), sc, 0.0)
        self.X, self.si, self.sj = X, i, j
        mat = self.mat[self.sol]
        self.smat = mat
        dX = X[j] - X[i]
        self.dX = dX
        diff = (self.h[sc[i]] ** 2 - _dot(dX, dX)).clamp(min=0.0)
        self.gW = (-6.0 * self.k[sc[i]] * diff ** 2)[:, None] * dX
        self.W = self.k[sc[i]] * diff ** 3
        self.V0 = (self.m["mass"] / self.m["start_den"])[mat]
        dim = self.dim[sc]
        C = torch.zeros(len(X), 3, 3, dtype=torch.float64, device=X.device)
        # column c, row r holds sum V gradW_r dX_c
        C.index_add_(0, i, self.V0[j][:, None, None] * (self.gW[:, :, None] * dX[:, None, :]))
        self.pad = (torch.arange(3, device=X.device)[None, :] >= dim[:, None])
        C = torch.where(torch.diag_embed(self.pad), torch.ones_like(C), C)
        self.L = torch.linalg.inv(C)
        self.same = mat[i] == mat[j]
        if stiffness is not None:
            s = torch.tensor(np.asarray(stiffness, np.float64), device=X.device)
            self.lam, self.mu = s[:, 0], s[:, 1]
        else:
            self.lam, self.mu = self.m["normal_stiffness"][mat], self.m["shear_stiffness"][mat]

    def _strain(self, F, Fd, order):
        Ft = F.transpose(1, 2)
        eye = torch.eye(3, dtype=torch.float64, device=F.device)
        C = torch.where(torch.diag_embed(self.pad), eye, Ft @ F)
        dC = Fd.transpose(1, 2) @ F
        dC = dC + dC.transpose(1, 2)
        if order == 2:
            return 0.5 * (C - eye), 0.5 * dC
        if order == 0:
            E, P = torch.zeros_like(C), eye.expand_as(C)
            for q in range(1, 6):
                P = P @ (C - eye)
                E = E + (1.0 if q & 1 else -1.0) / q * P
            return 0.5 * E, 0.5 * dC @ torch.linalg.inv(C)
        a = abs(order)
        m = a >> 1
        M = torch.linalg.matrix_power(C, m)
        if a & 1:
            w, U = torch.linalg.eigh(C)
            M = M @ (U * w.sqrt()[:, None, :]) @ U.transpose(1, 2)
        rate = torch.zeros_like(C)
        for q in range(m):
            rate = rate + torch.linalg.matrix_power(C, q) @ dC @ torch.linalg.matrix_power(C, m - 1 - q)
        rate = rate / order
        if order < 0:
            M = torch.linalg.inv(M)
            iC = torch.linalg.inv(C)
            rate = -iC @ rate @ iC
        return (M - eye) / order, rate

    def _solid(self, x, v, rho, ep, lam, mu):
        """The solids' acceleration (gravity included) and the plastic-strain rate (4 x 4)."""
        s, i, j = self.sol, self.si, self.sj
        sc = self.scene[s]
        xs, vs, rs = x[s], v[s], rho[s]
        n = len(s)
        mat = self.smat
        G = (self.L[i] @ self.gW[:, :, None])[:, :, 0]
        dx, dv = xs[j] - xs[i], vs[j] - vs[i]
        z = torch.zeros(n, 3, 3, dtype=torch.float64, device=x.device)
        F = z.index_add(0, i, self.V0[j][:, None, None] * dx[:, :, None] * G[:, None, :])
        Fd = z.index_add(0, i, self.V0[j][:, None, None] * dv[:, :, None] * G[:, None, :])
        E = torch.zeros(n, 4, 4, dtype=torch.float64, device=x.device)
        Ed = torch.zeros_like(E)
        for order in set(self.m["strain_order"][mat].long().tolist()):
            e3, r3 = self._strain(F, Fd, order)
            w = (self.m["strain_order"][mat].long() == order)[:, None, None].to(torch.float64)
            E = E + w * torch.nn.functional.pad(e3, (0, 1, 0, 1))
            Ed = Ed + w * torch.nn.functional.pad(r3, (0, 1, 0, 1))
        if ep is not None:
            E = E + ep
        on = ~self.pad
        eye4 = torch.eye(4, dtype=torch.float64, device=x.device)

        def hooke(e, a, b):
            tr = (torch.diagonal(e, dim1=1, dim2=2)[:, :3] * on).sum(-1)
            return (a * tr)[:, None, None] * eye4 + 2.0 * b[:, None, None] * e
        S = hooke(E, lam, mu) + hooke(Ed, self.m["normal_damp"][mat], self.m["shear_damp"][mat])
        A = F @ S[:, :3, :3].transpose(1, 2) @ self.L
        m1 = self.m["mass"][mat]
        c = torch.where(self.same, -(m1 / rs)[i] * (m1[i] / rs[j]), torch.zeros_like(rs[i]))
        f = c[:, None] * ((A[i] + A[j]) @ self.gW[:, :, None])[:, :, 0]
        f = f * on[i]
        # hourglass control over the reference pairs (all of them stay in neighboring cells here)
        hh = self.h[sc[i]]
        l2 = _dot(dx, dx)
        l = l2.sqrt()
        e = ((0.5 * (F[i] + F[j])) @ self.dX[:, :, None])[:, :, 0] - dx
        sh = (1e8 * m1[i] ** 2 / (rs[i] * rs[j])) * (0.5 * _dot(e, dx) / (l + hh)) / (l2 + 0.1 * hh * hh) * self.W
        u = torch.where(self.same, sh / (l + 0.1 * hh), torch.zeros_like(sh))
        f = f - u[:, None] * dx
        acc = torch.zeros(n, 3, dtype=torch.float64, device=x.device).index_add(0, i, f) / rs[:, None]
        acc = acc - self.g[sc][:, None] * torch.tensor([0.0, 1.0, 0.0], dtype=torch.float64, device=x.device)
        kep = None
        if ep is not None:
            sn = (S * S).sum((1, 2)).sqrt()
            Y = self.m["yield_strength"][mat]
            w = torch.where((self.m["plastic"][mat] != 0) & (Y <= sn), (sn - Y) / self.m["relaxation_time"][mat] / sn,
                            torch.zeros_like(sn))
            kep = w[:, None, None] * S
        return acc, kep

    def _pressure_term(self, rho, mat):
        eq, c, d0 = self.m["state_eq"][mat], self.m["sound_speed"][mat], self.m["target_den"][mat]
        tait = c * c * d0 / 7.0 * ((rho / torch.where(d0 != 0, d0, torch.ones_like(d0))) ** 7 - 1.0)
        p = torch.where(eq == 3, tait, torch.where(eq == 2, c * c * (rho - d0), torch.where(eq == 1, c * c, 0.0 * c)))
        return p / (rho * rho)

    def forces(self, x, v, rho, ep, lam=None, mu=None):
        """The derivative record: density rate, velocity the positions move with, acceleration, plastic rate."""
        n = self.n
        X, V, R = torch.cat([x, self.bx]), torch.cat([v, self.bv]), torch.cat([rho, self.br])
        with torch.no_grad():
            moved = math.inf if self.pairs is None else float((x - self.pair_x).norm(dim=1).max())
            if 2.0 * moved > 0.99 * self.slack * float(self.h.min()):
                self.pairs, self.pair_x = self._search(X.detach(), n, self.scene, self.slack), x.detach()
        pi, pj = self.pairs
        pt = self._pressure_term(R, self.mat)
        den = torch.zeros(n, dtype=torch.float64, device=x.device)
        acc = torch.zeros(n, 3, dtype=torch.float64, device=x.device)
        for i, j in zip(torch.split(pi, 1 << 23), torch.split(pj, 1 << 23)):
            dd, ff = self._fluid_pairs(i, j, X, V, R, pt)
            den = den.index_add(0, i, dd)
            acc = acc.index_add(0, i, ff)
        up = torch.tensor([0.0, 1.0, 0.0], dtype=torch.float64, device=x.device)
        a = acc / rho[:, None] - self.g[self.scene[:n]][:, None] * up
        vx = v
        kep = None
        if len(self.sol):
            sa, kep = self._solid(x, v, rho, ep, self.lam if lam is None else lam, self.mu if mu is None else mu)
            a = a.index_add(0, self.sol, sa)
            vx = v.index_add(0, self.sol, v[self.sol])  # both force terms carry dx/dt = v
        return den, vx, a, kep

    def _fluid_pairs(self, i, j, X, V, R, pt):
        sc = self.scene[i]
        h2, k = self.h[sc] ** 2, self.k[sc]
        mi, mj = self.mat[i], self.mat[j]
        m1, m2 = self.m["mass"][mi], self.m["mass"][mj]
        bnd = j >= self.n
        r = X[j] - X[i]
        r2 = _dot(r, r)
        gws = -6.0 * k * (h2 - r2).clamp(min=0.0) ** 2
        g = gws[:, None] * r
        v = V[j] - V[i]
        zero = torch.zeros_like(r2)
        den = torch.where(bnd, zero, m2 * _dot(v, g))
        f = (m1 * m2 * (pt[i] + pt[j]))[:, None] * g
        it = self.it[mi, mj]
        R1 = r2.sqrt()
        cp = torch.where(it[:, 0] == 2, it[:, 2] * (it[:, 1] - R1), zero)  # radius and strength swapped, as the shader has it
        cs = m2 * cp / R[j]
        f = f + cs[:, None] * g
        if float(self.it[:, :, 4].max()) > 0.0:
            fr = torch.where((self.stiff[i] | self.stiff[j] | bnd) & (mi != mj), it[:, 4], zero)
            u = v - (_dot(v, r) / r2)[:, None] * r
            ul = _dot(u, u).sqrt()
            t = torch.where((ul > 0)[:, None], u / torch.where(ul > 0, ul, torch.ones_like(ul))[:, None], torch.zeros_like(u))
            f = f + (fr * (cs * gws).abs() * R1)[:, None] * t
        denom = r2 + 0.1 * self.h[sc] ** 2
        vis = torch.where(bnd | self.stiff[i], zero, self.m["visc"][mi] + self.m["visc"][mj])
        f = f - (m1 * m2 * vis * _dot(r, g) / (R[i] * R[j] * denom))[:, None] * v
        bulk = torch.where(bnd, zero, torch.where(mi == mj, self.m["bulk_visc"][mi] + self.m["bulk_visc"][mj], it[:, 3]))
        f = f - (m1 * m2 * bulk * _dot(v, r) / ((R[i] + R[j]) * denom))[:, None] * g
        return den, f

    def advance(self, steps, y, lam=None, mu=None):
        """`steps` steps from y = (x, v, rho, ep)."""
        dt = self.dt
        ck = torch.utils.checkpoint.checkpoint if y[0].requires_grad else None

        def rate(s):
            if ck is None:
                return self.forces(*s)
            return ck(lambda x, v, r, a, b: self.forces(x, v, r, None, a, b), s[0], s[1], s[2], lam, mu,
                      use_reentrant=False)

        def moved(s, terms):
            x, v, r, e = s
            for c, (dr, dx, dv, de) in terms:
                x, v, r = x + c * dx, v + c * dv, r + c * dr
                e = e if e is None else e + c * de
            return x, v, r, e
        if self.integrator == "verlet":
            f = rate(y)
            for _ in range(steps):
                x, v, r, e = y
                v, r = v + 0.5 * dt * f[2], r + 0.5 * dt * f[0]
                e = e if e is None else e + 0.5 * dt * f[3]
                x = x + dt * v
                f = rate((x, v, r, e))
                y = (x, v + 0.5 * dt * f[2], r + 0.5 * dt * f[0], e if e is None else e + 0.5 * dt * f[3])
            return y
        a, b = _TABLEAUS[self.integrator]
        for _ in range(steps):
            ks = []
            for row in a:
                ks.append(rate(moved(y, [(c * dt, k) for c, k in zip(row, ks) if c])))
            y = moved(y, [(c * dt, k) for c, k in zip(b, ks) if c])
        return y


def exact(case, seed):
    k = case["kind"]
    if k in ("grid", "render"):
        return None  # whole numbers
    scs = _scenes_of(case, seed)
    grad = k in ("bargrad", "rtgrad")
    # a gradient keeps one pair list throughout (its stages are evaluated twice)
    S = _Step64(scs, scs[0].meta["stiffness"] if k == "bargrad" else None, 0.8 if grad else 0.05)
    ep = torch.zeros(len(S.sol), 4, 4, dtype=torch.float64, device=S.dev) if S.plastic else None
    if not grad:
        with torch.no_grad():
            x, v, r, _ = S.advance(case["steps"], (S.x0, S.v0, S.r0, ep))
        return {"den": r, "pos": x, "vel": v, "mat": None, "solid_id": None}
    y0 = [t.clone().requires_grad_(True) for t in (S.x0, S.v0, S.r0)]
    lm = [t.clone().requires_grad_(True) for t in (S.lam, S.mu)] if k == "bargrad" else [None, None]
    x, v, r, _ = S.advance(case["steps"], (*y0, None), *lm)
    w = torch.tensor(_grad_weights(S.n, seed, k == "rtgrad").astype(np.float64), device=S.dev)
    loss = (x * w[:, :3]).sum() + (r * w[:, 3]).sum() + (v * w[:, 4:7]).sum()
    got = torch.autograd.grad(loss, y0 + [t for t in lm if t is not None])
    g = torch.zeros(S.n, 8, dtype=torch.float64, device=S.dev)
    g[:, :3], g[:, 4:7], g[:, 3] = got[0], got[1], got[2]
    out = {"state": g}
    if k == "bargrad":
        out["stiffness"] = torch.stack(got[3:5], dim=1)
    return out
