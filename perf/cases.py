"""The work that users of this framework have it do, as cases to be timed.

A case is a scene with the calls a program makes on it: advance it by the steps
between two frames and read the frame (`Engine.update`), hook into every step
(`Engine.step`), exchange the state with another solver each step
(`Engine.update_io`), advance many scenes at once (`Batch`) or hand scenes to
the server (`Server`).  Scenes are those of the package's `scenes` module, over
the particle counts that its batched mix and serving stream draw (2k to 60k,
5k to 500k) and up to the 1.0M-fluid coupled dam break, and a packed bed of
grains.  A pass goes on from where the last one left the scene, as a
simulation does.

A frame is kept the way the frame files keep it, velocities, accelerations,
spins and densities as FP32 (what the engine's forces are computed in), but
positions stay in the FP64 that the download gives: a restart needs them.
"""
import math

import numpy as np
import torch

from __graft_entry__ import _package

ds = _package()
import dem_sphsource_gb300.scenes as scenes  # noqa: E402

# Steps or fluid periods between two frames, and the particle counts that
# draw() takes: (smallest, largest).
SPH_RANGE = (1_500, 420_000)
COUPLED_RANGE = (5_000, 500_000)
GRAINS_RANGE = (3_000, 210_000)


def listed():
    return [
        # A driver that looks at a small basin after every step: launches and latency are all there is.
        {"name": "basin_2k_step", "kind": "sph", "n": 2_000, "height": 0.3, "basin": True, "two": False, "steps": 1},
        # Two liquids (their own rest densities, sound speeds and smoothing lengths) side by side, a ragged count.
        {"name": "two_fluids_19k", "kind": "sph", "n": 9_501, "height": 0.27, "basin": False, "two": True, "steps": 20},
        # The plain benchmark scene: dx = 0.01 m.
        {"name": "dam_48k", "kind": "sph", "n": 48_000, "height": 0.3, "basin": False, "two": False, "steps": 20},
        # The upper end of what the serving stream draws.
        {"name": "dam_410k", "kind": "sph", "n": 410_000, "height": 0.3, "basin": False, "two": False, "steps": 8},
        # A driver that overrides update(): five stage calls a step.
        {"name": "stages_12k", "kind": "stages", "n": 12_000, "height": 0.3, "steps": 10},
        # Co-simulation: the whole state from the host and back every step.
        {"name": "exchange_47k", "kind": "exchange", "n": 47_000, "height": 0.31},
        # A small coupled scene of the batched mix alone: over a hundred DEM steps to a fluid step.
        {"name": "coupled_13k", "kind": "coupled", "n": 13_001, "height": 0.4, "periods": 2},
        # The coupled benchmark scene: 64 bonded cubes of 8^3 spheres, 0.6M wall particles.
        {"name": "coupled_1m", "kind": "coupled", "n": 1_000_000, "height": 0.4, "periods": 4},
        # A small bed of grains with clumps falling on it.
        {"name": "grains_6k", "kind": "grains", "n": 6_007, "clumps": 140, "steps": 50},
        # A bed of the granular benchmark's size, every grain in contact.
        {"name": "bed_200k", "kind": "grains", "n": 200_000, "clumps": 0, "steps": 40},
        # Scenes of the batched mix, one graph launch a round.
        {"name": "batch_8", "kind": "batch", "scenes": 8, "smallest": 2_000, "largest": 60_000, "steps": 40},
        # Requests of the serving stream's kinds, from submission to result (creation and set-up are part of it).
        {"name": "serve_6", "kind": "serve", "scenes": 6, "smallest": 5_000, "largest": 60_000, "steps": 120},
    ]


def _between(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(("sph", "sph", "coupled", "grains", "grains", "stages", "exchange", "batch", "serve"))
    height = round(rng.uniform(0.2, 0.5), 3)
    if kind == "sph":
        n = _between(rng, *SPH_RANGE)
        return {"kind": kind, "n": n, "height": height, "basin": rng.random() < 0.2, "two": rng.random() < 0.25,
                "steps": rng.randint(1, max(1, min(20, 3_500_000 // n)))}
    if kind == "coupled":
        n = _between(rng, *COUPLED_RANGE)
        return {"kind": kind, "n": n, "height": height, "periods": rng.randint(1, 3)}
    if kind == "grains":
        n = _between(rng, *GRAINS_RANGE)
        return {"kind": kind, "n": n, "clumps": rng.choice((0, n // 44)), "steps": rng.randint(1, 50)}
    if kind == "stages":
        return {"kind": kind, "n": _between(rng, 2_000, 60_000), "height": height, "steps": rng.randint(1, 12)}
    if kind == "exchange":
        return {"kind": kind, "n": _between(rng, 2_000, 200_000), "height": height}
    low, high = (2_000, 60_000) if kind == "batch" else (5_000, 60_000)
    return {"kind": kind, "scenes": rng.randint(2, 8), "smallest": low, "largest": high,
            "steps": rng.randint(3, 40) if kind == "batch" else rng.randint(50, 120)}


# ---------------------------------------------------------------- scenes

def _sph(case, seed):
    n, height = case["n"], case["height"]
    dx = (0.16 * height / n) ** (1.0 / 3.0)
    if case.get("basin"):  # liquid at rest, wall to wall
        r = scenes.dam_break(dx=dx, tank=(0.4, 0.4, height + 0.2), column=(0.4, 0.4, height), jitter=0.05, seed=seed)
    else:
        r = scenes.dam_break(dx=dx, column=(0.4, 0.4, height), jitter=0.05, seed=seed)
    if case.get("two"):
        rng = np.random.default_rng(seed + 1)
        size = (0.4, 0.4, 0.8 * height)
        x0 = 0.0 if case.get("basin") else 0.4
        p = scenes.regular_packed_points((x0, 0.0, height if case.get("basin") else 0.0), size, dx)
        p = p + rng.uniform(-0.05 * dx, 0.05 * dx, size=p.shape)
        if case.get("basin"):
            p = p[p[:, 2] < height + 0.15]
        r.addFluid(p, (0, 0, 0), 1.2 * dx, 1500.0, 25.0, 2.0e-6)
    return r


def _coupled(case, seed):
    return scenes.sized_coupled(case["n"], case["height"], seed=seed)


def _grains(case, seed):
    """Grains of about 1 mm radius, hexagonally packed on a floor wall with overlaps up to 1e-6 m (a bed under its
    own weight), one in five smaller and loose; clumps of four pebbles fall on the bed."""
    rng = np.random.default_rng(seed)
    n, clumps, r0 = case["n"], case["clumps"], 1.0e-3
    side = max(6, int(round((n / 1.5) ** (1.0 / 3.0))))
    layers = -(-n // (side * side))
    k, j, i = np.meshgrid(np.arange(layers), np.arange(side), np.arange(side), indexing="ij")
    i, j, k = (a.ravel()[:n].astype(np.float64) for a in (i, j, k))
    p = r0 * np.stack([1.0 + 2.0 * i + (j + k) % 2, 1.0 + math.sqrt(3.0) * (j + (k % 2) / 3.0),
                       1.0 + 2.0 * math.sqrt(6.0) / 3.0 * k], axis=1)
    radii = r0 * rng.uniform(0.9995, 1.0005, n)
    small = rng.random(n) < 0.2
    radii[small] = r0 * np.clip(np.exp(0.2 * rng.standard_normal(int(small.sum()))) - 0.2, 0.6, 0.98)
    r = scenes.Recipe("grains_%d" % n)
    box = (p.max(axis=0) + r0)
    m, rp, a = 6.0e-3, 1.0e-3, 0.8e-3
    pitch = 2 * (a + rp) * 1.05
    cx, cy = max(1, int(box[0] / pitch)), max(1, int(box[1] / pitch))
    height = box[2] + pitch * (-(-clumps // (cx * cy)))
    r.setDomain((-m, -m, -m), (box[0] + 2 * m, box[1] + 2 * m, height + 2 * m))
    Es, Gs = scenes.hertz_from_E_nu(1.0e8, 0.3)
    for u, v in ((0, 0), (0, 1), (1, 1)):
        r.setHertzianContactModel(u, v, Es, Gs, 0.5, 0.0, 0.0, 0.4, 0.0, 0.0)
    r.addCluster(p, radii, np.full(n, 2500.0), (0.02, -0.01, -0.05), 0)
    tet = np.array([[1, 1, 1], [1, -1, -1], [-1, 1, -1], [-1, -1, 1]], dtype=np.float64) / math.sqrt(3.0) * a
    rot = scenes._random_rotations(rng, clumps)
    for q in range(clumps):
        z, rest = divmod(q, cx * cy)
        c = np.array([(rest % cx + 0.5) * pitch, (rest // cx + 0.5) * pitch, box[2] + a + 1.05 * rp + z * pitch])
        peb = c + tet @ rot[q].T
        mass = 2500.0 * 4.0 / 3.0 * math.pi * rp ** 3 * 3.2
        pr = np.full(4, rp)
        r.addClump(peb, pr, c, (0, 0, -0.5), tuple(rng.uniform(-20, 20, 3)), mass,
                   scenes.clump_inertia(peb, pr, c, mass), 1)
    r.addInfiniteWall((0, 0, 0), (0, 0, 1), 0)
    t_r = math.pi * 0.6e-3 * math.sqrt(2500.0 * 2.6 / 1.0e8) / (0.1631 * 0.3 + 0.8766)
    r.setSimulationParameterTimeStep(0.1 * t_r)
    r.meta.update(dt=0.1 * t_r, gap=1)
    return r


def _mix(case, seed):
    """Recipes of the batched mix (SPH, coupled) or of the serving stream (SPH, DEM, coupled)."""
    rng = np.random.default_rng(seed)
    out = []
    for k in range(case["scenes"]):
        # spread evenly over the range: which scenes there are is the case's, what they hold the seed's
        n = int(case["smallest"] * (case["largest"] / case["smallest"]) ** ((k + 0.5) / case["scenes"]))
        height, s = 0.3, int(rng.integers(1 << 30))
        if case["kind"] == "serve" and k % 3 == 1:
            out.append(scenes.sized_granular(n, seed=s))
        elif k % 3 == 2 or (case["kind"] == "batch" and k % 5 == 1):
            out.append(scenes.sized_coupled(n, height, seed=s))
        else:
            out.append(scenes.sized_dam_break(n, height, seed=s))
    return out


def _recipes(case, seed):
    if case["kind"] in ("batch", "serve"):
        return _mix(case, seed)
    return [{"coupled": _coupled, "grains": _grains}.get(case["kind"], _sph)(case, seed)]


# ---------------------------------------------------------------- a program's calls

def _pinned(*shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True)


class _Sim:
    """One running simulation: its engine, the next step, and the host buffers that its frames are read into."""

    def __init__(self, recipe):
        self.builder, self.scene = ds.build_scene(recipe)
        self.engine = ds.Engine(self.scene)
        self.engine.initialize()
        self.dt, self.gap, self.next = self.scene.time_step, self.scene.fluid_integrate_gap, 1
        self.nf, self.ns = self.scene.n_fluid, self.scene.n_solid
        self.fluid = [_pinned(self.nf, 3), _pinned(self.nf, 3), _pinned(self.nf, 3), _pinned(self.nf)]
        # the walls of a plain dam break never move: its frames are the fluid's
        self.solids = any(fn in ("addCluster", "addClump", "addSolid") for fn, _ in recipe.calls)
        self.solid = {k: _pinned(self.ns, 3) for k in ("pos", "vel", "acc", "angvel")} if self.solids else {}

    def frame(self):
        out = {}
        if self.nf:
            self.engine.download_fluids([t.numpy() for t in self.fluid])
            pos, vel, acc, drho = self.fluid
            out.update(fluid_pos=pos, fluid_vel=vel.float(), fluid_acc=acc.float(), fluid_drho=drho.float())
        if self.solids:
            self.engine.download_solids({k: t.numpy() for k, t in self.solid.items()})
            out.update({"solid_" + k: t if k == "pos" else t.float() for k, t in self.solid.items()})
        return out


def prepare(case, seed):
    recipes = _recipes(case, seed)
    if case["kind"] == "serve":
        made = [ds.build_scene(r) for r in recipes]
        return {"case": case, "made": made, "server": ds.Server()}
    state = {"case": case, "sims": [_Sim(r) for r in recipes]}
    if case["kind"] == "batch":
        state["batch"] = ds.Batch()
        for sim in state["sims"]:  # a batch joins engines that have made their first step
            sim.engine.update(sim.dt, 1, 1, sim.gap)
            sim.next = 2
    if case["kind"] == "exchange":
        sim = state["sims"][0]
        p = np.concatenate([a[0] for fn, a in recipes[0].calls if fn == "addFluid"])
        sim.fluid[0].copy_(torch.from_numpy(p))
        sim.fluid[1].zero_()
        sim.fluid[3].zero_()
    torch.cuda.synchronize()
    return state


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "serve":
        server = state["server"]
        ids = [server.submit(scene, case["steps"]) for _, scene in state["made"]]
        out = []
        for rid in ids:
            server.wait(rid)
            got = server.fetch(rid)
            server.release(rid)
            out.append({k: v if k.endswith("pos") else torch.from_numpy(v).float() for k, v in got.items()
                        if len(v)})
        return out
    if kind == "batch":
        sims, n = state["sims"], case["steps"]
        state["batch"].update([s.engine for s in sims], [s.next for s in sims], [n] * len(sims), [s.dt for s in sims],
                              [s.gap for s in sims])
        out = []
        for s in sims:
            s.next += n
            f = s.frame()
            out.append({k: f[k] for k in ("fluid_pos", "fluid_vel", "fluid_drho", "solid_pos", "solid_vel") if k in f})
        return out
    sim = state["sims"][0]
    if kind == "exchange":
        pos, vel, acc, drho = (t.numpy() for t in sim.fluid)
        sim.engine.update_io(sim.dt, sim.next, 1, sim.gap, fluid_in=(pos, vel, drho), fluid_out=(pos, vel, drho))
        sim.next += 1
        return {"fluid_pos": sim.fluid[0], "fluid_vel": sim.fluid[1].float(), "fluid_drho": sim.fluid[3].float()}
    n = case["periods"] * sim.gap if kind == "coupled" else case["steps"]
    if kind == "stages":
        for s in range(sim.next, sim.next + n):
            sim.engine.step(sim.dt, s, sim.gap)
    else:
        sim.engine.update(sim.dt, sim.next, n, sim.gap)
    sim.next += n
    return sim.frame()


def _scene_work(kind, n, height, steps, clumps=0):
    """Bytes of the state read and written once, and the operations of its pair terms: about 74 fluid partners in
    the kernel's support (radius 2.6 spacings), 40 operations in each continuity term (two passes) and 60 in a
    momentum term; 250 in a contact, about four contacts a grain."""
    if kind == "grains":
        grains = n + 4 * clumps
        return {"bytes": 2 * 96.0 * grains + 96.0 * grains, "flops": steps * grains * 4 * 250.0}
    bytes_, flops = 2 * 52.0 * n + 80.0 * n, steps * n * 74 * 140.0
    return {"bytes": bytes_, "flops": flops}


def work(case):
    kind = case["kind"]
    if kind in ("batch", "serve"):
        total = {"bytes": 0.0, "flops": 0.0}
        for k in range(case["scenes"]):
            n = int(case["smallest"] * (case["largest"] / case["smallest"]) ** ((k + 0.5) / case["scenes"]))
            grains = kind == "serve" and k % 3 == 1
            coupled = not grains and (k % 3 == 2 or (kind == "batch" and k % 5 == 1))
            steps = case["steps"] / 40.0 if coupled else case["steps"]
            w = _scene_work("grains" if grains else "sph", n, 0.3, steps)
            total = {q: total[q] + w[q] for q in total}
        return total
    if kind == "grains":
        return _scene_work("grains", case["n"], 0.0, case["steps"], case["clumps"])
    if kind == "coupled":
        w = _scene_work("sph", case["n"], case["height"], case["periods"])
        solids = max(1, round(64 * case["n"] / 1.0e6)) * 512
        gap = 28 * max(1.0, (1.0e6 / case["n"]) ** (1.0 / 3.0))
        return {"bytes": w["bytes"] + 288.0 * solids, "flops": w["flops"] + case["periods"] * gap * solids * 4 * 500.0}
    n = case["n"] * (1.8 if case.get("two") else 1.0)
    return _scene_work("sph", n, case["height"], case.get("steps", 1))


# ---------------------------------------------------------------- the same steps in 64 bits

def _dot(a, b):
    return (a * b).sum(-1)


def _pairs(xa, xb, cut):
    """Index pairs (a, b) with |xa - xb| <= cut (a number), from cells of that size."""
    low = torch.minimum(xa.min(0).values, xb.min(0).values) - 1.5 * cut
    ca, cb = ((xa - low) / cut).long(), ((xb - low) / cut).long()
    dims = torch.maximum(ca.max(0).values, cb.max(0).values) + 2
    key, order = ((cb[:, 2] * dims[1] + cb[:, 1]) * dims[0] + cb[:, 0]).sort()
    found_a, found_b = [], []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):  # the three cells of a row are one range of the sorted order
            row = ((ca[:, 2] + dz) * dims[1] + ca[:, 1] + dy) * dims[0] + ca[:, 0]
            first, last = torch.searchsorted(key, row - 1), torch.searchsorted(key, row + 2)
            count = last - first
            a = torch.repeat_interleave(torch.arange(len(xa), device=xa.device), count)
            at = torch.arange(len(a), device=xa.device) - torch.repeat_interleave(count.cumsum(0) - count, count)
            b = order[first[a] + at]
            near = _dot(xa[a] - xb[b], xa[a] - xb[b]) <= cut * cut
            found_a.append(a[near])
            found_b.append(b[near])
    return torch.cat(found_a), torch.cat(found_b)


class _Exact:
    """The coupled step's fluid with fixed wall particles, or spheres under Hertz-Mindlin contacts with sliding
    springs on a floor, in FP64."""

    def __init__(self, recipe):
        f64 = dict(dtype=torch.float64, device="cuda")
        self.g = torch.tensor([0.0, 0.0, -9.81], **f64)
        fluid, walls, spheres, self.floor = [], [], [], None
        for fn, a in recipe.calls:
            if fn == "addFluid":
                fluid.append(a)
            elif fn == "addDummyParticleWall":
                walls.append(a)
            elif fn == "addCluster":
                spheres.append(a)
            elif fn == "setHertzianContactModel":
                self.E, self.G, self.res, self.mu = a[2], a[3], a[4], a[7]
        if fluid:
            self.x = torch.tensor(np.concatenate([a[0] for a in fluid]), **f64)
            h, rho0, c, nu = (torch.cat([torch.full((len(a[0]),), a[k], **f64) for a in fluid]) for k in (2, 3, 4, 5))
            self.h, self.rho0, self.c, self.nu, self.m = h, rho0, c, nu, (h / 1.3) ** 3 * rho0
            self.v, self.a, self.dr = torch.zeros_like(self.x), torch.zeros_like(self.x), torch.zeros_like(h)
            self.wx = torch.tensor(np.concatenate([a[0] for a in walls]), **f64)
            self.wr = torch.cat([torch.full((len(a[0]),), a[1], **f64) for a in walls])
            self.wn = self.normals(float(h.max()))
        if spheres:
            (p, r, rho, v, _), = spheres
            self.p, self.r = torch.tensor(p, **f64), torch.tensor(r, **f64)
            self.mass = 4.0 / 3.0 * math.pi * self.r ** 3 * torch.tensor(rho, **f64)
            self.pv = torch.tensor(v, **f64).expand_as(self.p).clone()
            self.pa, self.pw, self.pt = (torch.zeros_like(self.p) for _ in range(3))
            self.keys, self.springs = torch.zeros(0, dtype=torch.long, device="cuda"), torch.zeros(0, 3, **f64)
            self.floor = torch.zeros_like(self.p)

    @staticmethod
    def grad(r, h):  # G of grad W = -G r
        return (5 * 21 / (16 * math.pi)) * (1 - 0.5 * r / h).clamp(min=0) ** 3 / h ** 5

    def normals(self, h):
        near = ((self.wx >= self.x.min(0).values - 8 * h) & (self.wx <= self.x.max(0).values + 8 * h)).all(1)
        at = near.nonzero()[:, 0]  # only walls that fluid can reach matter
        a, b = _pairs(self.wx[at], self.wx, 2 * h)
        d = self.wx[at][a] - self.wx[b]
        n = torch.zeros_like(self.wx)
        s = torch.zeros_like(self.wx[at]).index_add_(0, a, (h / 1.3) ** 3 * self.grad(d.norm(dim=1), h)[:, None] * d)
        size = s.norm(dim=1, keepdim=True)
        n[at] = torch.where(size > 1e-10, s / size.clamp(min=1e-300), torch.zeros_like(s))
        return n

    def lists(self):
        i, j = _pairs(self.x, self.x, 2 * float(self.h.max()))
        keep = (i != j) & ((self.x[i] - self.x[j]).norm(dim=1) <= 2 * torch.maximum(self.h[i], self.h[j]))
        self.i, self.j = i[keep], j[keep]
        k, a = _pairs(self.x, self.wx, 2 * float(self.h.max()))
        keep = (self.x[k] - self.wx[a]).norm(dim=1) <= 2 * self.h[k]
        self.k, self.w = k[keep], a[keep]

    def chunks(self, count, size=1 << 24):
        return [slice(s, min(count, s + size)) for s in range(0, count, size)]

    def shepard(self, step):
        s = (21 / (16 * math.pi)) / self.h ** 3

        def W(d, h):
            q = d / h
            return torch.where(q < 2, (21 / (16 * math.pi)) / h ** 3 * (1 - 0.5 * q) ** 4 * (1 + 2 * q), 0 * q)
        for c in self.chunks(len(self.i)):
            i, j = self.i[c], self.j[c]
            s.index_add_(0, i, W((self.x[i] - self.x[j]).norm(dim=1), self.h[i]))
        k, w = self.k, self.w
        s.index_add_(0, k, W((self.x[k] - self.wx[w]).norm(dim=1), self.h[k]) * (2.6 * self.wr[w] / self.h[k]) ** 3)
        if step == 1:
            self.s0 = s
        else:
            self.dr = torch.maximum(self.rho0 + self.dr, self.rho0 * s / self.s0) - self.rho0

    def wall_terms(self):
        k, w = self.k, self.w
        d = self.x[k] - self.wx[w]
        r = d.norm(dim=1)
        h = 0.5 * (self.h[k] + 2.6 * self.wr[w])
        rho, P = self.rho0 + self.dr, self.dr * self.c ** 2
        Pa = P[k] + rho[k] * _dot(self.g, self.wn[w]).clamp(min=0) * _dot(d, self.wn[w])
        return k, w, d, r, self.grad(r, h), rho[k], P[k], Pa, Pa / self.c[k] ** 2 + self.rho0[k], (2 * self.wr[w]) ** 3

    def continuity(self, dt):
        rho, P, out = self.rho0 + self.dr, self.dr * self.c ** 2, torch.zeros_like(self.dr)
        for c in self.chunks(len(self.i)):
            i, j = self.i[c], self.j[c]
            d = self.x[i] - self.x[j]
            r = d.norm(dim=1)
            G = self.grad(r, 0.5 * (self.h[i] + self.h[j]))
            out.index_add_(0, i, -2 * rho[i] * self.m[j] / rho[j] * G / (rho[i] + rho[j]) * (
                rho[j] * _dot(self.v[i] - self.v[j], d) + (P[i] - P[j]) * r / (0.5 * (self.c[i] + self.c[j]))))
        k, w, d, r, G, rk, Pk, Pa, ra, Va = self.wall_terms()
        out.index_add_(0, k, -2 * rk * Va * G / (rk + ra) * (2 * ra * _dot(self.v[k], d) + (Pk - Pa) * r / self.c[k]))
        self.dr = self.dr + dt * out

    def momentum(self):
        rho, P, V = self.rho0 + self.dr, self.dr * self.c ** 2, self.m / (self.rho0 + self.dr)
        gam, out = self.nu * rho, torch.zeros_like(self.x)
        for c in self.chunks(len(self.i)):
            i, j = self.i[c], self.j[c]
            d, vij = self.x[i] - self.x[j], self.v[i] - self.v[j]
            r = d.norm(dim=1)
            G = self.grad(r, 0.5 * (self.h[i] + self.h[j]))
            dU = -_dot(vij, d) / r
            beta = torch.minimum(3 * dU.clamp(min=0), 0.5 * (self.c[i] + self.c[j]))
            Ps = (rho[i] * P[j] + rho[j] * P[i] + rho[i] * rho[j] * beta * dU) / (rho[i] + rho[j])
            vis = 2 * gam[i] * gam[j] / (gam[i] + gam[j])
            out.index_add_(0, i, (2 * V[i] * V[j] * G / self.m[i])[:, None] * (Ps[:, None] * d - vis[:, None] * vij))
        k, w, d, r, G, rk, Pk, Pa, ra, Va = self.wall_terms()
        dU = -2 * _dot(self.v[k], self.wn[w])
        beta = torch.minimum(3 * dU.clamp(min=0), self.c[k])
        Ps = (rk * Pa + ra * Pk + rk * ra * beta * dU) / (rk + ra)
        out.index_add_(0, k, (2 * V[k] * Va * G / self.m[k])[:, None] * (Ps[:, None] * d - 2 * gam[k][:, None] * self.v[k]))
        self.a = out + self.g

    def fluid_step(self, dt, step):
        self.lists()
        if step == 1 or step % 5 == 0:
            self.shepard(step)
        self.continuity(0.5 * dt)
        self.x = self.x + 0.5 * dt * self.v
        self.momentum()
        self.v = self.v + dt * self.a
        self.x = self.x + 0.5 * dt * self.v
        self.continuity(0.5 * dt)

    def hertz(self, vc, n, delta, m, R, spring, dt):
        """Force, and the sliding spring after the step, of contacts with overlap delta > 0."""
        log = math.log(self.res)
        damp = 2 * math.sqrt(5 / 6) * -log / math.sqrt(log * log + math.pi ** 2)
        kn, ks = 4 / 3 * self.E * (R * delta).sqrt(), 8 * self.G * (R * delta).sqrt()
        cn, cs = damp * (m * kn).sqrt(), damp * (m * ks).sqrt()
        vn = _dot(vc, n)[:, None] * n
        Fn, vs = (kn * delta)[:, None] * n - cn[:, None] * vn, vc - vn
        flat = spring - _dot(spring, n)[:, None] * n
        size = flat.norm(dim=1)
        scale = torch.where(size > 1e-10, spring.norm(dim=1) / size.clamp(min=1e-300), torch.ones_like(size))
        s = flat * scale[:, None] + vs * dt
        F = -ks[:, None] * s - cs[:, None] * vs
        f, most = F.norm(dim=1), self.mu * Fn.norm(dim=1)
        slip = f > most
        F2 = F * (most / f.clamp(min=1e-300))[:, None]
        s = torch.where(slip[:, None], -(F2 + cs[:, None] * vs) / ks[:, None], s)
        return Fn - ks[:, None] * s - cs[:, None] * vs, s

    def grain_step(self, dt):
        n_all = len(self.p)
        a, b = _pairs(self.p, self.p, 2.2 * float(self.r.max()))
        keep = (a < b) & (1.1 * (self.r[a] + self.r[b]) >= (self.p[a] - self.p[b]).norm(dim=1))
        key, order = (a[keep] * n_all + b[keep]).sort()
        a, b = a[keep][order], b[keep][order]
        spring = torch.zeros(len(key), 3, dtype=torch.float64, device="cuda")
        if len(self.keys):  # springs of pairs that were in the last step's list
            at = torch.searchsorted(self.keys, key).clamp(max=len(self.keys) - 1)
            same = self.keys[at] == key
            spring[same] = self.springs[at[same]]
        inertia = (0.4 * self.r ** 2 * self.mass)[:, None]
        self.pv = self.pv + 0.5 * dt * self.pa
        self.pw = self.pw + 0.5 * dt * self.pt / inertia
        self.p = self.p + 0.5 * dt * self.pv
        d = self.p[a] - self.p[b]
        dist = d.norm(dim=1)
        n, delta = d / dist[:, None], self.r[a] + self.r[b] - dist
        live = delta > 0
        F_all = torch.zeros_like(spring)
        new = torch.zeros_like(spring)
        A, B, n, delta = a[live], b[live], n[live], delta[live]
        rc = self.p[B] + (self.r[B] - 0.5 * delta)[:, None] * n
        arm_a, arm_b = rc - self.p[A], rc - self.p[B]
        vc = (self.pv[A] + torch.linalg.cross(self.pw[A], arm_a)) - (self.pv[B] + torch.linalg.cross(self.pw[B], arm_b))
        m = 1 / (1 / self.mass[A] + 1 / self.mass[B])
        F, s = self.hertz(vc, n, delta, m, self.r[A] * self.r[B] / (self.r[A] + self.r[B]), spring[live], dt)
        new[live] = s
        self.keys, self.springs = key, new
        total, torque = torch.zeros_like(self.p), torch.zeros_like(self.p)
        total.index_add_(0, A, F).index_add_(0, B, -F)
        torque.index_add_(0, A, torch.linalg.cross(arm_a, F)).index_add_(0, B, -torch.linalg.cross(arm_b, F))
        up = torch.tensor([0.0, 0.0, 1.0], dtype=torch.float64, device="cuda")
        over = self.r - self.p[:, 2]
        self.floor[over <= 0] = 0
        t = (over > 0).nonzero()[:, 0]
        if len(t):
            n = up.expand(len(t), 3)
            arm = -(self.r[t] - over[t])[:, None] * n
            vc = self.pv[t] + torch.linalg.cross(self.pw[t], arm)
            F, self.floor[t] = self.hertz(vc, n, over[t], self.mass[t], self.r[t], self.floor[t], dt)
            total.index_add_(0, t, F)
            torque.index_add_(0, t, torch.linalg.cross(arm, F))
        self.pa, self.pt = total / self.mass[:, None] + self.g, torque
        self.p = self.p + 0.5 * dt * self.pv
        self.pv = self.pv + 0.5 * dt * self.pa
        self.pw = self.pw + 0.5 * dt * self.pt / inertia


def exact(case, seed):
    kind = case["kind"]
    # bonds, clumps and mixes of scenes have no short restatement
    if kind in ("coupled", "batch", "serve") or case.get("clumps"):
        return None
    if case["n"] * case.get("steps", 1) > 9_000_000:
        return None
    recipe = _recipes(case, seed)[0]
    e, dt = _Exact(recipe), recipe.meta["dt"]
    for step in range(1, case.get("steps", 1) + 1):
        if kind == "grains":
            e.grain_step(dt)
        else:
            e.fluid_step(dt, step)
    if kind == "grains":
        return {"solid_pos": e.p, "solid_vel": e.pv, "solid_acc": e.pa, "solid_angvel": e.pw}
    if kind == "exchange":
        return {"fluid_pos": e.x, "fluid_vel": e.v, "fluid_drho": e.dr}
    return {"fluid_pos": e.x, "fluid_vel": e.v, "fluid_acc": e.a, "fluid_drho": e.dr}
