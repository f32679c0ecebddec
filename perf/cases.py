"""Timed cases of the substep framework: the work a user's program has it do.

Every case is one pass of such a program's loop through the public entry
points (``mpm_cuda_b200.sim.Simulation``, ``mpm_cuda_b200.surrogate``):

* ``read = "positions"``: a rendering or viewing loop, ``step(substeps)`` and
  the positions copied to page-locked host memory (a batch of scenes reads all
  of them in one asynchronous copy);
* ``read = "state"``: a run that hands its whole particle state on (analysis,
  harvesting, reproducible studies), ``step(substeps)`` and ``get_state``;
* ``read = "restart"``: a checkpoint loaded, advanced and saved again.

A simulation goes on from pass to pass, as in use.  ``exact`` replays the
first pass in 64 bits with plain torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from mpm_cuda_b200 import _lib as L
from mpm_cuda_b200.sim import Group, MaterialParams, Scene, Simulation
from mpm_cuda_b200.surrogate import StressSurrogate

# materials of the repository's workloads
MATERIALS = {
    "jello": dict(type=0, E=5e4, nu=0.3, rho=1000.0),
    "jello2d": dict(type=0, E=1e3, nu=0.2, rho=1.0),
    "snow": dict(type=1, E=1.4e5, nu=0.2, rho=400.0, xi=10.0, theta_c=2.5e-2, theta_s=7.5e-3),
    "water": dict(type=2, E=0.0, nu=0.0, rho=1000.0, bulk_k=1e4, gamma=7.0),
}
WALL = 3  # cells


def _case(name, **kw):
    c = dict(name=name, dim=3, body="cube", material="jello", nx=128, ny=128, nz=128, size=0.3, substeps=50, dt=1e-4,
             ppc=8, speed=2.0, scenes=1, p2g="atomic", pool=0, adaptive=False, learned=False, read="positions")
    c.update(kw)
    return c


def listed():
    return [
        # the smallest call: a live view of the 2D jello scene (9,000 particles), every substep shown
        _case("view_jello2d", dim=2, material="jello2d", nx=128, ny=128, nz=1, size=0.2, ppc=14, speed=1.0, substeps=1),
        # a 2D dam break on a grid of odd sides, one rendered frame of 100 substeps
        _case("frame_water2d", dim=2, body="column", material="water", nx=251, ny=187, nz=1, size=0.45, ppc=4,
              speed=0.0, substeps=100, dt=5e-5),
        # the 128^3 jello scene (about 450k particles), a rendered frame
        _case("frame_jello128", substeps=100),
        # the 256^3 snow collision (1.9M particles in two groups)
        _case("frame_snow256", body="spheres", material="snow", nx=256, ny=256, nz=256, size=0.24, speed=3.0, dt=5e-5),
        # the 256^3 jello scene (2M particles)
        _case("frame_jello256", nx=256, ny=256, nz=256, size=0.245),
        # a 3D dam break in a tank of three different odd sides
        _case("frame_water_tank", body="column", material="water", nx=149, ny=122, nz=83, size=0.45, speed=0.0,
              substeps=60),
        # a batch of small and middling scenes of the three materials in one handle (parameter studies)
        _case("batch_mixed", body="mixed", scenes=16, nx=96, ny=96, nz=96, size=0.3, speed=1.0, substeps=25),
        # one small object in a wide domain: the grid is paged
        _case("paged_snow", body="sphere", material="snow", nx=320, ny=200, nz=320, size=0.18, speed=1.0, dt=2e-5,
              pool=60000, substeps=40),
        # dt chosen on the device
        _case("adaptive_snow", body="sphere", material="snow", nx=70, ny=70, nz=70, size=0.33, speed=3.0, dt=2e-4,
              adaptive=True, substeps=80),
        # a run that has to be repeatable bit by bit, its state kept after every 20 substeps
        _case("reproducible_jello", nx=101, ny=101, nz=101, size=0.31, p2g="deterministic", substeps=20, read="state"),
        # a checkpoint of jello and water in one grid, loaded, advanced and saved
        _case("checkpoint", body="two", nx=118, ny=118, nz=118, size=0.26, speed=1.0, substeps=8, read="restart"),
        # the learned stress on the 128^3 jello scene
        _case("learned_jello", learned=True, substeps=40),
    ]


def draw(rng):
    """One more case of the listed ones' ranges."""
    log = lambda lo, hi: math.exp(rng.uniform(math.log(lo), math.log(hi)))  # noqa: E731
    kind = rng.choice(["jello", "jello", "snow", "snow", "water", "jello2d", "water2d", "batch", "paged", "adaptive",
                       "deterministic", "restart"])
    substeps = int(log(1, 100))
    if kind in ("jello2d", "water2d"):
        n = int(log(64, 400))
        c = _case("", dim=2, nx=n, ny=int(n * rng.uniform(0.8, 1.2)), nz=1, size=rng.uniform(0.15, 0.5),
                  ppc=rng.choice([4, 4, 9, 14]), substeps=substeps)
        if kind == "jello2d":
            c.update(material="jello2d", speed=rng.uniform(0.0, 1.0), dt=1e-4 * min(1.0, 128.0 / n))
        else:
            c.update(material="water", body="column", speed=0.0, dt=1e-4 * min(1.0, 128.0 / n))
    elif kind == "batch":
        n = int(log(48, 128))
        c = _case("", body="mixed", scenes=rng.randint(2, 24), nx=n, ny=n, nz=n, size=rng.uniform(0.15, 0.3), speed=1.0,
                  substeps=min(substeps, 40))
    else:
        n = int(log(48, 256))
        side = [int(n * rng.uniform(0.85, 1.0)) if rng.random() < 0.5 else n for _ in range(2)]
        c = _case("", nx=n, ny=side[0], nz=side[1], size=rng.uniform(0.15, 0.3), speed=rng.uniform(0.5, 3.0),
                  ppc=rng.choice([6, 8, 8, 8]), dt=1e-4 * min(1.0, 128.0 / n), substeps=substeps)
        if kind in ("snow", "paged"):
            c.update(material="snow", body=rng.choice(["sphere", "spheres"]) if kind == "snow" else "sphere",
                     size=rng.uniform(0.15, 0.25), dt=2.5e-5 * min(1.0, 256.0 / n), speed=rng.uniform(0.2, 1.5))
        if kind == "paged":
            c.update(pool=60000)
        if kind == "water":
            c.update(material="water", body="column", size=rng.uniform(0.25, 0.45), speed=0.0)
        if kind == "adaptive":
            c.update(adaptive=True, dt=3e-4 * min(1.0, 128.0 / n))
        if kind == "deterministic":
            c.update(p2g="deterministic", read="state", nx=min(n, 128), ny=min(side[0], 128), nz=min(side[1], 128),
                     substeps=min(substeps, 30))
        if kind == "restart":
            c.update(body="two", read="restart", nx=min(n, 128), ny=min(n, 128), nz=min(n, 128), size=rng.uniform(0.15, 0.26),
                     substeps=min(substeps, 16))
    del c["name"]
    return c


# ------------------------------------------------------------------- inputs

def _fill(lo, hi, h, ppc, inside, rng):
    """ppc jittered samples in every cell that [lo, hi] touches and whose centre is inside."""
    axes = [np.arange(int(math.floor(a / h)), int(math.ceil(b / h))) for a, b in zip(lo, hi)]
    cells = np.stack(np.meshgrid(*axes, indexing="ij"), axis=-1).reshape(-1, len(lo))
    cells = np.repeat(cells[inside((cells + 0.5) * h)], ppc, axis=0)
    return ((cells + rng.random(cells.shape)) * h).astype(np.float32)


def _in_box(lo, hi):
    return lambda x: np.all((x >= lo) & (x < hi), axis=1)


def _in_ball(c, r):
    return lambda x: np.sum((x - c) ** 2, axis=1) < r * r


def _scene_groups(case, index, rng):
    """[(material name, positions, velocity)] of one scene and its grid (sides, h)."""
    d = case["dim"]
    n = [case["nx"], case["ny"], case["nz"]][:d]
    body, size, material = case["body"], case["size"], case["material"]
    if body == "mixed":  # scenes of a batch differ in side, size and material
        scale = [1.0, 0.72, 1.31, 0.86, 1.13][index % 5]
        n = [int(v * scale) for v in n]
        size = size * [1.0, 0.9, 0.75, 1.05][index % 4]
        material = ["jello", "snow", "water"][index % 3]
        body = ["cube", "sphere", "column"][index % 3]
    h = 1.0 / max(n)
    top = np.array(n) * h
    ppc = case["ppc"]
    down = [0.0, -case["speed"], 0.0][:d]
    c = top * np.array([0.5, 0.6, 0.5][:d])
    if body == "cube":
        lo, hi = c - size / 2, c + size / 2
        return n, h, [(material, _fill(lo, hi, h, ppc, _in_box(lo, hi), rng), down)]
    if body == "sphere":
        return n, h, [(material, _fill(c - size / 2, c + size / 2, h, ppc, _in_ball(c, size / 2), rng), down)]
    if body == "column":  # a dam break, standing in a corner of the walls
        lo = np.full(d, (WALL + 1) * h)
        hi = lo + np.array([0.5, 1.0, 0.5][:d]) * size
        hi = np.minimum(hi, top - (WALL + 1) * h)
        return n, h, [(material, _fill(lo, hi, h, ppc, _in_box(lo, hi), rng), down)]
    out = []
    r = size / 2
    for k, s in enumerate((0.3, 0.7)):
        c = top * np.array([s, 0.5 + 0.02 * k, 0.5][:d])
        if body == "spheres":  # two balls that fly at each other
            v = [case["speed"] * (1 - 2 * k), 0.0, 0.0][:d]
            out.append((material, _fill(c - r, c + r, h, ppc, _in_ball(c, r), rng), v))
        else:  # "two": a jello cube and a water ball in one grid
            inside = _in_box(c - r, c + r) if k == 0 else _in_ball(c, r)
            out.append(("jello" if k == 0 else "water", _fill(c - r, c + r, h, ppc, inside, rng), down))
    return n, h, out


def _in_motion(material, x, v, rng):
    """(velocities, deformation gradients) of a body that moves and is strained already: smooth fields over the body."""
    d = x.shape[1]
    a, b, e = (np.float32(s * rng.standard_normal((d, d))) for s in (0.1, 1.0, 0.005 if material == "snow" else 0.015))
    wave = np.sin(8.0 * x @ b).astype(np.float32)
    v = np.float32(v) + wave @ a
    F = np.float32(np.eye(d)) + (0.0 if material == "water" else wave[:, :1, None]) * e
    return np.float32(v), np.array(np.broadcast_to(F, (len(x), d, d)), dtype=np.float32)


def _all_scenes(case, seed):
    """Per scene (sides, h, [(material, x, v, F)])."""
    out = []
    for i in range(case["scenes"]):
        rng = np.random.default_rng([seed, i])
        n, h, groups = _scene_groups(case, i, rng)
        out.append((n, h, [(m, x, *_in_motion(m, x, v, rng)) for m, x, v in groups]))
    return out


def _wall_type(case):
    return L.BC_SEPARATE if case["material"] == "jello2d" else L.BC_SLIP


def _scenes(case, seed):
    out = []
    d = case["dim"]
    for n, h, groups in _all_scenes(case, seed):
        vol = h ** d / case["ppc"]
        gs = []
        for material, x, v, F in groups:
            m = MaterialParams(**MATERIALS[material])
            gs.append(Group(material=m, p_mass=m.rho * vol, p_vol=vol, x=x, v=v, F=F))
        out.append(Scene(dim=d, n=tuple(n), h=h, dt=case["dt"], groups=gs, gravity=(0.0, -9.8, 0.0)[:d],
                         bc_type=_wall_type(case), bc_lo=WALL, bc_hi=WALL, mass_eps=0.0 if d == 2 else 2.2e-16))
    return out


def _checkpoint(case, seed):
    """The scene's state as a checkpoint holds it."""
    _, _, groups = _all_scenes(case, seed)[0]
    rng = np.random.default_rng([seed, 77])
    x, v, F = (np.concatenate([g[k] for g in groups]) for k in (1, 2, 3))
    C = np.float32(rng.standard_normal((3, 3))) + 0.1 * F
    water = np.concatenate([np.full(len(g[1]), g[0] == "water") for g in groups])
    aux = np.where(water, 1.0 + 0.02 * (x[:, 0] - 0.5), 1.0).astype(np.float32)
    return x, v, C, F, aux


def prepare(case, seed):
    scenes = _scenes(case, seed)
    mode = L.P2G_DETERMINISTIC if case["p2g"] == "deterministic" else L.P2G_ATOMIC
    sim = Simulation(scenes, p2g_mode=mode, adaptive_dt=case["adaptive"], grid_pool_blocks=case["pool"])
    state = {"case": case, "sim": sim}
    if case["learned"]:
        # the network of a program that trained it on strained states of its own material
        rng = np.random.default_rng(seed)
        F = np.eye(3) + 0.03 * rng.standard_normal((20000, 3, 3))
        net = StressSurrogate(seed=seed % 65536)
        net.train(F.astype(np.float32), n_samples=1 << 18, epochs=4)
        sim.set_stress_mode(L.STRESS_SURROGATE, net)
        state["net"] = net
    if case["read"] == "positions":
        n = sim.num_particles(-1)
        state["out"] = torch.empty((n, case["dim"]), dtype=torch.float32, pin_memory=True).numpy()
    if case["read"] == "restart":
        state["saved"] = _checkpoint(case, seed)
    return state


def run(state):
    case, sim = state["case"], state["sim"]
    if case["read"] == "restart":
        x, v, C, F, aux = state["saved"]
        sim.set_state(0, x=x, v=v, C_=C, F=F, aux=aux)
        sim.step(case["substeps"])
        return sim.get_state(0)
    if case["scenes"] > 1:
        sim.step_async(case["substeps"])
        ticket = sim.positions_async(state["out"], scene=-1)
        sim.synchronize()
        sim.wait_positions(ticket)
        return state["out"]
    sim.step(case["substeps"])
    if case["read"] == "state":
        return sim.get_state(0)
    return sim.positions(0, out=state["out"])


# --------------------------------------------------------------------- work

def _count(case):
    """Per material [particles, touched nodes], estimated from the shapes (no inputs are made)."""
    out = {}
    d = case["dim"]
    ppc = case["ppc"]
    for i in range(case["scenes"]):
        n = [case["nx"], case["ny"], case["nz"]][:d]
        size, body, material = case["size"], case["body"], case["material"]
        if body == "mixed":
            scale = [1.0, 0.72, 1.31, 0.86, 1.13][i % 5]
            n = [int(v * scale) for v in n]
            size = size * [1.0, 0.9, 0.75, 1.05][i % 4]
            material, body = ["jello", "snow", "water"][i % 3], ["cube", "sphere", "column"][i % 3]
        s = size * max(n)  # in cells
        ball = math.pi * s ** 3 / 6 if d == 3 else math.pi * s * s / 4
        cells = {"cube": s ** d, "sphere": ball, "column": s ** d * (0.25 if d == 3 else 0.5), "spheres": 2 * ball,
                 "two": s ** d + ball}[body]
        if body == "two":
            parts = [("jello", s ** d), ("water", ball)]
        else:
            parts = [(material, cells)]
        for m, k in parts:
            e = out.setdefault(m, [0.0, 0.0])
            e[0] += ppc * k
            e[1] += (k ** (1.0 / d) + 2) ** d
    return out


def work(case):
    """Per substep each particle's position, F (or J) read and written, each touched node's momentum written and its
    velocity read; the sums over the stencil in their separable form."""
    d = case["dim"]
    nbytes = flops = 0.0
    total = 0.0
    for m, (n, nodes) in _count(case).items():
        floats = d + {"jello": d * d, "jello2d": d * d, "snow": d * d + 1, "water": 1}[m]
        nbytes += n * 8 * floats + nodes * 32
        flops += n * (2000 if d == 3 else 500)
        total += n
    nbytes, flops = nbytes * case["substeps"], flops * case["substeps"]
    values = d if case["read"] == "positions" else 2 * d + 2 * d * d + 1
    nbytes += total * 4 * values * (2 if case["read"] == "restart" else 1)
    return {"bytes": nbytes, "flops": flops}


# -------------------------------------------------------------------- exact

def _mm(A, B):
    return (A.unsqueeze(-1) * B.unsqueeze(-3)).sum(-2)


def _det(F):
    if F.shape[-1] == 2:
        return F[:, 0, 0] * F[:, 1, 1] - F[:, 0, 1] * F[:, 1, 0]
    return (F[:, 0] * torch.linalg.cross(F[:, 1], F[:, 2])).sum(-1)


def _polar(F):
    """The rotation of F = R S."""
    if F.shape[-1] == 2:
        a, b = F[:, 0, 0] + F[:, 1, 1], F[:, 1, 0] - F[:, 0, 1]
        r = torch.sqrt(a * a + b * b)
        return torch.stack([a / r, -b / r, b / r, a / r], -1).reshape(-1, 2, 2)
    R = F
    for _ in range(12):  # Newton: R <- (R + R^-T) / 2
        cof = torch.stack([torch.linalg.cross(R[:, 1], R[:, 2]), torch.linalg.cross(R[:, 2], R[:, 0]),
                           torch.linalg.cross(R[:, 0], R[:, 1])], 1)
        new = 0.5 * (R + cof / (R[:, 0] * cof[:, 0]).sum(-1)[:, None, None])
        far = float((new - R).abs().max()) if len(R) else 0.0
        R = new
        if far < 1e-14:
            break
    return R


def _svd(F):
    """U, s, V of F = U diag(s) V^T with det F > 0, by Jacobi rotations of F^T F."""
    d = F.shape[-1]
    V = torch.eye(d, dtype=F.dtype, device=F.device).repeat(len(F), 1, 1)
    B = F.clone()  # F V
    for _ in range(8):
        worst = 0.0
        for p in range(d):
            for q in range(p + 1, d):
                a, b, c = (B[:, :, p] ** 2).sum(-1), (B[:, :, q] ** 2).sum(-1), (B[:, :, p] * B[:, :, q]).sum(-1)
                worst = max(worst, float((c.abs() / torch.sqrt(a * b)).max()) if len(F) else 0.0)
                th = 0.5 * torch.atan2(2 * c, a - b)
                cs, sn = torch.cos(th)[:, None], torch.sin(th)[:, None]
                for M in (B, V):
                    x, y = M[:, :, p].clone(), M[:, :, q].clone()
                    M[:, :, p] = cs * x + sn * y
                    M[:, :, q] = cs * y - sn * x
        if worst < 1e-15:
            break
    s = torch.sqrt((B ** 2).sum(1))
    return B / s[:, None, :], s, V


class _Exact:
    """One scene in 64 bits: dense grid, one pass over the stencil's offsets after the other."""

    def __init__(self, case, n, h, groups, dev):
        f = dict(dtype=torch.float64, device=dev)
        self.case, self.n, self.h, self.d, self.dev = case, n, h, case["dim"], dev
        self.dt = self.dt_next = self.dt_max = case["dt"]
        d = self.d
        self.vol = h ** d / case["ppc"]
        self.x = torch.cat([torch.as_tensor(g[1]).to(**f) for g in groups])
        self.v = torch.cat([torch.as_tensor(g[2]).to(**f) for g in groups])
        N = len(self.x)
        self.C = torch.zeros((N, d, d), **f)
        self.F = torch.cat([torch.as_tensor(g[3]).to(**f) for g in groups])
        self.aux = torch.ones(N, **f)
        self.parts, at, self.m = [], 0, torch.empty(N, **f)
        for material, x, _, _ in groups:
            p = dict(xi=10.0, theta_c=0.0, theta_s=0.0, bulk_k=0.0, gamma=7.0)
            p.update(MATERIALS[material])
            p["mu"] = p["E"] / (2 * (1 + p["nu"]))
            p["la"] = p["E"] * p["nu"] / ((1 + p["nu"]) * (1 - 2 * p["nu"]))
            p["wave"] = math.sqrt((p["bulk_k"] * p["gamma"] if p["type"] == 2 else p["la"] + 2 * p["mu"]) / p["rho"])
            self.parts.append((slice(at, at + len(x)), p))
            self.m[at:at + len(x)] = p["rho"] * self.vol
            at += len(x)
        if case["adaptive"]:
            fastest = max(p["wave"] + float(self.v[s].norm(dim=-1).max()) for s, p in self.parts)
            self.dt = self.dt_next = max(1e-4 * self.dt_max, min(self.dt_max, 0.5 * h / fastest))

    def stress(self):
        eye = torch.eye(self.d, dtype=torch.float64, device=self.dev)
        tau = torch.empty_like(self.F)
        for s, p in self.parts:
            F, aux = self.F[s], self.aux[s]
            if p["type"] == 2:
                tau[s] = (-p["bulk_k"] * (aux ** -p["gamma"] - 1) * aux)[:, None, None] * eye
                continue
            k = torch.exp(p["xi"] * (1 - aux))[:, None, None] if p["type"] == 1 else 1.0
            J = _det(F)[:, None, None]
            tau[s] = k * (2 * p["mu"] * _mm(F - _polar(F), F.transpose(1, 2)) + p["la"] * J * (J - 1) * eye)
        return tau

    def weights(self):
        g = self.x / self.h
        base = torch.floor(g - 0.5).long()
        f = g - base
        w = torch.stack([0.5 * (1.5 - f) ** 2, 0.75 - (f - 1) ** 2, 0.5 * (f - 0.5) ** 2])
        dw = torch.stack([f - 1.5, -2 * (f - 1), f - 0.5]) / self.h
        return base, f, w, dw

    def offsets(self, base, w, dw):
        d, stride = self.d, [1, self.n[0], self.n[0] * self.n[1]]
        for k in range(3 ** d):
            o = [k // 3 ** a % 3 for a in range(d)]
            at = sum((base[:, a] + o[a]) * stride[a] for a in range(d))
            wt = math.prod(w[o[a], :, a] for a in range(d))
            gw = torch.stack([math.prod((dw if a == b else w)[o[a], :, a] for a in range(d)) for b in range(d)], -1)
            yield torch.tensor(o, dtype=torch.float64, device=self.dev), at, wt, gw

    def step(self):
        d, h, case = self.d, self.h, self.case
        base, f, w, dw = self.weights()
        grid = torch.zeros((math.prod(self.n), d + 1), dtype=torch.float64, device=self.dev)
        A = -self.dt * self.vol * self.stress()
        mv = self.m[:, None] * self.v
        for o, at, wt, gw in self.offsets(base, w, dw):
            mom = mv + self.m[:, None] * (self.C * (h * (o - f))[:, None, :]).sum(-1)
            q = torch.cat([wt[:, None] * mom + (A * gw[:, None, :]).sum(-1), (wt * self.m)[:, None]], 1)
            grid.index_add_(0, at, q)
        m = grid[:, d]
        ok = m > (0.0 if d == 2 else 2.2e-16)
        vel = torch.where(ok[:, None], grid[:, :d] / torch.where(ok, m, torch.ones_like(m))[:, None], 0.0)
        vel[:, 1] -= self.dt * 9.8
        vel = torch.where(ok[:, None], vel, 0.0).reshape(*self.n[::-1], d)
        for a in range(d):
            lo, hi = vel.narrow(d - 1 - a, 0, WALL)[..., a], vel.narrow(d - 1 - a, self.n[a] - WALL, WALL)[..., a]
            if _wall_type(case) == L.BC_SLIP:
                lo.zero_()
                hi.zero_()
            else:
                lo.clamp_(min=0.0)
                hi.clamp_(max=0.0)
        vel = vel.reshape(-1, d)
        v, B, G = torch.zeros_like(self.v), torch.zeros_like(self.C), torch.zeros_like(self.C)
        for o, at, wt, gw in self.offsets(base, w, dw):
            vi = vel[at]
            v += wt[:, None] * vi
            B += (wt[:, None] * vi)[:, :, None] * (o - f)[:, None, :]
            G += vi[:, :, None] * gw[:, None, :]
        self.v, self.C = v, 4 / h * B
        fastest = 0.0
        for s, p in self.parts:
            if p["type"] == 2:
                self.aux[s] *= 1 + self.dt * G[s].diagonal(dim1=1, dim2=2).sum(-1)
            else:
                F = self.F[s] + self.dt * _mm(G[s], self.F[s])
                if p["type"] == 1:
                    U, sv, V = _svd(F)
                    sc = sv.clamp(1 - p["theta_c"], 1 + p["theta_s"])
                    F = _mm(U * sc[:, None, :], V.transpose(1, 2))
                    self.aux[s] *= sv.prod(-1) / sc.prod(-1)
                self.F[s] = F
            if case["adaptive"]:
                k = torch.exp(0.5 * p["xi"] * (1 - self.aux[s])) if p["type"] == 1 else 1.0
                fastest = max(fastest, float((v[s].norm(dim=-1) + p["wave"] * k).max()))
        self.x = self.x + self.dt * v
        if case["adaptive"]:
            self.dt, self.dt_next = self.dt_next, max(1e-4 * self.dt_max, min(self.dt_max, 0.5 * h / fastest))


def exact(case, seed):
    """The first pass in 64 bits (the learned stress stands for the exact one: its network is an approximation of it)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    sims = [_Exact(case, n, h, groups, dev) for n, h, groups in _all_scenes(case, seed)]
    if case["read"] == "restart":
        f = dict(dtype=torch.float64, device=dev)
        s = sims[0]
        s.x, s.v, s.C, s.F, s.aux = (torch.as_tensor(a).to(**f) for a in _checkpoint(case, seed))
    for s in sims:
        for _ in range(case["substeps"]):
            s.step()
    if case["read"] == "positions":
        return torch.cat([s.x for s in sims])
    s = sims[0]
    return {"x": s.x, "v": s.v, "C": s.C, "F": s.F, "aux": s.aux}
