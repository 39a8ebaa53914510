"""The work a user has this solver do, as measurable cases.

A pass advances a dam break by a few time steps through the public Python interface and reads
the state back into pinned host arrays, as a program does that watches or writes a run. The
scenes are a fluid column on a jittered lattice in an open tank; the seed draws the jitter and
the initial velocities.

``exact`` restates the time step in plain torch in 64 bits over pair lists: viscosity and
gravity, kick and drift, collisions, number density and equation of state, pressure gradient,
with the walls' mirror particles made twice per step. Its gradients come from torch.autograd.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from mps_cuda_b200 import F32, F64, F32_N64, MPS, MPSBatch, SceneDesc, dambreak_params
from mps_cuda_b200 import _lib as L
from mps_cuda_b200 import adjoint
from mps_cuda_b200.configs import batched_scenes

PRECISION = {"f32": F32, "f64": F64, "f32_n64": F32_N64}
FLUID, WALL, OBJECT = 0, 1, 2
SND, NU, G_Z, RHO = 20.0, 1e-6, -9.81, 1000.0
COL_RAT, DST_LMT_RAT = 0.2, 0.9
FIELDS = ("typ", "pos", "vel", "prs", "pav")


def _scene_case(name, l0, block, tank, dt, **more):
    case = {"kind": "scene", "l0": l0, "bx": block[0], "by": block[1], "bz": block[2],
            "tx": tank[0], "ty": tank[1], "tz": tank[2], "dt": dt, "precision": "f32",
            "steps": 10, "graph": False, "tune": False, "corrected": False, "plate": False,
            "upload": False, "methods": False, "vel_sigma": 0.0}
    case.update(more)
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # the smallest call: one step of a few hundred particles, then its result (a scene
        # under test, an interactive program); launches and latency
        _scene_case("scene_480_f32", 0.02, (8, 6, 10), (20, 10, 20), 2e-4, steps=1),
        # the small dam break in double precision, as one follows it for a thousand steps
        _scene_case("scene_6k_f64", 0.02, (20, 10, 30), (50, 10, 40), 2e-4, precision="f64",
                    graph=True),
        # an ordinary scene, no option touched
        _scene_case("scene_48k_f32", 0.01, (40, 20, 60), (100, 20, 80), 1e-4),
        # the standard dam break in both precisions, set up for a long run: captured step,
        # shapes tuned on the handle
        _scene_case("scene_384k_f32", 0.005, (80, 40, 120), (320, 40, 160), 5e-5, graph=True,
                    tune=True),
        _scene_case("scene_384k_f64", 0.005, (80, 40, 120), (320, 40, 160), 5e-5, graph=True,
                    tune=True, precision="f64", steps=5),
        # the largest scene, a state far larger than L2
        _scene_case("scene_6144k_f32", 0.0025, (160, 160, 240), (640, 160, 320), 2.5e-5,
                    graph=True, tune=True, steps=5),
        # the step called from a program that keeps the state on the host: up, one step, down
        _scene_case("host_state_384k_f32", 0.005, (80, 40, 120), (320, 40, 160), 5e-5, steps=1,
                    upload=True),
        # the reference's sequence of method calls, each on its own
        _scene_case("methods_48k_f32", 0.01, (40, 20, 60), (100, 20, 80), 1e-4, steps=1,
                    methods=True),
        # the corrected-matrix gradient on an odd-sized block that leaves a gap in the tank
        _scene_case("corrected_41k_f32", 0.0105, (39, 23, 47), (101, 31, 59), 9e-5, steps=5,
                    corrected=True),
        # a plate pushed through the fluid: walls that move and are bucketed every step
        _scene_case("plate_48k_f32", 0.01, (40, 20, 60), (100, 20, 80), 1e-4, steps=5,
                    plate=True, graph=True),
        # many independent scenes of uneven sizes advanced together
        {"name": "batch_64_f32_n64", "kind": "batch", "scenes": 64, "shapes": 2, "steps": 5,
         "graph": True, "precision": "f32_n64"},
        # a differentiated rollout: forward and backward
        dict(_scene_case("adjoint_48k_f64", 0.01, (40, 20, 60), (100, 20, 80), 1e-4,
                         precision="f64", steps=20, vel_sigma=0.05), kind="adjoint"),
    ]


def draw(rng):
    kind = rng.choice(["step"] * 7 + ["upload", "methods", "batch", "adjoint", "adjoint"])
    if kind == "batch":
        return {"kind": "batch", "scenes": rng.randint(3, 64), "shapes": rng.randrange(1 << 20),
                "steps": rng.choice([1, 2, 5]), "graph": rng.random() < 0.5,
                "precision": rng.choice(["f32", "f32_n64", "f64"])}
    precision = rng.choice(["f32", "f32", "f64", "f32_n64"])
    most = {"step": 3.0e6, "upload": 1.0e6, "methods": 4.0e5, "adjoint": 5.0e4}[kind]
    if precision == "f64" or kind == "adjoint":
        most = min(most, 4.0e5)
    n = math.exp(rng.uniform(math.log(400.0), math.log(most)))
    a, b = rng.uniform(0.5, 1.6), rng.uniform(0.5, 1.6)  # the column's width and depth to height
    bz = max(4, round((n / (a * b)) ** (1 / 3)))
    bx, by = max(3, round(a * bz)), max(3, round(b * bz))
    l0 = round(rng.uniform(0.2, 0.6) / bz, 5)
    umax = math.sqrt(2 * abs(G_Z) * (bz - 1) * l0)
    tank = (max(bx + 2, round(bx * rng.uniform(1.2, 4.0))),
            by if rng.random() < 0.6 else by + rng.randint(1, by), bz + rng.randint(2, 3 + bz // 2))
    steps = rng.choice([1, 2, 5, 10])
    case = _scene_case(None, l0, (bx, by, bz), tank, round(0.2 * l0 / (umax + SND), 9),
                       precision=precision, steps=steps, graph=rng.random() < 0.5,
                       vel_sigma=rng.choice([0.0, 0.05]))
    if kind == "step":
        case["corrected"] = rng.random() < 0.2
        case["plate"] = rng.random() < 0.2
    elif kind == "upload":
        case.update(upload=True, steps=1)
    elif kind == "methods":
        case.update(methods=True, graph=False, steps=min(steps, 2))
    else:
        case.update(kind="adjoint", precision="f64", steps=rng.randint(3, 20), vel_sigma=0.05)
    return case


# ---- scenes ---------------------------------------------------------------------------------
def _scene(l0, block, tank, rng, vel_sigma=0.0, plate=False):
    """typ (n,), pos, vel, nrm (3, n) in float64: the fluid block (x fastest), the walls of
    five faces (open top) with inward normals, and with `plate` a vertical OBJ plate that
    faces the fluid."""
    bx, by, bz = block
    cells = [int(round(t / l0)) for t in tank]
    k, j, i = np.meshgrid(np.arange(bz), np.arange(by), np.arange(bx), indexing="ij")
    pos = np.stack([i.ravel(), j.ravel(), k.ravel()]).astype(np.float64)
    pos += 0.5
    pos += rng.uniform(-0.01, 0.01, pos.shape)
    pos *= l0
    parts, normals, types = [pos], [np.zeros_like(pos)], [np.full(pos.shape[1], FLUID, np.int8)]

    def sheet(axis, at, sign, n1, n2, kind):
        q, p = np.meshgrid(np.arange(n2), np.arange(n1), indexing="ij")
        w, nv = np.zeros((3, p.size)), np.zeros((3, p.size))
        a1, a2 = [d for d in range(3) if d != axis]
        w[axis], w[a1], w[a2] = at, (p.ravel() + 0.5) * l0, (q.ravel() + 0.5) * l0
        nv[axis] = sign
        parts.append(w)
        normals.append(nv)
        types.append(np.full(p.size, kind, np.int8))

    for face in range(5):
        axis = face // 2
        n1, n2 = [cells[d] for d in range(3) if d != axis]
        sheet(axis, tank[axis] if face % 2 else 0.0, -1.0 if face % 2 else 1.0, n1, n2, WALL)
    if plate:
        sheet(0, (bx + 0.6) * l0, -1.0, cells[1], min(cells[2], bz + 2), OBJECT)
    pos, nrm, typ = np.concatenate(parts, 1), np.concatenate(normals, 1), np.concatenate(types)
    vel = np.zeros_like(pos)
    if vel_sigma:
        nf = bx * by * bz
        vel[:, :nf] = vel_sigma * rng.standard_normal((3, nf))
    return typ, pos, vel, nrm


def _of_case(case, seed):
    """(l0, block, tank, dt, scene) of every scene of a case."""
    if case["kind"] == "batch":
        out = []
        for k, (d, dt) in enumerate(batched_scenes(case["scenes"], seed=case["shapes"])):
            rng = np.random.default_rng([seed, k])
            out.append((d.l0, d.block, d.tank, dt, _scene(d.l0, d.block, d.tank, rng)))
        return out
    l0, block = case["l0"], (case["bx"], case["by"], case["bz"])
    tank = tuple(case[t] * l0 for t in ("tx", "ty", "tz"))
    sc = _scene(l0, block, tank, np.random.default_rng(seed), case["vel_sigma"], case["plate"])
    return [(l0, block, tank, case["dt"], sc)]


def _params(l0, block, tank, dt, precision):
    return dambreak_params(SceneDesc(l0, tank, block), snd=SND, dt=dt, nu=NU, g_z=G_Z,
                           precision=precision)


def _pinned(n, real):
    one = {"typ": ((n,), np.int8), "pos": ((3, n), real), "vel": ((3, n), real),
           "prs": ((n,), real), "pav": ((n,), real)}
    kinds = {np.int8: torch.int8, np.float32: torch.float32, np.float64: torch.float64}
    return {k: torch.empty(s, dtype=kinds[d], pin_memory=True).numpy() for k, (s, d) in one.items()}


# ---- passes ---------------------------------------------------------------------------------
def prepare(case, seed):
    scenes = _of_case(case, seed)
    precision = PRECISION[case["precision"]]
    if case["kind"] == "adjoint":
        l0, block, tank, dt, (typ, pos, vel, nrm) = scenes[0]
        problem = adjoint.RolloutProblem(SceneDesc(l0, tank, block), dt, case["steps"],
                                         precision=precision)
        problem.typ, problem.pos, problem.vel, problem.nrm = typ, pos, vel, nrm
        problem.fluid = np.nonzero(typ == FLUID)[0]
        return {"case": case, "problem": problem, "vel0": vel[:, problem.fluid].copy(),
                "target": _target(pos[:, problem.fluid])}
    real = np.float64 if precision == F64 else np.float32
    params = [_params(*s[:4], precision) for s in scenes]
    typ = np.concatenate([s[4][0] for s in scenes])
    pos, vel, nrm = (np.concatenate([s[4][k] for s in scenes], 1).astype(real) for k in (1, 2, 3))
    if case["kind"] == "batch":
        h = MPSBatch(params, typ, pos, vel, nrm, counts=[s[4][0].size for s in scenes])
    else:
        h = MPS(params[0], typ, pos, vel, nrm)
        if case["plate"]:
            l0 = case["l0"]
            h.set_wall_motion(OBJECT, center=((case["bx"] + 0.6) * l0, 0.5 * case["ty"] * l0, 0.0),
                              axis=(0.0, 0.0, 1.0), omega=0.05, velocity=(-0.02, 0.0, 0.0))
        if case["corrected"]:
            h.set_option(L.OPT_GRADIENT, L.GRAD_CORRECTED)
        if case["tune"]:
            h.autotune(3)
    if case["graph"]:
        h.set_option(L.OPT_GRAPH, 1)
    state = {"case": case, "h": h, "out": _pinned(typ.size, real)}
    if case.get("upload"):
        up = _pinned(typ.size, real)
        up["typ"][:], up["pos"][:], up["vel"][:], up["prs"][:], up["pav"][:] = typ, pos, vel, 0, 0
        state["up"] = up
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "adjoint":
        nu = torch.tensor(NU, dtype=torch.float64, requires_grad=True)
        vel0 = torch.from_numpy(state["vel0"]).requires_grad_(True)
        pos, vel, alive = adjoint.rollout(nu, vel0, state["problem"])
        loss = adjoint.dambreak_loss(pos, alive, state["target"])
        loss.backward()
        return {"loss": loss.detach(), "pos": pos.detach(), "vel": vel.detach(), "alive": alive,
                "grad_nu": nu.grad, "grad_vel0": vel0.grad}
    h = state["h"]
    if case.get("upload"):
        up = state["up"]
        h.set_state(typ=up["typ"], pos=up["pos"], vel=up["vel"], pav=up["pav"])
    if case.get("methods"):
        for _ in range(case["steps"]):
            h.step_by_methods()
    else:
        h.step(case["steps"])
    return h.state(state["out"])


def work(case):
    """Every step reads each fluid particle's type, position, velocity and mean pressure and
    writes them and the pressure; the walls' places and normals are read once a step. 122 and
    32 lattice neighbours lie inside the two radii; a viscosity pair costs about 20 operations,
    a collision, density and gradient pair 40, a backward step about twice its forward one."""
    s = 8 if case["precision"] == "f64" else 4
    if case["kind"] == "batch":
        fluid = wall = 0
        for d, _ in batched_scenes(case["scenes"], seed=case["shapes"]):
            c = [int(round(t / d.l0)) for t in d.tank]
            fluid += d.block[0] * d.block[1] * d.block[2]
            wall += 2 * c[1] * c[2] + 2 * c[0] * c[2] + c[0] * c[1]
    else:
        c = [case["tx"], case["ty"], case["tz"]]
        fluid = case["bx"] * case["by"] * case["bz"]
        wall = 2 * c[1] * c[2] + 2 * c[0] * c[2] + c[0] * c[1]
    moved = case["steps"] * (fluid * ((7 + 8) * s + 2) + wall * 6 * s)
    flops = case["steps"] * fluid * (122 * 20 + 32 * 40)
    if case["kind"] == "adjoint":
        moved, flops = 3 * moved, 3 * flops
    return {"bytes": moved, "flops": flops}


# ---- the step in 64 bits --------------------------------------------------------------------
def _pairs(a, b, r):
    """(i, j) of every pair |a_i - b_j| <= r; a, b are (n, 3)."""
    with torch.no_grad():
        lo = torch.minimum(a.min(0).values, b.min(0).values) - 2 * r
        size = ((torch.maximum(a.max(0).values, b.max(0).values) - lo) / r).long() + 3
        num = lambda p: (lambda c: (c[:, 2] * size[1] + c[:, 1]) * size[0] + c[:, 0])(((p - lo) / (r * (1 + 1e-9))).long())
        ka = num(a)
        kb, order = num(b).sort()
        out_i, out_j = [], []
        for dz in (-1, 0, 1):
            for dy in (-1, 0, 1):
                mid = ka + (dz * size[1] + dy) * size[0]
                first = torch.searchsorted(kb, mid - 1)
                count = torch.searchsorted(kb, mid + 1, right=True) - first
                i = torch.repeat_interleave(torch.arange(a.shape[0], device=a.device), count)
                at = torch.arange(i.shape[0], device=a.device) - (count.cumsum(0) - count)[i]
                j = order[first[i] + at]
                keep = ((a[i] - b[j]) ** 2).sum(1) <= r * r
                out_i.append(i[keep])
                out_j.append(j[keep])
        return torch.cat(out_i), torch.cat(out_j)


def _lowest(index, value, n, big):
    return torch.full((n,), big, dtype=value.dtype, device=value.device).scatter_reduce(
        0, index, value, "amin")


class _Exact:
    def __init__(self, l0, block, tank, dt, scene, device):
        typ, pos, _, nrm = scene
        dev = lambda v: torch.as_tensor(np.ascontiguousarray(v), device=device)
        self.l0, self.dt = l0, dt
        self.r, self.rp, self.rlim = 3.1 * l0, 2.1 * l0, DST_LMT_RAT * l0
        height = (block[2] - 1) * l0
        self.umax, self.pmax = math.sqrt(2 * abs(G_Z) * height), RHO * abs(G_Z) * height
        self.wpos, self.wnrm = dev(pos[:, typ != FLUID].T), dev(nrm[:, typ != FLUID].T)
        g = np.arange(-10, 10) * l0
        d2 = (g[:, None, None] ** 2 + g[:, None] ** 2 + g ** 2).ravel()
        d = np.sqrt(d2[d2 > 0])
        self.n0 = (self.r / d + d / self.r - 2)[d < self.r].sum()
        self.n0g = (self.rp / d - d / self.rp)[d < self.rp].sum()
        # the walls' order of visit (bucket, then id), the planes they form, and their edges
        size = [int((t + 6.2 * l0) / self.r) + 3 for t in tank]
        c = ((self.wpos + self.r) / self.r).long() + 1
        nw = self.wpos.shape[0]
        order = ((c[:, 2] * size[1] + c[:, 1]) * size[0] + c[:, 0]).argsort(stable=True)
        self.by_rank, self.rank = order, torch.empty_like(order)
        self.rank[order] = torch.arange(nw, device=device)
        self.normals, self.plane = self.wnrm.unique(dim=0, return_inverse=True)
        i, j = _pairs(self.wpos, self.wpos, l0 * (1 - 1e-6))
        self.edge = torch.zeros(nw, dtype=torch.bool, device=device)
        self.edge[i[self.plane[i] != self.plane[j]]] = True

    def mirrors(self, x):
        """(owner, slot, position) of the mirror particles of fluid at x."""
        n, big, k = x.shape[0], self.wpos.shape[0], self.normals.shape[0]
        i, j = _pairs(x, self.wpos, self.r)
        first = _lowest(i * k + self.plane[j], self.rank[j], n * k, big).view(n, k)
        e = self.edge[j]
        ie, je = i[e], j[e]
        efirst = _lowest(ie * k + self.plane[je], self.rank[je], n * k, big).view(n, k)
        owner, p = (first < big).nonzero(as_tuple=True)
        slot = owner * 10 + (first[owner] < first[owner, p][:, None]).sum(1)
        parts = [(owner, slot, self.by_rank[first[owner, p]], self.normals[p])]
        # corner mirrors: through the nearest Edge wall of the last plane met where there are
        # two, through the first one met where there are more
        ne = (efirst < big).sum(1)
        last = torch.where(efirst < big, efirst, -1).argmax(1)
        sel = self.plane[je] == last[ie]
        i2, j2 = ie[sel], je[sel]
        d2 = ((x.detach()[i2] - self.wpos[j2]) ** 2).sum(1)
        best = _lowest(i2, d2, n, math.inf)
        near = d2 == best[i2]
        nearest = _lowest(i2[near], self.rank[j2[near]], n, big)
        owner = (ne >= 2).nonzero()[:, 0]
        s = ((efirst[owner] < big).double() @ self.normals)
        s = s / s.norm(dim=1, keepdim=True)
        through = torch.where(ne[owner] == 2, nearest[owner], efirst[owner, last[owner]])
        parts.append((owner, owner * 10 + (first[owner] < big).sum(1), self.by_rank[through], s))
        owner, slot, wall, nv = (torch.cat(v) for v in zip(*parts))
        off = ((x[owner] - self.wpos[wall]) * nv).sum(1)
        pos = x[owner] - 2 * off[:, None] * nv
        # those that their nearest wall has on its own side are dropped
        keep = off.detach() >= 0
        i, j = _pairs(pos.detach(), self.wpos, self.r)
        d2 = ((pos.detach()[i] - self.wpos[j]) ** 2).sum(1)
        near = d2 == _lowest(i, d2, pos.shape[0], math.inf)[i]
        wall = _lowest(i[near], self.rank[j[near]], pos.shape[0], big)
        w = self.by_rank[wall.clamp(max=big - 1)]
        inside = ((pos.detach() - self.wpos[w]) * self.wnrm[w]).sum(1) >= 0
        keep &= ~((wall < big) & inside)
        return owner[keep], slot[keep], pos[keep]

    def clamp(self, v):
        speed = v.norm(dim=1, keepdim=True)
        return torch.where(speed > self.umax, v * (self.umax / speed.clamp(min=1e-300)), v)

    def step(self, x, v, nu):
        n, dt = x.shape[0], self.dt
        add = lambda i, val: torch.zeros((n,) + val.shape[1:], dtype=x.dtype, device=x.device).index_add(0, i, val)
        # viscosity and gravity, kick and drift
        owner, _, m1 = self.mirrors(x)
        acc = 0.0
        for y, u in ((x, v), (m1, torch.zeros_like(m1))):
            i, j = _pairs(x, y, self.r)
            if y is x:
                i, j = i[i != j], j[i != j]
            d = ((y[j] - x[i]) ** 2).sum(1).sqrt()
            acc = acc + add(i, (u[j] - v[i]) * (2 * self.l0 / d ** 3)[:, None])
        acc = nu / self.n0 * acc + torch.tensor([0.0, 0.0, G_Z], dtype=x.dtype, device=x.device)
        v = v + acc * dt
        x = x + v * dt
        v = self.clamp(v)
        # collisions, and the number density with the equation of state
        kick, dens = 0.0, 0.0
        rc = max(self.rp, self.rlim)
        for y, u, r in ((x, v, rc), (self.wpos, torch.zeros_like(self.wpos), 0.45 * self.l0),
                        (m1, torch.zeros_like(m1), rc)):
            i, j = _pairs(x, y, r)
            if y is x:
                i, j = i[i != j], j[i != j]
            e = y[j] - x[i]
            d2 = (e ** 2).sum(1)
            f = ((v[i] - u[j]) * e).sum(1)
            hit = (f > 0) & (d2 < min(self.rlim, r) ** 2)
            kick = kick + add(i[hit], -e[hit] * (f[hit] * 0.5 * (1 + COL_RAT) / d2[hit])[:, None])
            if y is not self.wpos:
                d = d2.sqrt()
                inside = d < self.rp
                dens = dens + add(i[inside], (self.rp / d - d / self.rp)[inside])
        v = v + kick
        prs = ((dens - self.n0g) * (SND * SND / self.n0g) * RHO).clamp(0.0, self.pmax)
        # pressure gradient, kick and drift
        owner, slot, m2 = self.mirrors(x)
        i, j = _pairs(x, x, self.rp)
        inside = (i != j) & (((x[j] - x[i]) ** 2).sum(1) < self.rp ** 2).detach()
        i, j = i[inside], j[inside]
        low = prs.scatter_reduce(0, i, prs[j], "amin")
        acc = 0.0
        for y, p, i, j in ((x, prs, i, j), (m2, prs[owner]) + _pairs(x, m2, self.rp)):
            if y is m2:
                other = slot[j] != i
                i, j = i[other], j[other]
            e = y[j] - x[i]
            d2 = (e ** 2).sum(1)
            d = d2.sqrt()
            w = (self.rp / d - d / self.rp) / d2
            acc = acc + add(i, e * (w * (p[j] - low[i]))[:, None])
        acc = acc * (-1 / RHO * 3 / self.n0g)
        v = v + acc * dt
        x = x + acc * dt * dt
        return x, self.clamp(v), prs


def _target(pos):
    """Where the loss wants the fluid: its centroid moved by a column's width; no height."""
    c = pos.mean(1)
    return (c[0] + pos[0].max(), c[1], c[2], 0.0)


def exact(case, seed):
    fluid_steps = work(case)["flops"] / 3720
    if case.get("plate") or case.get("corrected") or fluid_steps > 6e6 or not torch.cuda.is_available():
        return None
    device = "cuda"
    single = case["precision"] != "f64"
    parts = []
    for l0, block, tank, dt, scene in _of_case(case, seed):
        typ, pos, vel, nrm = scene
        if single:
            pos, vel = pos.astype(np.float32).astype(np.float64), vel.astype(np.float32).astype(np.float64)
        fluid = typ == FLUID
        e = _Exact(l0, block, tank, dt, (typ, pos, vel, nrm), device)
        start = torch.as_tensor(pos[:, fluid].T.copy(), device=device)
        v0 = torch.as_tensor(vel[:, fluid].T.copy(), device=device)
        nu = torch.tensor(NU, dtype=torch.float64, device=device)
        if case["kind"] == "adjoint":
            nu.requires_grad_(True)
            v0.requires_grad_(True)
        x, v, pav = start, v0, torch.zeros(start.shape[0], dtype=torch.float64, device=device)
        for _ in range(case["steps"]):
            x, v, prs = e.step(x, v, nu)
            pav = pav + prs
        if case["kind"] == "adjoint":
            loss = adjoint.dambreak_loss(x.T, torch.ones(x.shape[0], dtype=torch.bool, device=device),
                                         _target(pos[:, fluid]))
            loss.backward()
            return {"loss": loss.detach().cpu(), "pos": x.detach().T.cpu(),
                    "vel": v.detach().T.cpu(), "alive": None, "grad_nu": nu.grad.cpu(),
                    "grad_vel0": v0.grad.T.cpu()}
        got = {"pos": pos.copy(), "vel": vel.copy(), "prs": np.zeros(typ.size), "pav": np.zeros(typ.size)}
        got["pos"][:, fluid], got["vel"][:, fluid] = x.T.cpu().numpy(), v.T.cpu().numpy()
        got["prs"][fluid], got["pav"][fluid] = prs.cpu().numpy(), pav.cpu().numpy()
        parts.append(got)
    return dict({k: np.concatenate([p[k] for p in parts], -1) for k in FIELDS[1:]}, typ=None)
