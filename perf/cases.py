"""Performance cases of the PBF engine: the work its users have it do.

kind    what a user's program does
step    one solver step of one scene from a given state (coupled solvers and
        frame loops load positions and velocities, step, read them back)
hash    the spatial hash and neighbour counts of a point set
batch   one step of many independent scenes of uneven size
grad    a differentiable rollout: forward steps, then the gradient of a loss
        with respect to the initial state and the scene parameters
frame   an interactive frame: mouse pulse, step, rendered image

States are jittered lattices at rest spacing (0.5 h) with random velocities:
jitter 0.01 h at rest is how the benchmark workloads start; jitter 0.2 h with
speeds of about 1 m/s stands for a flow that has lost its lattice order.
Sizes are those of mtlphys_b200/configs.py (2,000 to 1,003,520 particles in a
scene, up to 256 scenes), with odd ones in between.
"""
from __future__ import annotations

import math

import numpy as np
import torch

H = 0.1
SPACING = 0.5 * H
BOX = 86 * H
DT = 1.0 / 120.0


# ---- the cases -----------------------------------------------------------------

def listed():
    step = dict(kind="step", jitter=0.01, speed=0.0, k=0.1, eps=100.0, iterations=3, graph=True)
    return [
        # the smallest scene of the cube ensemble: launches and latency count
        dict(step, name="step cube 2k", shape="cube", n=2197),
        # the cube drop benchmark (46^3)
        dict(step, name="step cube 97k", shape="cube", n=97336),
        # the dam break benchmark, its first step
        dict(step, name="step dam 1m", shape="dam", n=1003520, iterations=5),
        # the same scene in motion, a ragged count
        dict(step, name="step dam 1m moving", shape="dam", n=999983, iterations=5, jitter=0.2, speed=1.0),
        # a mid-size calm scene at the reference's solver constants, launched without a graph
        dict(step, name="step dam 250k direct", shape="dam", n=250007, iterations=5, k=1e-4, eps=800.0,
             jitter=0.05, speed=0.3, graph=False),
        # buildSpatialHash for a neighbour query
        dict(kind="hash", name="hash 500k", shape="dam", n=500009, jitter=0.2, speed=0.0),
        # a handful of small scenes
        dict(kind="batch", name="batch 12 small", scenes=12, lo=2000, hi=8000, k=0.1, iterations=3, jitter=0.01,
             speed=0.0),
        # the ensemble benchmark: 256 cube drops, 4.5M particles
        dict(kind="batch", name="batch 256", scenes=256, lo=2000, hi=64000, k=0.1, iterations=3, jitter=0.01,
             speed=0.0),
        # the differentiable cube, 20^3 as the gradient checks run it and 46^3 as the benchmark does
        dict(kind="grad", name="grad cube 8k", shape="cube", scenes=1, lo=8000, hi=8000, k=1e-4, eps=1e4,
             iterations=3, steps=10, every=5, jitter=0.01, speed=0.5),
        dict(kind="grad", name="grad cube 97k", shape="cube", scenes=1, lo=97336, hi=97336, k=1e-4, eps=1e5,
             iterations=3, steps=10, every=10, jitter=0.01, speed=0.5),
        # an ensemble of sphere drops, gradients to the sphere and s_corr of every scene
        dict(kind="grad", name="grad lakes 8", shape="lake", scenes=8, lo=20000, hi=80000, k=1e-4, eps=1e4,
             iterations=3, steps=4, every=2, jitter=0.01, speed=0.1),
        # the app's frame: 200,000 particles with the sphere, rendered
        dict(kind="frame", name="frame 200k", n=200000, width=960, height=540, jitter=0.05, speed=0.2),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) | 1

    kind = rng.choice(["step", "step", "step", "hash", "batch", "grad", "frame"])
    calm = rng.random() < 0.5
    solver = dict(k=1e-4 if calm else 0.1, iterations=rng.choice([3, 4, 5]))
    order = dict(jitter=0.01, speed=0.0) if rng.random() < 0.5 else dict(jitter=round(rng.uniform(0.05, 0.2), 3),
                                                                           speed=round(rng.uniform(0.1, 1.0), 3))
    if kind == "step":
        return dict(kind=kind, shape=rng.choice(["cube", "dam"]), n=size(1500, 1000000),
                    eps=800.0 if calm else 100.0, graph=rng.random() < 0.7, **solver, **order)
    if kind == "hash":
        return dict(kind=kind, shape=rng.choice(["cube", "dam"]), n=size(1500, 1000000), **order)
    if kind == "batch":
        lo = size(1500, 16000)
        return dict(kind=kind, scenes=size(2, 60), lo=lo, hi=lo * rng.choice([2, 4]), **solver, **order)
    if kind == "grad":
        lake = rng.random() < 0.5
        return dict(kind=kind, shape="lake" if lake else "cube", scenes=rng.choice([1, 2, 3, 5]),
                    lo=4001, hi=size(6000, 60000), k=1e-4, eps=1e4, iterations=rng.choice([2, 3]),
                    steps=rng.choice([3, 4, 6]), every=rng.choice([2, 3, 6]), jitter=0.01,
                    speed=round(rng.uniform(0.1, 0.5), 3))
    return dict(kind=kind, n=size(20000, 200000), width=rng.choice([640, 961, 1280]),
                height=rng.choice([361, 540, 720]), jitter=0.05, speed=0.2)


# ---- inputs ----------------------------------------------------------------------

def _rest_density():
    """Poly6 density of an interior lattice site."""
    r = np.arange(-3, 4) * SPACING
    d2 = (r[:, None, None] ** 2 + r[None, :, None] ** 2 + r[None, None, :] ** 2).ravel()
    d2 = d2[d2 < H * H]
    return float(315.0 / (64.0 * math.pi * H ** 9) * ((H * H - d2) ** 3).sum())


def _layout(shape, n):
    """(lattice dims, first site, box size) of n particles."""
    if shape == "cube":
        side = math.ceil(round(n ** (1.0 / 3.0), 9))
        return (side, side, side), (20 * H, 30 * H, 20 * H), (BOX, BOX, BOX)
    if shape == "dam":  # a column of the dam break's proportions against the x = 0 wall
        f = (n / 1003520.0) ** (1.0 / 3.0)
        nx, ny = max(1, round(64 * f)), max(1, round(160 * f))
        nz = -(-n // (nx * ny))
        return (nx, ny, nz), (0.5 * H, 0.5 * H, 0.5 * (BOX - (nz - 1) * SPACING)), (BOX, BOX, BOX)
    side = math.ceil(math.sqrt(n / 40.0))  # a lake 20 h deep in a box that hugs it
    width = (side - 1) * SPACING + H
    return (side, 40, side), (0.5 * H, 0.5 * H, 0.5 * H), (width, 40 * H, width)


def _points(shape, n, jitter, speed, gen, dev):
    dims, first, _ = _layout(shape, n)
    i = torch.arange(n, device=dev)
    site = torch.stack([i % dims[0], i // (dims[0] * dims[2]), (i // dims[0]) % dims[2]], 1).double()
    move = (torch.rand(n, 3, generator=gen, device=dev, dtype=torch.float64) * 2 - 1) * (jitter * H)
    pos = torch.ones(n, 4, device=dev)
    pos[:, :3] = (torch.tensor(first, device=dev, dtype=torch.float64) + site * SPACING + move).float()
    vel = torch.zeros(n, 4, device=dev)
    vel[:, :3] = torch.randn(n, 3, generator=gen, device=dev) * speed
    return pos, vel


def _scenes(case):
    """Per-scene counts, dts and epsilons of a case: part of the case, not of the seed."""
    if case["kind"] in ("step", "hash"):
        return [case["n"]], [DT], [case.get("eps", 100.0)]
    if case["kind"] == "frame":
        return [case["n"]], [DT], [800.0]
    rng = np.random.Generator(np.random.MT19937(3))
    n = case["scenes"]
    counts = np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]), size=n)).astype(int).tolist()
    if case["lo"] == case["hi"]:
        counts = [case["lo"]] * n
    if case["kind"] == "grad":
        return counts, [DT] * n, [case["eps"]] * n
    return counts, rng.uniform(1 / 240, 1 / 120, size=n).tolist(), rng.uniform(50.0, 200.0, size=n).tolist()


def _spheres(counts):
    """One sphere per lake, half immersed and sinking: centers, velocities, radii."""
    c, v, r = [], [], []
    for n in counts:
        width = _layout("lake", n)[2][0]
        rad = 8 * H * min(1.0, width / (2.5 * 16 * H))
        c.append([0.5 * width, 21 * H, 0.5 * width])
        v.append([0.0, -1.0, 0.0])
        r.append(rad)
    return c, v, r


FRAME_BOX = ((-3.0, -3.0, -3.0), (3.0, 6.0, 3.0))  # the reference engine's
FRAME_SPHERE = ([0.0, -2.4, 0.0], [0.0, 0.0, 0.0], 0.6)
PULSE = dict(origin=(0.0, 1.0, 5.0), direction=(0.0, -0.6, -0.8), force=(1.5, 0.5, 0.0), radius=0.8)


def _state(case, seed):
    """Positions and velocities of all scenes, from the seed alone."""
    dev = torch.device("cuda", torch.cuda.current_device())
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    if case["kind"] == "frame":
        n = case["n"]
        i = torch.arange(n, device=dev)
        nx = 117  # a layer of the default box at rest spacing
        site = torch.stack([i % nx, i // (nx * nx), (i // nx) % nx], 1).double()
        move = (torch.rand(n, 3, generator=gen, device=dev, dtype=torch.float64) * 2 - 1) * (case["jitter"] * H)
        pos = torch.ones(n, 4, device=dev)
        pos[:, :3] = (site * SPACING + move - 2.95 + SPACING * 0.5).float()
        vel = torch.zeros(n, 4, device=dev)
        vel[:, :3] = torch.randn(n, 3, generator=gen, device=dev) * case["speed"]
        return pos, vel
    counts = _scenes(case)[0]
    parts = [_points(case.get("shape", "cube"), n, case["jitter"], case["speed"], gen, dev) for n in counts]
    return torch.cat([p for p, _ in parts]), torch.cat([v for _, v in parts])


def _params(case, eps, box):
    from mtlphys_b200 import _abi

    p = _abi.default_params()
    if case["kind"] == "frame":
        return p  # the reference engine's
    return p.set(h=H, cell_size=H, rest_density=_rest_density(), epsilon=eps, gravity=(0.0, -9.8, 0.0),
                 bounds_min=(0.0, 0.0, 0.0), bounds_max=box, scorr_k=case.get("k", 0.1), scorr_n=4, scorr_dq=0.2,
                 solver_iterations=case.get("iterations", 3))


class _State:
    pass


def prepare(case, seed):
    from mtlphys_b200 import Engine, _abi
    from mtlphys_b200.batch import Batch

    s = _State()
    s.case = case
    s.pos0, s.vel0 = _state(case, seed)
    counts, dts, eps = _scenes(case)
    shape = case.get("shape", "cube")
    ids = {"cube": 0, "dam": 1, "lake": 2}
    dev = s.pos0.device
    s.stream = torch.cuda.current_stream(dev)
    if case["kind"] in ("batch", "grad"):
        s.b = Batch(dev.index)
        s.b.reset(counts, [_params(case, e, _layout(shape, n)[2]) for n, e in zip(counts, eps)], dts,
                  [ids[shape]] * len(counts))
        s.b.set_graph_mode(True)
        owner = s.b
    else:
        s.e = Engine(dev.index)
        s.e.set_params(_params(case, eps[0], (BOX, BOX, BOX)))
        s.e.reset(counts[0], 2 if case["kind"] == "frame" else ids[shape])
        s.e.set_graph_mode(bool(case.get("graph", True)))
        owner = s.e
    view = lambda which: owner.tensor(which)  # noqa: E731
    s.pos, s.vel = view(_abi.MP_BUF_POSITIONS), view(_abi.MP_BUF_VELOCITIES)
    s.lam, s.foam, s.count = view(_abi.MP_BUF_LAMBDAS), view(_abi.MP_BUF_FOAM), view(_abi.MP_BUF_NEIGHBOR_COUNTS)
    if case["kind"] == "hash":
        s.pos.copy_(s.pos0)
        s.hashes = {k: view(w) for k, w in (("hash", _abi.MP_BUF_CELL_HASHES), ("start", _abi.MP_BUF_CELL_START),
                                            ("index", _abi.MP_BUF_SORTED_INDEX), ("counts", _abi.MP_BUF_NEIGHBOR_COUNTS),
                                            ("sorted", _abi.MP_BUF_SORTED_POSITIONS))}
    if case["kind"] == "frame":
        s.e.set_sphere(*FRAME_SPHERE)
        s.image = _abi.default_render_params(width=case["width"], height=case["height"])
    if case["kind"] == "grad":
        gen = torch.Generator(device=dev)
        gen.manual_seed(seed + 7919)
        s.target = _target(s.pos0, gen)
        s.pos0.requires_grad_(True)
        s.vel0.requires_grad_(True)
        s.k = torch.full((len(counts),), case["k"], device=dev, requires_grad=True)
        s.sphere = None
        if shape == "lake":
            s.sphere = tuple(torch.tensor(x, device=dev, dtype=torch.float32, requires_grad=True)
                             for x in _spheres(counts))
    return s


def _target(pos0, gen):
    t = pos0.detach().clone()
    t[:, :3] += torch.randn(t.shape[0], 3, generator=gen, device=t.device) * 0.1
    return t


# ---- one pass ----------------------------------------------------------------------

def run(s):
    c = s.case
    if c["kind"] == "hash":
        s.e.build_spatial_hash(s.stream)
        return s.hashes
    if c["kind"] == "grad":
        from mtlphys_b200.autograd import rollout

        p, v = rollout(s.b, c["steps"], s.pos0, s.vel0, s.k, s.sphere, checkpoint_every=c["every"])
        loss = (p - s.target).square().sum() / p.shape[0]
        inputs = [s.pos0, s.vel0, s.k] + list(s.sphere or ())
        return {"pos": p.detach(), "vel": v.detach(), "grads": list(torch.autograd.grad(loss, inputs))}
    s.pos.copy_(s.pos0)
    s.vel.copy_(s.vel0)
    out = {"pos": s.pos, "vel": s.vel, "lambda": s.lam, "foam": s.foam, "count": s.count}
    if c["kind"] == "batch":
        s.b.step(s.stream)
    elif c["kind"] == "step":
        s.e.step(DT, s.stream)
    else:
        s.e.apply_mouse_pulse(PULSE["origin"], PULSE["direction"], PULSE["force"], PULSE["radius"], s.stream)
        s.e.step(DT, s.stream)
        out["image"] = s.e.render(s.image, s.stream)
    return out


def work(case):
    """Inputs read once, outputs written once; about 30 neighbours a particle, each needing a distance and
    the pair term of both solver passes (about 60 operations) in every iteration."""
    n = float(sum(_scenes(case)[0]))
    pairs = 30.0 * n
    if case["kind"] == "hash":
        return {"bytes": (16 + 4 + 4 + 4 + 16) * n + 4.0 * 86 ** 3, "flops": 9 * pairs}
    k = case.get("iterations", 5)
    step = 60.0 * pairs * k
    if case["kind"] == "grad":  # the gradient repeats the forward's pair terms and their derivatives
        return {"bytes": (32 + 16 + 32 + 32) * n, "flops": case["steps"] * step * 4}
    px = float(case["width"] * case["height"]) if case["kind"] == "frame" else 0.0
    return {"bytes": (32 + 32 + 12) * n + 16 * px, "flops": step + 100 * px}


# ---- the same in 64 bits, in plain torch ---------------------------------------------

class _Model:
    """The PBF step of S scenes in FP64: per-particle constants, cells of positions rounded to FP32."""

    def __init__(self, scene, dt, eps, box_lo, box_hi, p):
        self.scene, self.dt, self.eps, self.lo, self.hi, self.p = scene, dt, eps, box_lo, box_hi, p
        f32 = lambda x: float(np.float32(x))  # noqa: E731
        self.h = f32(H)
        self.rho0 = f32(p["rho0"])
        self.inv = float(np.float32(1.0) / np.float32(H))
        self.dims = torch.ceil((box_hi - box_lo).float() / torch.full_like(box_hi, H).float()).long()
        cells = self.dims.prod(1)
        sizes = torch.zeros(int(scene.max()) + 1, dtype=torch.long, device=scene.device)
        sizes[scene] = cells
        self.base = (torch.cumsum(sizes, 0) - sizes)[scene]
        self.total = int(sizes.sum())

    def cells(self, x):
        q = torch.floor((x.float() - self.lo.float()) * self.inv)
        return torch.minimum(torch.clamp(q, min=0).long(), self.dims - 1)

    def cell_id(self, c):
        return self.base + c[:, 0] + self.dims[:, 0] * (c[:, 1] + self.dims[:, 1] * c[:, 2])

    def pairs(self, x, order, start):
        """i, j of every j != i within h of i whose hash cell is in the 27 cells around i's cell."""
        c = self.cells(x)
        lo, hi = torch.clamp(c - 1, min=0), torch.minimum(c + 1, self.dims - 1)
        found = []
        me = torch.arange(x.shape[0], device=x.device)
        for dz in range(-1, 2):
            for dy in range(-1, 2):
                y, z = c[:, 1] + dy, c[:, 2] + dz
                ok = (y >= 0) & (y < self.dims[:, 1]) & (z >= 0) & (z < self.dims[:, 2])
                row = self.base + self.dims[:, 0] * (y + self.dims[:, 1] * z)
                i = me[ok]
                a, b = start[(row + lo[:, 0])[ok]], start[(row + hi[:, 0])[ok] + 1]
                while i.numel():
                    more = a < b
                    i, a, b = i[more], a[more], b[more]
                    j = order[a]
                    near = ((x[i] - x[j]).square().sum(1) < self.h ** 2) & (i != j)
                    found.append(torch.stack([i[near], j[near]]))
                    a = a + 1
        return torch.cat(found, 1)

    def step(self, pos, vel, k, sphere):
        p, h = self.p, self.h
        dt = self.dt[:, None]
        v = vel + dt * torch.tensor(p["gravity"], device=pos.device, dtype=torch.float64)
        x = pos + v * dt
        x = x + (x.float().double() - x).detach()  # the hash and the solver start from FP32 predictions
        if sphere is not None:
            sphere = self.advance(sphere)
        with torch.no_grad():
            home = self.cell_id(self.cells(x))
            order = torch.argsort(home, stable=True)
            start = torch.zeros(self.total + 1, dtype=torch.long, device=pos.device)
            start[1:] = torch.cumsum(torch.bincount(home, minlength=self.total), 0)
        w6, sp = 315.0 / (64.0 * math.pi * h ** 9), 45.0 / (math.pi * h ** 6)
        wq = w6 * (h * h - (p["dq"] * h) ** 2) ** 3
        count = None
        for _ in range(p["iterations"]):
            with torch.no_grad():
                i, j = self.pairs(x.detach(), order, start)
                if count is None:
                    count = torch.bincount(i, minlength=x.shape[0])
            r = x[i] - x[j]
            r2 = r.square().sum(1)
            d = h * h - r2
            zero = r2 <= 1e-12
            rl = torch.sqrt(torch.where(zero, torch.ones_like(r2), r2))
            g = torch.where(zero, torch.zeros_like(rl), -sp * torch.clamp(h - rl, min=0.0) ** 2 / rl)[:, None] * r
            sums = torch.zeros(x.shape[0], 5, device=x.device, dtype=torch.float64)
            sums = sums.index_add(0, i, torch.cat([(w6 * d ** 3)[:, None], g, g.square().sum(1, keepdim=True)], 1))
            dens = sums[:, 0] + w6 * h ** 6
            lam = -(dens / self.rho0 - 1) / ((sums[:, 1:4].square().sum(1) + sums[:, 4]) / self.rho0 ** 2 + self.eps)
            s = -k[self.scene[i]] * (w6 * d ** 3 / wq) ** 4
            dx = torch.zeros_like(x).index_add(0, i, (lam[i] + lam[j] + s)[:, None] * g) / self.rho0
            dl = torch.sqrt(torch.clamp(dx.square().sum(1, keepdim=True), min=1e-30))
            most = 0.3 * h
            x = x + torch.where(dl > most, dx * (most / dl), dx)
            x = torch.minimum(torch.maximum(x, self.lo), self.hi)
            if sphere is not None:
                c, _, rad = sphere
                e = x - c[self.scene]
                e2 = e.square().sum(1, keepdim=True)
                rr = rad[self.scene][:, None]
                x = torch.where(e2 < rr * rr, c[self.scene] + e * (rr / torch.sqrt(torch.clamp(e2, min=1e-8))), x)
        return self.finish(pos, x, lam, count, sphere)

    def finish(self, pos, x, lam, count, sphere):
        p, h = self.p, self.h
        v = (x - pos) * (p["damping"] / self.dt)[:, None]
        low, high = x <= self.lo + 1e-3, x >= self.hi - 1e-3
        v = torch.where(low, torch.clamp(v, min=0.0), v)
        v = torch.where(high, torch.clamp(v, max=0.0), v)
        floor = low[:, 1:2]
        wall = (low | high).any(1, keepdim=True) & ~floor
        horizontal = torch.tensor([True, False, True], device=x.device)
        v = torch.where(floor & horizontal, v * 0.55, torch.where(wall, v * 0.97, v))
        most = (h / self.dt)[:, None]
        speed = torch.sqrt(torch.clamp(v.square().sum(1, keepdim=True), min=1e-30))
        v = torch.where(speed > most, v * (most / speed), v)
        t = torch.clamp((torch.minimum(speed, most)[:, 0] - 1.2) / (4.5 - 1.2), 0.0, 1.0)
        foam = (1 - torch.clamp(count / 96.0, 0.0, 1.0)) * t * t * (3 - 2 * t)
        return x, v, lam, foam, sphere

    def advance(self, sphere):
        c, v, r = sphere
        first = torch.searchsorted(self.scene, torch.arange(c.shape[0], device=c.device))
        dt, lo, hi = self.dt[first][:, None], self.lo[first], self.hi[first]
        v = (v + dt * torch.tensor([0.0, -9.81, 0.0], device=c.device, dtype=torch.float64)) * 0.998
        c = c + v * dt
        rr = r[:, None]
        under = c - rr < lo
        c, v = torch.where(under, lo + rr, c), torch.where(under, -0.4 * v, v)
        over = c + rr > hi
        return torch.where(over, hi - rr, c), torch.where(over, -0.4 * v, v), r


def exact(case, seed):
    if case["kind"] == "hash":
        return None  # whole numbers and copies
    pos0, vel0 = _state(case, seed)
    dev = pos0.device
    counts, dts, eps = _scenes(case)
    n = torch.tensor(counts, device=dev)
    scene = torch.repeat_interleave(torch.arange(len(counts), device=dev), n)
    f64 = lambda x: torch.tensor(np.asarray(x, np.float32), device=dev).double()  # noqa: E731
    if case["kind"] == "frame":
        lo, hi = f64([FRAME_BOX[0]]), f64([FRAME_BOX[1]])
        p = dict(rho0=8000.0, gravity=(0.0, float(np.float32(-9.81)), 0.0), dq=0.2, iterations=5)
        k = f64([1e-4])
    else:
        hi = f64([_layout(case.get("shape", "cube"), c)[2] for c in counts])
        lo = torch.zeros_like(hi)
        p = dict(rho0=_rest_density(), gravity=(0.0, float(np.float32(-9.8)), 0.0), dq=float(np.float32(0.2)),
                 iterations=case["iterations"])
        k = f64([case["k"]] * len(counts))
    p["damping"] = float(np.float32(0.996))
    m = _Model(scene, f64(dts)[scene], f64(eps)[scene], lo[scene], hi[scene], p)
    pos, vel = pos0[:, :3].double(), vel0[:, :3].double()
    four = lambda x, w: torch.cat([x, torch.full_like(x[:, :1], w)], 1)  # noqa: E731
    if case["kind"] == "grad":
        sphere = None
        leaves = [pos.requires_grad_(True), vel.requires_grad_(True), k.requires_grad_(True)]
        if case["shape"] == "lake":
            sphere = tuple(f64(x).requires_grad_(True) for x in _spheres(counts))
            leaves += list(sphere)
        x, v = pos, vel
        for _ in range(case["steps"]):
            x, v, _, _, sphere = m.step(x, v, k, sphere)
        gen = torch.Generator(device=dev)
        gen.manual_seed(seed + 7919)
        target = _target(pos0, gen)[:, :3].double()
        loss = (x - target).square().sum() / x.shape[0]
        g = torch.autograd.grad(loss, leaves)
        return {"pos": four(x.detach(), 1.0), "vel": four(v.detach(), 0.0),
                "grads": [four(g[0], 0.0), four(g[1], 0.0)] + list(g[2:])}
    sphere = None
    with torch.no_grad():
        if case["kind"] == "frame":
            sphere = tuple(f64([x]) for x in FRAME_SPHERE)
            o, d, f = (f64([PULSE[w]]) for w in ("origin", "direction", "force"))
            t = ((pos - o) * d).sum(1, keepdim=True)
            r2 = (pos - (o + d * t)).square().sum(1, keepdim=True)
            big = float(np.float32(PULSE["radius"])) ** 2
            push = torch.exp(-r2 / (big * 0.4)) * ((t > 0) & (r2 < big))
            vel = vel + f * push
        x, v, lam, foam, _ = m.step(pos, vel, k, sphere)
    out = {"pos": four(x, 1.0), "vel": four(v, 0.0), "lambda": lam, "foam": foam, "count": None}
    if case["kind"] == "frame":
        out["image"] = None
    return out
