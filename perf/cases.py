"""The work this package is timed on: its force solvers and integrators through
their public entry points, from the smallest call to the largest.

The sizes are those of the package's own workloads: a Plummer sphere of 1,000
to 262,144 particles for the direct sums (1k..64k for a served job),
clusters of 256 to 16,384 particles for a batch, a collision of two disc
galaxies of 10,000 to 2,000,000 particles for the tree. ``draw`` gives more
cases of the same ranges. Inputs are made on the GPU from a seed.
"""
import math
from types import SimpleNamespace

import numpy as np
import torch

import orrery_b200 as ob
from orrery_b200 import simulation

STATE = ("x", "y", "z", "vx", "vy", "vz", "ax", "ay", "az")


def listed():
    return [
        # One velocity-Verlet step of a small direct system, the call a live
        # display or a small served job makes step by step: latency.
        dict(name="step-direct-1k", kind="steps", solver="direct", precision="fp32", n=1000,
             integrator="vv", steps=1, softening=0.01),
        # The plain direct configuration: 4096 particles, 100 steps per call.
        dict(name="steps-direct-4096", kind="steps", solver="direct", precision="fp32", n=4096,
             integrator="vv", steps=100, softening=0.01),
        # A force evaluation on device arrays inside a caller's own integrator,
        # at a ragged size in the middle of the direct range.
        dict(name="forces-direct-20011", kind="forces", solver="direct", precision="fp32",
             n=20011, softening=0.01),
        # The same at the largest direct size.
        dict(name="forces-direct-262144", kind="forces", solver="direct", precision="fp32",
             n=262144, softening=0.01),
        # A Yoshida-4 step in the precision form, the largest served direct job.
        dict(name="yoshida-split-65536", kind="steps", solver="direct", precision="split",
             n=65536, integrator="yoshida4", steps=1, softening=0.01),
        # The batched form: clusters of uneven size advanced together by ten
        # Yoshida-4 steps, every member's state then read.
        dict(name="batch-128", kind="batch", systems=128, smallest=256, largest=16384,
             integrator="yoshida4", steps=10, softening=0.01),
        # The reference's own call, compute_accelerations(configuration,
        # particles), on host particles with the bit-exact FP64 direct sum.
        dict(name="call-direct-fp64-4096", kind="call", solver="direct", precision="fp64",
             n=4096, softening=0.01),
        # A small tree on device arrays, monopoles only (the solver's default).
        dict(name="forces-tree-10k", kind="forces", solver="tree", precision="fp32", n=10000,
             softening=0.02, angle=0.5, leaf=32, quadrupole=False, model="plummer"),
        # The ForceSolver drop-in over host arrays, at a served tree job's size.
        dict(name="host-tree-200k", kind="host", solver="tree", precision="fp32", n=200000,
             softening=0.02, angle=0.5, leaf=32, quadrupole=True, model="collision"),
        # The headline: one velocity-Verlet step of the 2M two-disc collision.
        dict(name="step-tree-2m", kind="steps", solver="tree", precision="fp32", n=2000000,
             integrator="vv", steps=1, softening=0.02, angle=0.5, leaf=32, quadrupole=True,
             model="collision"),
        # The FP64 parity walk (forces bit-identical to the reference's).
        dict(name="forces-tree-fp64-100k", kind="forces", solver="tree", precision="fp64",
             n=100000, softening=0.02, angle=0.5, leaf=32, quadrupole=True, model="collision"),
        # The conserved quantities a run logs at each record point.
        dict(name="diagnostics-32k", kind="diagnostics", solver="direct", precision="fp32",
             n=32768, softening=0.01),
    ]


def draw(rng):
    def size(lo, hi):
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        return min(hi, n | 1 if rng.random() < 0.5 else n)

    def tree(n):
        return dict(n=n, softening=rng.choice([0.01, 0.02, 0.05]),
                    angle=rng.choice([0.5, 0.6, 0.7, 0.9]), leaf=rng.choice([8, 16, 32, 48]),
                    quadrupole=rng.random() < 0.6, model=rng.choice(["plummer", "collision"]))

    kind = rng.choice(["steps-direct", "forces-direct", "split", "batch", "direct-fp64",
                       "forces-tree", "host-tree", "steps-tree", "tree-fp64", "diagnostics"])
    integrator = rng.choice(["vv", "yoshida4"])
    if kind == "steps-direct":
        n = size(256, 32768)
        return dict(kind="steps", solver="direct", precision="fp32", n=n, integrator=integrator,
                    steps=rng.randint(1, 20), softening=0.01)
    if kind == "forces-direct":
        return dict(kind="forces", solver="direct", precision="fp32", n=size(256, 250000),
                    softening=rng.choice([0.01, 0.05]))
    if kind == "split":
        return dict(kind="steps", solver="direct", precision="split", n=size(512, 60000),
                    integrator=integrator, steps=1, softening=0.01)
    if kind == "batch":
        return dict(kind="batch", systems=rng.randint(4, 128), smallest=256,
                    largest=size(2048, 16384), integrator=integrator, steps=rng.randint(1, 4),
                    softening=0.01)
    if kind == "direct-fp64":
        return dict(kind=rng.choice(["call", "host"]), solver="direct", precision="fp64",
                    n=size(256, 32768), softening=0.01)
    if kind == "forces-tree":
        return dict(kind="forces", solver="tree", precision="fp32", **tree(size(1000, 1500000)))
    if kind == "host-tree":
        return dict(kind=rng.choice(["host", "call"]), solver="tree", precision="fp32",
                    **tree(size(1000, 500000)))
    if kind == "steps-tree":
        return dict(kind="steps", solver="tree", precision="fp32", integrator="vv",
                    steps=rng.randint(1, 3), **tree(size(1000, 500000)))
    if kind == "tree-fp64":
        return dict(kind=rng.choice(["forces", "call"]), solver="tree", precision="fp64",
                    **tree(size(1000, 200000)))
    return dict(kind="diagnostics", solver="direct", precision="fp32", n=size(512, 65536),
                softening=0.01)


# --------------------------------------------------------------------- inputs

DT = 1e-3


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


class _Random:
    def __init__(self, seed):
        self.device = _device()
        self.g = torch.Generator(device=self.device)
        self.g.manual_seed(int(seed))

    def uniform(self, *shape):
        return torch.rand(*shape, generator=self.g, device=self.device, dtype=torch.float64)

    def normal(self, *shape):
        return torch.randn(*shape, generator=self.g, device=self.device, dtype=torch.float64)

    def directions(self, n):
        v = self.normal(n, 3)
        return v / v.norm(dim=1, keepdim=True)


def _plummer(r, n, radius=1.0):
    """A Plummer sphere of unit mass: enclosed-mass radii, speeds from the
    distribution function q^2 (1 - q^2)^{7/2} by its tabulated integral."""
    frac = 0.999 * r.uniform(n).clamp(min=1e-12)
    d = radius / torch.sqrt(frac ** (-2.0 / 3.0) - 1.0)
    grid = torch.linspace(0.0, 1.0, 4097, device=r.device, dtype=torch.float64)
    pdf = grid ** 2 * (1.0 - grid ** 2).clamp(min=0.0) ** 3.5
    cdf = torch.cumsum(pdf, 0) / pdf.sum()
    q = grid[torch.searchsorted(cdf, r.uniform(n)).clamp(max=4096)]
    speed = q * torch.sqrt(2.0 / torch.sqrt(d * d + radius * radius))
    return d[:, None] * r.directions(n), speed[:, None] * r.directions(n)


def _disc(r, n, mass, length, inclination):
    """An exponential disc with a Hernquist bulge of a fifth of its mass, on
    about circular orbits."""
    bulge = n // 5
    radius = -length * torch.log((1.0 - r.uniform(n - bulge)) * (1.0 - r.uniform(n - bulge)))
    radius = torch.where(radius > 7.0 * length, radius % (7.0 * length), radius)
    phi = 2.0 * math.pi * r.uniform(n - bulge)
    height = -0.1 * length * torch.log(1.0 - r.uniform(n - bulge))
    height = torch.where(r.uniform(n - bulge) < 0.5, -height, height)
    su = torch.sqrt(0.995 * r.uniform(bulge))
    core = 0.2 * length * su / (1.0 - su)
    x = torch.cat([torch.stack([radius * torch.cos(phi), radius * torch.sin(phi), height], 1),
                   core[:, None] * r.directions(bulge)])
    speed = torch.sqrt(mass * radius / (radius + length) ** 2)
    v = torch.cat([torch.stack([-speed * torch.sin(phi), speed * torch.cos(phi),
                                torch.zeros_like(phi)], 1),
                   0.3 * math.sqrt(mass / length) * r.normal(bulge, 3)])
    c, s = math.cos(inclination), math.sin(inclination)
    turn = torch.tensor([[1, 0, 0], [0, c, s], [0, -s, c]], dtype=torch.float64,
                        device=r.device)
    return x @ turn, v @ turn


def _collision(r, n):
    """Two discs of mass ratio 3:1 at 30 degrees, 20 scale lengths apart on a
    bound grazing orbit."""
    first = n - n // 4
    a, va = _disc(r, first, 0.75, 1.0, 0.0)
    b, vb = _disc(r, n - first, 0.25, math.sqrt(1.0 / 3.0), math.radians(30.0))
    apart = torch.tensor([20.0, 12.0, 0.0], dtype=torch.float64, device=r.device)
    speed = torch.tensor([-0.23, 0.0, 0.0], dtype=torch.float64, device=r.device)
    return (torch.cat([a - 0.25 * apart, b + 0.75 * apart]),
            torch.cat([va - 0.25 * speed, vb + 0.75 * speed]))


def _inputs(case, seed):
    r = _Random(seed)
    n = case["n"]
    x, v = (_collision if case.get("model") == "collision" else _plummer)(r, n)
    m = torch.full((n,), 1.0 / n, dtype=torch.float64, device=r.device)
    return x - x.mean(0), v - v.mean(0), m


def _sizes(case):
    """Particles of each system of a batch, about log-uniform: the same for
    every seed, so that a batch's work depends on its case alone."""
    lo, hi = math.log(case["smallest"]), math.log(case["largest"])
    return [int(math.exp(lo + (hi - lo) * ((0.5 + 0.6180339887498949 * k) % 1.0)))
            for k in range(case["systems"])]


def _clusters(case, seed):
    """(softening, x, v, m) of each system of a batch."""
    r = _Random(seed)
    sizes = _sizes(case)
    radii = (0.5 + 1.5 * r.uniform(len(sizes))).tolist()
    x, v = _plummer(r, sum(sizes))
    out, at = [], 0
    for n, a in zip(sizes, radii):
        out.append((case["softening"] * a, x[at:at + n] * a, v[at:at + n] / math.sqrt(a),
                    torch.full((n,), 1.0 / n, dtype=torch.float64, device=r.device)))
        at += n
    return out


# ---------------------------------------------------------------- preparation

def _host(t):
    return t.cpu().numpy()


def _columns(t):
    return [np.ascontiguousarray(c) for c in _host(t).T]


def _solver(case):
    if case["solver"] == "direct":
        return ob.B200DirectSolver(case["softening"], case["precision"])
    return ob.B200TreeSolver(case["softening"], case["angle"], case["leaf"], case["quadrupole"],
                             case["precision"])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        members = _clusters(case, seed)
        batch = ob.DeviceBatch([len(c[3]) for c in members], [c[0] for c in members])
        for k, (_, x, v, m) in enumerate(members):
            batch.set_state(k, *_columns(x), *_columns(v), _host(m))
        batch.refresh()
        return dict(case=case, batch=batch, systems=len(members))
    x, v, m = _inputs(case, seed)
    n = case["n"]
    if kind == "forces":
        out = torch.empty(3, n, dtype=torch.float64, device=x.device)
        return dict(case=case, solver=_solver(case), x=x.t().contiguous(), m=m, out=out,
                    n=n)
    if kind == "host":
        return dict(case=case, solver=_solver(case), x=_columns(x), m=_host(m),
                    out=[np.empty(n) for _ in range(3)])
    if kind == "call":
        settings = SimpleNamespace(kind="direct" if case["solver"] == "direct" else "barnes-hut",
                                   softening=case["softening"],
                                   opening_angle=case.get("angle", 0.5),
                                   leaf_capacity=case.get("leaf", 32),
                                   quadrupole=case.get("quadrupole", False))
        px, py, pz = _columns(x)
        particles = SimpleNamespace(position_x=px, position_y=py, position_z=pz, mass=_host(m),
                                    acceleration_x=np.empty(n), acceleration_y=np.empty(n),
                                    acceleration_z=np.empty(n))
        return dict(case=case, configuration=SimpleNamespace(solver=settings),
                    particles=particles)
    solver = ob.SOLVER_DIRECT if case["solver"] == "direct" else ob.SOLVER_TREE
    system = ob.DeviceSystem(n, case["softening"], solver, case["precision"],
                             case.get("angle", 0.5), case.get("leaf", 32),
                             case.get("quadrupole", False))
    system.set_state(*_columns(x), *_columns(v), _host(m))
    views = {k: torch.as_tensor(a, device=x.device)
             for k, a in simulation.device_arrays(system).items()}
    if kind == "steps":
        # Such a program steps many times: its step graph is captured by now
        # (a call of no steps leaves the state as it is).
        system.step_kernels(DT, case["integrator"])
    return dict(case=case, system=system, views=views)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "steps":
        state["system"].step(DT, case["steps"], case["integrator"])
        return [state["views"][k] for k in STATE]
    if kind == "forces":
        x, out = state["x"], state["out"]
        stream = torch.cuda.current_stream().cuda_stream
        state["solver"].evaluate_device(state["n"], x[0], x[1], x[2], state["m"], out[0], out[1],
                                        out[2], stream)
        return out
    if kind == "host":
        state["solver"].evaluate(tuple(state["x"]), state["m"], state["out"])
        return state["out"]
    if kind == "call":
        p = state["particles"]
        ob.compute_accelerations(state["configuration"], p, precision=case["precision"])
        return [p.acceleration_x, p.acceleration_y, p.acceleration_z]
    if kind == "batch":
        state["batch"].step(DT, case["steps"], case["integrator"])
        members = [state["batch"].state(k) for k in range(state["systems"])]
        return [np.concatenate([s[k] for s in members]) for k in STATE]
    d = state["system"].diagnostics()
    return [d["kinetic_energy"], d["potential_energy"], d["linear_momentum"],
            d["angular_momentum"]]


# ----------------------------------------------------------------------- work

# Conventional operations of one softened pair term, one monopole cell term
# and one quadrupole cell term (a square root or a division counts as one).
PAIR, MONOPOLE, QUADRUPOLE = 19, 19, 57


def _evaluations(case):
    return case.get("steps", 1) * (3 if case.get("integrator") == "yoshida4" else 1)


# ln(terms per target) of the theta walk as a quadratic in L = ln(n / 2e6) with
# A = ln(angle / 0.5), F = ln(leaf / 32): coefficients of 1, L, L^2, A, F, A L, F L,
# fitted to the solver's own counts from 1,000 to 2,000,000 particles (cells
# within a quarter, pairs within a factor of 1.8).
_TERMS = {
    "plummer": ((6.949, -0.269, -0.04, -3.5, 1.221, -0.235, 0.074),
                (7.905, 0.064, -0.055, -2.399, 0.018, -0.301, 0.074)),
    "collision": ((7.618, -0.234, -0.064, -3.575, 1.274, -0.354, 0.099),
                  (7.913, 0.261, -0.041, -1.818, -0.086, -0.229, 0.06)),
}


def _tree_terms(case):
    """Pair and cell terms per target (estimates)."""
    size = math.log(case["n"] / 2e6)
    angle, leaf = math.log(case["angle"] / 0.5), math.log(case["leaf"] / 32)
    basis = (1.0, size, size * size, angle, leaf, angle * size, leaf * size)
    return tuple(min(float(case["n"]), math.exp(sum(c * b for c, b in zip(fit, basis))))
                 for fit in _TERMS[case["model"]])


def work(case):
    kind = case["kind"]
    if kind == "batch":
        sizes = _sizes(case)
        pairs = sum(n * (n - 1.0) for n in sizes)
        return dict(bytes=152.0 * sum(sizes), flops=_evaluations(case) * PAIR * pairs)
    n = float(case["n"])
    if kind == "diagnostics":
        # Each pair once: an inverse distance and its weighted sum.
        return dict(bytes=56.0 * n, flops=11.0 * n * (n - 1.0) / 2.0 + 40.0 * n)
    if case["solver"] == "direct":
        flops = PAIR * n * (n - 1.0)
    else:
        pairs, cells = _tree_terms(case)
        flops = n * (PAIR * pairs + (QUADRUPOLE if case["quadrupole"] else MONOPOLE) * cells)
    if kind == "steps":
        # State and masses read once, positions, velocities, accelerations written.
        return dict(bytes=152.0 * n, flops=_evaluations(case) * flops)
    return dict(bytes=56.0 * n, flops=flops)


def tolerance(case):
    if case["kind"] == "diagnostics" or case.get("precision") == "fp64":
        return "exact"  # bit-identical to the reference's FP64 results
    if case["kind"] == "batch" or case["precision"] == "split":
        return {"rel": 2e-7}   # 1.7e-8 to 4.7e-8 from 64 bits as measured
    if case["solver"] == "tree":
        return {"rel": 1e-6}   # 4e-8 (quadrupoles) to 2.3e-7 (small, monopoles)
    return {"rel": 4e-6}       # FP32 sums: 2.5e-7 to 1.3e-6


# ------------------------------------------------- the same results in 64 bits

def _direct(x, m, eps2):
    """Softened accelerations over all pairs (the own term is zero)."""
    out = torch.empty_like(x)
    rows = max(1, (1 << 26) // x.shape[0])
    for at in range(0, x.shape[0], rows):
        t = x[at:at + rows]
        r2 = torch.full((t.shape[0], x.shape[0]), eps2, dtype=x.dtype, device=x.device)
        for k in range(3):
            d = t[:, k, None] - x[None, :, k]
            r2.addcmul_(d, d)
        w = r2.pow_(-1.5).mul_(m)
        for k in range(3):
            out[at:at + rows, k] = (x[None, :, k] - t[:, k, None]).mul_(w).sum(1)
    return out


def _potential(x, m, eps2):
    total = 0.0
    rows = max(1, (1 << 26) // x.shape[0])
    for at in range(0, x.shape[0], rows):
        t = x[at:at + rows]
        r2 = torch.full((t.shape[0], x.shape[0]), eps2, dtype=x.dtype, device=x.device)
        for k in range(3):
            d = t[:, k, None] - x[None, :, k]
            r2.addcmul_(d, d)
        w = r2.rsqrt_().mul_(m)
        own = torch.arange(t.shape[0], device=x.device)
        w[own, at + own] = 0.0
        total -= 0.5 * float((m[at:at + rows] * w.sum(1)).sum())
    return total


def _spread_bits(v):
    out = torch.zeros_like(v)
    for b in range(21):
        out |= ((v >> b) & 1) << (3 * b)
    return out


class _Tree:
    """Barnes-Hut in plain torch: Morton-ordered particles, cells split while
    they hold more than `leaf` particles, moments and acceptance radii, and the
    walk as one frontier of (target, cell) pairs per level."""

    LEVELS = 21

    def __init__(self, x, m, angle, leaf, quadrupole):
        lo, hi = x.amin(0), x.amax(0)
        edge = float((hi - lo).max()) or 1.0
        centre = (lo + hi) / 2.0
        grid = ((x - (centre - edge / 2.0)) * (2097152.0 / edge)).long().clamp(0, 2097151)
        code = (_spread_bits(grid[:, 0]) << 2) | (_spread_bits(grid[:, 1]) << 1) | _spread_bits(
            grid[:, 2])
        code, self.order = torch.sort(code, stable=True)
        self.x, self.m = x[self.order], m[self.order]
        n, device = x.shape[0], x.device
        parts = dict(first=[], count=[], com=[], mass=[], r2=[], quad=[], child=[], kids=[])
        inside = torch.arange(n, device=device)     # particles of this level's cells
        nodes = 0
        for level in range(self.LEVELS + 1):
            prefix = code[inside] >> (3 * (self.LEVELS - level))
            _, owner, count = torch.unique_consecutive(prefix, return_inverse=True,
                                                       return_counts=True)
            cells = count.numel()
            first = inside[torch.cumsum(count, 0) - count]
            mi, xi = self.m[inside], self.x[inside]
            mass = torch.zeros(cells, dtype=x.dtype, device=device).index_add_(0, owner, mi)
            com = torch.zeros(cells, 3, dtype=x.dtype, device=device).index_add_(
                0, owner, xi * mi[:, None]) / mass[:, None]
            size = edge / 2.0 ** level
            corner = torch.floor((self.x[first] - (centre - edge / 2.0)) / size).clamp(
                0, 2 ** level - 1)
            middle = (centre - edge / 2.0) + (corner + 0.5) * size
            radius = size / angle + (com - middle).norm(dim=1)
            quad = torch.zeros(cells, 6, dtype=x.dtype, device=device)
            if quadrupole:
                d = xi - com[owner]
                trace = (d * d).sum(1)
                terms = torch.stack([3 * d[:, 0] ** 2 - trace, 3 * d[:, 0] * d[:, 1],
                                     3 * d[:, 0] * d[:, 2], 3 * d[:, 1] ** 2 - trace,
                                     3 * d[:, 1] * d[:, 2], 3 * d[:, 2] ** 2 - trace], 1)
                quad.index_add_(0, owner, terms * mi[:, None])
            split = (count > leaf) & (level < self.LEVELS)
            # A split cell's children follow those of the split cells before it.
            inner = split[owner]
            inside = inside[inner]
            kids = torch.zeros(cells, dtype=torch.long, device=device)
            if inside.numel():
                finer = code[inside] >> (3 * (self.LEVELS - level - 1))
                new = torch.ones_like(finer, dtype=torch.bool)
                new[1:] = finer[1:] != finer[:-1]
                kids.index_add_(0, owner[inner], new.long())
            base = nodes + cells
            for key, value in (("first", first), ("count", torch.where(split, 0, count)),
                               ("com", com), ("mass", mass), ("r2", radius * radius),
                               ("quad", quad), ("kids", kids),
                               ("child", base + torch.cumsum(kids, 0) - kids)):
                parts[key].append(value)
            nodes = base
            if not inside.numel():
                break
        for key, value in parts.items():
            setattr(self, key, torch.cat(value))
        self.quadrupole = quadrupole

    @staticmethod
    def _expand(who, first, count):
        """Every (who, first + k) for k below count."""
        owner = torch.repeat_interleave(torch.arange(who.numel(), device=who.device), count)
        k = torch.arange(owner.numel(), device=who.device) - (torch.cumsum(count, 0) - count)[owner]
        return who[owner], first[owner] + k

    def forces(self, eps2, chunk=8192):
        out = torch.zeros_like(self.x)
        device = self.x.device
        n = self.x.shape[0]
        for at in range(0, n, chunk):
            target = torch.arange(at, min(n, at + chunk), device=device)
            node = torch.zeros_like(target)
            while target.numel():
                d = self.com[node] - self.x[target]
                d2 = (d * d).sum(1)
                take = d2 >= self.r2[node]
                self._cells(out, target[take], node[take], d[take], d2[take], eps2)
                target, node = target[~take], node[~take]
                leaf = self.count[node] > 0
                self._pairs(out, target[leaf], node[leaf], eps2)
                target, node = target[~leaf], node[~leaf]
                target, node = self._expand(target, self.child[node], self.kids[node])
        back = torch.empty_like(out)
        back[self.order] = out
        return back

    def _cells(self, out, target, node, d, d2, eps2):
        inv = torch.rsqrt(d2 + eps2)
        inv2 = inv * inv
        a = d * (self.mass[node] * inv2 * inv)[:, None]
        if self.quadrupole:
            q = self.quad[node]
            qd = torch.stack([q[:, 0] * d[:, 0] + q[:, 1] * d[:, 1] + q[:, 2] * d[:, 2],
                              q[:, 1] * d[:, 0] + q[:, 3] * d[:, 1] + q[:, 4] * d[:, 2],
                              q[:, 2] * d[:, 0] + q[:, 4] * d[:, 1] + q[:, 5] * d[:, 2]], 1)
            inv5 = inv2 * inv2 * inv
            a = a - qd * inv5[:, None] + d * (2.5 * (d * qd).sum(1) * inv5 * inv2)[:, None]
        out.index_add_(0, target, a)

    def _pairs(self, out, target, node, eps2):
        step = 1 << 20
        for at in range(0, target.numel(), step):
            t, v = target[at:at + step], node[at:at + step]
            i, j = self._expand(t, self.first[v], self.count[v])
            keep = i != j
            i, j = i[keep], j[keep]
            d = self.x[j] - self.x[i]
            inv = torch.rsqrt((d * d).sum(1) + eps2)
            out.index_add_(0, i, d * (self.m[j] * inv ** 3)[:, None])


def _field(case):
    """x, m -> accelerations in 64 bits."""
    eps2 = case["softening"] * case["softening"]
    if case["solver"] == "direct":
        return lambda x, m: _direct(x, m, eps2)
    return lambda x, m: _Tree(x, m, case["angle"], case["leaf"], case["quadrupole"]).forces(eps2)


def _integrate(case, field, x, v, m):
    """The integrator's steps; x, v, a after them as nine columns."""
    outer = 1.0 / (2.0 - 2.0 ** (1.0 / 3.0))
    weights = [outer, 1.0 - 2.0 * outer, outer] if case["integrator"] == "yoshida4" else [1.0]
    a = field(x, m)
    for _ in range(case["steps"]):
        for w in weights:
            v = v + (0.5 * w * DT) * a
            x = x + (w * DT) * v
            a = field(x, m)
            v = v + (0.5 * w * DT) * a
    return [_host(t[:, k]) for t in (x, v, a) for k in range(3)]


def exact(case, seed):
    kind = case["kind"]
    if work(case)["flops"] > 4e12:
        return None  # over about 20 seconds
    if kind == "batch":
        parts = []
        for eps, x, v, m in _clusters(case, seed):
            parts.append(_integrate(case, lambda p, w: _direct(p, w, eps * eps), x, v, m))
        return [np.concatenate(column) for column in zip(*parts)]
    x, v, m = _inputs(case, seed)
    if kind == "diagnostics":
        momentum = (v * m[:, None]).sum(0)
        spin = (torch.linalg.cross(x, v) * m[:, None]).sum(0)
        kinetic = 0.5 * float((m * (v * v).sum(1)).sum())
        # The momenta are zero but for rounding (the inputs are centred).
        return [kinetic, _potential(x, m, case["softening"] ** 2), None, _host(spin)]
    if kind == "steps":
        return _integrate(case, _field(case), x, v, m)
    a = _field(case)(x, m)
    return a.t().contiguous() if kind == "forces" else [_host(a[:, k]) for k in range(3)]
