"""The workloads this library's speed is measured on, and what each computes.

A case is one pass of a user's program over the public Python entry points:
load a state into a world, advance it a few steps, read the state back (WCSPH
in both precisions and batched, PBF, DFSPH), or evaluate or differentiate the
learned surrogate on a particle graph. Scenes are dam breaks: a jittered
lattice block, set in motion, in a one-layer boundary shell. `exact` restates
each solver in 64-bit torch from its equations.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "physics-engine_b200"))
import physics_engine_rs as pe  # noqa: E402
from physics_engine_rs.surrogate import Surrogate  # noqa: E402

DX = 0.01
RHO0, C0, GAMMA, ALPHA, VISC_EPS, XSPH, GRAVITY = 1000.0, 20.0, 7.0, 0.01, 0.01, 0.25, 9.81
DT, SOLVER_DT = 1e-4, 1e-3
CUBIC, WENDLAND, POLY6, SPIKY = 0, 1, 2, 3
WIDTH = 128


def _wcsph(name, n, box, steps=20, precision="f64", kernel=CUBIC, visc_beta=0.0, h_over_dx=2.0, tanks=1, graph=False):
    return {"name": name, "form": "wcsph", "dim": 3 if n[2] > 1 else 2, "nx": n[0], "ny": n[1], "nz": n[2],
            "bx": box[0], "by": box[1], "bz": box[2], "steps": steps, "precision": precision, "kernel": kernel,
            "visc_beta": visc_beta, "h_over_dx": h_over_dx, "tanks": tanks, "graph": graph}


def _solver(name, form, n, box, steps):
    return {"name": name, "form": form, "dim": 3, "nx": n[0], "ny": n[1], "nz": n[2], "bx": box[0], "by": box[1],
            "bz": box[2], "steps": steps, "h_over_dx": 2.0, "tanks": 1}


def _net(name, form, n):
    return {"name": name, "form": form, "nx": n[0], "ny": n[1], "nz": n[2]}


def listed():
    return [
        # The smallest world: 256 fluid particles in a shell, 20 steps, h = 2.2 dx (the shape of the
        # fluid crate's own WCSPH benchmark). Launches and their gaps are all there is.
        _wcsph("wcsph tiny", (8, 8, 4), (12, 12, 8), h_over_dx=2.2, graph=True),
        # A 2-D tank, as used for validation against shallow-water and sloshing solutions.
        _wcsph("wcsph 2d", (160, 100, 1), (400, 160, 1)),
        # The 32^3 dam break of the parity runs: an interactive-size scene.
        _wcsph("wcsph 32k", (32, 32, 32), (100, 40, 60)),
        # A mid-size tank with odd extents, another kernel and both viscosity terms.
        _wcsph("wcsph 152k wendland", (61, 47, 53), (199, 77, 101), kernel=WENDLAND, visc_beta=0.02),
        # The flagship: the 1M-particle dam break.
        _wcsph("wcsph 1m", (100, 100, 100), (400, 160, 240), steps=10),
        # The single-precision form at an interactive size with odd extents, and at 1M.
        _wcsph("wcsph f32 60k", (41, 39, 37), (127, 63, 79), precision="f32"),
        _wcsph("wcsph f32 1m", (100, 100, 100), (400, 160, 240), steps=10, precision="f32"),
        # Many independent tanks of uneven size in one world (parameter sweeps, training data).
        _wcsph("wcsph 24 tanks", (40, 36, 34), (100, 70, 70), steps=12, tanks=24, graph=True),
        # The sibling solvers on a mid-size tank.
        _solver("pbf 64k", "pbf", (40, 40, 40), (120, 60, 80), 10),
        _solver("dfsph 46k", "dfsph", (37, 35, 36), (110, 60, 80), 5),
        # The learned surrogate's inference and one training step's loss and gradients, on a tank's graph.
        _net("surrogate forward", "forward", (48, 48, 44)),
        _net("surrogate gradients", "gradients", (25, 23, 24)),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _block(rng, count):
    """A lattice of about `count` points whose sides differ by at most a factor of about two."""
    a, b = rng.uniform(0.7, 1.4), rng.uniform(0.7, 1.4)
    side = count ** (1.0 / 3.0)
    return tuple(max(3, int(round(s))) for s in (side * a, side * b, side / (a * b)))


def draw(rng):
    kind = rng.choice(("wcsph", "wcsph", "wcsph", "f32", "f32", "2d", "tanks", "pbf", "dfsph", "forward", "gradients"))
    steps = rng.randint(6, 20)
    if kind == "2d":
        n = _log_uniform(rng, 500, 60000)
        a = rng.uniform(0.6, 1.8)
        nx, ny = int(math.sqrt(n) * a) + 3, int(math.sqrt(n) / a) + 3
        c = _wcsph("", (nx, ny, 1), (int(nx * rng.uniform(1.3, 3.0)) + 3, ny + rng.randint(3, 60), 1), steps)
    elif kind in ("wcsph", "f32"):
        n = _block(rng, _log_uniform(rng, 200, 400000))
        box = tuple(int(k * rng.uniform(1.1, f)) + 3 for k, f in zip(n, (3.5, 1.6, 2.0)))
        f32 = kind == "f32"
        c = _wcsph("", n, box, min(steps, 10) if n[0] * n[1] * n[2] > 100000 else steps, "f32" if f32 else "f64",
                   CUBIC if f32 else rng.choice((CUBIC, CUBIC, WENDLAND)), rng.choice((0.0, 0.0, 0.02)),
                   rng.choice((2.0, 2.0, 2.2)), graph=rng.random() < 0.3)
    elif kind == "tanks":
        t = rng.randint(3, 40)
        n = _block(rng, _log_uniform(rng, 2048, 600000 / t))
        c = _wcsph("", n, tuple(int(k * rng.uniform(1.2, 2.0)) + 3 for k in n), min(steps, 10),
                   rng.choice(("f64", "f32")), tanks=t, graph=True)
    elif kind in ("pbf", "dfsph"):
        n = _block(rng, _log_uniform(rng, 1000, 100000 if kind == "pbf" else 50000))
        c = _solver("", kind, n, tuple(int(k * rng.uniform(1.2, 2.5)) + 6 for k in n), rng.randint(2, 6))
    else:
        c = _net("", kind, _block(rng, _log_uniform(rng, 1000, 90000 if kind == "forward" else 15000)))
    del c["name"]
    return c


# ---------------------------------------------------------------------------
# Scenes
# ---------------------------------------------------------------------------
def _tank_blocks(case):
    """The fluid lattice of each tank: the case's block, smaller from tank to tank when there are several."""
    n = (case["nx"], case["ny"], case["nz"])
    return [tuple(max(3, k - (t * 7 + a) % max(1, k // 3)) for a, k in enumerate(n)) if case["tanks"] > 1 else n
            for t in range(case["tanks"])]


def _origin(case):
    """The block starts one spacing off the walls, two for the position-based and divergence-free solvers."""
    o = DX if case["form"] == "wcsph" else 2.0 * DX
    return np.array([o, o, o if case["dim"] == 3 else 0.0])


def _box(case):
    return np.array([case["bx"], case["by"], case["bz"] if case["dim"] == 3 else 0]) * DX


def _shell(case):
    """The one-layer boundary shell in `fill_box_boundary`'s order: pairs of opposite face points."""
    hi = _box(case)
    x, y, z = (np.arange(int(round(e / DX)) + 1) * DX for e in hi)

    def faces(axes, points, across):
        grid = np.stack(np.meshgrid(*points, indexing="ij"), -1).reshape(-1, len(points))
        p = np.zeros((len(grid), 2, 3))
        p[:, :, axes] = grid[:, None]
        p[:, 1, across] = hi[across]
        return p.reshape(-1, 3)

    if case["dim"] == 2:
        return np.concatenate([faces([0], [x], 1), faces([1], [y[1:-1]], 0)])
    return np.concatenate([faces([0, 1], [x, y], 2), faces([0, 2], [x, z[1:-1]], 1),
                           faces([1, 2], [y[1:-1], z[1:-1]], 0)])


def _scene(case, seed):
    """Positions, velocities, kinds (0 fluid, 1 boundary) and tank numbers, in the builders' order."""
    rng = np.random.default_rng(seed)
    shell, o, dim = _shell(case), _origin(case), case["dim"]
    xs, vs, kinds, tanks = [], [], [], []
    for t, (nx, ny, nz) in enumerate(_tank_blocks(case)):
        iz, iy, ix = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
        f = o + np.stack([ix, iy, iz], -1).reshape(-1, 3) * DX
        jitter, noise = rng.uniform(-1e-4, 1e-4, f.shape), rng.normal(0.0, 0.02, f.shape)
        drift = rng.uniform(-0.2, 0.2, 3)
        if dim == 2:
            jitter[:, 2], noise[:, 2], drift[2] = 0.0, 0.0, 0.0
        xs += [f + jitter, shell]
        vs += [drift + noise, np.zeros_like(shell)]
        kinds += [np.zeros(len(f), np.uint8), np.ones(len(shell), np.uint8)]
        tanks.append(np.full(len(f) + len(shell), t))
    return np.concatenate(xs), np.concatenate(vs), np.concatenate(kinds), np.concatenate(tanks)


def _gravity(case):
    return (0.0, 0.0, -GRAVITY) if case["dim"] == 3 else (0.0, -GRAVITY, 0.0)


def _particles(case):
    h = case["h_over_dx"] * DX
    if case["form"] == "dfsph":
        mass = pe.mass_calibrated_to_rest(RHO0, DX, h, case["dim"])
    else:
        mass = pe.mass_from_spacing(RHO0, DX, case["dim"])
    parts = []
    for n in _tank_blocks(case):
        p = pe.Particles(case["dim"], RHO0, mass, h)
        p.fill_box(_origin(case), *n, DX)
        p.fill_box_boundary((0.0, 0.0, 0.0), _box(case), DX, 1)
        parts.append(p)
    return parts


# The network's layers: (name, inputs, outputs, has a bias).
def _mlp(name, k, n):
    return [(name + ".0", k, WIDTH, True), (name + ".1", WIDTH, WIDTH, True), (name + ".2", WIDTH, n, True)]


LAYERS = _mlp("enc", 8, WIDTH)
for _hop in ("hop1", "hop2"):
    LAYERS += [(_hop + ".edge.a", WIDTH, WIDTH, False), (_hop + ".edge.b", WIDTH, WIDTH, False),
               (_hop + ".edge.0", 16, WIDTH, True), (_hop + ".edge.1", WIDTH, WIDTH, True),
               (_hop + ".edge.2", WIDTH, WIDTH, True)] + _mlp(_hop + ".node", 2 * WIDTH, WIDTH)
LAYERS += _mlp("dec", WIDTH, 4)


def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _graph(case, seed):
    """A tank's message graph (edges within h = 2 dx, grouped by destination), its features (values a
    bfloat16 holds), weights and targets."""
    dev = _device()
    g = torch.Generator(device="cpu").manual_seed(seed)
    n = (case["nx"], case["ny"], case["nz"])
    k = torch.stack(torch.meshgrid(*[torch.arange(m) for m in n], indexing="ij"), -1).reshape(-1, 3).to(dev)
    x = k * DX + ((torch.rand(k.shape, generator=g, dtype=torch.float64) - 0.5) * 2e-3).to(dev)
    # the outermost lattice layer stands for boundary samples: they send messages and receive none
    top = torch.tensor(n, device=dev) - 1
    fluid = ((k > 0) & (k < top)).all(1)
    dst, src = [], []
    index = (k[:, 0] * n[1] + k[:, 1]) * n[2] + k[:, 2]
    for a in range(-2, 3):
        for b in range(-2, 3):
            for c in range(-2, 3):
                if (a, b, c) == (0, 0, 0):
                    continue
                q = k + torch.tensor([a, b, c], device=dev)
                ok = fluid & ((q >= 0) & (q <= top)).all(1)
                j = (index + (a * n[1] + b) * n[2] + c)[ok]
                i = index[ok]
                near = ((x[j] - x[i]) ** 2).sum(1) <= (2.0 * DX) ** 2
                dst.append(i[near])
                src.append(j[near])
    dst, src = torch.cat(dst), torch.cat(src)
    by = torch.argsort(dst * len(x) + src)
    dst, src = dst[by], src[by]
    v = (0.1 * torch.randn(k.shape, generator=g, dtype=torch.float64)).to(dev)
    rho = (0.2 * torch.randn(len(x), generator=g, dtype=torch.float64)).to(dev)
    p = 0.7 * rho
    bnd = (~fluid).double()
    f = torch.stack([v[:, 0], v[:, 1], v[:, 2], rho, p, bnd, 0 * rho, 0 * rho], 1)
    r = (x[src] - x[dst]) / (2.0 * DX)
    w = v[src] - v[dst]
    xe = torch.cat([r, r.norm(dim=1, keepdim=True), w, rho[dst, None], rho[src, None], p[dst, None], p[src, None],
                    bnd[src, None], torch.zeros(len(src), 4, device=dev, dtype=torch.float64)], 1)
    row = torch.zeros(len(x) + 1, dtype=torch.int64, device=dev)
    row[1:] = torch.cumsum(torch.bincount(dst, minlength=len(x)), 0)
    target = torch.randn(len(x), 4, generator=g).to(dev) * fluid[:, None]
    params = {}
    for name, kin, out, bias in LAYERS:
        sd = math.sqrt(2.0 / kin) * (0.3 if name == "dec.2" else 1.0)
        params[name + ".W"] = (sd * torch.randn(kin, out, generator=g)).bfloat16().float()
        if bias:
            params[name + ".b"] = 0.05 * torch.randn(out, generator=g)
    return {"f": f.bfloat16().float(), "xe": xe.bfloat16().float(), "dst": dst, "src": src, "row": row,
            "fluid": fluid, "target": target, "params": params}


# ---------------------------------------------------------------------------
# The measured path
# ---------------------------------------------------------------------------
def prepare(case, seed):
    if case["form"] in ("forward", "gradients"):
        g = _graph(case, seed)
        net = Surrogate(seed=1)
        net.set_params({k: v.numpy() for k, v in g["params"].items()})
        net.set_graph(*(g[k].cpu().numpy() for k in ("f", "xe", "row", "src", "fluid")))
        if case["form"] == "gradients":
            net.set_targets(g["target"].cpu().numpy())
        return {"case": case, "net": net}
    x, v, _, _ = _scene(case, seed)
    parts = _particles(case)
    g = _gravity(case)
    if case["form"] == "wcsph":
        prm = pe.WcsphParams.water(RHO0, C0, g)
        prm.adapt_sound_speed = False
        prm.density_kernel, prm.visc_beta = case["kernel"], case["visc_beta"]
        f32 = case["precision"] == "f32"
        cfg = pe.WcsphConfig(precision=pe.PRECISION_F32 if f32 else pe.PRECISION_F64, use_graph=case["graph"])
        world = pe.WcsphWorld.from_tanks(prm, parts, cfg) if case["tanks"] > 1 else pe.WcsphWorld(parts[0], prm, cfg)
    elif case["form"] == "pbf":
        world = pe.PbfWorld(parts[0], pe.PbfParams(gravity=g, iterations=4, epsilon_lambda=0.01, art_pressure_k=0.0,
                                                   viscosity_eps=0.01, vorticity_eps=0.0))
    else:
        parts[0].recomputed_akinci_psi()
        world = pe.DfsphWorld(parts[0], pe.DfsphParams(
            gravity=g, particle_diameter=DX, density_error_tol=0.01, divergence_error_tol=0.01, max_density_iters=8,
            max_divergence_iters=8, xsph_epsilon=0.05, adaptive_dt=False, warm_start=True, solver_omega=1.0,
            max_velocity_correction=0.5))
    return {"case": case, "world": world, "x": x, "v": v}


def run(state):
    case = state["case"]
    if case["form"] == "forward":
        return state["net"].forward()
    if case["form"] == "gradients":
        loss = state["net"].train_step(0.0)
        return {"loss": loss, "gradients": state["net"].get_params(grads=True)}
    world = state["world"]
    world.set_positions(state["x"])
    world.set_velocities(state["v"])
    if case["form"] == "dfsph":
        world.rebuild_neighbours()
        world.compute_density()
        world.compute_alpha()
    world.run(DT if case["form"] == "wcsph" else SOLVER_DT, case["steps"])
    return {"x": world.positions(), "v": world.velocities(), "rho": world.densities()}


def _counts(case):
    fluid = sum(a * b * c for a, b, c in _tank_blocks(case))
    return fluid, len(_shell(case)) * case["tanks"]


def work(case):
    """Bytes: per step the state each pass has to read and write once (252 bytes a fluid and 108 a boundary
    particle for WCSPH in 64 bits, half of it in 32; the solvers' passes likewise), and the state in and out.
    Operations: those of the pairs inside the support."""
    if case["form"] in ("forward", "gradients"):
        n = case["nx"] * case["ny"] * case["nz"]
        inner = (case["nx"] - 2) * (case["ny"] - 2) * (case["nz"] - 2)
        edges = 32 * inner
        flops = edges * 2 * 2 * (16 * 128 + 2 * 128 * 128) + n * 2 * (10 * 128 * 128 + 2 * 5 * 128 * 128)
        nbytes = n * (16 + 16 + 1) + edges * (32 + 4)
        weights = 4 * sum(k * o + o for _, k, o, _ in LAYERS)
        return {"bytes": nbytes + (2 if case["form"] == "gradients" else 1) * weights,
                "flops": flops * (3 if case["form"] == "gradients" else 1)}
    nf, nb = _counts(case)
    size = 4 if case.get("precision") == "f32" else 8
    ratio = case["h_over_dx"]
    io = (nf + nb) * 8 * 13
    if case["form"] == "pbf":  # support h: lists once, 4 iterations of density, lambda and correction; density, viscosity
        pairs, per_step, ops = 4.19 * ratio ** 3, 4 * 200 + 300, 4 * 90 + 50
    elif case["form"] == "dfsph":  # support 2h: XSPH, density, alpha, at least 3 iterations and 2 warm starts
        pairs, per_step, ops = 33.5 * ratio ** 3, 400 + 5 * 150, 100 + 3 * 90 + 2 * 45
    else:
        pairs = 33.5 * ratio ** 3 if case["dim"] == 3 else 12.6 * ratio ** 2
        per_step, ops = 252 * size / 8, 114
    return {"bytes": io + case["steps"] * (nf * per_step + nb * 108 * size / 8),
            "flops": case["steps"] * nf * pairs * ops}


# ---------------------------------------------------------------------------
# The same in 64-bit torch
# ---------------------------------------------------------------------------
def _support(kernel, h):
    return 2.0 * h if kernel in (CUBIC, WENDLAND) else h


def _kernel(kernel, h, dim):
    """W(r) and dW/dr."""
    pi = math.pi
    if kernel == CUBIC:
        a = 10 / (7 * pi * h ** 2) if dim == 2 else 1 / (pi * h ** 3)

        def w(r):
            q = r / h
            return a * torch.where(q < 1, 1 - 1.5 * q * q + 0.75 * q ** 3, 0.25 * (2 - q).clamp(min=0) ** 3)

        def dw(r):
            q = r / h
            return a / h * torch.where(q < 1, -3 * q + 2.25 * q * q, -0.75 * (2 - q).clamp(min=0) ** 2)
    elif kernel == WENDLAND:
        a = 7 / (4 * pi * h ** 2) if dim == 2 else 21 / (16 * pi * h ** 3)

        def w(r):
            return a * (1 - 0.5 * r / h).clamp(min=0) ** 4 * (2 * r / h + 1)

        def dw(r):
            return a / h * -5 * (r / h) * (1 - 0.5 * r / h).clamp(min=0) ** 3
    elif kernel == POLY6:
        a = 4 / (pi * h ** 8) if dim == 2 else 315 / (64 * pi * h ** 9)

        def w(r):
            return a * (h * h - r * r).clamp(min=0) ** 3

        def dw(r):
            return -6 * a * r * (h * h - r * r).clamp(min=0) ** 2
    else:
        a = 10 / (pi * h ** 5) if dim == 2 else 15 / (pi * h ** 6)

        def w(r):
            return a * (h - r).clamp(min=0) ** 3

        def dw(r):
            return -3 * a * (h - r).clamp(min=0) ** 2
    return w, dw


class _Pairs:
    """Ordered pairs (i, j != i) with i from `centres`, of points in the same or adjacent grid cells of the
    same tank, closer than the cell unless `all_candidates`."""

    def __init__(self, x, tank, centres, cell, dim, all_candidates=False):
        key = torch.floor(x / cell).long()
        if dim == 2:
            key[:, 2] = 0
        key = key - key.min(0).values + 1
        ext = key.max(0).values + 2
        stride = torch.stack([ext[1] * ext[2], ext[2], torch.ones_like(ext[2])])
        cid = (key * stride).sum(1) + tank * ext.prod()
        order = torch.argsort(cid)
        count = torch.bincount(cid, minlength=int(ext.prod()) * (int(tank.max()) + 1) + 1)
        start = torch.cumsum(count, 0) - count
        out_i, out_j = [], []
        for dx in (-1, 0, 1):
            for dy in (-1, 0, 1):
                for dz in (-1, 0, 1) if dim == 3 else (0,):
                    c = cid[centres] + dx * stride[0] + dy * stride[1] + dz
                    k = count[c]
                    i = torch.repeat_interleave(centres, k)
                    at = torch.arange(len(i), device=x.device) - torch.repeat_interleave(torch.cumsum(k, 0) - k, k)
                    j = order[torch.repeat_interleave(start[c], k) + at]
                    keep = i != j
                    if not all_candidates:
                        keep &= ((x[j] - x[i]) ** 2).sum(1) < (cell * (1 + 1e-9)) ** 2
                    out_i.append(i[keep])
                    out_j.append(j[keep])
        self.i, self.j, self.n = torch.cat(out_i), torch.cat(out_j), len(x)

    def geometry(self, x):
        self.d = x[self.j] - x[self.i]
        self.r = self.d.norm(dim=1)
        return self

    def grad(self, dw):
        """grad_i W of every pair."""
        s = torch.where(self.r < 1e-30, 0.0, -dw(self.r) / self.r.clamp(min=1e-30))
        return self.d * s[:, None]

    def sum(self, t):
        return torch.zeros((self.n,) + t.shape[1:], dtype=t.dtype, device=t.device).index_add_(0, self.i, t)


def _exact_wcsph(case, x, v, kind, tank):
    dim, h, beta = case["dim"], case["h_over_dx"] * DX, case["visc_beta"]
    w, dw = _kernel(case["kernel"], h, dim)
    mass, psi = RHO0 * DX ** dim, DX ** dim
    fluid = kind == 0
    centres = torch.nonzero(fluid)[:, 0]
    g = torch.tensor(_gravity(case), dtype=torch.float64, device=x.device)
    share = mass * fluid.double() + RHO0 * psi * (~fluid).double()

    def neighbours(x):
        return _Pairs(x, tank, centres, _support(case["kernel"], h), dim).geometry(x)

    def density(q):
        rho = mass * w(torch.zeros(1, dtype=torch.float64, device=x.device)) + q.sum(share[q.j] * w(q.r))
        return torch.where(fluid, rho, RHO0)

    q = neighbours(x)
    rho = density(q)
    for _ in range(case["steps"]):
        p = RHO0 * C0 * C0 / GAMMA * ((rho / RHO0) ** GAMMA - 1)
        pr = torch.where(fluid, p / rho ** 2, 0.0)
        vr = -((v[q.i] - v[q.j]) * q.d).sum(1)
        mu = h * vr / (q.r ** 2 + VISC_EPS * h * h)
        visc = (-ALPHA * C0 * mu + beta * mu * mu) / (0.5 * (rho[q.i] + rho[q.j]))
        coef = -share[q.j] * (pr[q.i] + pr[q.j] + torch.where((vr < 0) & fluid[q.j], visc, 0.0))
        a = q.sum(q.grad(dw) * coef[:, None])
        v = torch.where(fluid[:, None], v + (a + g) * DT, v)
        x = torch.where(fluid[:, None], x + v * DT, x)
        q = neighbours(x)
        rho = density(q)
        f = torch.where(fluid[q.j], mass / (0.5 * (rho[q.i] + rho[q.j])) * w(q.r), 0.0)
        v = v + XSPH * q.sum((v[q.j] - v[q.i]) * f[:, None])
    return x, v, rho


def _exact_pbf(case, x, v, kind, tank):
    dim, h, dt = case["dim"], case["h_over_dx"] * DX, SOLVER_DT
    w, _ = _kernel(POLY6, h, dim)
    _, dw = _kernel(SPIKY, h, dim)
    mass, psi = RHO0 * DX ** dim, DX ** dim
    fluid = kind == 0
    centres = torch.nonzero(fluid)[:, 0]
    g = torch.tensor(_gravity(case), dtype=torch.float64, device=x.device)
    share = mass / RHO0 * fluid.double() + psi * (~fluid).double()

    def density(q):
        rho = mass * w(torch.zeros(1, dtype=torch.float64, device=x.device)) + q.sum(RHO0 * share[q.j] * w(q.r))
        return torch.where(fluid, rho, RHO0)

    for _ in range(case["steps"]):
        v = torch.where(fluid[:, None], v + g * dt, v)
        new = torch.where(fluid[:, None], x + v * dt, x)
        q = _Pairs(new, tank, centres, h, dim, all_candidates=True)
        for _ in range(4):
            q.geometry(new)
            c = q.grad(dw) * share[q.j][:, None]
            total = q.sum(c)
            squares = q.sum(torch.where(fluid[q.j], (c * c).sum(1), 0.0)) + (total * total).sum(1)
            lam = torch.where(fluid, -(density(q) / RHO0 - 1) / (squares + 0.01), 0.0)
            dp = q.sum(c * (lam[q.i] + lam[q.j])[:, None])
            size = dp.norm(dim=1, keepdim=True)
            new = new + torch.where(size > 0.4 * h, dp * (0.4 * h / size.clamp(min=1e-300)), dp)
        v = torch.where(fluid[:, None], (new - x) / dt, v)
        x = new
        q = _Pairs(x, tank, centres, h, dim).geometry(x)
        rho = density(q)
        f = torch.where(fluid[q.j], mass / (0.5 * (rho[q.i] + rho[q.j])) * w(q.r), 0.0)
        v = v + 0.01 * q.sum((v[q.j] - v[q.i]) * f[:, None])
    return x, v, rho


def _exact_dfsph(case, x, v, kind, tank):
    dim, h, dt = case["dim"], case["h_over_dx"] * DX, SOLVER_DT
    w, dw = _kernel(CUBIC, h, dim)
    w0 = float(w(torch.zeros(1, dtype=torch.float64)))
    k = torch.arange(-5, 6, dtype=torch.float64) * DX
    r = torch.stack(torch.meshgrid(k, k, k, indexing="ij"), -1).norm(dim=-1)
    mass = RHO0 / float(w(r).sum())  # the lattice sums to the rest density
    fluid = kind == 0
    centres, walls = torch.nonzero(fluid)[:, 0], torch.nonzero(~fluid)[:, 0]
    b = _Pairs(x[walls], tank[walls], torch.arange(len(walls), device=x.device), 2 * h, dim).geometry(x[walls])
    share = torch.full_like(x[:, 0], mass)
    share[walls] = RHO0 / (w0 + b.sum(w(b.r)))
    n_fluid = len(centres)
    floor = max(1e-6 * (mass / h ** 4) ** 2, 1e-12)

    def state(x):
        q = _Pairs(x, tank, centres, 2 * h, dim).geometry(x)
        rho = torch.where(fluid, mass * w0 + q.sum(share[q.j] * w(q.r)), RHO0)
        q.mg = q.grad(dw) * share[q.j][:, None]
        total = q.sum(q.mg)
        squares = (total * total).sum(1) + q.sum((q.mg * q.mg).sum(1))
        return q, rho, torch.where(fluid, rho / squares.clamp(min=floor), 0.0)

    def push(q, v, rho, kappa):
        kr = torch.where(fluid, kappa / rho, 0.0)
        dv = -dt * q.sum(q.mg * (kr[q.i] + kr[q.j])[:, None])
        size = dv.norm(dim=1, keepdim=True)
        return v + torch.where(size > 0.5, dv * (0.5 / size.clamp(min=1e-300)), dv)

    def solve(q, v, rho, alpha, warm, divergence):
        v = push(q, v, rho, warm)
        warm = torch.zeros_like(warm)
        for it in range(1, 9):
            rate = q.sum(((v[q.i] - v[q.j]) * q.mg).sum(1))
            err = torch.where(fluid, (rate if divergence else rho + dt * rate - RHO0).clamp(min=0), 0.0)
            kappa = err * alpha * (1 / dt if divergence else 1 / dt ** 2)
            warm = warm + kappa
            v = push(q, v, rho, kappa)
            if float(err.sum()) / RHO0 / n_fluid <= 0.01 and it >= (1 if divergence else 2):
                break
        return v, warm

    g = torch.tensor(_gravity(case), dtype=torch.float64, device=x.device)
    warm_rho, warm_div = torch.zeros_like(x[:, 0]), torch.zeros_like(x[:, 0])
    q, rho, alpha = state(x)
    for _ in range(case["steps"]):
        v = torch.where(fluid[:, None], v + g * dt, v)
        f = torch.where(fluid[q.j], mass / (0.5 * (rho[q.i] + rho[q.j])) * w(q.r), 0.0)
        v = v + 0.05 * q.sum((v[q.j] - v[q.i]) * f[:, None])
        v, warm_rho = solve(q, v, rho, alpha, warm_rho, False)
        x = torch.where(fluid[:, None], x + v * dt, x)
        q, rho, alpha = state(x)
        v, warm_div = solve(q, v, rho, alpha, warm_div, True)
    return x, v, rho


def _exact_net(case, seed):
    g = _graph(case, seed)
    dev = g["f"].device
    p = {k: v.to(dev).double() for k, v in g["params"].items()}
    train = case["form"] == "gradients"
    for t in p.values():
        t.requires_grad_(train)
    f, xe, dst, src, fluid = g["f"].double(), g["xe"].double(), g["dst"], g["src"], g["fluid"].double()[:, None]

    def linear(name, x):
        y = x @ p[name + ".W"]
        return y + p[name + ".b"] if name + ".b" in p else y

    def mlp(name, x):
        return linear(name + ".2", torch.relu(linear(name + ".1", torch.relu(linear(name + ".0", x)))))

    def messages(hop, h):
        a, b = linear(hop + ".edge.a", h), linear(hop + ".edge.b", h)
        total = torch.zeros_like(h)
        for part in torch.arange(len(dst), device=dev).split(len(dst) if train else 1 << 20):
            z = torch.relu(a[dst[part]] + b[src[part]] + linear(hop + ".edge.0", xe[part]))
            m = linear(hop + ".edge.2", torch.relu(linear(hop + ".edge.1", z)))
            total = total.index_add(0, dst[part], m)
        return total

    with torch.set_grad_enabled(train):
        h = mlp("enc", f)
        for hop in ("hop1", "hop2"):
            h = h + fluid * mlp(hop + ".node", torch.cat([h, messages(hop, h) / 16.0], 1))
        y = mlp("dec", h)
        if not train:
            return y.cpu().numpy()
        loss = (((y - g["target"].double()) * fluid) ** 2).sum() / fluid.sum()
        loss.backward()
    return {"loss": float(loss), "gradients": {k: t.grad.cpu().numpy() for k, t in p.items()}}


def exact(case, seed):
    if case["form"] in ("forward", "gradients"):
        return _exact_net(case, seed)
    dev = _device()
    x, v, kind, tank = (torch.from_numpy(a).to(dev) for a in _scene(case, seed))
    form = {"wcsph": _exact_wcsph, "pbf": _exact_pbf, "dfsph": _exact_dfsph}[case["form"]]
    x, v, rho = form(case, x, v, kind, tank)
    return {"x": x.cpu().numpy(), "v": v.cpu().numpy(), "rho": rho.cpu().numpy()}
