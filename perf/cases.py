"""Performance cases of the PF-FLIP framework: the work its users have it do.

Four kinds of work, each through the public entry points of ``pfflip``:

* ``step``   load a particle state into a ``Simulator``, advance it by a few
  steps of fixed dt, read the particles back (device tensors throughout);
* ``solve``  ``MGPCG.build_hierarchy`` + ``MGPCG.solve``, the standalone
  variable-coefficient pressure solve;
* ``grad``   ``DiffSim.rollout`` and the gradient of a linear functional of the
  final particles with respect to the initial ones (forward + backward);
* ``phase``  ``DiffSim.phase_field`` and its gradient.

``exact`` restates the same mathematics in plain binary64 torch, without this
repository's code.
"""

import math
import os
import sys

import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "implementation-of-adaptive-phase-field-flip_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

DEV = "cuda:0"
G = 9.81


# ------------------------------------------------------------------ the cases
def listed():
    def step(name, res, ppc, scene, steps, **more):
        c = {"name": name, "kind": "step", "nx": res[0], "ny": res[1], "nz": res[2], "dx": 1.0 / max(res), "ppc": ppc,
             "scene": scene, "steps": steps, "tol": 1e-4, "k_div": 0.0, "droplets": False, "precision": "fp32"}
        return {**c, **more}

    def solve(name, res, tol, precision="fp32", stencil="flux"):
        return {"name": name, "kind": "solve", "nx": res[0], "ny": res[1], "nz": res[2], "tol": tol,
                "precision": precision, "stencil": stencil}

    def grad(name, res, steps, scene="asteroid", ppc=8):
        return {"name": name, "kind": "grad", "nx": res[0], "ny": res[1], "nz": res[2], "dx": 1.0 / max(res),
                "ppc": ppc, "scene": scene, "steps": steps, "tol": 1e-6}

    return [
        # the smallest simulations (smoke test, unit tests, parameter scans): latency and launches
        step("step_dam_16", (16, 16, 16), 8, "dam", 4),
        # a ragged grid with an obstacle and a spacing that is no power of two
        step("step_tower_ragged", (60, 44, 36), 8, "tower", 2),
        # an ordinary production step: the default Config (64^3, dx = 1, 8 ppc, droplets on)
        step("step_dam_64_droplets", (64, 64, 64), 8, "dam", 1, dx=1.0, droplets=True),
        # the headline benchmark: 128^3 / 27 ppc dam break, 56.6 M particles
        step("step_dam_128_27ppc", (128, 128, 128), 27, "dam", 2),
        # the largest: 256^3 / 8 ppc heavy-over-light, 134 M particles
        step("step_rt_256", (256, 256, 256), 8, "rt", 1),
        # pressure solves: a small grid to the production tolerance, a ragged box with the
        # 16-bit hierarchy, the 128^3 benchmark problem to 1e-6
        solve("solve_32", (32, 32, 32), 1e-4),
        solve("solve_ragged_fp16", (96, 64, 80), 1e-6, "fp16"),
        solve("solve_128", (128, 128, 128), 1e-6),
        # gradients: a unit-test size and the differentiable asteroid (one checkpoint block)
        grad("grad_24", (24, 24, 24), 2),
        grad("grad_64", (64, 64, 64), 5),
        # the loss on the phase field of the Rayleigh-Taylor gradient, 16.8 M particles
        {"name": "phase_128", "kind": "phase", "nx": 128, "ny": 128, "nz": 128, "dx": 1.0 / 128, "ppc": 8,
         "scene": "rt", "steps": 0, "tol": 1e-4},
    ]


def _size(rng, lo, hi):
    """One edge length, spread over the logarithm: multiples of 4 (the grid coarsens
    at least twice), below 22 now and then an odd one (no coarsening on that axis)."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    if n < 22 and rng.random() < 0.4:
        return max(lo, int(n) | 1)
    return max(lo, 4 * round(n / 4))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "solve", "solve", "grad", "phase"])
    top = {"step": 160, "solve": 160, "grad": 72, "phase": 128}[kind]
    nx = _size(rng, 12, top)
    if rng.random() < 0.5:
        ny = nz = nx
    else:  # a box: the other edges within a factor of two
        ny, nz = (_size(rng, max(12, nx // 2), min(top, 2 * nx)) for _ in range(2))
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz}
    if kind == "solve":
        c["precision"] = rng.choice(["fp32", "fp32", "fp16", "bf16"])
        c["stencil"] = "reference" if c["precision"] == "fp32" and max(nx, ny, nz) <= 64 and rng.random() < 0.3 else "flux"
        c["tol"] = 1e-4 if c["stencil"] == "reference" else rng.choice([1e-4, 1e-6])
        return c
    c["ppc"] = 27 if kind == "step" and rng.random() < 0.4 else 8
    c["dx"] = rng.choice([1.0 / max(nx, ny, nz), 1.0 / nx, 1.0, 0.1])
    c["scene"] = rng.choice({"step": ["dam", "pool", "rt", "tower"], "grad": ["asteroid", "rt"], "phase": ["rt", "asteroid"]}[kind])
    c["steps"] = {"step": rng.choice([1, 2, 3]), "grad": rng.choice([1, 2, 3]), "phase": 0}[kind]
    c["tol"] = 1e-6 if kind == "grad" else 1e-4
    if kind == "step":
        c["k_div"] = rng.choice([0.0, 0.0, 0.5]) if c["scene"] != "tower" else 0.0
        c["droplets"] = c["k_div"] == 0.0 and rng.random() < 0.3
        c["precision"] = rng.choice(["fp32", "fp32", "fp32", "fp16"])
        if c["droplets"]:
            c["steps"] = 1
        # no dearer than the 134 M particles of the largest listed one
        c["steps"] = max(1, min(c["steps"], 130_000_000 // _particles(c)))
    return c


def _particles(c):
    return c["nx"] * c["ny"] * c["nz"] * c["ppc"]


def work(c):
    cells = c["nx"] * c["ny"] * c["nz"]
    if c["kind"] == "solve":
        # three face arrays and b in, p out; about 25 iterations of a V-cycle (six smoothing
        # sweeps of 20 operations on 8/7 of the cells, the transfers) and the CG vectors
        return {"bytes": 20 * cells, "flops": 25 * cells * 200}
    n = _particles(c)
    if c["kind"] == "phase":
        # positions in, gradient out, phi out and its weights in; the cell weights of eight
        # nodes, and their gradients
        return {"bytes": 24 * n + 8 * cells, "flops": n * 8 * 30}
    # positions, velocities and types in, positions and velocities out; every step reads and
    # writes the state, splats 32 weights of 10 operations and takes 15 trilinear samples
    steps = c["steps"]
    w = {"bytes": 52 * n + steps * (48 * n + 60 * cells), "flops": steps * (n * (32 * 10 + 15 * 16) + 20 * cells * 200)}
    if c["kind"] == "grad":  # the same again, replayed, and the adjoint of each step
        w = {k: 3 * v for k, v in w.items()}
    return w


def tolerance(c):
    """About four times what the path shows against ``exact`` (2-norm of the worst output)."""
    if c["kind"] == "phase":  # a cell within rounding of phi = 0 or 1 has a gradient or none
        return {"rel": 6e-4, "max": 0.5}
    if c["kind"] == "solve":
        # the stopping test bounds the residual, and a stop one iteration earlier or later moves
        # the solution by its own error
        return {"rel": 5e-4 if c["tol"] > 1e-5 else 4e-5}
    if c["kind"] == "grad":
        # a particle within rounding of a cell face takes its gradient from the neighbouring cell
        return {"rel": 2e-2, "max": 0.9}
    # the pressure is solved to 1e-4; a cell within rounding of phi = 0.5 can change its phase
    return {"rel": 3e-3, "max": 0.9}


# ------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _extent(c):
    return tuple(c[k] * c["dx"] for k in ("nx", "ny", "nz"))


def _speed(c):
    return math.sqrt(2 * G * 0.6 * max(_extent(c)))


def _dt(c):
    return 0.5 * c["dx"] / _speed(c)


def _flow(X, modes):
    """A divergence-free field on the unit box (unit coordinates X), tangent to the walls."""
    (a, m), (b, n) = modes
    x, y, z = (math.pi * X[:, d] for d in range(3))
    u = a * torch.sin(m * x) * torch.cos(m * y)
    v = -a * torch.cos(m * x) * torch.sin(m * y) + b * torch.sin(n * y) * torch.cos(n * z)
    w = -b * torch.cos(n * y) * torch.sin(n * z)
    return torch.stack((u, v, w), 1)


def _liquid(scene, X):
    x, y, z = X.unbind(1)
    if scene == "dam":
        return (x < 0.4) & (y < 0.6)
    if scene == "pool":
        return y < 0.5
    if scene == "rt":  # heavy over light
        return y > 0.5 + 0.02 * (torch.cos(2 * math.pi * x) + torch.cos(2 * math.pi * z))
    if scene == "asteroid":
        return (y < 0.3) | ((x - 0.5) ** 2 + (y - 0.7) ** 2 + (z - 0.5) ** 2 < 0.01)
    return (y < 0.22) | ((x < 0.26) & (y < 0.72))  # tower: a surge towards the obstacle


def _tower(c):
    """The cylindrical obstacle of the tower scene on the cell grid (True = solid)."""
    i = (torch.arange(c["nx"], device=DEV) + 0.5) / c["nx"]
    k = (torch.arange(c["nz"], device=DEV) + 0.5) / c["nz"]
    disc = (i[:, None] - 0.62) ** 2 + (k[None, :] - 0.5) ** 2 < 0.075**2
    s = disc[:, None, :].expand(c["nx"], c["ny"], c["nz"]).clone()
    s[:, -2:, :] = False
    return s


def _state(c, seed):
    """Particles in the middle of a flow: the jittered seeding lattice (in lattice order, as
    the scenes give it) carried a cell or two by a divergence-free flow, moving with that flow
    and a little noise; types by the scene's liquid region."""
    g = _gen(seed)
    pa = round(c["ppc"] ** (1 / 3))
    res = torch.tensor([c["nx"], c["ny"], c["nz"]], device=DEV)
    site = res * pa
    n = _particles(c)
    L = torch.tensor(_extent(c), device=DEV, dtype=torch.float32)
    r = torch.rand(4, generator=g, device=DEV).tolist()
    drift = 2.0 / max(c["nx"], c["ny"], c["nz"])
    modes = ((drift * (0.5 + r[0]), 1 + int(3 * r[1])), (drift * (0.5 + r[2]), 1 + int(3 * r[3])))
    x = torch.empty((n, 3), device=DEV)
    v = torch.empty((n, 3), device=DEV)
    t = torch.empty(n, dtype=torch.int32, device=DEV)
    keep = torch.ones(n if c["scene"] == "tower" else 0, dtype=torch.bool, device=DEV)
    s1, s2 = int(site[1]), int(site[2])
    for lo in range(0, n, 1 << 24):
        e = torch.arange(lo, min(n, lo + (1 << 24)), device=DEV)
        idx = torch.stack((e // (s1 * s2), e // s2 % s1, e % s2), 1)
        X = (idx + 0.5 + 0.8 * (torch.rand(idx.shape, generator=g, device=DEV) - 0.5)) / site
        t[lo:lo + len(e)] = _liquid(c["scene"], X).to(torch.int32)
        if c["scene"] == "tower":  # no seeding inside the obstacle (by site: the same number for every seed)
            S = (idx + 0.5) / site
            keep[lo:lo + len(e)] = (S[:, 0] - 0.62) ** 2 + (S[:, 2] - 0.5) ** 2 >= 0.075**2
        for _ in range(4):
            X = X + 0.25 * _flow(X + 0.125 * _flow(X, modes), modes)
        u = _flow(X, modes) * (0.4 * _speed(c) / drift)
        v[lo:lo + len(e)] = u + 0.02 * _speed(c) * torch.randn(u.shape, generator=g, device=DEV)
        eps = 1e-4 * c["dx"]
        x[lo:lo + len(e)] = torch.minimum((X * L).clamp_min(eps), L - eps)
    if c["scene"] == "tower":
        x, v, t = x[keep], v[keep], t[keep]
    return x, v, t


def _system(c, seed):
    """Face coefficients beta = 1/rho of a smoothed phase field (a wavy surface and a drop,
    1000:1, zero on the walls) and a zero-mean right-hand side."""
    g = _gen(seed)
    res = (c["nx"], c["ny"], c["nz"])
    dx = 1.0 / max(res)
    X, Y, Z = torch.meshgrid(*((torch.arange(m, device=DEV, dtype=torch.float64) + 0.5) / m for m in res), indexing="ij")
    r = torch.rand(3, generator=g, device=DEV).tolist()
    h = 0.4 + 0.2 * r[0] + 0.03 * torch.cos(2 * math.pi * (X + r[1])) * torch.cos(2 * math.pi * (Z + r[2]))
    slab = 0.5 * (1 - torch.tanh((Y - h) / (2 * dx)))
    drop = 0.5 * (1 - torch.tanh((torch.sqrt((X - 0.5) ** 2 + (Y - 0.8) ** 2 + (Z - 0.5) ** 2) - 0.12) / (2 * dx)))
    phi = torch.maximum(slab, drop)
    faces = []
    for a in range(3):
        inner = 0.5 * (phi.narrow(a, 0, res[a] - 1) + phi.narrow(a, 1, res[a] - 1))
        beta = torch.zeros([m + (d == a) for d, m in enumerate(res)], dtype=torch.float64, device=DEV)
        beta.narrow(a, 1, res[a] - 1).copy_(1.0 / ((1 - inner) * 1.0 + inner * 1000.0))
        faces.append(beta.float())
    b = torch.randn(res, generator=g, device=DEV)
    return faces, (b - b.mean()).contiguous()


def _config(c):
    from pfflip import Config

    grad = c["kind"] in ("grad", "phase")
    return Config(res=(c["nx"], c["ny"], c["nz"]), dx=c["dx"], ppc=c["ppc"], droplets=bool(c.get("droplets", False)),
                  pcg_tol=c["tol"], pcg_max_iter=400 if grad else 200, k_div=c.get("k_div", 0.0),
                  precision=c.get("precision", "fp32"), device=DEV)


def prepare(c, seed):
    if c["kind"] == "solve":
        from pfflip.poisson import MGPCG

        beta, b = _system(c, seed)
        # the V-cycle of Config's defaults (three sweeps each way)
        s = MGPCG(b.shape, DEV, pre=3, post=3, precision=c["precision"], stencil=c["stencil"])
        return {"case": c, "solver": s, "beta": beta, "b": b, "p": torch.zeros_like(b)}
    x, v, t = _state(c, seed)
    st = {"case": c, "x": x, "v": v, "t": t, "dt": _dt(c)}
    if c["kind"] == "step":
        from pfflip import Simulator

        st["sim"] = Simulator(_config(c))
        if c["scene"] == "tower":
            st["sim"].set_solids(_tower(c).cpu().numpy())
        st["x_out"], st["v_out"] = torch.empty_like(x), torch.empty_like(v)
        return st
    from pfflip.adjoint import DiffSim

    st["sim"] = DiffSim(_config(c), t, st["dt"], adjoint_tol=1e-6)
    g = _gen(seed + 1)
    if c["kind"] == "phase":
        st["w"] = torch.randn((c["nx"], c["ny"], c["nz"]), generator=g, device=DEV)
    else:  # the loss: <wx, x_T> / dx + <wv, v_T> / speed
        st["wx"] = torch.randn(x.shape, generator=g, device=DEV) / c["dx"]
        st["wv"] = torch.randn(x.shape, generator=g, device=DEV) / _speed(c)
    return st


# ------------------------------------------------------------------ one pass
def run(st):
    c = st["case"]
    if c["kind"] == "solve":
        s = st["solver"]
        s.build_hierarchy(*st["beta"])
        s.solve(st["b"], st["p"], tol=c["tol"])
        return {"p": st["p"]}
    if c["kind"] == "phase":
        x = st["x"].detach().requires_grad_(True)
        phi = st["sim"].phase_field(x)
        (gx,) = torch.autograd.grad(phi, x, st["w"])
        return {"phi": phi.detach(), "gx": gx}
    if c["kind"] == "grad":
        x, v = st["x"].detach().requires_grad_(True), st["v"].detach().requires_grad_(True)
        xT, vT = st["sim"].rollout(x, v, c["steps"])
        gx, gv = torch.autograd.grad((xT, vT), (x, v), (st["wx"], st["wv"]))
        return {"x": xT.detach(), "v": vT.detach(), "gx": gx, "gv": gv}
    sim = st["sim"]
    sim.step_index = 0  # the droplet stage draws from (seed, step)
    sim.set_particles(st["x"], st["v"], st["t"])
    for _ in range(c["steps"]):
        sim.step(st["dt"])
    sim.read_particles(st["x_out"], st["v_out"])
    out = {"x": st["x_out"], "v": st["v_out"], "u": [a.tensor for a in sim.vel], "phi": sim.phi_cell.tensor}
    if c["scene"] != "tower":  # inside an obstacle the pressure has no meaning
        out["p"] = sim.pressure.tensor
    return out


# ------------------------------------------------------------------ binary64 restatement
class _A64:
    """The 7-point operator of three face arrays, its coarse operators (sums of faces) and a
    multigrid-preconditioned flexible CG, all in binary64."""

    def __init__(self, beta):
        self.lev = [[b.detach().double() for b in beta]]
        while True:
            bx, by, bz = self.lev[-1]
            n = (bx.shape[0] - 1, by.shape[1] - 1, bz.shape[2] - 1)
            if min(n) < 8 or any(m % 2 for m in n):
                break
            pair = lambda f, a: f.unfold(a, 2, 2).sum(-1)  # noqa: E731
            self.lev.append([pair(pair(bx[::2], 1), 2), pair(pair(by[:, ::2], 0), 2), pair(pair(bz[:, :, ::2], 0), 1)])
        self.diag = [sum(b.narrow(a, 0, b.shape[a] - 1) + b.narrow(a, 1, b.shape[a] - 1) for a, b in enumerate(l))
                     for l in self.lev]
        self.inv = [torch.where(d > 0, 0.8 / d.clamp_min(1e-300), torch.zeros_like(d)) for d in self.diag]

    def mul(self, p, l=0):
        out = torch.zeros_like(p)
        for a, b in enumerate(self.lev[l]):
            m = p.shape[a] - 1
            f = b.narrow(a, 1, m) * (p.narrow(a, 1, m) - p.narrow(a, 0, m))
            out.narrow(a, 1, m).add_(f)
            out.narrow(a, 0, m).sub_(f)
        return out

    def cycle(self, b, l=0):
        last = l + 1 == len(self.lev)
        p = self.inv[l] * b
        for _ in range(150 if last else 2):
            p = p + self.inv[l] * (b - self.mul(p, l))
        if not last:
            r = b - self.mul(p, l)
            for a in range(3):
                r = r.unfold(a, 2, 2).sum(-1)
            e = self.cycle(r, l + 1)
            for a in range(3):
                e = e.repeat_interleave(2, a)
            p = p + 1.5 * e
            for _ in range(3):
                p = p + self.inv[l] * (b - self.mul(p, l))
        return p

    def solve(self, b, tol=1e-12, most=300):
        live = self.diag[0] > 0
        off = lambda v: torch.where(live, v - v.sum() / v.numel(), torch.zeros_like(v))  # noqa: E731
        b = off(b)
        x, r = torch.zeros_like(b), b
        z = self.cycle(r)
        q, rz = z, (r * z).sum()
        end = tol * float(b.abs().max())
        for k in range(most):
            Aq = self.mul(q)
            al = rz / (q * Aq).sum()
            x = x + al * q
            old, r = r, r - al * Aq
            if float(r.abs().max()) <= end:
                break
            z = self.cycle(r)
            new = (r * z).sum()
            q, rz = z + ((new - (old * z).sum()) / rz).clamp_min(0.0) * q, new
        return x - x.mean()


class _Solve(torch.autograd.Function):
    @staticmethod
    def forward(ctx, b, *beta):
        A = _A64(beta)
        p = A.solve(b)
        ctx.A, ctx.p = A, p
        return p

    @staticmethod
    def backward(ctx, g):
        lam, p = ctx.A.solve(g), ctx.p
        gb = []
        for a, f in enumerate(ctx.A.lev[0]):
            m = p.shape[a] - 1
            d = torch.zeros_like(f)
            d.narrow(a, 1, m).copy_(-(lam.narrow(a, 1, m) - lam.narrow(a, 0, m)) * (p.narrow(a, 1, m) - p.narrow(a, 0, m)))
            gb.append(d)
        return (lam, *gb)


def _offsets(x, dx, shape, node):
    """Per axis the lower tap and the fraction of x within a grid whose nodes sit at
    (n + node) dx; shape is the grid's."""
    lo, fr = [], []
    for d in range(3):
        q = x[:, d] / dx - node[d]
        i = torch.floor(q.detach()).long()
        lo.append(i)
        fr.append(q - i)
    return lo, fr


def _corners():
    return [(a, b, c) for a in (0, 1) for b in (0, 1) for c in (0, 1)]


class _Ref:
    """One simulation in binary64: P2G, phase field, forces, solve, projection, extrapolation,
    G2P and Ralston RK3 (differentiable in the particles)."""

    def __init__(self, c):
        self.c, self.dx, self.dt = c, float(torch.tensor(c["dx"])), _dt(c)
        self.n = (c["nx"], c["ny"], c["nz"])
        self.rho_l, self.rho_g = 1000.0, 1.0
        pa = round(c["ppc"] ** (1 / 3))
        o2 = ((torch.arange(-pa - 1, pa + 1, dtype=torch.float64) + 0.5) / pa) ** 2
        t = (1 - (o2[:, None, None] + o2[None, :, None] + o2[None, None, :])).clamp_min(0)
        self.rho0 = float((t**3).sum())
        self.rho_0l, self.rho_min = self.rho0 * self.rho_l, math.log(1000.0) * self.rho_g * self.rho0
        self.solid = _tower(c) if c["scene"] == "tower" else None

    def shape(self, a):
        return tuple(m + (d == a) for d, m in enumerate(self.n))

    def node(self, a):
        return tuple(0.0 if d == a else 0.5 for d in range(3))

    def chunks(self, x):
        step = len(x) if x.requires_grad else 1 << 23
        return range(0, len(x), step), step

    def splat(self, x, vals, a):
        """Sums of w * val on grid a (3 = cells) for each val; w = (1 - d^2/dx^2)^3."""
        sh = self.shape(a)
        outs = [torch.zeros(sh[0] * sh[1] * sh[2], dtype=torch.float64, device=DEV) for _ in vals]
        rng, step = self.chunks(x)
        for s in rng:
            lo, fr = _offsets(x[s:s + step], self.dx, sh, self.node(a))
            for cr in _corners():
                d2 = sum((f - o) ** 2 for f, o in zip(fr, cr))
                w = (1 - d2).clamp_min(0) ** 3
                i = [l + o for l, o in zip(lo, cr)]
                ok = torch.ones_like(w, dtype=torch.bool)
                for q, m in zip(i, sh):
                    ok &= (q >= 0) & (q < m)
                at = torch.where(ok, (i[0] * sh[1] + i[1]) * sh[2] + i[2], torch.zeros_like(i[0]))
                w = torch.where(ok, w, torch.zeros_like(w))
                outs = [o.index_add(0, at, w * v[s:s + step]) if x.requires_grad else o.index_add_(0, at, w * v[s:s + step])
                        for o, v in zip(outs, vals)]
        return [o.view(sh) for o in outs]

    def phase(self, rho):
        q = (rho - self.rho_min) / self.rho_0l
        on = q > 0
        return torch.where(on, torch.sqrt(torch.where(on, q, torch.ones_like(q))).clamp_max(1.0), torch.zeros_like(q))

    def wall(self, a):
        w = torch.zeros(self.shape(a), dtype=torch.bool, device=DEV)
        w.narrow(a, 0, 1).fill_(True)
        w.narrow(a, self.n[a], 1).fill_(True)
        if self.solid is not None:
            w.narrow(a, 0, self.n[a]).logical_or_(self.solid)
            w.narrow(a, 1, self.n[a]).logical_or_(self.solid)
        return w

    def sample(self, f, a, x):
        """Trilinear sample of face grid a at x, taps clamped to the grid."""
        sh = f.shape
        lo, fr = _offsets(x, self.dx, sh, self.node(a))
        flat, out = f.reshape(-1), 0.0
        for cr in _corners():
            i = [(l + o).clamp(0, m - 1) for l, o, m in zip(lo, cr, sh)]
            w = 1.0
            for t, o in zip(fr, cr):
                w = w * (t if o else 1 - t)
            out = out + w * flat[(i[0] * sh[1] + i[1]) * sh[2] + i[2]]
        return out

    def extrapolate(self, u, a, liq):
        known = torch.zeros(self.shape(a), dtype=torch.bool, device=DEV)
        known.narrow(a, 0, self.n[a]).logical_or_(liq)
        known.narrow(a, 1, self.n[a]).logical_or_(liq)
        f = torch.where(known, u, torch.zeros_like(u))
        for _ in range(3):
            kd = known.double()
            acc, cnt = torch.zeros_like(f), torch.zeros_like(kd)
            for d in range(3):
                m = f.shape[d] - 1
                pad = [0, 0, 0, 0, 0, 0]
                up, dn = list(pad), list(pad)
                up[2 * (2 - d)], dn[2 * (2 - d) + 1] = 1, 1
                fk = torch.where(known, f, torch.zeros_like(f))
                for p_, lo in ((up, 0), (dn, 1)):
                    acc = acc + torch.nn.functional.pad(fk.narrow(d, lo, m), p_)
                    cnt = cnt + torch.nn.functional.pad(kd.narrow(d, lo, m), p_)
            new = ~known & (cnt > 0)
            f = torch.where(new, acc / cnt.clamp_min(1), f)
            known = known | new
        return f

    def step(self, x, v, liquid):
        n, dx, dt = self.n, self.dx, self.dt
        mp = torch.where(liquid, self.rho_l, self.rho_g).double()
        cm, cw = self.splat(x, [mp, torch.ones_like(mp)], 3)
        phi = self.phase(cm)
        liq = phi.detach() >= 0.5
        u, us, beta = [], [], []
        for a in range(3):
            m, q = self.splat(x, [mp, mp * v[:, a]], a)
            ok = m.detach() > 1e-12 * self.rho_0l
            ua = torch.where(ok, q / torch.where(ok, m, torch.ones_like(m)), torch.zeros_like(m))
            A, B = torch.zeros_like(ok), torch.zeros_like(ok)
            B.narrow(a, 0, n[a]).copy_(liq)
            A.narrow(a, 1, n[a]).copy_(liq)
            A.narrow(a, 0, 1).copy_(B.narrow(a, 0, 1))
            B.narrow(a, n[a], 1).copy_(A.narrow(a, n[a], 1))
            ph = torch.where(A & B, torch.ones_like(m), torch.where(A ^ B, self.phase(m), torch.zeros_like(m)))
            wall = self.wall(a)
            beta.append(torch.where(wall, torch.zeros_like(m), 1 / ((1 - ph) * self.rho_g + ph * self.rho_l)))
            ua = torch.where(wall, torch.zeros_like(m), ua)
            us.append(ua)
            u.append(torch.where(wall, ua, ua + (-G * dt if a == 1 else 0.0)))
        div = sum(f.narrow(a, 1, n[a]) - f.narrow(a, 0, n[a]) for a, f in enumerate(u))
        b = -(dx / dt) * div
        if self.c.get("k_div", 0.0) > 0:
            b = b - dx * dx * self.c["k_div"] * ((cw - self.rho0) / self.rho0).clamp_min(0) / dt
        p = _Solve.apply(b, *beta)
        for a in range(3):
            g = torch.nn.functional.pad(p.narrow(a, 1, n[a] - 1) - p.narrow(a, 0, n[a] - 1),
                                        [1 if (2 - k // 2) == a else 0 for k in range(6)])
            u[a] = u[a] - dt * beta[a] * g / dx
        if self.c.get("droplets", False):
            return None, None, u, phi, p
        ul = [self.extrapolate(u[a], a, liq) for a in range(3)]
        xs, vs = [], []
        rng, size = self.chunks(x)
        for s in rng:
            y, w = self.move(x[s:s + size], v[s:s + size], liquid[s:s + size], u, us, ul)
            xs.append(y)
            vs.append(w)
        return torch.cat(xs), torch.cat(vs), u, phi, p

    def move(self, x, v, liquid, u, us, ul):
        dt, dx = self.dt, self.dx
        al = torch.where(liquid, 0.985, 0.96).double()
        vn = []
        for a in range(3):
            pic, old = self.sample(u[a], a, x), self.sample(us[a], a, x)
            vn.append(al * (v[:, a] + pic - old) + (1 - al) * pic)

        def vel(y):
            return torch.stack([torch.where(liquid, self.sample(ul[a], a, y), self.sample(u[a], a, y)) for a in range(3)], 1)

        k1 = vel(x)
        k2 = vel(x + 0.5 * dt * k1)
        k3 = vel(x + 0.75 * dt * k2)
        y = x + dt * (2 * k1 + 3 * k2 + 4 * k3) / 9
        eps = 1e-4 * dx
        out = []
        for a in range(3):
            hi = self.n[a] * dx - eps
            ya, w = y[:, a].clamp(eps, hi), vn[a]
            w = torch.where(ya <= eps, w.clamp_min(0), torch.where(ya >= hi, w.clamp_max(0), w))
            out.append((ya, w))
        y, w = torch.stack([o[0] for o in out], 1), torch.stack([o[1] for o in out], 1)
        return self.push_out(y, w) if self.solid is not None else (y, w)

    def push_out(self, x, v):
        """Particles inside the obstacle leave along the axis of the nearest free cell."""
        n, dx = self.n, self.dx
        cell = [(x[:, d] / dx).long().clamp(0, n[d] - 1) for d in range(3)]
        inside = self.solid[cell[0], cell[1], cell[2]]
        best = torch.full_like(x[:, 0], 1e9)
        ax, sg = torch.zeros_like(cell[0]), torch.ones_like(x[:, 0])
        for d in range(6):
            a, s = d // 2, -1 if d % 2 == 0 else 1
            found = torch.full_like(best, 1e9)
            for t in range(7, 0, -1):
                q = list(cell)
                q[a] = q[a] + s * t
                ok = (q[a] >= 0) & (q[a] < n[a])
                q[a] = q[a].clamp(0, n[a] - 1)
                found = torch.where(ok & ~self.solid[q[0], q[1], q[2]], torch.full_like(best, float(t)), found)
            better = found < best
            best, ax, sg = torch.where(better, found, best), torch.where(better, a, ax), torch.where(better, float(s), sg)
        go = inside & (best < 1e8)
        one = torch.nn.functional.one_hot(ax, 3).bool() & go[:, None]
        x = torch.where(one, x + ((best + 0.5) * dx * sg)[:, None], x)
        return x, torch.where(one & (sg[:, None] * v < 0), torch.zeros_like(v), v)


def exact(c, seed):
    if c["kind"] == "solve":
        beta, b = _system(c, seed)
        b = b.double()
        return {"p": _A64(beta).solve(b - b.mean())}
    x, v, t = _state(c, seed)
    liquid, ref = t == 1, _Ref(c)
    if c["kind"] == "step":
        with torch.no_grad():
            x, v = x.double(), v.double()
            for _ in range(c["steps"]):
                x, v, u, phi, p = ref.step(x, v, liquid)
        out = {"x": x, "v": v, "u": u, "phi": phi}  # with droplets x and v follow a random stream: no such value
        return out if c["scene"] == "tower" else {**out, "p": p}
    g = _gen(seed + 1)
    if c["kind"] == "phase":
        if len(x) > 20_000_000:
            return None
        w = torch.randn(ref.n, generator=g, device=DEV).double()
        x = x.double().requires_grad_(True)
        (cm,) = ref.splat(x, [torch.where(liquid, ref.rho_l, ref.rho_g).double()], 3)
        phi = ref.phase(cm)
        (gx,) = torch.autograd.grad(phi, x, w)
        return {"phi": phi.detach(), "gx": gx}
    if len(x) > 4_000_000:
        return None
    wx = torch.randn(x.shape, generator=g, device=DEV) / c["dx"]
    wv = torch.randn(x.shape, generator=g, device=DEV) / _speed(c)
    x, v = x.double(), v.double()
    at = []
    with torch.no_grad():  # the states, then each step again with its gradient
        for _ in range(c["steps"]):
            at.append((x, v))
            x, v = ref.step(x, v, liquid)[:2]
    gx, gv = wx.double(), wv.double()
    for a, b in reversed(at):
        a, b = a.detach().requires_grad_(True), b.detach().requires_grad_(True)
        y, w = ref.step(a, b, liquid)[:2]
        gx, gv = torch.autograd.grad((y, w), (a, b), (gx, gv))
    return {"x": x, "v": v, "gx": gx, "gv": gv}
