"""The work that a user of this framework has it do, as measurable cases.

A case is one stretch of simulation through the public entry points: a driver
loop steps a job (or a batch of jobs, or a server's requests) and then reads
the points' position, velocity and stress back, as it does between frames.
``GPUExplicitUSL`` is the replacement of one job's solver, ``GPUBatch`` steps
many independent jobs, ``GPUServer`` admits requests that arrive together and
returns each one's result.

Sizes are those of the workloads in ``mpm_3d_b200.inputs`` (the block drop in
2D, the two-body collision, the column collapse, the ensemble of block drops,
the serving stream, the sand column, the blocks on a slip floor) and sizes
between them. Every body is seeded: points are moved by up to 1 % of a cell
(the column's own jitter) and the body gets a velocity gradient, a slow spin
and stretch, so that its stress is that of a moving solid from the first step
on and not the rounding of a free flight.
"""
import math

import numpy as np
import torch

from mpm_3d_b200 import inputs
from mpm_3d_b200.native import GPUBatch, GPUExplicitUSL, GPUServer

FIELDS = ("x", "x_t", "T")


def listed():
    return [
        # the smallest job: 144 points in 2D, where launches are everything
        {"name": "drop_2d", "kind": "drop", "dim": 2, "mode": "fp64", "n": 20, "steps": 400},
        # one small job in 3D, the low end of the ensemble's grids, alone
        {"name": "drop_small", "kind": "drop", "dim": 3, "mode": "fp64", "n": 24, "steps": 400},
        # an odd grid with the granular material of the reference's own examples
        {"name": "sand_column", "kind": "sand", "dim": 3, "mode": "fp64", "n": 70, "steps": 300},
        # two neo-Hookean blocks sliding into each other on a slip floor:
        # the reflected contact normal and the other elastic material
        {"name": "slip_walls", "kind": "walls", "dim": 3, "mode": "fp64", "n": 61, "steps": 300},
        # the two-body collision at its full size, the ordinary call
        {"name": "collision", "kind": "collision", "dim": 3, "mode": "fp64", "n": 128, "steps": 800},
        # the same collision in the mixed form on a smaller odd grid
        {"name": "collision_mixed", "kind": "collision", "dim": 3, "mode": "mixed", "n": 97, "steps": 150},
        # the column collapse at full size: 3.1 million points, the largest
        {"name": "column", "kind": "column", "dim": 3, "mode": "fp64", "n": 256, "steps": 1000},
        # the column in the mixed form, half the cells per axis
        {"name": "column_mixed", "kind": "column", "dim": 3, "mode": "mixed", "n": 128, "steps": 300},
        # the bit-reproducible form on the quarter-size column
        {"name": "column_exact_sums", "kind": "column", "dim": 3, "mode": "fp64_deterministic", "n": 64, "steps": 300},
        # independent block drops of uneven size stepped together
        {"name": "batch", "kind": "batch", "dim": 3, "mode": "fp64", "n": 128, "jobs": 21, "steps": 300},
        # more and smaller jobs in the mixed form, one more than a power of two
        {"name": "batch_mixed", "kind": "batch", "dim": 3, "mode": "mixed", "n": 72, "jobs": 21, "steps": 100},
        # requests of the serving stream served together, a tenth of them
        # two-body collisions, each with its own step count
        {"name": "serve", "kind": "serve", "dim": 3, "mode": "mixed", "n": 96, "jobs": 14, "steps": 160},
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another case of the same ranges. Step counts fall with the size, so
    that no case costs more than the full-size column."""
    kind = rng.choice(["drop", "drop", "sand", "walls", "collision", "column", "batch", "serve"])
    case = {"kind": kind, "dim": 3}
    if kind == "drop":
        case["dim"] = rng.choice([2, 3])
        case["mode"] = rng.choice(["fp64", "mixed"])
        case["n"] = _between(rng, 20, 200) if case["dim"] == 2 else _between(rng, 16, 128)
        case["steps"] = rng.randint(200, 500)
    elif kind == "sand":
        case["dim"] = rng.choice([2, 3])
        case["mode"] = "fp64"
        case["n"] = 10 * _between(rng, 2, 20 if case["dim"] == 2 else 12)
        case["steps"] = rng.randint(100, 400)
    elif kind == "walls":
        case["mode"] = "fp64"
        case["n"] = _between(rng, 16, 100)
        case["steps"] = rng.randint(100, 400)
    elif kind == "collision":
        case["mode"] = rng.choice(["fp64", "mixed"])
        case["n"] = _between(rng, 20, 150)
        case["steps"] = rng.randint(200, 600) if case["mode"] == "fp64" else rng.randint(80, 150)
    elif kind == "column":
        case["mode"] = rng.choice(["fp64", "fp64", "mixed", "fp64_deterministic"])
        case["n"] = 8 * _between(rng, 4, 24 if case["mode"] != "fp64_deterministic" else 14)
        case["steps"] = rng.randint(100, 300)
    else:
        case["mode"] = rng.choice(["fp64", "mixed"])
        case["n"] = _between(rng, 40, 128)
        case["jobs"] = rng.randint(5, 21) if kind == "batch" else rng.randint(4, 14)
        case["steps"] = rng.randint(60, 160)
    return case


# ---- inputs ----


def _block(n, dim, layout):
    """A block drop on an n^dim grid: the ensemble's in 3D, the 2D block drop
    scaled to the grid (0.3 m block of 2 points per cell and axis)."""
    if dim == 3:
        return inputs.block_drop_ensemble(1, layout, n_range=(n, n))[0]
    h = (1.0 / n,) * 2
    side = int(round(0.3 / (h[0] / 2.0)))
    body = inputs.block_points((0.35, 0.45), (side, side), h, 1000.0, (0.0, -1.0), name="block")
    return inputs.Case(name="block_drop_2d", dim=2, L=(1.0, 1.0), N=(n, n), dt=1e-4 * 20 / n, steps=0, bodies=[body])


def _column(n, seed):
    """The column collapse at n x n x n/2 cells (the workload's 2 x 2 x 1 m box)."""
    N = (n, n, n // 2)
    h = (2.0 / n,) * 3
    counts = tuple(int(round(s / (h[0] / 2.0))) for s in (0.5, 0.5, 0.75))
    body = inputs.block_points((0.75, 0.75, 0.0), counts, h, 1500.0, (0.0, 0.0, 0.0), name="column", E=1e6, nu=0.3)
    return inputs.Case(name="column", dim=3, L=(2.0, 2.0, 1.0), N=N, dt=1e-5 * 256 / n, steps=0, bodies=[body])


def _stirred(case, rng):
    """The case with its bodies' points moved by up to 1 % of a cell, and a
    velocity gradient of up to 0.3 / s on each body."""
    d = case.dim
    for b in case.bodies:
        h = np.asarray(case.h)
        x = b.x[:, :d] + rng.uniform(-0.01, 0.01, (b.n, d)) * h
        b.x[:, :d] = np.clip(x, 1e-3 * h, np.asarray(case.L[:d]) - 1e-3 * h)
        b.x_t[:, :d] += (b.x[:, :d] - b.x[:, :d].mean(0)) @ rng.uniform(-0.3, 0.3, (d, d))
    return case


def _jobs(case, seed):
    """[(job, steps)] of a case. Block sizes come from the case alone (so that
    a case is the same work for every seed), everything else from the seed."""
    rng = np.random.default_rng(seed)
    kind, n, dim, steps = case["kind"], case["n"], case["dim"], case["steps"]
    if kind == "drop":
        jobs = [(_block(n, dim, n), steps)]
    elif kind == "sand":
        jobs = [(inputs.sand_column(dim, n), steps)]
        jobs[0][0].dt = 1e-4 * 20 / n
    elif kind == "walls":
        jobs = [(inputs.wall_collision(dim, n, reflected=True), steps)]
        jobs[0][0].dt = 1e-4 * 16 / n
        for b in jobs[0][0].bodies:
            b.material_class = "CompressibleNeohookeanElasticity"
    elif kind == "collision":
        jobs = [(inputs.two_body_collision_3d(n, gap=0.0), steps)]
        jobs[0][0].dt = 2e-5 * 128 / n
    elif kind == "column":
        jobs = [(_column(n, seed), steps)]
    else:
        size = np.random.default_rng(n)
        jobs = []
        for k in range(case["jobs"]):
            m = int(round(16 * (n / 16) ** size.random()))
            s = steps if kind == "batch" else max(1, int(steps * size.uniform(0.25, 1.0)))
            if kind == "serve" and k % 10 == 5:
                c = inputs.two_body_collision_3d(m, gap=0.0, mu=0.3)
                c.dt = 2e-5 * 128 / m
                jobs.append((c, s))
            else:
                jobs.append((_block(m, 3, 1000 * n + k), s))
    return [(_stirred(c, rng), s) for c, s in jobs]


def prepare(case, seed):
    jobs = _jobs(case, seed)
    state = {"kind": case["kind"], "steps": case["steps"], "jobs": jobs}
    if case["kind"] == "serve":
        # a service keeps its server; the requests are what arrives
        state["server"] = GPUServer(40 << 30, mode=case["mode"])
    elif case["kind"] == "batch":
        batch = GPUBatch(dim=case["dim"], mode=case["mode"])
        state["ids"] = [batch.add(c, steps=1 << 40) for c, _ in jobs]
        state["batch"] = batch
    else:
        state["solver"] = GPUExplicitUSL(jobs[0][0], mode=case["mode"])
    return state


def run(state):
    if state["kind"] == "serve":
        server = state["server"]
        ids = [server.submit(c, s) for c, s in state["jobs"]]
        out, left = [None] * len(ids), set(ids)
        while left:
            server.advance(20)
            for rid in server.poll():
                if rid not in left:
                    continue
                left.discard(rid)
                k = ids.index(rid)
                out[k] = [{f: server.result(rid, b, f) for f in FIELDS} for b in range(len(state["jobs"][k][0].bodies))]
                server.release(rid)
        return out
    if state["kind"] == "batch":
        batch = state["batch"]
        batch.step(state["steps"])
        return {f: batch.points_many(state["ids"], 0, f) for f in FIELDS}
    solver = state["solver"]
    solver.step(state["steps"])
    return [{f: solver.points(b, f) for f in FIELDS} for b in range(len(state["jobs"][0][0].bodies))]


# ---- work ----


def work(case):
    """Each step reads a point's state and writes what changed (276 bytes in
    FP64; 192 in the mixed form, whose position, velocity and mass are two
    words), and accumulates and reads 7 values of each node with mass (about
    0.15 nodes per point in 3D, 0.35 in 2D). A point takes about 700
    floating-point operations per step in 3D and 250 in 2D."""
    dim = case["dim"]
    state = 192 if case["mode"] == "mixed" else 276
    if dim == 2:
        state = state * 2 // 3
    per = state + 112 * (0.15 if dim == 3 else 0.35)
    bytes_, flops = 0.0, 0.0
    for c, s in _sizes(case):
        bytes_ += c * (s * per + 15 * 8)
        flops += c * s * (700 if dim == 3 else 250)
    return {"bytes": bytes_, "flops": flops}


def _sizes(case):
    """[(points, steps)] of the case's jobs."""
    return [(c.n_points, s) for c, s in _jobs(case, 0)]


# ---- the step in 64 bits ----


def exact(case, seed):
    jobs = _jobs(case, seed)
    # up to 8e-8 s per point and step, plus 4 ms per step
    if sum(c.n_points * s * 8e-8 + s * 4e-3 for c, s in jobs) > 16.0:
        return None
    out = [_simulate(c, s) for c, s in jobs]
    if case["kind"] == "batch":
        return {f: [o[0][f] for o in out] for f in FIELDS}
    return out if case["kind"] == "serve" else out[0]


def _axis(x, a, corner, h, L, N):
    """One axis of the shape functions: base node, and the three nodes'
    weights W and (signed, unscaled) gradient weights G."""
    hat = lambda r: (1.0 - r.abs())  # noqa: E731
    lo, hi = x - a, x + a
    el, eh, ex = (torch.floor(v / L * N) for v in (lo, hi, x))
    open_ = hi < L   # a corner on the upper face has no element
    eh = torch.where(open_, eh, el)
    rl, rh = lo / h - el, hi / h - eh
    wl0, wl1 = hat(rl), hat(rl - 1)
    wh0, wh1 = hat(rh) * open_, hat(rh - 1) * open_
    wide = eh > el
    z = torch.zeros_like(x)
    Wc = [torch.where(wide, wl0, wl0 + wh0), torch.where(wide, wl1 + wh0, wl1 + wh1), torch.where(wide, wh1, z)]
    Gc = [torch.where(wide, -wl0, wh0 - wl0), torch.where(wide, wh0 - wl1, wh1 - wl1), torch.where(wide, wh1, z)]
    r = x / h - ex
    Wp, Gp = [hat(r), hat(r - 1), z], [z - 1.0 / h, z + 1.0 / h, z]
    pick = lambda c, p: torch.stack([torch.where(corner, u, v) for u, v in zip(c, p)], -1)  # noqa: E731
    return torch.where(corner, el, ex).long(), pick(Wc, Wp), pick(Gc, Gp)


class _Body64:
    def __init__(self, case, b, dev):
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)  # noqa: E731
        d = case.dim
        self.b, self.case, self.d = b, case, d
        self.m, self.vol, self.x, self.v = t(b.m), t(b.v), t(b.x[:, :d]), t(b.x_t[:, :d])
        self.ext = 0.5 * self.vol ** (1.0 / d)
        self.T = torch.zeros(b.n, 3, 3, dtype=torch.float64, device=dev)
        self.F = torch.eye(3, dtype=torch.float64, device=dev).expand(b.n, 3, 3).clone()

    def map(self):
        """Node ids [n, K], values S [n, K] and gradients [n, K, d]."""
        c, d = self.case, self.d
        a = 0.5 * self.ext
        corner = torch.ones_like(a, dtype=torch.bool)
        for k in range(d):
            corner &= (self.x[:, k] - a >= 0) & (self.x[:, k] + a <= c.L[k])
        ax = [_axis(self.x[:, k], a, corner, c.h[k], c.L[k], c.N[k]) for k in range(d)]
        cp = 2 ** d
        sS = torch.where(corner, 1.0 / cp, 1.0)
        sG = torch.where(corner, 1.0 / (cp / 2 * self.ext), torch.ones_like(a))
        ids, S, g = 0, 1.0, [1.0] * d
        stride = 1
        for k, (base, W, G) in enumerate(ax):
            shape = [-1] + [1] * d
            shape[d - k] = 3     # the first axis runs fastest
            node = (base[:, None] + torch.arange(3, device=base.device)).clamp(max=c.N[k])
            ids = ids + (node * stride).reshape(shape)
            S = S * W.reshape(shape)
            g = [gi * (G if i == k else W).reshape(shape) for i, gi in enumerate(g)]
            stride *= c.N[k] + 1
        n = self.m.shape[0]
        flat = lambda q: q.expand(n, *([3] * d)).reshape(n, -1)  # noqa: E731
        return flat(ids), flat(S) * sS[:, None], torch.stack([flat(gi) for gi in g], -1) * sG[:, None, None]

    def stress(self, L, dt):
        b = self.b
        G = b.E / (2 * (1 + b.nu))
        K = b.E / (3 * (1 - 2 * b.nu))
        lam = K - 2 * G / 3
        eye = torch.eye(3, dtype=torch.float64, device=L.device)
        if b.material_class == "CompressibleNeohookeanElasticity":
            self.F = self.F + dt * (L @ self.F)
            B = self.F @ self.F.transpose(1, 2)
            J = torch.det(self.F)[:, None, None]
            self.T = G / J * (B - eye) + lam * torch.log(J) / J * eye
            return
        D, W = 0.5 * (L + L.transpose(1, 2)), 0.5 * (L - L.transpose(1, 2))
        tr = torch.einsum("nii->n", D)[:, None, None]
        T = self.T + dt * (2 * G * D + lam * tr * eye + W @ self.T - self.T @ W)
        if b.material_class == "Sand_SachithLocal":
            (grain, mu_s, rho_s, rho_c, mu_2, i_0), _ = inputs.sand_params(b)
            p = -torch.einsum("nii->n", T) / 3
            t0 = T + p[:, None, None] * eye
            tau = (t0 * t0).sum((1, 2)).sqrt() / math.sqrt(2.0)
            loose = (self.m / self.vol < rho_c) | (p <= 0)
            q = torch.where(p > 0, p, torch.ones_like(p))
            S0, S2 = mu_s * q, mu_2 * q
            al = G * i_0 * dt * (q / rho_s).sqrt() / grain
            bb, cc = S2 + tau + al, S2 * tau + S0 * al
            root = 2 * cc / (bb + (bb * bb - 4 * cc).sqrt())
            scale = torch.where(tau <= S0, torch.ones_like(tau), root / tau)
            T = scale[:, None, None] * t0 - p[:, None, None] * eye
            T = torch.where(loose[:, None, None], torch.zeros_like(T), T)
        self.T = T


def _contact(case, c, nodes, nrm, faces):
    """ContactHuang (implicit form) on the two bodies' nodal (m, mx, f)."""
    (m1, p1, f1), (m2, p2, f2) = nodes[c.b1], nodes[c.b2]
    n = nrm
    if c.reflected:
        n = torch.where(faces & (m1 > 0)[:, None], torch.zeros_like(n), n)
    n = n / n.norm(dim=1, keepdim=True)
    both = (m1 > 0) & (m2 > 0)
    a1 = torch.where(both, m1, torch.ones_like(m1))[:, None]
    dt = case.dt
    q1, q2 = p1 + dt * f1, p2 + dt * f2
    vcm = (q1 + q2) / torch.where(both, m1 + m2, torch.ones_like(m1))[:, None]
    rel = vcm - q1 / a1
    touch = both & ((-rel * n).sum(1) > 0)
    fn = a1[:, 0] / dt * (rel * n).sum(1)
    s = a1 / dt * rel - fn[:, None] * n
    ft = s.norm(dim=1)
    s = s / torch.where(ft > 0, ft, torch.ones_like(ft))[:, None]
    fc = fn.clamp(max=0.0)[:, None] * n + torch.minimum(c.mu * fn.abs(), ft)[:, None] * s
    fc = torch.where(touch[:, None], fc, torch.zeros_like(fc))
    nodes[c.b1] = (m1, p1, f1 + fc)
    nodes[c.b2] = (m2, p2, f2 - fc)


def _simulate(case, steps):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    d, dt = case.dim, case.dt
    bodies = [_Body64(case, b, dev) for b in case.bodies]
    nn = case.n_nodes
    i = torch.arange(nn, device=dev)
    faces = []
    for k in range(d):
        ik = i % (case.N[k] + 1)
        i = i // (case.N[k] + 1)
        faces.append((ik == 0) | (ik == case.N[k]))
    faces = torch.stack(faces, 1)
    grav = torch.zeros(d, dtype=torch.float64, device=dev)
    grav[1 if d == 2 else 2] = -9.81
    first = {c.b1 for c in case.contacts}
    for _ in range(steps):
        maps, nodes, normals = [], [], {}
        for k, b in enumerate(bodies):
            ids, S, g = b.map()
            maps.append((ids, S, g))
            vT = (b.vol[:, None, None] * b.T)[:, :d, :d]
            val = torch.cat([(S * b.m[:, None])[..., None], (S * b.m[:, None])[..., None] * b.v[:, None, :],
                             -torch.einsum("nkb,nab->nka", g, vT)], -1)
            if k in first:
                val = torch.cat([val, g * b.m[:, None, None]], -1)
            acc = torch.zeros(nn, val.shape[-1], dtype=torch.float64, device=dev)
            acc.index_add_(0, ids.reshape(-1), val.reshape(-1, val.shape[-1]))
            m = acc[:, 0]
            nodes.append((m, acc[:, 1:1 + d], acc[:, 1 + d:1 + 2 * d] + m[:, None] * grav))
            if k in first:
                normals[k] = acc[:, 1 + 2 * d:]
        for c in case.contacts:
            _contact(case, c, nodes, normals[c.b1], faces)
        for b, (ids, S, g), (m, p, f) in zip(bodies, maps, nodes):
            wall = faces if inputs.boundary_class(b.b) == "CartesianSmoothBox" else faces.any(1, keepdim=True)
            p, f = p * ~wall, f * ~wall
            inv = torch.where(m > 0, 1.0 / m, torch.zeros_like(m))[:, None]
            v, dv = (p + dt * f) * inv, dt * f * inv
            vk = v[ids]
            b.x = b.x + dt * torch.einsum("nk,nkd->nd", S, vk)
            b.v = b.v + torch.einsum("nk,nkd->nd", S, dv[ids])
            L = torch.zeros(b.m.shape[0], 3, 3, dtype=torch.float64, device=dev)
            L[:, :d, :d] = torch.einsum("nka,nkb->nab", vk, g)
            b.vol = b.vol * torch.exp(dt * torch.einsum("nii->n", L))
            b.stress(L, dt)
    pad = lambda a: torch.nn.functional.pad(a, (0, 3 - d))  # noqa: E731
    return [{"x": pad(b.x).cpu().numpy(), "x_t": pad(b.v).cpu().numpy(), "T": b.T.reshape(-1, 9).cpu().numpy()} for b in bodies]
