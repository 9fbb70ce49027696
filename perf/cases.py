"""The work that users of this framework have it do, as cases for timing.

Every case goes through the package's public Python API on seeded synthetic packings
(bidisperse, R = 0.5 and 0.7 alternating, spines at least a tenth of the radius sum
apart, as the package's generators make them).  ``exact`` repeats the computation in
64 bits with plain torch operations.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from spherocyls_gb300 import BoxBatch

PI = 3.14159265358979  # the reference's pi
DEV = "cuda"
F64 = torch.float64


def listed():
    shear = dict(kind="shear", contacts=1, aor=1.0, rate=1e-4, dt=0.02, pad=0.2, gamma=0.0,
                 se_every=0)
    fire = dict(kind="fire", contacts=2, phi=0.90, pad=0.1, iters=50)
    return [
        # One force and stress evaluation of a small packing (analysis of a saved file).
        dict(name="stress_fp64_n256", kind="stress", precision="fp64", contacts=1, n=256, phi=0.85,
             aor=1.0, pad=0.1, gamma=0.2),
        # The plain FP64 shear run of the validation configuration, one saved record.
        dict(shear, name="shear_fp64_n1024", precision="fp64", n=1024, phi=0.85, rate=1e-5,
             steps=100, se_every=100),
        # The precision comparison's system: stress and energy recorded at every step.
        dict(shear, name="shear_mixed_n16384", precision="mixed", n=16384, phi=0.86, gamma=0.25,
             steps=20, se_every=1),
        # The headline: large sheared system, mixed form, device-resident.
        dict(shear, name="shear_mixed_n1048576", precision="mixed", n=1 << 20, phi=0.84, steps=20),
        # The same system in the plain FP64 form.
        dict(shear, name="shear_fp64_n1048576", precision="fp64", n=1 << 20, phi=0.84, steps=4),
        # An ensemble of independent systems of uneven size, shape, packing and rate.
        dict(name="ensemble_mixed_512", kind="ensemble", precision="mixed", nsys=512, nmin=64,
             nmax=8192, sizes=2, dt=0.02, pad=0.2, steps=20),
        # Relaxation of jamming replicas, two-point contacts: mixed sweeps, FP64 refinement.
        dict(fire, name="fire_mixed_128x4096", precision="mixed", nsys=128, n=4096),
        dict(fire, name="fire_fp64_32x4096", precision="fp64", nsys=32, n=4096),
        # The reference's minimiser on one jamming replica.
        dict(name="cg_fp64_n4096", kind="cg", contacts=2, nsys=1, n=4096, phi=0.90, pad=0.1,
             iters=10),
        # Slow box compression and expansion, an odd number of particles.
        dict(name="resize_mixed_n49999", kind="resize", precision="mixed", contacts=1, n=49999,
             phi=0.80, aor=0.5, dt=0.02, pad=0.2, resize=1e-5, steps=20),
        # Elongated particles in FP64 at a middle, odd size and a sheared start.
        dict(shear, name="shear_fp64_n30011", precision="fp64", n=30011, phi=0.82, aor=2.0,
             rate=1e-3, gamma=-0.3, steps=10, se_every=10),
        # End to end: a box made from host arrays, advanced, its stress and state read back.
        dict(name="endtoend_mixed_n1048576", kind="endtoend", precision="mixed", contacts=1,
             n=1 << 20, phi=0.84, aor=1.0, rate=1e-4, dt=0.02, pad=0.2, gamma=0.0, steps=20),
    ]


def draw(rng):
    def log(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choice(["shear", "shear", "shear", "ensemble", "fire", "resize", "stress", "cg",
                       "endtoend"])
    precision = rng.choice(["mixed", "fp64"])
    case = dict(kind=kind, precision=precision, contacts=rng.choice([1, 1, 2]),
                phi=round(rng.uniform(0.70, 0.90), 3), pad=round(rng.uniform(0.1, 0.5), 3))
    if kind in ("shear", "resize", "endtoend"):
        case["n"] = int(log(100, 600000 if precision == "mixed" else 200000))
        most = max(1, int((1 << 23 if precision == "mixed" else 1 << 20) / case["n"]))
        case["steps"] = min(int(log(2, 60)), most)
        case["aor"] = round(rng.uniform(0.2, 2.0), 2)
        case["dt"] = 0.02
    if kind in ("shear", "endtoend"):
        case["rate"] = log(1e-6, 1e-3)
        case["gamma"] = round(rng.uniform(-0.45, 0.45), 3)
    if kind == "shear":
        case["se_every"] = rng.choice([0, 1, case["steps"]])
    if kind == "resize":
        case["resize"] = log(1e-6, 1e-5)
    if kind == "stress":
        case.update(n=int(log(50, 200000)), aor=round(rng.uniform(0.2, 2.0), 2),
                    gamma=round(rng.uniform(-0.45, 0.45), 3))
    if kind == "ensemble":
        case = dict(kind=kind, precision=precision, nsys=int(log(8, 300)), nmin=rng.randint(20, 200),
                    nmax=int(log(500, 4000)), sizes=rng.randint(0, 999), dt=0.02, pad=case["pad"],
                    steps=rng.randint(5, 20) if precision == "mixed" else rng.randint(2, 5))
    if kind in ("fire", "cg"):
        case.update(phi=round(rng.uniform(0.89, 0.92), 3), nsys=int(log(1, 48 if kind == "fire" else 4)),
                    n=int(log(200, 4096)), iters=rng.choice([20, 50]) if kind == "fire" else 5)
        if kind == "cg":
            del case["precision"]
    return case


# ---- inputs ----

def _systems(case):
    """Per-system sizes, packing fractions, aspect ratios and strain rates."""
    kind = case["kind"]
    if kind == "ensemble":
        rng = np.random.default_rng(case["sizes"])
        k = case["nsys"]
        ns = (np.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"]), k)) / 2).round()
        return (ns.astype(np.int64) * 2, rng.uniform(0.75, 0.90, k), rng.uniform(0.2, 2.0, k),
                np.exp(rng.uniform(math.log(1e-6), math.log(1e-3), k)))
    if kind in ("fire", "cg"):
        k = case["nsys"]
        aor = np.array([0.25, 0.5, 1.0, 2.0])[(4 * np.arange(k)) // k]
        return np.full(k, case["n"]), np.full(k, case["phi"]), aor, np.zeros(k)
    one = np.ones(1)
    return one.astype(np.int64) * case["n"], one * case["phi"], one * case["aor"], \
        one * case.get("rate", 0.0)


class _Packing:
    """Seeded packings of all systems of a case, one after the other, on the GPU.

    Centres start clear of the box faces by more than they move in a pass, so that
    no position is wrapped in it."""

    def __init__(self, case, seed):
        ns, phis, aors, rates = _systems(case)
        self.ns, self.rates = ns, torch.tensor(rates, dtype=F64, device=DEV)
        self.nsys, self.n = len(ns), int(ns.sum())
        cnt = torch.tensor(ns, device=DEV)
        self.cnt = cnt
        self.sys = torch.repeat_interleave(torch.arange(self.nsys, device=DEV), cnt)
        self.p0 = torch.cumsum(cnt, 0) - cnt
        k = torch.arange(self.n, device=DEV) - self.p0[self.sys]
        self.R = torch.where(k % 2 == 0, 0.5, 0.7).to(F64)
        self.A = self.R * torch.tensor(aors, dtype=F64, device=DEV)[self.sys]
        area = torch.zeros(self.nsys, dtype=F64, device=DEV)
        area.index_add_(0, self.sys, PI * self.R ** 2 + 4 * self.A * self.R)
        # the same bits from every run, whatever the order of the sums
        self.L = ((area / torch.tensor(phis, dtype=F64, device=DEV)).sqrt() * 2 ** 20).round() / 2 ** 20
        g = torch.Generator(device=DEV).manual_seed(int(seed))
        L = self.L[self.sys]
        edge = torch.clamp(0.05 * L, max=3.0 if case["kind"] in ("fire", "cg") else 1.0)
        x, y, p = (torch.zeros(self.n, dtype=F64, device=DEV) for _ in range(3))
        todo = torch.ones(self.n, dtype=torch.bool, device=DEV)
        gamma = torch.full_like(self.L, case.get("gamma", 0.0))
        # minimisers start part of the way down, from spines that did not cross on it
        sep = 0.22 if case["kind"] in ("fire", "cg") else 0.1
        for _ in range(600):
            u = torch.rand(3, self.n, dtype=F64, device=DEV, generator=g)
            x = torch.where(todo, edge + u[0] * (L - 2 * edge), x)
            y = torch.where(todo, edge + u[1] * (L - 2 * edge), y)
            p = torch.where(todo, (u[2] - 0.5) * math.pi, p)
            i, j = _near_pairs(self, x, y, gamma, self.A + sep * self.R, 0.0)
            D = _displacement(self, x, y, gamma, i, j)
            q = _Spines(D, p[i], p[j], self.A[i], self.A[j])
            s, t = q.closest()
            near = q.gap2(s, t) < (sep * (self.R[i] + self.R[j])) ** 2
            todo = torch.zeros_like(todo)
            todo[torch.maximum(i, j)[near]] = True
            if not bool(todo.any()):
                break
        self.x, self.y, self.p = x, y, p
        if case["kind"] in ("fire", "cg"):
            e = _Exact(case, seed, self)
            e.descend(80, 0.06, 0.02)
            self.x, self.y, self.p = e.x, e.y, e.p


def _near_pairs(pk, x, y, gamma, half, slack):
    """Pairs (i < j) of one system whose centres, in the sheared frame, are closer than
    half[i] + half[j] + slack; candidates from cells, all pairs in small boxes."""
    top = torch.zeros(pk.nsys, dtype=F64, device=DEV).scatter_reduce_(0, pk.sys, half, "amax")
    reach = 2 * top + slack
    cols = torch.floor(pk.L / (reach * (1 + gamma.abs()))).long()
    rows = torch.floor(pk.L / reach).long()
    grid = (cols >= 3) & (rows >= 3)
    got = []
    cols, rows = cols.clamp(min=1), rows.clamp(min=1)
    if bool(grid.any()):
        c0 = torch.cumsum(cols * rows, 0) - cols * rows
        L = pk.L[pk.sys]
        cx = torch.floor((x % L) / L * cols[pk.sys]).long().clamp(min=0)
        cy = torch.floor((y % L) / L * rows[pk.sys]).long().clamp(min=0)
        cx, cy = torch.minimum(cx, cols[pk.sys] - 1), torch.minimum(cy, rows[pk.sys] - 1)
        cell = c0[pk.sys] + cy * cols[pk.sys] + cx
        order = torch.argsort(cell, stable=True)
        fill = torch.bincount(cell, minlength=int((cols * rows).sum()))
        start = torch.cumsum(fill, 0) - fill
        who = torch.arange(pk.n, device=DEV)
        inside = grid[pk.sys]
        for dx, dy in ((0, 0), (1, 0), (-1, 1), (0, 1), (1, 1)):
            nx, ny = (cx + dx) % cols[pk.sys], (cy + dy) % rows[pk.sys]
            c = c0[pk.sys] + ny * cols[pk.sys] + nx
            k = torch.where(inside, fill[c], 0)
            i = torch.repeat_interleave(who, k)
            off = torch.arange(len(i), device=DEV) - torch.repeat_interleave(torch.cumsum(k, 0) - k, k)
            j = order[start[c][i] + off]
            if dx == 0 and dy == 0:
                i, j = i[i < j], j[i < j]
            got.append(_keep_near(pk, x, y, gamma, half, slack, i, j))
    for s in torch.nonzero(~grid).flatten().tolist():
        m = int(pk.ns[s])
        i, j = torch.triu_indices(m, m, 1, device=DEV)
        p0 = int(pk.p0[s])
        got.append(_keep_near(pk, x, y, gamma, half, slack, i + p0, j + p0))
    i, j = torch.cat([g[0] for g in got]), torch.cat([g[1] for g in got])
    return torch.minimum(i, j), torch.maximum(i, j)


def _keep_near(pk, x, y, gamma, half, slack, i, j):
    dx, dy = _displacement(pk, x, y, gamma, i, j)
    keep = dx * dx + dy * dy < (half[i] + half[j] + slack) ** 2
    return i[keep], j[keep]


def _displacement(pk, x, y, gamma, i, j, L=None):
    """Minimum-image displacement i - j with the Lees-Edwards shift."""
    s = pk.sys[i]
    L = (pk.L if L is None else L)[s]
    dx, dy = x[i] - x[j], y[i] - y[j]
    dx = dx + L * ((dx < -0.5 * L).to(F64) - (dx > 0.5 * L).to(F64))
    dy = dy + L * ((dy < -0.5 * L).to(F64) - (dy > 0.5 * L).to(F64))
    return dx + gamma[s] * dy, dy


# ---- the 64-bit computation ----

def _clamp(v):
    return torch.clamp(torch.nan_to_num(v, nan=-1.0), -1.0, 1.0)


class _Spines:
    """Two spines: P + s u and Q + t v, with P - Q = D."""

    def __init__(self, D, pp, pq, ap, aq):
        self.X, self.Y = D
        self.ux, self.uy = ap * torch.cos(pp), ap * torch.sin(pp)
        self.vx, self.vy = aq * torch.cos(pq), aq * torch.sin(pq)
        self.a, self.c = ap * ap, aq * aq
        self.b = -(self.ux * self.vx + self.uy * self.vy)
        self.d = self.ux * self.X + self.uy * self.Y
        self.e = -self.vx * self.X - self.vy * self.Y
        self.delta = self.a * self.c - self.b * self.b

    def gap(self, s, t):
        return self.X + s * self.ux - t * self.vx, self.Y + s * self.uy - t * self.vy

    def gap2(self, s, t):
        gx, gy = self.gap(s, t)
        return gx * gx + gy * gy

    def s_at(self, t):
        return -(self.b * t + self.d) / self.a

    def t_at(self, s):
        return -(self.b * s + self.e) / self.c

    def closest(self):
        t = _clamp((self.b * self.d - self.a * self.e) / self.delta)
        s = self.s_at(t)
        t = torch.where(s.abs() > 1, _clamp(self.t_at(_clamp(s))), t)
        return _clamp(s), t

    def two(self):
        """Both contacts of the two-point rule (crossing directions): s1, t1, s2, t2 and
        whether the second is another one."""
        w = torch.where
        t1 = _clamp((self.b * self.d - self.a * self.e) / self.delta)
        s1 = self.s_at(t1)
        end = s1.abs() >= 1
        s1 = _clamp(s1)
        t1 = w(end, _clamp(self.t_at(s1)), t1)
        flip = self.b < 0
        # the first contact at an end of P
        s2 = -s1
        t2 = self.t_at(s2)
        out = t2.abs() > 1
        t2 = _clamp(t2)
        s2 = w(out, _clamp(self.s_at(t2)), s2)
        t3 = w(flip, -s1, s1)
        s3 = self.s_at(t3)
        t3 = w(s3.abs() >= 1, _clamp(self.t_at(_clamp(s3))), t3)
        s3, t3 = w(out, s2, _clamp(s3)), w(out, t2, t3)
        # inside P
        t2b = -t1
        s2b = self.s_at(t2b)
        outb = s2b.abs() > 1
        s2b = _clamp(s2b)
        t2b = w(outb, _clamp(self.t_at(s2b)), t2b)
        s3b = w(flip, -t1, t1)
        t3b = self.t_at(s3b)
        s3b = w(t3b.abs() >= 1, _clamp(self.s_at(_clamp(t3b))), s3b)
        s3b, t3b = w(outb, s2b, s3b), w(outb, t2b, _clamp(t3b))
        s2, t2, s3, t3 = w(end, s2, s2b), w(end, t2, t2b), w(end, s3, s3b), w(end, t3, t3b)
        other = (s1 != s2) & (t1 != t2)
        nearer = other & (s3 != s1) & (s3 != s2) & (self.gap2(s3, t3) < self.gap2(s2, t2))
        return s1, t1, w(nearer, s3, s2), w(nearer, t3, t2), other


class _Exact:
    """Forces, stress and the protocols of a packing in 64 bits."""

    def __init__(self, case, seed, pk=None):
        self.case, self.pk = case, pk or _Packing(case, seed)
        pk = self.pk
        self.x, self.y, self.p = pk.x, pk.y, pk.p
        self.gamma = torch.full((pk.nsys,), case.get("gamma", 0.0), dtype=F64, device=DEV)
        self.L = pk.L
        al = pk.A / pk.R
        C = 3 * PI + 24 * al + 6 * PI * al ** 2 + 8 * al ** 3
        self.inertia = pk.R ** 4 * C / (6 * pk.R * (PI * pk.R + 4 * pk.A))
        self.rc = (8 * al + 6 * PI * al ** 2 + 8 * al ** 3) / C
        self.pairs = None

    def near(self):
        """Candidate pairs, renewed when something has moved a quarter of their slack."""
        if self.pairs is not None:
            dx, dy, dp = self.x - self.at[0], self.y - self.at[1], self.p - self.at[2]
            if float((dx.abs() + dy.abs() + self.pk.A * dp.abs()).max()) < 0.1:
                return self.pairs
        self.at = self.x, self.y, self.p
        self.pairs = _near_pairs(self.pk, self.x, self.y, self.gamma, self.pk.R + self.pk.A, 0.5)
        return self.pairs

    def forces(self, x, y, p, gamma, L, stress=False):
        pk, (i, j) = self.pk, self.near()
        two = self.case.get("contacts", 1) == 2
        D = _displacement(pk, x, y, gamma, i, j, L)
        sig = pk.R[i] + pk.R[j]
        q = _Spines(D, p[i], p[j], pk.A[i], pk.A[j])
        if two:
            s1, t1, s2, t2, other = q.two()
            contacts = [(s1, t1, torch.ones_like(other)), (s2, t2, other)]
        else:
            contacts = [(*q.closest(), torch.ones_like(i, dtype=torch.bool))]
        f = [torch.zeros(pk.n, dtype=F64, device=DEV) for _ in range(3)]
        se = torch.zeros(5, pk.nsys, dtype=F64, device=DEV) if stress else None
        for s, t, on in contacts:
            gx, gy = q.gap(s, t)
            r2 = gx * gx + gy * gy
            k = torch.nonzero(on & (r2 < sig * sig)).flatten()
            ik, jk, sk, tk, gx, gy, r, sg = i[k], j[k], s[k], t[k], gx[k], gy[k], r2[k].sqrt(), sig[k]
            ux, uy, vx, vy = q.ux[k], q.uy[k], q.vx[k], q.vy[k]
            dv = (1 - r / sg) / sg
            fx, fy = gx * dv / r, gy * dv / r
            to = (torch.cat([ik, jk]),)  # a sum in the same order every time
            f[0].index_put_(to, torch.cat([fx, -fx]), accumulate=True)
            f[1].index_put_(to, torch.cat([fy, -fy]), accumulate=True)
            f[2].index_put_(to, torch.cat([sk * (ux * fy - uy * fx), tk * (vy * fx - vx * fy)]),
                            accumulate=True)
            if stress:
                sy = pk.sys[ik]
                LL = (L * L)[sy]
                cxa, cya = sk * ux - 0.5 * gx, sk * uy - 0.5 * gy
                cxb = tk * vx + 0.5 * gx
                # one-point contacts: the reference's own sums, its slips included
                cyb = tk * (vy if two else vx) + 0.5 * gy
                pxx = fx * (cxa - cxb) - (0 if two else fy * cxb)
                pxy = fy * (cxa - (cxb if two else 0))
                terms = (dv * sg * (1 - r / sg) / (2 * pk.cnt[sy]), pxx / LL, fy * (cya - cyb) / LL,
                         pxy / LL, fx * (cya - cyb) / LL)
                for m, v in enumerate(terms):
                    se[m].index_add_(0, sy, v)
        return f, (se.T.contiguous() if stress else None)

    def stress(self):
        f, se = self.forces(self.x, self.y, self.p, self.gamma, self.L, True)
        return f, se

    def turn(self, p):
        return self.pk.rates[self.pk.sys] * 0.5 * (1 - self.rc * torch.cos(2 * p))

    def shear(self, steps, dt, se_every=0):
        pk, sy, got = self.pk, self.pk.sys, []
        for k in range(1, steps + 1):
            f, _ = self.forces(self.x, self.y, self.p, self.gamma, self.L)
            v0 = f[0] - self.gamma[sy] * f[1], f[1], f[2] / self.inertia - self.turn(self.p)
            g1 = self.gamma + dt * pk.rates
            xt, yt, pt = self.x + dt * v0[0], self.y + dt * v0[1], self.p + dt * v0[2]
            f, _ = self.forces(xt, yt, pt, g1, self.L)
            v1 = f[0] - g1[sy] * f[1], f[1], f[2] / self.inertia - self.turn(pt)
            self.x = self.x + 0.5 * dt * (v0[0] + v1[0])
            self.y = self.y + 0.5 * dt * (v0[1] + v1[1])
            self.p = self.p + 0.5 * dt * (v0[2] + v1[2])
            self.gamma = g1
            if se_every and k % se_every == 0:
                got.append(self.stress()[1])
        return got

    def descend(self, steps, dt, most):
        """Steepest descent, no spine end moving further than `most` in a step."""
        for _ in range(steps):
            f, _ = self.forces(self.x, self.y, self.p, self.gamma, self.L)
            turn = f[2] / self.inertia
            far = dt * ((f[0] ** 2 + f[1] ** 2).sqrt() + self.pk.A * turn.abs())
            h = dt * torch.clamp(most / far, max=1.0)
            self.x, self.y, self.p = self.x + h * f[0], self.y + h * f[1], self.p + h * turn

    def resize(self, steps, dt, rate):
        f = (1.0 - rate) ** dt
        for _ in range(steps):
            f0, _ = self.forces(self.x, self.y, self.p, self.gamma, self.L)
            xt, yt = (self.x + dt * f0[0]) * f, (self.y + dt * f0[1]) * f
            pt = self.p + dt * f0[2] / self.inertia
            f1, _ = self.forces(xt, yt, pt, self.gamma, self.L)
            self.x = (self.x + 0.5 * dt * (f0[0] + f1[0])) * f
            self.y = (self.y + 0.5 * dt * (f0[1] + f1[1])) * f
            self.p = self.p + 0.5 * dt * (f0[2] + f1[2]) / self.inertia
            self.L = self.L * f

    def fire(self, iters, dt0=1e-2, dt_max=0.2):
        pk, m = self.pk, self.pk.nsys
        I = self.inertia.view(m, -1)
        v = [torch.zeros_like(I) for _ in range(3)]
        dt = torch.full((m, 1), dt0, dtype=F64, device=DEV)
        alpha, npos = torch.full_like(dt, 0.1), torch.zeros_like(dt)
        for _ in range(iters):
            f, _ = self.forces(self.x, self.y, self.p, self.gamma, self.L)
            fx, fy, tq = (a.view(m, -1) for a in f)
            P = (fx * v[0] + fy * v[1] + tq * v[2]).sum(1, keepdim=True)
            vv = (v[0] ** 2 + v[1] ** 2 + I * v[2] ** 2).sum(1, keepdim=True)
            ff = (fx ** 2 + fy ** 2 + tq ** 2 / I).sum(1, keepdim=True)
            c1, c2 = 1 - alpha, alpha * (vv / ff).sqrt()
            up = P > 0
            npos = torch.where(up, npos + 1, 0.0)
            fast = up & (npos > 5)
            dt = torch.where(fast, torch.clamp(dt * 1.1, max=dt_max), torch.where(up, dt, dt * 0.5))
            alpha = torch.where(fast, alpha * 0.99, torch.where(up, alpha, 0.1))
            a = fx, fy, tq / I
            v = [torch.where(up, c1 * w + c2 * g, 0.0) + dt * g for w, g in zip(v, a)]
            self.x = self.x + (dt * v[0]).reshape(-1)
            self.y = self.y + (dt * v[1]).reshape(-1)
            self.p = self.p + (dt * v[2]).reshape(-1)


def exact(case, seed):
    kind = case["kind"]
    if kind == "cg":  # its path is decided by comparisons of equal energies
        return None
    e = _Exact(case, seed)
    if kind == "stress":
        f, se = e.stress()
        return {"se": se.cpu().numpy(), "f": tuple(v.cpu().numpy() for v in f)}
    se = None
    if kind in ("shear", "ensemble"):
        got = e.shear(case["steps"], case["dt"], case.get("se_every", 0))
        se = torch.stack(got).cpu().numpy() if got else None
    elif kind == "endtoend":
        e.shear(case["steps"], case["dt"])
        se = e.stress()[1].cpu().numpy()
    elif kind == "resize":
        e.resize(case["steps"], case["dt"], case["resize"])
    elif kind == "fire":
        e.fire(case["iters"])
    out = {"x": e.x, "y": e.y, "phi": e.p}
    if se is not None:
        out["se"] = se
    return out


# ---- the calls ----

def prepare(case, seed):
    pk = _Packing(case, seed)
    pad = case["pad"]
    host = [v.cpu().pin_memory().numpy() for v in (pk.x, pk.y, pk.p, pk.A, pk.R)]
    state = {"case": case, "grow": False, "L": pk.L.cpu().numpy(), "ns": pk.ns, "host": host,
             "rates": pk.rates.cpu().numpy(),
             "out": tuple(torch.empty(pk.n, dtype=F64, pin_memory=True).numpy() for _ in range(3))}
    if case["kind"] != "endtoend":
        state["box"] = _box(state, pad)
    return state


def _box(state, pad):
    case = state["case"]
    x, y, p, A, R = state["host"]
    box = BoxBatch(state["ns"], state["L"], x, y, p, A, R, pad,
                   precision=case.get("precision", "fp64"), contacts=case.get("contacts", 1))
    if case["kind"] in ("shear", "ensemble", "endtoend"):
        for s, r in enumerate(state["rates"]):
            box.set_strain_rate(float(r), sys=s)
    if "dt" in case:
        box.set_step(case["dt"])
    if "resize" in case:
        box.set_resize_rate(case["resize"])
    if case.get("gamma"):
        box.set_gamma(case["gamma"])
    return box


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "endtoend":
        with _box(state, case["pad"]) as box:
            box.strain_steps(case["steps"])
            se = box.calc_se()
            x, y, p = box.state(out=state["out"])
        return {"x": x, "y": y, "phi": p, "se": se}
    box = state["box"]
    if kind == "stress":
        return {"se": box.calc_se(), "f": box.forces()}
    more = {}
    if kind in ("shear", "ensemble"):
        se = box.strain_steps(case["steps"], case.get("se_every", 0))
        if se is not None:
            more["se"] = se
    elif kind == "resize":
        box.resize_steps(case["steps"], shrink=not state["grow"])
        state["grow"] = not state["grow"]
    elif kind == "fire":
        more["iters"], _, _ = box.fire_minimize(1e-14, case["iters"])
    elif kind == "cg":
        more["iters"], more["energy"], more["why"] = box.cg_minimize(case["iters"])
    x, y, p = box.state(out=state["out"])
    return {"x": x, "y": y, "phi": p, **more}


def work(case):
    """Each force evaluation reads the state (x, y, phi, R, A) and writes what follows from
    it (three values) once; about 2.5 contacts a particle of 100 operations each."""
    kind = case["kind"]
    n = case["n"] * case.get("nsys", 1) if "n" in case else \
        case["nsys"] * (case["nmax"] - case["nmin"]) / math.log(case["nmax"] / case["nmin"])
    evals = {"stress": 1, "fire": case.get("iters", 1), "cg": 30 * case.get("iters", 1)}.get(
        kind, 2 * case.get("steps", 1))
    if kind == "endtoend":
        evals += 2
    return {"bytes": 64.0 * n * evals, "flops": 250.0 * n * evals}
