"""Timed workloads of the library, through its public entry points.

A case is a dict of plain values: what is simulated (``model``), its size,
the arithmetic mode (``precision``) and what one pass does (``call``):

  steps     the next ``steps`` velocity-Verlet steps, then a read of the
            positions, velocities and damage (what a program does between
            two file writes); with contacts the neighbour lists are rebuilt
            every ``neigh`` steps, as ``run`` does
  evaluate  one ``save_state``: a force evaluation and the damage, then a
            read of the accelerations
  minimize  one quasi-static load increment (``QSDrag``)

A pass continues from the state the previous one left, as a simulation
does.  Sizes follow ``peridyn_b200.configs``; the seed sets the jitter, the
pulses, the critical stretches and the loading rates.  Velocities and
accelerations of the "fp32c" mode are held in 32 bits and returned so.
"""
import math
import random

import numpy as np
import torch

import peridyn_b200 as pb
from peridyn_b200 import configs, lattice

SPACING = 1.0e-3


def listed():
    return [
        # a small study in the default arithmetic (bit-identical to the serial loop): latency and launches
        {"name": "cube_1k_serial", "model": "pmb", "nx": 9, "ny": 10, "nz": 11, "precision": "fp64_serial",
         "call": "steps", "steps": 20},
        # the tensile bar in the default arithmetic: the parity run of a state-based solid
        {"name": "bar_40k_serial", "model": "bar", "nx": 100, "ny": 20, "nz": 20, "precision": "fp64_serial",
         "call": "steps", "steps": 20},
        # one quasi-static load increment of a bar (always serial arithmetic)
        {"name": "bar_9k_quasistatic", "model": "bar", "nx": 61, "ny": 13, "nz": 12, "precision": "fp64_serial",
         "call": "minimize", "steps": 40},
        # the single jittered cube of 8,000 particles: launch latency of the throughput mode
        {"name": "cube_8k_fp32c", "model": "pmb", "nx": 20, "ny": 20, "nz": 20, "precision": "fp32c",
         "call": "steps", "steps": 200},
        # the tensile bar in the throughput mode: dilatation and force passes, boundary conditions
        {"name": "bar_40k_fp32c", "model": "bar", "nx": 100, "ny": 20, "nz": 20, "precision": "fp32c",
         "call": "steps", "steps": 200},
        # an ordinary state-based body with odd edges in plain FP64
        {"name": "lps_71k_fp64", "model": "lps", "nx": 47, "ny": 41, "nz": 37, "precision": "fp64",
         "call": "steps", "steps": 50},
        # the batched study: 256 uneven specimens of 12 to 32 per edge, the largest call
        {"name": "batch_256_fp32c", "model": "batch", "nspec": 256, "lo": 12, "hi": 32, "layout": 4,
         "precision": "fp32c", "call": "steps", "steps": 400},
        # a smaller batch in plain FP64
        {"name": "batch_64_fp64", "model": "batch", "nspec": 64, "lo": 12, "hi": 32, "layout": 7,
         "precision": "fp64", "call": "steps", "steps": 100},
        # a stiff sphere striking a disk: contact forces and neighbour updates between steps
        {"name": "impact_fp32c", "model": "impact", "radius": 0.02, "layers": 8, "sphere": 0.004,
         "precision": "fp32c", "call": "steps", "steps": 100, "neigh": 50},
        # an elasto-plastic (Von Mises) bar pulled past its yield stress
        {"name": "ep_bar_10k_fp32c", "model": "ep", "nx": 50, "ny": 14, "nz": 14, "precision": "fp32c",
         "call": "steps", "steps": 50},
        # one file write of a state-based body: a single force evaluation
        {"name": "lps_139k_evaluate", "model": "lps", "nx": 61, "ny": 53, "nz": 43, "precision": "fp32c",
         "call": "evaluate", "steps": 1},
        # a large state-based body in the throughput mode
        {"name": "lps_402k_fp32c", "model": "lps", "nx": 80, "ny": 75, "nz": 67, "precision": "fp32c",
         "call": "steps", "steps": 60},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _edges(rng, n):
    """Three uneven edges of a body of about n particles."""
    a, b = rng.uniform(0.7, 1.4), rng.uniform(0.7, 1.4)
    e = n ** (1.0 / 3.0)
    return [max(4, int(round(e * s))) for s in (a, b, 1.0 / (a * b))]


def draw(rng):
    kind = rng.choice(["pmb", "pmb", "bar", "lps", "lps", "batch", "batch", "minimize", "evaluate", "impact", "ep"])
    precision = rng.choice(["fp64_serial", "fp64", "fp32c", "fp32c"])
    top = {"fp64_serial": 6.0e4, "fp64": 4.0e5, "fp32c": 1.5e6}[precision]
    if kind in ("pmb", "lps", "evaluate"):
        n = _log_int(rng, 500, top)
        e = _edges(rng, n)
        c = {"model": rng.choice(["pmb", "lps"]) if kind == "evaluate" else kind, "nx": e[0], "ny": e[1], "nz": e[2],
             "precision": precision, "call": "evaluate" if kind == "evaluate" else "steps"}
        c["steps"] = 1 if kind == "evaluate" else max(5, min(300, int(3.0e6 / n)))
        return c
    if kind in ("bar", "ep"):
        w = rng.randint(6, 22)
        h = rng.randint(6, 22)
        return {"model": kind, "nx": rng.randint(20, 120), "ny": w, "nz": h, "precision": precision, "call": "steps",
                "steps": rng.randint(10, 40 if kind == "ep" or precision == "fp64_serial" else 200)}
    if kind == "minimize":
        return {"model": "bar", "nx": rng.randint(20, 90), "ny": rng.randint(5, 16), "nz": rng.randint(5, 16),
                "precision": "fp64_serial", "call": "minimize", "steps": rng.randint(5, 60)}
    if kind == "batch":
        nspec = _log_int(rng, 4, {"fp64_serial": 16, "fp64": 64, "fp32c": 200}[precision])
        lo = rng.randint(8, 14)
        return {"model": "batch", "nspec": nspec, "lo": lo, "hi": rng.randint(lo + 4, 30),
                "layout": rng.randint(1, 10 ** 6), "precision": precision, "call": "steps",
                "steps": rng.randint(5, 20) if precision == "fp64_serial" else rng.randint(20, 120)}
    return {"model": "impact", "radius": round(rng.uniform(0.006, 0.022), 4), "layers": rng.randint(3, 10),
            "sphere": round(rng.uniform(0.0015, 0.004), 5), "precision": rng.choice(["fp64", "fp32c"]),
            "call": "steps", "steps": rng.choice([40, 60, 100]), "neigh": rng.choice([10, 20, 50])}


# ---------------------------------------------------------------------------
# workloads
# ---------------------------------------------------------------------------
def _specimen_edges(case):
    r = random.Random(case["layout"])
    return [[r.randint(case["lo"], case["hi"]) for _ in range(3)] for _ in range(case["nspec"])]


def _pulsed(model, dims, rng, seed, **kw):
    """A jittered cuboid with a velocity pulse: peak and critical stretch as
    in the batched study."""
    cs, peak = rng.uniform(0.002, 0.01), rng.uniform(5.0, 50.0)
    if model == "lps":
        return configs.lps_cube(tuple(dims), cs=cs, peak=peak, seed=seed)
    return configs.pmb_cube(dims=dims, cs=cs, peak=peak, seed=seed, **kw)


def _workload(case, seed):
    rng = random.Random(seed)
    s = rng.randrange(1 << 40)
    if case["model"] in ("pmb", "lps"):
        w = _pulsed(case["model"], (case["nx"], case["ny"], case["nz"]), rng, s)
        if case["call"] == "evaluate":  # a body already set moving by its pulse
            gen = w["materials"][0].general
            gen.y += 2.0e-7 * gen.velocity
            gen.deformed = [True]
        return w
    if case["model"] == "batch":
        mats = []
        for k, e in enumerate(_specimen_edges(case)):
            w = _pulsed("pmb", e, rng, s + k, origin=(k * 40 * SPACING, 0.0, 0.0), type_id=k + 1,
                        name="specimen%d" % k)
            mats += w["materials"]
        return {"materials": mats, "contacts": [], "bcs": [], "dt": w["dt"]}
    if case["model"] == "bar":
        return configs.lps_bar(nx=case["nx"], ny=case["ny"], nz=case["nz"], E=rng.uniform(60e9, 80e9),
                               pull=rng.uniform(1.0, 3.0))
    if case["model"] == "ep":
        # stretched to near the yield strain, so that the pulled bar yields within the pass
        w = configs.ep_bar(nx=case["nx"], ny=case["ny"], nz=case["nz"], yield_stress=rng.uniform(1e6, 3e6))
        gen = w["materials"][0].general
        gen.y[0] *= 1.0 + rng.uniform(1e-5, 4e-5)
        gen.deformed = [True]
        return w
    # impact: the sphere starts inside the contact distance of the disk
    return configs.disk_impact(radius=case["radius"], thickness=case["layers"] * 2.5e-4,
                               sphere_radius=case["sphere"], speed=rng.uniform(30.0, 60.0))


def prepare(case, seed):
    w = _workload(case, seed)
    env = pb.Env(1, w["materials"], w["contacts"], w["bcs"], w["dt"], precision=case["precision"])
    pb.update_neighs(env)
    pb.apply_bc_at0(env, 0)
    pb.update_acc(env)
    solver = None
    if case["call"] == "minimize":
        solver = pb.QSDrag(5.0e-8, 1.0e3, max_iter=case["steps"], x_tol=1e-14, f_tol=1e-3)
    return {"case": case, "env": env, "solver": solver}


def _rate(case, a):
    return a.astype(np.float32) if case["precision"] == "fp32c" else a


def run(state):
    case, env = state["case"], state["env"]
    if case["call"] == "evaluate":
        damage = pb.save_state(env)
        return {"f": _rate(case, env.f), "damage": damage}
    if case["call"] == "minimize":
        it = pb.minimize(env, state["solver"])
        return {"iterations": it, "y": env.y, "f": env.f}
    neigh = case.get("neigh", case["steps"])
    for k in range(0, case["steps"], neigh):
        pb.velocity_verlet_step(env, nsteps=min(neigh, case["steps"] - k))
        if env.short_range_contact:
            pb.update_neighs(env)
    return {"y": env.y, "v": _rate(case, env.v), "damage": pb.cal_damage(env)}


# ---------------------------------------------------------------------------
# the work of one pass
# ---------------------------------------------------------------------------
def _lattice_bonds(nx, ny, nz, factor):
    """Directed bonds of a lattice: offsets shorter than factor spacings."""
    r, n = int(math.ceil(factor)), 0
    for i in range(-r, r + 1):
        for j in range(-r, r + 1):
            for k in range(-r, r + 1):
                if 0 < i * i + j * j + k * k < factor * factor:
                    n += max(0, nx - abs(i)) * max(0, ny - abs(j)) * max(0, nz - abs(k))
    return n


def _parts(case):
    """(particles, directed bonds, law, force evaluations) of every body."""
    n = case["steps"]
    if case["model"] in ("pmb", "lps", "bar", "ep"):
        d = (case["nx"], case["ny"], case["nz"])
        return [(d[0] * d[1] * d[2], _lattice_bonds(*d, 3.0 if case["model"] in ("bar", "ep") else 3.015),
                 case["model"], n)]
    if case["model"] == "batch":
        return [(math.prod(e), _lattice_bonds(*e, 3.015), "pmb", n) for e in _specimen_edges(case)]
    e = 2.5e-4
    disk = math.pi * (case["radius"] / e) ** 2
    ball = 4.0 / 3.0 * math.pi * (case["sphere"] / e) ** 3
    # bonds of an infinite plate of that many layers
    side = 64
    per = _lattice_bonds(side, side, case["layers"], 3.015) / (side * side * case["layers"])
    return [(int(disk * case["layers"]), int(disk * case["layers"] * per), "pmb", n),
            (int(ball), int(ball * 105), "pmb", n)]


def work(case):
    """Per force evaluation: the reference position and weight read, the
    displacement and velocity read and written, one flag bit per directed
    bond; every undirected bond evaluated once per pass over the bonds."""
    real = 4 if case["precision"] == "fp32c" else 8
    moved = flops = 0.0
    for n, bonds, law, evals in _parts(case):
        state = 4 * real + 2 * (3 * real + 24)
        moved += evals * (n * state + bonds / 8.0)
        if law in ("bar", "lps"):
            moved += evals * n * 2 * real
        if law == "ep":
            moved += evals * (n * 3 * real + 2 * 8 * bonds)
        flops += evals * (bonds / 2.0) * {"pmb": 40.0, "bar": 75.0, "lps": 75.0, "ep": 150.0}[law]
    return {"bytes": moved, "flops": flops}


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def _family(x, spacing, horizon):
    """Directed bonds (i, j) of points near a lattice of that spacing."""
    lo = x.min(dim=1, keepdim=True).values
    c = torch.round((x - lo) / spacing).long()
    r = int(math.ceil(horizon / spacing))
    dims = [int(v) + 1 + 2 * r for v in c.max(dim=1).values]
    c = c + r
    cell = torch.full((dims[0] * dims[1] * dims[2],), -1, dtype=torch.long, device=x.device)
    at = c[0] + dims[0] * (c[1] + dims[1] * c[2])
    cell[at] = torch.arange(x.shape[1], device=x.device)
    ii, jj = [], []
    for dz in range(-r, r + 1):
        for dy in range(-r, r + 1):
            for dx in range(-r, r + 1):
                if dx == dy == dz == 0:
                    continue
                j = cell[at + dx + dims[0] * (dy + dims[1] * dz)]
                i = torch.nonzero(j >= 0).reshape(-1)
                j = j[i]
                d = x[:, i] - x[:, j]
                keep = (d[0] * d[0] + d[1] * d[1]) + d[2] * d[2] < horizon * horizon
                ii.append(i[keep])
                jj.append(j[keep])
    i, j = torch.cat(ii), torch.cat(jj)
    order = torch.argsort(i, stable=True)
    return i[order], j[order]


class _Body:
    """One block: its bonds and constants."""

    def __init__(self, mat, dev):
        gen, spc = mat.general, mat.specific
        put = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
        self.kind = type(spc).__name__
        self.x, self.vol = put(gen.x), put(gen.volume)
        self.n = gen.n
        self.rho = float(spc.density[0])
        spacing = float(gen.volume[0]) ** (1.0 / 3.0)
        self.i, self.j = _family(self.x, spacing, gen.horizon)
        X = self.x[:, self.j] - self.x[:, self.i]
        self.X = X.square().sum(dim=0).sqrt()
        self.live = torch.ones(self.i.shape[0], dtype=torch.bool, device=dev)
        self.count0 = torch.bincount(self.i, minlength=self.n)
        self.deformed = bool(gen.deformed[0])
        self.cs = float(spc.critical_stretch[0, 0])
        if self.kind == "BondBasedSpecific":
            self.c = float(spc.bond_stiffness[0, 0])
        else:
            K, G = float(spc.bulk_modulus[0, 0]), float(spc.shear_modulus[0, 0])
            self.k = 3 * K if self.kind == "ElastoPlasticSolidSpecific" else 3 * K - 5 * G
            self.g = 15 * G
            self.m = self._sum(self.X * self.vol[self.j])
        if self.kind == "ElastoPlasticSolidSpecific":
            self.psi2 = 2 * float(spc.psi[0, 0])
            self.edp = torch.zeros_like(self.X)
            key = self.i * self.n + self.j
            back = self.j * self.n + self.i
            key, order = torch.sort(key)
            self.reverse = order[torch.searchsorted(key, back)]

    def _sum(self, t):
        return torch.zeros(self.n, dtype=torch.float64, device=t.device).index_add_(0, self.i, t)

    def force(self, y):
        if not self.deformed:
            a = y - y[:, :1] + self.x[:, :1]
            self.deformed = not bool((a - self.x).norm() <= 2.0 ** -26 * max(a.norm(), self.x.norm()))
        if not self.deformed:
            return torch.zeros_like(y)
        Y = y[:, self.j] - y[:, self.i]
        L = Y.square().sum(dim=0).sqrt()
        e = L - self.X
        s = e / self.X
        vj = self.vol[self.j]
        if self.kind != "BondBasedSpecific":
            theta = 3.0 / self.m * self._sum(torch.where(self.live, e * vj, torch.zeros_like(e)))
        self.live &= s < self.cs
        if self.kind == "BondBasedSpecific":
            t = self.c * s
        elif self.kind == "OrdinaryStateBasedSpecific":
            tm = theta / self.m
            t = self.k * (tm[self.i] + tm[self.j]) + self.g * s * (1 / self.m[self.i] + 1 / self.m[self.j])
        else:
            a, b = 1 / (self.X * self.m[self.i]), 1 / (self.X * self.m[self.j])
            tw = theta[self.i] * a + theta[self.j] * b
            ede = e - tw / (a + b) * self.X / 3 - self.edp
            trial = self.g * (a + b) * ede
            td2 = self._sum(torch.where(self.live, trial.square() * vj, torch.zeros_like(e)))
            C = (self.psi2 / td2[self.i]).sqrt()
            plastic = ~(C > 1)
            own = self.k * self.X * tw + torch.where(plastic, C * trial, trial)
            t = 0.5 * (own + own[self.reverse])
            self.edp = torch.where(self.live & plastic, self.edp + ede * (1 - C), self.edp)
        w = torch.where(self.live, t / L * vj / self.rho, torch.zeros_like(t))
        return torch.stack([self._sum(w * Y[d]) for d in range(3)])

    def damage(self):
        return 1.0 - self._sum(self.live.double()) / self.count0


class _System:
    """All blocks of an environment, with its boundary conditions and contact."""

    def __init__(self, w, dev):
        self.bodies = [_Body(m, dev) for m in w["materials"]]
        self.dt, self.contact = w["dt"], (w["contacts"] or [None])[0]
        self.at = np.cumsum([0] + [b.n for b in self.bodies])
        gens = [m.general for m in w["materials"]]
        put = lambda a: torch.from_numpy(np.ascontiguousarray(np.concatenate(a, axis=1))).to(dev)  # noqa: E731
        self.y, self.v = put([g.y for g in gens]), put([g.velocity for g in gens])
        self.f = torch.zeros_like(self.y)
        self.bcs = [(torch.from_numpy(np.nonzero(bc.bool)[0]).to(dev), torch.from_numpy(bc.rate).to(dev).view(3, 1))
                    for bc in w["bcs"]]
        self.last = [self.y[:, m].clone() for m, _ in self.bcs]
        self.size = gens[0].particle_size
        self.pairs = None
        self.neighbours()

    def span(self, b):
        return slice(int(self.at[b]), int(self.at[b + 1]))

    def neighbours(self):
        """Two-block contact (first block to second): within the search
        distance, the largest indices first, at most max_neighs of them."""
        if self.contact is None:
            return
        a, b, d = self.y[:, self.span(0)], self.y[:, self.span(1)], self.contact.distance
        lo = torch.maximum(a.min(dim=1).values, b.min(dim=1).values).view(3, 1) - d
        hi = torch.minimum(a.max(dim=1).values, b.max(dim=1).values).view(3, 1) + d
        ia, ib = (torch.nonzero(((p > lo) & (p < hi)).all(dim=0)).reshape(-1) for p in (a, b))
        pi, pj = [], []
        for part in torch.split(ia, 512):
            D = a[:, part].unsqueeze(2) - b[:, ib].unsqueeze(1)
            near = (D[0] * D[0] + D[1] * D[1]) + D[2] * D[2] < d * d
            rank = near.long().flip(1).cumsum(1).flip(1)
            r, c = torch.nonzero(near & (rank <= self.contact.max_neighs), as_tuple=True)
            pi.append(part[r])
            pj.append(ib[c] + int(self.at[1]))
        self.pairs = (torch.cat(pi), torch.cat(pj)) if pi else None

    def evaluate(self):
        self.f = torch.cat([b.force(self.y[:, self.span(k)]) for k, b in enumerate(self.bodies)], dim=1)
        if self.pairs is None:
            return
        i, j = self.pairs
        c = self.contact
        D = self.y[:, i] - self.y[:, j]
        r = D.square().sum(dim=0).sqrt()
        strain = (c.equi_dist - r) / c.equi_dist
        s = torch.where(strain >= 0, c.stifness * strain.clamp(min=0) ** c.exponent / (r + 1e-10),
                        torch.zeros_like(r))
        A, B = self.bodies[0], self.bodies[1]
        self.f.index_add_(1, i, s * D * B.vol[j - int(self.at[1])] / A.rho)
        self.f.index_add_(1, j, -s * D * A.vol[i] / B.rho)

    def place(self):
        for k, (m, rate) in enumerate(self.bcs):
            self.last[k] = self.last[k] + self.dt * rate
            self.y[:, m] = self.last[k]

    def hold(self):
        for m, rate in self.bcs:
            self.v[:, m] = rate

    def step(self):
        self.v = self.v + self.dt / 2 * self.f
        self.y = self.y + self.dt * self.v
        self.place()
        self.evaluate()
        self.v = self.v + self.dt / 2 * self.f
        self.hold()

    def minimize(self, solver):
        self.place()
        self.hold()
        free = torch.ones(self.y.shape[1], dtype=torch.bool, device=self.y.device)
        for m, _ in self.bcs:
            free[m] = False
        o = torch.zeros_like(self.y[:, free])
        h, a = solver.step_size, self.size / 10
        for it in range(1, solver.max_iter + 1):
            self.evaluate()
            g = self.f[:, free]
            force = g - solver.drag * o * (1.0 + solver.drag / 10 * o.abs())
            dy = (0.5 * force * (h * h) + o * h).clamp(-a, a)
            o = o + h * force
            self.y[:, free] += dy
            if float(g.abs().max()) < solver.f_tol and float(dy.abs().max()) < solver.x_tol:
                break
        return it

    def damage(self):
        return torch.cat([b.damage() for b in self.bodies])


def exact(case, seed):
    parts = _parts(case)
    if sum(b * e for _, b, _, e in parts) > 8.0e9 or sum(b for _, b, _, _ in parts) > 9.0e7:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    with torch.no_grad():
        s = _System(_workload(case, seed), dev)
        s.evaluate()
        if case["call"] == "evaluate":
            s.evaluate()
            return {"f": s.f, "damage": s.damage()}
        if case["call"] == "minimize":
            it = s.minimize(pb.QSDrag(5.0e-8, 1.0e3, max_iter=case["steps"], x_tol=1e-14, f_tol=1e-3))
            return {"iterations": it, "y": s.y, "f": s.f}
        for k in range(case["steps"]):
            s.step()
            if (k + 1) % case.get("neigh", case["steps"]) == 0:
                s.neighbours()
        return {"y": s.y, "v": s.v, "damage": s.damage()}
