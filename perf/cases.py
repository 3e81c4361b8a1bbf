"""Workloads by which the speed of the explicit step is judged.

A case is one stretch of a run as a program drives it through the public
entry points: the particle state goes from page-locked host buffers to the
device (``Solver.upload``), the loop advances a number of iterations (fused
``run``, the split ``step`` of a host driver, a ``Batch`` of bodies, or a
gradient), and the state or the gradients come back to page-locked buffers.
Every pass starts from the same uploaded state, so passes repeat.

The decks are those of ``mcmtop_b200.deck``: the Taylor bar, the fluid column
with its ghost-particle walls, the calibration ensemble, the bar of two
materials.  The seed draws the lattice jitter (and the fluid's velocities).
Bodies have 2 thousand to 700 thousand particles: a neighbour table several
times the L2 cache at the upper end, and linked-list grids within the 65 536
cells that a handle has room for from the start.

The FP64 forms return FP64 results.  The mixed form sums pairs in FP32, and
the programs here keep its results in single precision, as for plotting.

``exact`` advances the same decks with plain torch in FP64.
"""
from __future__ import annotations

import math

import numpy as np
import torch
import torch.utils.checkpoint

from mcmtop_b200 import _abi
from mcmtop_b200.deck import VEL, fluid_column, taylor_bar, taylor_ensemble, two_material_bar
from mcmtop_b200.solver import Batch, Solver

PRECISION = {"exact": _abi.PREC_FP64_EXACT, "fp64": _abi.PREC_FP64, "mixed": _abi.PREC_MIXED}

# what a host driver keeps of a particle: the state to restart from, and the
# fields it reads at an output time
STATE = ("x", "v", "mass", "h", "hold", "rho", "e", "p", "c", "vabs", "efps", "pcut", "p_cut", "fail", "sigma", "mat")
RESULT = ("x", "v", "rho", "e", "p", "efps", "sigma")

BAR_RADIUS, BAR_LENGTH = 3.2e-3, 32.4e-3


def listed():
    return [
        # A host driver's split loop on the smallest bar of the tests, every
        # energy read back: many small launches and one wait per call.
        dict(name="bar_2k_exact_split", kind="bar", dx=0.8e-3, precision="exact", loop="split", steps=40,
             diagnostics=True, reorder=0),
        # The program's own defaults (reference order and arithmetic, diagnostic
        # fields on) on the bar at dx = 0.4 mm: the everyday deck.
        dict(name="bar_17k_exact", kind="bar", dx=0.4e-3, precision="exact", loop="run", steps=40,
             diagnostics=True, reorder=0),
        # Two materials in kernel contact, own material's neighbours first.
        dict(name="bar2mat_31k_exact", kind="bar2", dx=0.32e-3, precision="exact", loop="run", steps=30,
             diagnostics=True, reorder=0),
        # Corrected SPH (disctype 1) on a bar of ordinary size.
        dict(name="bar_70k_exact_corrected", kind="bar", dx=0.25e-3, precision="exact", loop="run", steps=20,
             diagnostics=False, reorder=0, disctype=1),
        # One body of a parameter study in the mixed form.
        dict(name="bar_40k_mixed", kind="bar", dx=0.3e-3, precision="mixed", loop="run", steps=60,
             diagnostics=False, reorder=0),
        # The differentiated bar at dx = 0.2 mm: gradient of a misfit with
        # respect to the material and the initial state.
        dict(name="gradient_132k_fp64", kind="gradient", dx=0.2e-3, precision="fp64", steps=8, every=4),
        # A calibration ensemble, uneven bodies, one graph launch per iteration.
        dict(name="ensemble_24_mixed", kind="ensemble", bodies=24, precision="mixed", lanes=16, steps=50),
        # The collapsing column with five ghost walls, small in the program's
        # default arithmetic and large in the mixed form.
        dict(name="column_16k_exact", kind="column", dx=20.0e-3, precision="exact", loop="run", steps=40,
             diagnostics=True, reorder=0),
        dict(name="column_450k_mixed", kind="column", dx=6.5e-3, precision="mixed", loop="run", steps=60,
             diagnostics=False, reorder=20),
        # The large bar as the benchmark runs it: fused, re-sorted, in the
        # three arithmetics.
        dict(name="bar_690k_fp64", kind="bar", dx=0.115e-3, precision="fp64", loop="run", steps=50,
             diagnostics=False, reorder=20),
        dict(name="bar_690k_exact", kind="bar", dx=0.115e-3, precision="exact", loop="run", steps=40,
             diagnostics=False, reorder=20),
        dict(name="bar_690k_mixed", kind="bar", dx=0.115e-3, precision="mixed", loop="run", steps=80,
             diagnostics=False, reorder=20),
    ]


def draw(rng):
    kind = rng.choice(["bar", "bar", "bar", "bar2", "column", "column", "ensemble", "gradient", "corrected"])
    if kind == "ensemble":
        return dict(kind="ensemble", bodies=rng.randint(4, 24), precision=rng.choice(["mixed", "fp64", "exact"]),
                    lanes=rng.choice([4, 8, 16]), steps=rng.randint(10, 40))
    if kind == "gradient":
        n = math.exp(rng.uniform(math.log(2.0e3), math.log(1.3e5)))
        return dict(kind="gradient", dx=_bar_dx(n), precision=rng.choice(["fp64", "exact"]),
                    steps=rng.randint(4, 8), every=rng.choice([2, 4]))
    if kind == "corrected":
        n = math.exp(rng.uniform(math.log(2.0e3), math.log(1.0e5)))
        return dict(kind="bar", dx=_bar_dx(n), precision="exact", loop=rng.choice(["run", "split"]),
                    steps=rng.randint(10, 20), diagnostics=rng.choice([True, False]), reorder=0, disctype=1)
    n = math.exp(rng.uniform(math.log(2.0e3), math.log(4.4e5 if kind == "column" else 6.5e5)))
    big = n > 1.0e5
    # past a few hundred thousand particles programs fuse, re-sort and turn the diagnostics off
    steps = rng.randint(10, 20) if big else rng.randint(20, 50)
    c = dict(kind=kind, precision=rng.choice(["mixed", "fp64", "exact"]),
             loop="run" if big else rng.choice(["run", "run", "split"]), steps=steps,
             diagnostics=False if big else rng.choice([True, False]), reorder=20 if big else rng.choice([0, 20]))
    if kind == "column":
        c["dx"] = round((0.5 * 0.25 * 1.0 / n) ** (1.0 / 3.0), 6)
    else:
        c["dx"] = _bar_dx(n)
    return c


def _bar_dx(n):
    return round((math.pi * BAR_RADIUS ** 2 * BAR_LENGTH / n) ** (1.0 / 3.0), 9)


# ------------------------------------------------------------------- decks
def _decks(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        # the study's bodies are given; the seed moves their particles
        rng = np.random.default_rng(seed)
        return [d.replace(x=d.x + rng.uniform(-0.01, 0.01, size=d.x.shape) * (d.materials[0].h / 1.3))
                for d in taylor_ensemble(nbodies=case["bodies"])]
    if kind == "column":
        deck = fluid_column(dx=case["dx"], box=(1.0, 0.25, 1.2), seed=seed)
        # water already in motion, up to 0.1 m/s
        v = np.random.default_rng(seed + 1).uniform(-0.1, 0.1, size=deck.x.shape) * VEL
        return [deck.replace(v=v)]
    if kind == "bar2":
        return [two_material_bar(dx=case["dx"], seed=seed)]
    return [taylor_bar(dx=case["dx"], seed=seed, disctype=case.get("disctype", 0))]


def _pinned(n, width, dtype):
    return torch.zeros((n, width) if width > 1 else (n,), dtype=dtype, pin_memory=torch.cuda.is_available())


def _width(name):
    return _abi.FIELD_WIDTH.get(name, 1)


def _target(deck):
    """Where the particles of a gradient's misfit were measured: the bar moved by 1 % of its length."""
    t = np.array(deck.x)
    t[:, 2] *= 0.99
    return t


def prepare(case, seed):
    decks = _decks(case, seed)
    gradient = case["kind"] == "gradient"
    sols = [Solver(d, PRECISION[case["precision"]], reorder_interval=case.get("reorder", 0)) for d in decks]
    ends = np.cumsum([0] + [s.n for s in sols])
    n = int(ends[-1])
    ints = ("mat",)
    init = {f: _pinned(n, _width(f), torch.int32 if f in ints else torch.float64) for f in STATE}
    out = {f: _pinned(n, _width(f), torch.float64) for f in RESULT}

    def views(buffers, k):
        return {f: t[int(ends[k]):int(ends[k + 1])].numpy() for f, t in buffers.items()}

    bodies = []
    for k, s in enumerate(sols):
        s.set_diagnostics(bool(case.get("diagnostics", gradient)))
        mine = views(init, k)
        s.download_into(mine)
        bodies.append((s, mine, views(out, k), (s.dt, s.dtold, s.ptime)))
    state = {"case": case, "bodies": bodies, "init": init, "out": out}
    if case["precision"] == "mixed" and not gradient:
        state["single"] = {f: torch.zeros(t.shape, dtype=torch.float32) for f, t in out.items()}
    if case["kind"] == "ensemble":
        state["batch"] = Batch(sols, lanes=case["lanes"])
    if gradient:
        # the step sizes of a nominal run, and the measured positions
        s, mine = bodies[0][0], bodies[0][1]
        dts = [s.dt]
        for _ in range(case["steps"]):
            s.step_a()
            s.dt_update()
            dts.append(s.dt)
            s.step_b(False)
            s.step_c()
        state["dts"], state["target"] = dts, _target(decks[0])
    return state


def run(state):
    case = state["case"]
    for s, init, _, (dt, dtold, ptime) in state["bodies"]:
        s.upload(init, fortran_layout=True)
        s.dt, s.dtold, s.ptime, s.ended, s.timestep = dt, dtold, ptime, False, 1
    if case["kind"] == "gradient":
        s = state["bodies"][0][0]
        s.adjoint_forward(state["dts"], case["every"])
        x = s.download(["x"])["x"]
        theta, x0, v0 = s.adjoint_backward(x - state["target"], None)
        return {"theta": theta, "x0": x0, "v0": v0}
    if case["kind"] == "ensemble":
        state["batch"].run(case["steps"])
    elif case["loop"] == "split":
        s = state["bodies"][0][0]
        for _ in range(case["steps"]):
            s.step()
    else:
        state["bodies"][0][0].run(case["steps"])
    for s, _, out, _ in state["bodies"]:
        s.download_into(out)
    if "single" in state:
        for f, t in state["single"].items():
            t.copy_(state["out"][f])
        return state["single"]
    return state["out"]


def _particles(case):
    kind = case["kind"]
    if kind == "ensemble":
        return case["bodies"] * 21800          # mean of 4k..64k, log-uniform
    if kind == "column":
        return int(0.125 / case["dx"] ** 3)
    return int(math.pi * BAR_RADIUS ** 2 * BAR_LENGTH / case["dx"] ** 3)


def work(case):
    # Per particle and step the state is read and written once (x v 6, h m rho
    # e p c efps q 8, sigma 6, vabs 1 in; all but h and m out: 320 bytes).  With
    # about 78 neighbours a pair costs a distance (8 operations), a velocity
    # gradient (about 45) and an acceleration (about 50), the corrected form
    # three walks of each, and the per-particle update about 400.  A gradient
    # advances each step twice (once to record) and sweeps it back at about
    # twice a step's cost.
    per_step = 78 * (8 + 95 * (3 if case.get("disctype") else 1)) + 400
    steps = case["steps"] * (4 if case["kind"] == "gradient" else 1)
    n = _particles(case)
    moved = 8 * n * (sum(_width(f) for f in STATE) + sum(_width(f) for f in RESULT))
    return {"bytes": float(n * steps * 320 + moved), "flops": float(n) * steps * per_step}


# ------------------------------------------------- the same in FP64 torch
SKIN = 0.3          # reach kept beyond 2h between rebuilds of the lists, in h
CHUNK = 1 << 24     # pairs worked on at a time


class _Lists:
    """For every particle the indices of everything within (2 + SKIN) h of it,
    ghost images included: rows padded with the particle itself."""

    def __init__(self, r, x):
        dev = x.device
        n = x.shape[0]
        self.parent = torch.arange(n, device=dev)
        self.mult = torch.ones((n, 3), dtype=x.dtype, device=dev)
        self.add = torch.zeros((n, 3), dtype=x.dtype, device=dev)
        reach = (2.0 + SKIN) * r.h
        for d, _, b in r.planes:
            at = x[self.parent] * self.mult + self.add
            near = torch.nonzero((at[:, d] - b).abs() <= reach[self.parent]).flatten()
            m, a = self.mult[near].clone(), self.add[near].clone()
            m[:, d] *= -1.0
            a[:, d] = 2.0 * b - a[:, d]
            self.parent = torch.cat([self.parent, self.parent[near]])
            self.mult = torch.cat([self.mult, m])
            self.add = torch.cat([self.add, a])
        at = x[self.parent] * self.mult + self.add
        body, rr = r.body[self.parent], reach[self.parent]
        low = torch.full((r.bodies, 3), 1e30, dtype=x.dtype, device=dev)
        low = low.scatter_reduce(0, body[:, None].expand(-1, 3), at, "amin")
        cell = ((at - low[body]) / rr[:, None]).long() + 1
        nx, ny, nz = (int(v) + 2 for v in cell.max(0).values)
        key = ((body * nz + cell[:, 2]) * ny + cell[:, 1]) * nx + cell[:, 0]
        order = torch.argsort(key)
        keys = key[order]
        rows = torch.tensor([(dz * ny + dy) * nx for dz in (-1, 0, 1) for dy in (-1, 0, 1)], device=dev)
        found, widest = [], 1
        for s in range(0, n, 100_000):
            e = min(n, s + 100_000)
            k = key[s:e, None] + rows
            lo = torch.searchsorted(keys, k - 1)
            cnt = torch.searchsorted(keys, k + 1, right=True) - lo
            tot = cnt.flatten()
            first = torch.cumsum(tot, 0) - tot
            i = torch.repeat_interleave(torch.arange(tot.numel(), device=dev), tot)
            j = order[lo.flatten()[i] + torch.arange(i.numel(), device=dev) - first[i]]
            i = i // 9
            d = at[s + i] - at[j]
            keep = ((d * d).sum(1) < reach[s + i] ** 2) & (j != s + i)
            i, j = i[keep], j[keep]
            each = torch.bincount(i, minlength=e - s)
            found.append((s, i, j, torch.arange(i.numel(), device=dev) - (torch.cumsum(each, 0) - each)[i]))
            widest = max(widest, int(each.max()))
        self.j = torch.arange(n, device=dev)[:, None].repeat(1, widest)
        for s, i, j, at_k in found:
            self.j[s + i, at_k] = j

    def image(self, x):
        return x[self.parent] * self.mult + self.add


class _Reference:
    """The explicit step of one or several bodies that do not meet."""

    def __init__(self, case, seed):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        decks = _decks(case, seed)
        put = lambda parts: torch.as_tensor(np.concatenate(parts), device=self.dev)   # noqa: E731
        self.disc = decks[0].disctype
        self.bodies = len(decks)
        self.body = put([np.full(d.np, k, dtype=np.int64) for k, d in enumerate(decks)])
        self.x0 = put([np.asarray(d.x, dtype=np.float64) for d in decks])
        self.v0 = put([np.asarray(d.v, dtype=np.float64) for d in decks])
        per = lambda f: put([np.array([f(d, m) for m in d.materials], dtype=np.float64)[d.mat - 1]  # noqa: E731
                             for d in decks])
        total = put([np.bincount(d.mat)[d.mat].astype(np.float64) for d in decks])
        self.mass = per(lambda d, m: m.mass) / total
        self.h = per(lambda d, m: m.h)
        self.rho0 = per(lambda d, m: m.rho)
        self.av_l, self.av_q = decks[0].materials[0].av_l, decks[0].materials[0].av_q
        self.fluid = decks[0].materials[0].model == 9
        self.theta = [per(lambda d, m, k=k: m.strinput[k]) for k in range(3)] + [per(lambda d, m: m.eosinput[1])]
        self.cut = decks[0].materials[0].strinput[0] if self.fluid else -1.0e30
        self.c0 = decks[0].materials[0].eosinput[0]
        self.gamma0 = decks[0].materials[0].eosinput[4]
        d = decks[0]
        self.planes = [(p // 2, p % 2, d.sym_x[p]) for p in range(6) if d.sym_flag[p] == 1]
        self.base = torch.tensor([d.base_a[k] if d.nthp[k] == 1 else 0.0 for k in range(3)], dtype=torch.float64,
                                 device=self.dev)
        self.tssf = d.tssf

    def start(self):
        z = torch.zeros_like(self.mass)
        c = torch.sqrt(self.theta[3] / self.rho0) if self.fluid else torch.full_like(z, self.c0)
        return dict(x=self.x0, v=self.v0, rho=self.rho0.clone(), e=z, p=z, c=c, efps=z,
                    sigma=torch.zeros((z.numel(), 3, 3), dtype=torch.float64, device=self.dev))

    def least(self, s):
        """Critical timestep of every body."""
        crit = self.h / (s["c"] + s["v"].norm(dim=1))
        return torch.full((self.bodies,), 1e20, dtype=torch.float64, device=self.dev).scatter_reduce(
            0, self.body, crit, "amin")

    # pair sums: fn(rows, j, f, w, d) over chunks of rows; f d = grad W, x_i - x_j = d
    def _sums(self, ls, x_now, x_pair_i, x_pair_all, fn):
        n, width = ls.j.shape
        at = ls.image(x_now)
        outs = []
        for s in range(0, n, max(1, CHUNK // width)):
            rows = slice(s, min(n, s + max(1, CHUNK // width)))
            j = ls.j[rows]
            h = self.h[rows, None]
            gap = (x_now[rows, None] - at[j]).detach()
            inside = ((gap * gap).sum(2) < 4.0 * h * h) & (j != torch.arange(n, device=self.dev)[rows, None])
            d = x_pair_i[rows, None] - x_pair_all[j]
            r2 = (d * d).sum(2)
            r = torch.sqrt(torch.where(inside, r2, torch.ones_like(r2)))
            z = r / h
            unit = 1.0 / (math.pi * h ** 3)
            dw = torch.where(z < 1.0, unit * (2.25 * z - 3.0) * z,
                             torch.where(z < 2.0, -0.75 * unit * (2.0 - z) ** 2, torch.zeros_like(z)))
            f = torch.where(inside, dw / (h * r), torch.zeros_like(r))
            w = None
            if self.disc == 1:
                w = torch.where(z < 1.0, unit * ((0.75 * z - 1.5) * z * z + 1.0),
                                torch.where(z < 2.0, 0.25 * unit * (2.0 - z) ** 3, torch.zeros_like(z)))
                w = torch.where(inside, w, torch.zeros_like(w))
            outs.append(fn(rows, j, f, w, d))
        return torch.cat(outs)

    def _correction(self, vol_j, vol_i, f, w, d, sign):
        """Corrected kernel gradients of the chunk's pairs and of the self
        entry, and the inverse of the gradient correction."""
        w0 = (1.0 / (math.pi * self.h[0] ** 3))
        g = f[..., None] * d * sign
        sw = (vol_j * w).sum(1) + vol_i * w0
        sg = (vol_j[..., None] * g).sum(1)
        cg = (g * sw[:, None, None] - w[..., None] * sg[:, None]) / (sw * sw)[:, None, None]
        cs = -w0 * sg / (sw * sw)[:, None]
        b = torch.einsum("ik,ikn,ikm->inm", vol_j, -d, cg)
        det = torch.linalg.det(b)
        fine = det.abs() >= 1.0e-8
        eye = torch.eye(3, dtype=b.dtype, device=b.device).expand_as(b)
        return cg, cs, torch.where(fine[:, None, None], torch.linalg.inv(torch.where(fine[:, None, None], b, eye)), eye)

    def step(self, s, ls, dt, dtold=None, dtnew=None):
        """One loop iteration; dt per body.  Returns the new state and its step."""
        par, n = ls.parent, s["x"].shape[0]
        dti = dt[self.body][:, None]
        ghost = par[n:]
        x, v, rho_was = s["x"], s["v"], s["rho"]
        xs = x - 0.5 * v * dti
        xs_all = torch.cat([xs, ls.image(x)[n:]])
        v_all = v[par] * ls.mult
        vol = (self.mass / rho_was)[par]

        def strain(rows, j, f, w, d):
            if self.disc == 0:
                return torch.einsum("ikn,ikm->inm", vol[j][..., None] * (v_all[j] - v[rows, None]), f[..., None] * d)
            cg, cs, inv = self._correction(vol[j], vol[rows], f, w, d, 1.0)
            g = torch.einsum("ik,ikn,ikl->inl", vol[j], v_all[j], cg) + (vol[rows, None] * v[rows])[:, :, None] * cs[:, None]
            return torch.einsum("inl,iml->inm", g, inv)

        gv = self._sums(ls, x, xs, xs_all, strain)
        new = self._material(s, gv, dt[self.body])
        q = new.pop("q")
        if dtnew is None:
            dtold = dt
            dtnew = torch.minimum(self.tssf * self.least(dict(c=new["c"], v=v)), 1.1 * dt)
        eye = torch.eye(3, dtype=q.dtype, device=q.device)
        core = new["sigma"] - q[:, None, None] * eye
        a_real = core / (new["rho"] ** 2)[:, None, None]
        off = 2.0 * eye - 1.0
        a_all = torch.cat([a_real, core[ghost] * off / (rho_was[ghost] ** 2)[:, None, None]])
        x_all = ls.image(x)
        vol2 = self.mass[par] / torch.cat([new["rho"], rho_was[ghost]])

        def force(rows, j, f, w, d):
            both = a_all[j] + a_real[rows, None]
            if self.disc == 0:
                return torch.einsum("ik,ikmn,ikm->in", self.mass[par[j]], both, f[..., None] * d)
            cg, cs, inv = self._correction(vol2[j], vol2[rows], f, w, d, -1.0)
            ds = torch.einsum("ikmn,ikl->imnl", both, cg)
            return self.mass[rows, None] * torch.einsum("imnl,ilm->in", ds, inv)

        acc = self._sums(ls, x, x, x_all, force) + self.base
        dtn = dtnew[self.body][:, None]
        v = v + acc * (0.5 * (dtn + dtold[self.body][:, None]))
        x = x + v * dtn
        for d, side, b in self.planes:
            out = x[:, d] < b if side == 0 else x[:, d] > b
            flip = torch.zeros_like(x, dtype=torch.bool)
            flip[:, d] = out
            x, v = torch.where(flip, 2.0 * b - x, x), torch.where(flip, -v, v)
        return dict(new, x=x, v=v), dtnew

    def _material(self, s, gv, dt):
        gg, qs, qh, slope = self.theta
        n = dt.numel()
        eye = torch.eye(3, dtype=torch.float64, device=self.dev)
        rod = 0.5 * (gv + gv.transpose(1, 2))
        spin = 0.5 * (gv - gv.transpose(1, 2))
        tr = rod.diagonal(dim1=1, dim2=2).sum(1)
        rho_was, rho0, mass = s["rho"], self.rho0, self.mass
        rho = rho_was * (1.0 - tr * dt)
        # Jaumann rotation by the exponential map
        wz, wy, wx = -0.5 * dt * spin[:, 0, 1], 0.5 * dt * spin[:, 0, 2], -0.5 * dt * spin[:, 1, 2]
        w2 = wx * wx + wy * wy + wz * wz
        some = w2 > 0.0
        m = torch.sqrt(torch.where(some, w2, torch.ones_like(w2)))
        dd = torch.where(some, torch.tan(0.5 * m), torch.zeros_like(m))
        q4 = 0.25 * w2
        cc = torch.where(torch.where(some, m, torch.zeros_like(m)) < float(np.float32(1.0e-3)),
                         0.5 * (1.0 + q4 * (1 / 3 + q4 * (2 / 15 + q4 * (17 / 315 + q4 * (62 / 2835))))), dd / m)
        bb = 2.0 * cc / (1.0 + dd * dd)
        aa = bb * cc
        w = torch.stack([wx, wy, wz], 1)
        zero = torch.zeros_like(wx)
        skew = torch.stack([zero, -wz, wy, wz, zero, -wx, -wy, wx, zero], 1).view(n, 3, 3)
        rot = eye + bb[:, None, None] * skew + aa[:, None, None] * (w[:, :, None] * w[:, None] - w2[:, None, None] * eye)
        sig = rot @ s["sigma"] @ rot.transpose(1, 2)
        p_was = -sig.diagonal(dim1=1, dim2=2).sum(1) / 3.0
        mu = rho / rho0 - 1.0
        vol_was, vol, vol0 = mass / rho_was, mass / rho, mass / rho0
        if self.fluid:
            dev = torch.zeros_like(sig)
            efps = s["efps"]
            c = torch.sqrt(slope / rho0)
        else:
            g2 = 2.0 * dt * gg
            # the trial deviator adds (not subtracts) the mean rate, the shears take half
            dev = sig + p_was[:, None, None] * eye + g2[:, None, None] * torch.where(
                eye.bool(), rod + (tr / 3.0)[:, None, None], 0.5 * rod)
            j2 = 0.5 * (dev * dev).sum((1, 2))
            loaded = j2 > 0.0
            sj = torch.where(loaded, torch.sqrt(3.0 * torch.where(loaded, j2, torch.ones_like(j2))), torch.zeros_like(j2))
            ak = qs + qh * s["efps"]
            third = 1.0 / (3.0 * gg)
            more = torch.clamp(sj - ak, min=0.0) / (1.0 + third * qh)
            more = third * torch.minimum(sj, more)
            efps = s["efps"] + more
            ak = torch.clamp(ak + qh * more, min=0.0)
            dev = dev * (ak / torch.maximum(ak, sj))[:, None, None]
            ao = rho0 * self.c0 ** 2
            k1 = slope - 1.0
            bo, co = ao * (1.0 + 2.0 * k1), ao * (2.0 * k1 + 3.0 * k1 * k1)
            gam = self.gamma0 * rho0 / rho
            f = gam * mu
            e1 = s["e"] / mass
            squeezed = ao * (1.0 - f) + bo * (2.0 - 1.5 * f) * mu + co * (3.0 - 2.0 * f) * mu * mu
            c2 = torch.where(mu > 0.0, squeezed, ao * (1.0 - f)) / rho0 + gam * e1 + gam * rho * p_was / rho ** 2
            c = torch.sqrt(c2)
        ht = self.h * tr
        q = torch.where(tr < 0.0, self.av_l * rho * c * self.h * tr.abs() + self.av_q * rho * ht * ht, torch.zeros_like(tr))
        # energy trial; the viscosity's own mean drops out of the deviatoric part
        work_ = (rod * 0.5 * (sig + p_was[:, None, None] * eye + dev)).sum((1, 2))
        etry = s["e"] + dt * 0.5 * (vol + vol_was) * work_ - (vol - vol_was) * (0.5 * p_was + q)
        dvol = vol - vol_was
        if self.fluid:
            p = slope * mu
        else:
            ph = torch.where(mu > 0.0, ao * mu + bo * mu ** 2 + co * mu ** 3, ao * mu)
            p = (ph * (1.0 - 0.5 * f) + rho * gam * etry / mass) / (1.0 + 0.5 * rho * gam * dvol / vol0)
        low = p < self.cut
        p = torch.where(low, torch.full_like(p, self.cut), p)
        e = torch.where(low, s["e"], etry - 0.5 * dvol * p)
        rho = torch.where(low, rho / (1.0 - tr * dt), rho)
        return dict(rho=rho, e=e, p=p, c=c, efps=efps, sigma=dev - p[:, None, None] * eye, q=q)

    def lists_for(self, x, ls, x_at):
        """The lists again once some particle may have come into reach."""
        if ls is not None and not bool(((x - x_at).norm(dim=1) > 0.49 * SKIN * self.h).any()):
            return ls, x_at
        return _Lists(self, x), x


def exact(case, seed):
    r = _Reference(case, seed)
    if case["kind"] == "gradient":
        return _exact_gradient(case, seed, r)
    with torch.no_grad():
        s = r.start()
        dt = r.tssf * r.least(s)
        ls = x_at = None
        for _ in range(case["steps"]):
            ls, x_at = r.lists_for(s["x"], ls, x_at)
            s, dt = r.step(s, ls, dt)
    out = {f: s[f].cpu() for f in RESULT}
    out["sigma"] = out["sigma"].reshape(-1, 9)
    return out


def _exact_gradient(case, seed, r):
    # the step sizes are given numbers, each step's neighbours are fixed
    with torch.no_grad():
        s = r.start()
        dts, lists = [r.tssf * r.least(s)], []
        ls = x_at = None
        for _ in range(case["steps"]):
            ls, x_at = r.lists_for(s["x"], ls, x_at)
            lists.append(ls)
            s, dt = r.step(s, ls, dts[-1])
            dts.append(dt)
    theta = [t[:1].clone().requires_grad_() for t in r.theta]
    r.theta = [t.expand(r.mass.numel()) for t in theta]
    r.x0.requires_grad_()
    r.v0.requires_grad_()
    s = r.start()
    names = list(s)
    for k in range(case["steps"]):
        def one(*vals, k=k):
            new, _ = r.step(dict(zip(names, vals)), lists[k], dts[k], dts[k], dts[k + 1])
            return tuple(new[f] for f in names)
        s = dict(zip(names, torch.utils.checkpoint.checkpoint(one, *(s[f] for f in names), use_reentrant=False)))
    target = torch.as_tensor(_target(_decks(case, seed)[0]), device=r.dev)
    (0.5 * (s["x"] - target).square().sum()).backward()
    return {"theta": torch.stack([t.grad[0] for t in theta])[None].cpu(), "x0": r.x0.grad.cpu(), "v0": r.v0.grad.cpu()}
