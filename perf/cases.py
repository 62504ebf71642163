"""The work this framework is used for, as cases that can be timed and checked.

A case is a small dict.  `prepare` makes the inputs and the solver context that a program keeps,
`run` is one job through the public entry points (set the state, advance a number of time steps,
read the state; or one loss with its gradient; or a queue of host-buffer steps), and `exact` is
the same job in 64-bit torch, from the equations alone.

Every job starts from the initial temperature, as the documented workloads do: the layered slab,
the point source cube, the batched sweep of uneven grids, the inclusion grid, the slab with
temperature-dependent properties and the inverse problem.  The seed moves the heating, the layers
and the random materials.
"""
import ctypes as C
import math

import numpy as np
import torch

from heatflow_gb300 import abi
from heatflow_gb300.adjoint import AdjointModel, ProbeMisfit
from heatflow_gb300.problem import Problem
from heatflow_gb300.solver import HeatFlow

DX, DT, T0 = 1e-9, 1e-13, 300.0
SI, POLY = (149.0, 2329.0, 710.0), (0.2, 1190.0, 1200.0)      # kappa, rho, c

TRUE = dict(criterion="true", tol=1e-10)


def listed():
    return [
        # the reference's deck size (25 x 25 x 1) as the host program runs it: its own stopping
        # rule in FP64, the loop in one graph; small calls, latency is all
        dict(name="deck 25x25x1 reference rule", kind="point", nx=25, ny=25, nz=1, steps=10, cattaneo=0,
             precision="fp64", rule="recursive", graph=1, io="host"),
        # a program that couples to simulate() step by step with every option at its default
        dict(name="cube 20 default simulate", kind="point", nx=20, ny=20, nz=20, steps=4, cattaneo=1,
             precision="fp64", rule="recursive", graph=0, io="simulate"),
        # small device-resident runs: the layered slab on a 64^3 grid, mixed precision
        dict(name="slab 64 mixed", kind="slab", nx=64, ny=64, nz=64, steps=20, cattaneo=1,
             precision="mixed", rule="true", graph=1, io="device"),
        # odd sizes, Fourier mode, FP64
        dict(name="ragged 97x61x45 fp64", kind="lognormal", nx=97, ny=61, nz=45, steps=10, cattaneo=0,
             precision="fp64", rule="true", graph=1, io="device"),
        # the layered slab at its stated 128^3
        dict(name="slab 128 mixed", kind="slab", nx=128, ny=128, nz=128, steps=20, cattaneo=1,
             precision="mixed", rule="true", graph=1, io="device"),
        # the benchmark's grid with the options that its autotuner picks
        dict(name="slab 256 mixed", kind="slab", nx=256, ny=256, nz=256, steps=12, cattaneo=1,
             precision="mixed", rule="true", graph=1, io="device", inner_tol=1e-6, depth=32),
        # the FP64 path at a size that fills the memory system, rows that are no multiple of 4
        dict(name="slab 190x192x192 fp64", kind="slab", nx=190, ny=192, nz=192, steps=8, cattaneo=1,
             precision="fp64", rule="true", graph=1, io="device"),
        # the batched sweep: uneven grids of 16..96 cells an edge in one context
        dict(name="sweep 64 grids mixed", kind="sweep", count=64, lo=16, hi=96, steps=20, cattaneo=1,
             precision="mixed", rule="true", graph=1, io="host"),
        # many CG iterations on a large periodic grid: random inclusions
        dict(name="inclusions 320x320x256 mixed", kind="inclusions", nx=320, ny=320, nz=256, steps=5, cattaneo=1,
             precision="mixed", rule="true", graph=1, io="device"),
        # temperature-dependent properties: the operator rebuilt after every step
        dict(name="tables 96x100x90 mixed", kind="tables", nx=96, ny=100, nz=90, steps=10, cattaneo=1,
             precision="mixed", rule="true", graph=1, io="device"),
        # one loss and gradient of the inverse problem (forward, checkpoints, adjoint solves), as
        # the adjoint's own program sets it up
        dict(name="adjoint 48 mixed", kind="adjoint", nx=48, ny=48, nz=48, steps=20, cattaneo=1,
             precision="mixed", rule="true", graph=2, io="gradient"),
        # a host program that keeps the fields in pinned host arrays and queues its steps
        dict(name="host steps 160 mixed", kind="slab", nx=160, ny=160, nz=160, steps=10, cattaneo=1,
             precision="mixed", rule="true", graph=1, io="queue"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["point", "slab", "slab", "lognormal", "sweep", "inclusions", "tables", "adjoint", "queue"])
    precision = rng.choice(["mixed", "fp64"])
    base = dict(kind=kind, cattaneo=rng.choice([1, 1, 0]), precision=precision, rule="true", graph=1, io="device")
    if kind == "point":
        rule = rng.choice(["recursive", "true"])
        return dict(base, nx=_log(rng, 8, 60), ny=_log(rng, 8, 60), nz=_log(rng, 1, 40), steps=rng.randint(2, 12),
                    rule=rule, precision="fp64" if rule == "recursive" else precision,
                    graph=rng.choice([0, 1, 1, 3]), io=rng.choice(["host", "simulate"]))
    if kind == "sweep":
        lo = rng.randint(8, 24)
        return dict(base, count=_log(rng, 3, 48), lo=lo, hi=rng.randint(lo + 4, 80), steps=rng.randint(4, 12), io="host")
    if kind == "adjoint":
        return dict(base, nx=_log(rng, 12, 56), ny=_log(rng, 12, 56), nz=_log(rng, 12, 56), steps=rng.randint(4, 16),
                    graph=rng.choice([1, 2]), io="gradient")
    top = 230 if kind == "slab" else 160
    c = dict(base, nx=_log(rng, 24, top), ny=_log(rng, 24, top), nz=_log(rng, 16, top), steps=rng.randint(4, 12))
    if kind == "queue":
        c.update(kind="slab", io="queue", precision="mixed")
    elif kind == "inclusions":
        c.update(nx=max(c["nx"], 40), ny=max(c["ny"], 40), nz=max(c["nz"], 32))
    return c


# ---- inputs: plain numpy arrays and numbers, x fastest --------------------------------------------
def _layers(nz, layer, phase):
    return ((np.arange(nz) + phase) // layer) % 2 == 1


def _by_plane(values, ny, nx):
    return np.broadcast_to(values[:, None, None], (len(values), ny, nx))


def _grid(case, rng):
    """One grid: its cells' kappa, rho, c, heater power (per cell; heated: where) and its faces."""
    kind, nx, ny, nz = case["kind"], case["nx"], case["ny"], case["nz"]
    shape, kb, periodic = (nz, ny, nx), 149.0, (0, 0, 0)
    power, total = None, None
    rho, cap = 2329.0, 710.0
    if kind == "point":
        kappa = 149.0
        power = np.zeros(shape)
        at = [int(rng.integers(n // 3, n - n // 3)) for n in shape]
        power[tuple(at)] = 1e-6 * rng.uniform(0.5, 1.5)
    elif kind in ("slab", "tables"):
        poly = _layers(nz, 16, int(rng.integers(0, 16)))
        kappa, rho, cap = (_by_plane(np.where(poly, p, s), ny, nx) for s, p in zip(SI, POLY))
        power = np.zeros(shape)
        cx = (nx - 1) / 2 + nx * rng.uniform(-0.1, 0.1)
        cy = (ny - 1) / 2 + ny * rng.uniform(-0.1, 0.1)
        gx, gy = (np.exp(-(np.arange(n) - m) ** 2 / 50.0) for n, m in ((nx, cx), (ny, cy)))
        power[-1] = 1e-5 * rng.uniform(0.5, 1.0) * gy[:, None] * gx[None, :]
    elif kind == "inclusions":
        poly = _balls(shape, rng)
        kappa, rho, cap = (np.where(poly, p, s) for s, p in zip(SI, POLY))
        periodic = (1, 1, 0)
        heated = 8 * nx * ny
        total = 1e-9 * heated * rng.uniform(0.5, 1.5)
    else:                                                         # lognormal, sweep, adjoint
        kb = 50.0
        n = nx * ny * nz
        kappa = np.exp(math.log(50.0) + (0.5 if kind == "adjoint" else 1.0) * rng.standard_normal(shape))
        rho, cap = (2000.0 if kind == "adjoint" else rng.uniform(1e3, 3e3, size=shape)), 1000.0
        cells = rng.choice(n, size=8 if kind == "adjoint" else int(rng.integers(1, 5)), replace=False)
        power = np.zeros(n)
        power[cells] = rng.uniform(1e-7, 1e-5, size=len(cells))
        power = power.reshape(shape)
    if power is not None:
        heat = power > 0
    else:
        heat = np.zeros(shape, bool)
        heat[:8] = True
    return dict(nx=nx, ny=ny, nz=nz, kappa=kappa, rho=rho, cap=cap, power=power, total=total, heat=heat, kb=kb,
                periodic=periodic, cattaneo=case["cattaneo"])


def _balls(shape, rng, frac=0.05):
    """Random spheres of radius 3..10 (periodic in x and y) until `frac` of the cells are covered."""
    poly = np.zeros(shape, bool)
    nz, ny, nx = shape
    count, target = 0, frac * poly.size
    while count < target:
        r = int(rng.integers(3, 11))
        cz, cy, cx = (int(v) for v in rng.integers(0, shape))
        zs, ys, xs = np.ogrid[-r:r + 1, -r:r + 1, -r:r + 1]
        ball = zs * zs + ys * ys + xs * xs <= r * r
        zi = np.arange(cz - r, cz + r + 1)
        keep = (zi >= 0) & (zi < nz)
        at = np.ix_(zi[keep], np.arange(cy - r, cy + r + 1) % ny, np.arange(cx - r, cx + r + 1) % nx)
        new = poly[at] | ball[keep]
        count += int(new.sum() - poly[at].sum())
        poly[at] = new
    return poly


def _grids(case, seed):
    rng = np.random.default_rng(1000 + seed)
    if case["kind"] != "sweep":
        return [_grid(case, rng)]
    edges = np.random.default_rng(case["count"]).integers(case["lo"], case["hi"] + 1, size=(case["count"], 3))
    return [_grid(dict(case, nx=int(a), ny=int(b), nz=int(c)), rng) for a, b, c in edges]


def _tables():
    t = np.array([250.0, 290.0, 300.0, 305.0, 320.0, 400.0, 600.0])
    return [np.c_[t, 150.0 - 0.2 * (t - 250.0), 2300.0 - 0.1 * (t - 250.0), 700.0 + 0.8 * (t - 250.0)],
            np.c_[t, 0.3 - 0.0003 * (t - 250.0), 1200.0 - 0.1 * (t - 250.0), 1100.0 + 0.5 * (t - 250.0)]]


def _cell_table(g):
    return np.where(np.broadcast_to(np.asarray(g["kappa"]), (g["nz"], g["ny"], g["nx"])) > 1.0, 0, 1).astype(np.int32).reshape(-1)


def _problem(g):
    n = g["nx"] * g["ny"] * g["nz"]
    flat = lambda a: np.reshape(a, -1) if np.ndim(a) else a  # noqa: E731
    return Problem(nx=g["nx"], ny=g["ny"], nz=g["nz"], lx=g["nx"] * DX, ly=g["ny"] * DX, lz=g["nz"] * DX,
                   kappa=flat(g["kappa"]), rho=flat(g["rho"]), heat_capacity=flat(g["cap"]), tau=1e-12, em=0.0,
                   iheater=g["heat"].reshape(n).astype(np.int64), power=None if g["power"] is None else g["power"].reshape(n),
                   power_in=g["total"] or 0.0, time_step=DT, icattaneo=g["cattaneo"], periodic=g["periodic"],
                   qdens_mode=abi.HF_QDENS_HEATED_VOLUME if g["power"] is None else abi.HF_QDENS_CELL_VOLUME,
                   kappa_bound=(g["kb"],) * 6, t_bath_face=(T0,) * 6, t_bath=T0)


def _options(case):
    if case["rule"] == "recursive":
        return {} if case["graph"] == 0 else dict(use_graph=case["graph"])
    o = dict(TRUE, precision=case["precision"], use_graph=case["graph"])
    if "inner_tol" in case:
        o.update(inner_tol=case["inner_tol"])
    if "depth" in case:
        o.update(task_depth=case["depth"])
    return o


def _adjoint_inputs(case, seed):
    g = _grids(case, seed)[0]
    rng = np.random.default_rng(5000 + seed)
    n = g["kappa"].size
    sources = np.flatnonzero(g["heat"].reshape(-1))
    probes = rng.choice(np.setdiff1d(np.arange(n), sources), size=min(64, n // 4), replace=False)
    amps = g["power"].reshape(-1)[sources] * rng.uniform(0.6, 0.9, size=len(sources))
    observed = T0 + rng.uniform(0.0, 2.0, size=(case["steps"], len(probes)))
    return g, sources, probes, amps, observed


# ---- the job ---------------------------------------------------------------------------------------
class State:
    pass


def prepare(case, seed):
    s = State()
    s.case, s.steps = case, case["steps"]
    if case["io"] == "gradient":
        g, sources, probes, amps, observed = _adjoint_inputs(case, seed)
        s.model = AdjointModel(_problem(g), probes, sources, s.steps, 10, **_options(case))
        s.log_kappa = torch.tensor(np.log(g["kappa"]).reshape(-1), device="cuda", requires_grad=True)
        s.amps = torch.tensor(amps, device="cuda", requires_grad=True)
        s.observed = torch.tensor(observed, device="cuda")
        return s
    grids = _grids(case, seed)
    probs = [_problem(g) for g in grids]
    s.hf = HeatFlow(probs if case["kind"] == "sweep" else probs[0], **_options(case))
    if case["kind"] == "tables":
        s.hf.set_property_tables(_tables(), _cell_table(grids[0]))
    n = s.hf.n
    if case["io"] == "device":
        s.start = torch.full((n,), T0, dtype=torch.float64, device="cuda")
        s.out = [torch.empty_like(s.start) for _ in range(2)]
        torch.cuda.synchronize()
    else:
        s.pinned = [torch.full((n,), T0, dtype=torch.float64).pin_memory() for _ in range(4)]
        s.host = [t.numpy() for t in s.pinned]
    return s


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def run(s):
    case, K = s.case, s.steps
    if case["io"] == "gradient":
        s.log_kappa.grad = s.amps.grad = None
        loss = ProbeMisfit.apply(s.log_kappa, s.amps, s.model, s.observed)
        loss.backward()
        return [loss.detach(), s.log_kappa.grad, s.amps.grad]
    hf = s.hf
    if case["io"] == "device":
        abi.check(hf.lib.hf_set_state_device(hf.h, _ptr(s.start), _ptr(s.start)), "hf_set_state_device")
        hf.run(1, K)
        abi.check(hf.lib.hf_get_state_device(hf.h, _ptr(s.out[0]), _ptr(s.out[1])), "hf_get_state_device")
        return s.out
    if case["io"] == "queue":
        start, ring = s.host[0], s.host[1:]
        new, prev = start, start                      # T^n and T^(n-1) in pinned host arrays
        for k in range(K):
            out = ring[k % 3]
            hf.step_host_async(1 + k, new, prev, out)
            new, prev = out, new
        hf.host_sync()
        return [new, prev]
    hf.set_state(s.host[0], s.host[0])
    if case["io"] == "simulate":
        for k in range(K):
            hf.simulate(1 + k)
    else:
        hf.run(1, K)
    return list(hf.get_state(out=(s.host[1], s.host[2])))


# ---- work --------------------------------------------------------------------------------------
#: CG iterations of a step, about: what its materials and time step ask for at the job's tolerance.
ITERATIONS = {"point": 25, "slab": 4, "lognormal": 15, "sweep": 15, "inclusions": 14, "tables": 15, "adjoint": 15}


def work(case):
    """Per cell and step: T^n, T^(n-1) and three material properties read, T^(n+1) written (48
    bytes), once; a right-hand side and a residual (22 operations) and 22 per CG iteration.  A
    gradient runs the steps forward twice (checkpoints) and one adjoint solve per step."""
    if case["kind"] == "sweep":
        edges = np.random.default_rng(case["count"]).integers(case["lo"], case["hi"] + 1, size=(case["count"], 3))
        cells = float(np.prod(edges, axis=1).sum())
    else:
        cells = float(case["nx"] * case["ny"] * case["nz"])
    solves = cells * case["steps"] * (3 if case["io"] == "gradient" else 1)
    return {"bytes": 48 * solves, "flops": (22 + 22 * ITERATIONS[case["kind"]]) * solves}


# ---- the same job from the equations, in 64 bits ---------------------------------------------------
# Per cell  div(kappa grad T') - rc/dt (T' - T) - tau rc/dt^2 (T' - 2 T + Told) + Q = 0  with
# harmonic-mean face conductances (half cells to the bath of the outer faces): H T' = S.
class _Grid:
    def __init__(self, g, device):
        self.g, self.device = g, device
        self.shape = (g["nz"], g["ny"], g["nx"])
        full = lambda a: torch.tensor(np.array(np.broadcast_to(np.asarray(a, np.float64), self.shape)), device=device)  # noqa: E731
        self.kappa, self.rc = full(g["kappa"]), full(g["rho"]) * full(g["cap"])
        self.tau = 1e-12 / DT ** 2 if g["cattaneo"] else 0.0
        vol = DX ** 3
        if g["power"] is None:
            heated = float(g["heat"].sum()) * vol
            self.q = torch.tensor(g["heat"], device=device).double() * (g["total"] / heated)
        else:
            self.q = torch.tensor(g["power"], device=device) / vol
        self.len = [DX, DX, DX]                                     # z, y, x

    def faces(self, kappa):
        """Per axis (z, y, x) the conductance to the + neighbour, and of the two outer faces."""
        per = self.g["periodic"][::-1]
        inner, outer = [], []
        for a in range(3):
            L2, n = self.len[a] ** 2, self.shape[a]
            lo, hi = kappa.narrow(a, 0, n - 1), kappa.narrow(a, 1, n - 1)
            inner.append(2 * lo * hi / (lo + hi) / L2)
            ends = [kappa.narrow(a, 0, 1), kappa.narrow(a, n - 1, 1)]
            if per[a]:
                outer.append(2 * ends[0] * ends[1] / (ends[0] + ends[1]) / L2)
            else:
                outer.append([2 * self.g["kb"] * e / (self.g["kb"] + e) / L2 for e in ends])
        return inner, outer

    def assemble(self):
        self.inner, self.outer = self.faces(self.kappa)
        self.a0, self.c0 = -self.rc / DT - 2 * self.tau * self.rc, self.tau * self.rc
        ones = torch.ones_like(self.kappa)
        self.diag = self.rc / DT + self.tau * self.rc                    # of -H
        self.bath = torch.zeros_like(self.kappa)
        for a in range(3):
            n = self.shape[a]
            self.diag.narrow(a, 0, n - 1).add_(self.inner[a])
            self.diag.narrow(a, 1, n - 1).add_(self.inner[a])
            o = self.outer[a]
            for k, at in enumerate((0, n - 1)):
                v = o[k] if isinstance(o, list) else o
                self.diag.narrow(a, at, 1).add_(v)
                if isinstance(o, list):
                    self.bath.narrow(a, at, 1).add_(v * T0 * ones.narrow(a, at, 1))

    def apply(self, x):
        """-H x."""
        y = self.diag * x
        for a in range(3):
            n, c = self.shape[a], self.inner[a]
            y.narrow(a, 0, n - 1).sub_(c * x.narrow(a, 1, n - 1))
            y.narrow(a, 1, n - 1).sub_(c * x.narrow(a, 0, n - 1))
            o = self.outer[a]
            if not isinstance(o, list):
                y.narrow(a, 0, 1).sub_(o * x.narrow(a, n - 1, 1))
                y.narrow(a, n - 1, 1).sub_(o * x.narrow(a, 0, 1))
        return y

    def solve(self, b, x):
        """-H x = b by Jacobi-CG, restarted twice from the true residual."""
        inv, norm = 1 / self.diag, float(b.norm())
        for _ in range(3):
            r = b - self.apply(x)
            z = inv * r
            p, rho = z.clone(), float((r * z).sum())
            for _ in range(400):
                if float(r.norm()) <= 1e-15 * norm or rho == 0.0:
                    break
                q = self.apply(p)
                alpha = rho / float((p * q).sum())
                x = x + alpha * p
                r = r - alpha * q
                z = inv * r
                rho, old = float((r * z).sum()), rho
                p = z + (rho / old) * p
        return x

    def step(self, t, told):
        s = self.a0 * t + self.c0 * told - self.q - self.bath
        return self.solve(-s, 2 * t - told)


def _retabulate(grid, tables, cells, t):
    for k, rows in enumerate(tables):
        r = torch.tensor(rows, device=t.device)
        T = r[:, 0].contiguous()
        v = t.clamp(float(T[0]), float(T[-1]))
        i = (torch.searchsorted(T, v, right=True) - 1).clamp(0, len(T) - 2)
        f = (v - T[i]) / (T[i + 1] - T[i])
        cols = [r[i, c] + f * (r[i + 1, c] - r[i, c]) for c in (1, 2, 3)]
        grid.kappa = torch.where(cells == k, cols[0], grid.kappa)
        grid.rc = torch.where(cells == k, cols[1] * cols[2], grid.rc)


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if case["io"] == "gradient":
        return _exact_gradient(case, seed, device)
    new, old = [], []
    for g in _grids(case, seed):
        grid = _Grid(g, device)
        grid.assemble()
        t = torch.full(grid.shape, T0, dtype=torch.float64, device=device)
        told = t.clone()
        cells = torch.tensor(_cell_table(g), device=device).reshape(grid.shape) if case["kind"] == "tables" else None
        for _ in range(case["steps"]):
            t, told = grid.step(t, told), t
            if cells is not None:
                _retabulate(grid, _tables(), cells, t)
                grid.assemble()
        new.append(t.reshape(-1))
        old.append(told.reshape(-1))
    return [torch.cat(new), torch.cat(old)]


def _exact_gradient(case, seed, device):
    """The adjoint equations H l_k = dJ/dT_k + a l_(k+1) + c l_(k+2); the derivative of
    sum_k l_k (S_k - H T_k) with respect to log kappa and the source powers by autograd."""
    g, sources, probes, amps, observed = _adjoint_inputs(case, seed)
    power = g["power"].copy().reshape(-1)
    power[sources] = amps
    grid = _Grid(dict(g, power=power.reshape(g["kappa"].shape)), device)
    grid.assemble()
    probes, observed = torch.tensor(probes, device=device), torch.tensor(observed, device=device)
    t = torch.full(grid.shape, T0, dtype=torch.float64, device=device)
    fields, told = [t], t.clone()
    for _ in range(case["steps"]):
        t, told = grid.step(t, told), t
        fields.append(t)
    off = torch.stack([f.reshape(-1)[probes] for f in fields[1:]]) - observed
    log_kappa = torch.tensor(np.log(g["kappa"]), device=device, requires_grad=True)
    grad_k = torch.zeros_like(t)
    grad_q = torch.zeros_like(t)
    l1, l2 = torch.zeros_like(t), torch.zeros_like(t)
    for k in range(case["steps"], 0, -1):
        b = torch.zeros_like(t).reshape(-1).index_add(0, probes, 2 * off[k - 1]).reshape(t.shape)
        b = b + grid.a0 * l1 + grid.c0 * l2
        lam = grid.solve(-b, l1)
        kappa = log_kappa.exp()
        inner, outer = grid.faces(kappa)
        x, form = fields[k], 0.0
        for a in range(3):
            n = grid.shape[a]
            d = x.narrow(a, 1, n - 1) - x.narrow(a, 0, n - 1)
            dl = lam.narrow(a, 1, n - 1) - lam.narrow(a, 0, n - 1)
            form = form + (inner[a] * d * dl).sum()
            for j, at in enumerate((0, n - 1)):
                form = form + (outer[a][j] * lam.narrow(a, at, 1) * (x.narrow(a, at, 1) - T0)).sum()
        grad_k += torch.autograd.grad(form, log_kappa)[0]
        grad_q -= lam / DX ** 3
        l1, l2 = lam, l1
    return [(off ** 2).sum(), grad_k.reshape(-1), grad_q.reshape(-1)[torch.tensor(sources, device=device)]]
