"""The framework's work as a user has it done, as cases that can be timed and
compared: the MHD step of one grid through the solver (from latency-bound to
the benchmark's size, each reconstruction, boundary mode, even and odd
grids), the learned step, batches of independent grids, the per-kernel launch
interface, and the training of the troubled-cell indicator.

A pass of a solver case is a short run: the state is seeded from pinned host
arrays, stepped, and gathered into device tensors, so every pass does the
same work.  Initial states are analytic, made from the seed:

  flow    smooth multi-mode fields with pressure and density disks, field
          Bx(y), By(x), Bz(x, y): no uniform region, as in a developed flow
  rotor   a dense spinning disk in a uniform gas with Bx (the benchmark)
  blast   a pressure disk in a uniform gas with Bx and By

In-plane fields of this form are divergence-free to the bit, as the solver
requires of a seeded state; walls take flow without an in-plane field.
"""
from __future__ import annotations

import math
import os

import numpy as np
import torch

COMPONENTS = ("rho", "mx", "my", "mz", "energy", "bx_face", "by_face", "bz_cell")
ORDERS = {"muscl_minmod": 2, "mp5": 5, "mp7": 7}
GHOSTS = {2: 2, 5: 3, 7: 4}
MODES = {"periodic": 0, "outflow": 1, "wall": 2}
CFL = 0.4

# Algorithmic FLOPs per zone and step (add, multiply, divide, square root one
# each; compares none), the step's phases summed: profiles/flop_counts.json
# for MP5 and MP7; MUSCL from its formulas.
STEP_FLOPS = {2: 6000.0, 5: 49932.0, 7: 45142.0}


# ---- cases -------------------------------------------------------------------
def _solver(name, ic, nx, ny, scheme, bc, steps, loop="auto", learned=False):
    return dict(name=name, kind="solver", ic=ic, nx=nx, ny=ny, scheme=scheme, bc=bc, steps=steps,
                loop=loop, learned=learned)


def listed():
    return [
        # a student's or a test's grid, host loop as in the reference's CLI:
        # launches and the read-back of dt are what it waits for
        _solver("api_64_mp5", "flow", 64, 64, "mp5", "periodic", 16, loop="api"),
        # a small production grid, odd sides ratio, device-resident loop
        _solver("auto_200x150_mp7", "blast", 200, 150, "mp7", "outflow", 16),
        # the ordinary 2-D run
        _solver("auto_512_mp5", "flow", 512, 512, "mp5", "periodic", 8),
        # odd sides (odd pitch, ragged tiles in every kernel), walls, host loop
        _solver("api_1023x517_mp7_wall", "flow", 1023, 517, "mp7", "wall", 4, loop="api"),
        # a large run of a flow without uniform regions
        _solver("auto_2048_mp7", "flow", 2048, 2048, "mp7", "periodic", 4),
        # the benchmark's own workload: rotor 4096^2 MP7, outflow
        _solver("auto_rotor_4096_mp7", "rotor", 4096, 4096, "mp7", "outflow", 3),
        # second-order runs: quick looks and parameter scans
        _solver("auto_1024_muscl", "flow", 1024, 1024, "muscl_minmod", "outflow", 8),
        # the learned step with the shipped indicator
        _solver("learned_rotor_2048_mp7", "rotor", 2048, 2048, "mp7", "outflow", 3, learned=True),
        # an ensemble: independent grids of uneven sides stepped together
        dict(name="batch_32_mp5", kind="batch", count=32, lo=64, hi=512, scheme="mp5", steps=8,
             learned=False),
        dict(name="batch_32_mp5_learned", kind="batch", count=32, lo=64, hi=512, scheme="mp5",
             steps=8, learned=True),
        # another solver's driver on the per-kernel launch interface: the
        # residual and stage combine of one Runge-Kutta stage
        dict(name="seam_768x1024_mp5", kind="seam", ic="flow", nx=768, ny=1024, scheme="mp5",
             bc="periodic"),
        # training the troubled-cell indicator on the cells of two states
        dict(name="train_2x384", kind="train", n=384, states=2, scheme="mp5", tiles_per_step=128),
    ]


def draw(rng):
    """One more case of the same ranges: solver runs most often."""
    log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))  # noqa: E731
    kind = rng.choice(["solver"] * 5 + ["batch", "seam", "train"])
    scheme = rng.choice(["mp5", "mp7", "mp7"])
    if kind == "solver":
        if rng.random() < 0.15:
            scheme = "muscl_minmod"
        nx, ny = log(48, 2600), log(48, 2600)
        bc = rng.choice(["periodic", "outflow", "wall"])
        ic = "flow" if bc != "outflow" else rng.choice(["flow", "rotor", "blast"])
        steps = max(2, min(16, int(6e6 / (nx * ny))))
        learned = scheme != "muscl_minmod" and bc != "wall" and rng.random() < 0.2
        c = _solver("", ic, nx, ny, scheme, bc, steps, loop=rng.choice(["auto", "auto", "api"]),
                    learned=learned)
    elif kind == "batch":
        lo = rng.choice([48, 64, 96])
        c = dict(kind="batch", count=log(4, 40), lo=lo, hi=log(lo + 32, 512), scheme=scheme,
                 steps=rng.randint(4, 8), learned=rng.random() < 0.5)
    elif kind == "seam":
        bc = rng.choice(["periodic", "outflow"])
        c = dict(kind="seam", ic="flow", nx=log(96, 1600), ny=log(96, 1600), scheme=scheme, bc=bc)
    else:
        c = dict(kind="train", n=log(96, 512), states=rng.randint(1, 2),
                 scheme=rng.choice(["mp5", "mp7"]), tiles_per_step=rng.choice([64, 128, 256]))
    c.pop("name", None)
    return c


# ---- initial states ----------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _state(ic, nx, ny, order, bc, rng, lx, ly, device, gamma=5.0 / 3.0):
    """Padded conserved components [8, ny + 2g, nx + 2g] of an initial state
    drawn from `rng` (a numpy Generator)."""
    g = GHOSTS[order]
    f8 = dict(dtype=torch.float64, device=device)
    x = ((torch.arange(-g, nx + g, **f8) + 0.5) / nx)[None, :]
    y = ((torch.arange(-g, ny + g, **f8) + 0.5) / ny)[:, None]
    one = torch.ones(ny + 2 * g, nx + 2 * g, **f8)
    two_pi = 2.0 * math.pi

    def modes(count, kmax):
        """Sum of plane waves with random wave numbers and phases, |sum| <= 1."""
        s = torch.zeros_like(one)
        for _ in range(count):
            k, m = int(rng.integers(0, kmax + 1)), int(rng.integers(0, kmax + 1))
            s = s + torch.sin(two_pi * (k * x + m * y) + float(rng.uniform(0, two_pi)))
        return s / count

    def line(v, kmax):
        s = torch.zeros_like(v)
        for k in range(1, kmax + 1):
            s = s + torch.sin(two_pi * k * v + float(rng.uniform(0, two_pi))) / k
        return s

    r = torch.hypot((x - 0.5) * lx, (y - 0.5) * ly) / min(lx, ly)
    if ic == "rotor":
        r0 = float(rng.uniform(0.08, 0.14))
        f = ((1.15 * r0 - r) / (0.15 * r0)).clamp(0.0, 1.0)
        rho, p = 1.0 + 9.0 * f, one.clone()
        sp = torch.where(r <= r0, one * (2.0 / r0), f * 2.0 / r.clamp_min(1e-9))
        vx, vy, vz = -sp * (y - 0.5) * one, sp * (x - 0.5) * one, 0.0 * one
        bx, by, bz = one * (5.0 / math.sqrt(4.0 * math.pi)), 0.0 * one, 0.0 * one
    elif ic == "blast":
        rho, vx, vy, vz = one.clone(), 0.0 * one, 0.0 * one, 0.0 * one
        p = torch.where(r < float(rng.uniform(0.08, 0.16)), 10.0 * one, 0.1 * one)
        b = float(rng.uniform(0.5, 1.0))
        bx, by, bz = b * one, b * one, 0.3 * one
    else:
        rho = 1.0 + 0.3 * modes(4, 5)
        p = 0.6 + 0.2 * modes(4, 5)
        for _ in range(3):  # disks with a jump
            cx, cy = float(rng.uniform(0.2, 0.8)), float(rng.uniform(0.2, 0.8))
            disk = torch.hypot(x - cx, y - cy) < float(rng.uniform(0.05, 0.12))
            rho, p = torch.where(disk, 1.7 * rho, rho), torch.where(disk, 2.2 * p, p)
        vx = -torch.sin(two_pi * y) + 0.4 * modes(4, 4)
        vy = torch.sin(two_pi * x) + 0.4 * modes(4, 4)
        vz = 0.3 * modes(3, 4)
        s = 0.0 if bc == "wall" else 1.0
        bx = s * (0.2 + 0.3 * line(y, 3)) * one
        by = s * (-0.1 + 0.3 * line(x, 3)) * one
        bz = 0.25 + 0.15 * modes(3, 4)
    e = p / (gamma - 1.0) + 0.5 * rho * (vx * vx + vy * vy + vz * vz) + 0.5 * (bx * bx + by * by + bz * bz)
    return torch.stack([rho, rho * vx, rho * vy, rho * vz, e, bx, by, bz])


def _sides(case, seed):
    """The batch's grid sides and families; the sides depend on the case
    alone, so that every seed is the same amount of work."""
    rng = np.random.default_rng(1000 * case["count"] + case["hi"] + case["lo"])
    out = []
    for _ in range(case["count"]):
        nx, ny = (int(round(math.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]))))) for _ in range(2))
        out.append((nx, ny, ("flow", "flow", "blast")[int(rng.integers(0, 3))]))
    return out


def _lengths(nx, ny):
    """Square cells on a box whose shorter side is 1."""
    m = min(nx, ny)
    return nx / m, ny / m


def _host(state):
    """Pinned float64 numpy arrays of the eight components."""
    return [c.cpu().pin_memory().numpy().reshape(-1) if torch.cuda.is_available()
            else c.cpu().numpy().reshape(-1) for c in state]


def _indicator(order):
    from quasar_b200 import indicator
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    z = np.load(os.path.join(root, "quasar_b200", "data", f"indicator_mp{order}.npz"))
    ind = indicator.TroubledCellIndicator()
    ind.set_params(z["params"])
    return ind, float(z["threshold"])


def _config(nx, ny, scheme, bc):
    from quasar_b200 import mhd
    c = mhd.MhdConfig()
    lx, ly = _lengths(nx, ny)
    c.grid = mhd.Grid2D(nx, ny, lx, ly)
    c.reconstruction, c.cfl, c.gamma = scheme, CFL, 5.0 / 3.0
    c.boundary = mhd.MhdBoundarySpec([bc] * 4, [bc] * 4)
    return c


def _case_state(case, seed):
    order = ORDERS[case["scheme"]]
    return _state(case["ic"], case["nx"], case["ny"], order, case["bc"],
                  np.random.default_rng(seed), *_lengths(case["nx"], case["ny"]), _device())


# ---- what a program holds before the call --------------------------------------
def prepare(case, seed):
    return {"solver": _prepare_solver, "batch": _prepare_batch, "seam": _prepare_seam,
            "train": _prepare_train}[case["kind"]](case, seed)


def _prepare_solver(case, seed):
    from quasar_b200 import mhd
    order, nx, ny = ORDERS[case["scheme"]], case["nx"], case["ny"]
    s = mhd.MhdSolver2D(_config(nx, ny, case["scheme"], case["bc"]))
    n = (nx + 2 * GHOSTS[order]) * (ny + 2 * GHOSTS[order])
    host = _host(_case_state(case, seed))
    if case["learned"]:
        ind, threshold = _indicator(order)
        ind.attach(s, threshold)
    return dict(case=case, solver=s, host=host, idx=torch.arange(n, device="cuda"),
                out=torch.empty(8, n, dtype=torch.float64, device="cuda"))


def _prepare_batch(case, seed):
    from quasar_b200 import indicator, mhd
    order = ORDERS[case["scheme"]]
    sides = _sides(case, seed)
    bcs = ["outflow" if ic == "blast" else "periodic" for _, _, ic in sides]
    b = mhd.MhdBatch2D([_config(nx, ny, case["scheme"], bc) for (nx, ny, _), bc in zip(sides, bcs)])
    host, idx, out = [], [], []
    for k, ((nx, ny, ic), bc) in enumerate(zip(sides, bcs)):
        rng = np.random.default_rng([seed, k])
        host.append(_host(_state(ic, nx, ny, order, bc, rng, *_lengths(nx, ny), "cuda")))
        n = host[-1][0].size
        idx.append(torch.arange(n, device="cuda"))
        out.append(torch.empty(8, n, dtype=torch.float64, device="cuda"))
    if case["learned"]:
        ind, threshold = _indicator(order)
        indicator.attach_batch(ind, b, threshold)
    return dict(case=case, batch=b, host=host, idx=idx, out=out)


def _prepare_seam(case, seed):
    from quasar_b200 import launch as L
    order, nx, ny = ORDERS[case["scheme"]], case["nx"], case["ny"]
    ng = GHOSTS[order]
    lx, ly = _lengths(nx, ny)
    n = (nx + 2 * ng) * (ny + 2 * ng)
    f8 = dict(dtype=torch.float64, device="cuda")
    new = lambda k: torch.zeros(k, n, **f8)  # noqa: E731
    u = _case_state(case, seed).reshape(8, n).contiguous()
    return dict(case=case, L=L, grid=L.Grid(nx, ny, ng, lx / nx, ly / ny), u=u, next=u.clone(),
                dudt=new(8), fx=new(8), fy=new(8), ix=new(16), iy=new(16), cb=new(2), tab=new(4),
                nj=torch.zeros(2, n, dtype=torch.int32, device="cuda"),
                flags=L.flags([MODES[case["bc"]]] * 4), dt=0.1 * (lx / nx), order=order)


def _prepare_train(case, seed):
    from quasar_b200 import indicator, mhd
    order = ORDERS[case["scheme"]]
    ind = indicator.TroubledCellIndicator(seed=seed)
    s = mhd.MhdSolver2D(_config(case["n"], case["n"], case["scheme"], "periodic"))
    for k in range(case["states"]):
        rng = np.random.default_rng([seed, k])
        for name, a in zip(COMPONENTS, _host(_state("flow", case["n"], case["n"], order, "periodic",
                                                    rng, 1.0, 1.0, "cuda"))):
            s.seed_state(name, a)
        ind.collect(s, tol=1e-4)
    return dict(case=case, ind=ind, solver=s, start=ind.params())


# ---- one pass ------------------------------------------------------------------
def run(state):
    return {"solver": _run_solver, "batch": _run_batch, "seam": _run_seam,
            "train": _run_train}[state["case"]["kind"]](state)


def _run_solver(st):
    s, case = st["solver"], st["case"]
    for name, a in zip(COMPONENTS, st["host"]):
        s.seed_state(name, a)
    if case["loop"] == "api":
        t = 0.0
        for _ in range(case["steps"]):
            dt = s.cfl_limit()
            s.step_unchecked(dt)
            t += dt
    else:
        t, _ = s.advance_auto(0.0, float("inf"), case["steps"])
    for k, name in enumerate(COMPONENTS):
        s.gather_live(name, st["idx"], st["out"][k])
    return {"t": t, "state": st["out"]}


def _run_batch(st):
    b, case = st["batch"], st["case"]
    for k, host in enumerate(st["host"]):
        s = b.instance(k)
        for name, a in zip(COMPONENTS, host):
            s.seed_state(name, a)
    done = b.advance(case["steps"])
    for k, (idx, out) in enumerate(zip(st["idx"], st["out"])):
        s = b.instance(k)
        for c, name in enumerate(COMPONENTS):
            s.gather_live(name, idx, out[c])
    return {"done": done, "state": st["out"]}


def _run_seam(st):
    L, grid, order, fl = st["L"], st["grid"], st["order"], st["flags"]
    gamma = 5.0 / 3.0
    u, d = L.field(st["u"]), L.field(st["dudt"])
    fx, fy = L.field(st["fx"]), L.field(st["fy"])
    ix, iy = L.iface(st["ix"][:8], st["ix"][8:]), L.iface(st["iy"][:8], st["iy"][8:])
    table = L.emf(st["tab"][0], st["tab"][1], st["nj"][0], st["nj"][1], st["tab"][2], st["tab"][3])
    L.fill_ghosts(grid, u, list(fl))
    st["dudt"].zero_()
    L.reconstruct(grid, u, st["cb"][0], st["cb"][1], 0, ix, order, fl, gamma)
    L.hlld_flux(grid, ix, 0, fx, fl, gamma, order)
    L.reconstruct(grid, u, st["cb"][0], st["cb"][1], 1, iy, order, fl, gamma)
    L.hlld_flux(grid, iy, 1, fy, fl, gamma, order)
    L.flux_difference(grid, fx, 0, d)
    L.flux_difference(grid, fy, 1, d)
    L.ct_emf_prepare(grid, u, st["cb"][0], st["cb"][1], ix, iy, fl, table, gamma, order)
    L.ct_emf_finish(grid, fl, table, order)
    L.emf_curl_rate(grid, table, d)
    L.rk_stage(grid, L.field(st["next"]), u, u, d, 1.0, 0.0, st["dt"])
    return {"dudt": st["dudt"], "next": st["next"]}


def _run_train(st):
    case, ind = st["case"], st["ind"]
    ind.set_params(st["start"])
    loss = ind.train(epochs=1, tiles_per_step=case["tiles_per_step"], lr=1e-3, pos_weight=8.0,
                     holdout=20, seed=1)
    return {"loss": loss, "params": ind.params()}


# ---- what a pass cannot do without -----------------------------------------------
def _zones(case):
    if case["kind"] == "batch":
        return sum(nx * ny for nx, ny, _ in _sides(case, 0))
    if case["kind"] == "train":
        return case["n"] ** 2 * case["states"]
    return case["nx"] * case["ny"]


def work(case):
    z = _zones(case)
    if case["kind"] == "train":
        # forward, and twice that backward, of 200-64-64-1 per row; a row is
        # 200 BF16 features and a label
        return {"bytes": z * 401.0, "flops": z * 6.0 * (200 * 64 + 64 * 64 + 64)}
    order = ORDERS[case["scheme"]]
    if case["kind"] == "seam":
        return {"bytes": z * 8.0 * 24, "flops": z * STEP_FLOPS[order] / 3.0}
    # eight components read and written by each step; the learned step keeps
    # the flux and CT work and does most faces without the characteristic one
    per = STEP_FLOPS[order] - (25000.0 if case["learned"] else 0.0)
    return {"bytes": z * case["steps"] * 128.0, "flops": z * case["steps"] * per}


def tolerance(case):
    """Binary64 results.  The eigenvector weights of a fan without transverse
    field are square roots of rounding-level differences (rotor, blast: their
    uniform regions), and a characteristic variable's limiter switches on the
    sign of rounding noise where it is zero: another order of the sums moves
    isolated faces by far more than the last bit."""
    if case["kind"] == "train":
        # BF16 operands, and Adam's first steps are nearly sign(gradient)
        return {"rel": 1e-2, "max": 0.5}
    if case.get("learned"):
        # a flag may change at the threshold; flags choose between two
        # interpolations that agree to the training tolerance of 1e-4
        return {"rel": 1e-6, "max": 1e-3}
    if case["kind"] == "batch" or case["ic"] != "flow":
        # measured against exact(): 8e-10 in t, 1e-10 in the state (rotor)
        return {"rel": 4e-9, "max": 4e-6}
    # measured against exact(): 2e-16, one small step's rounding
    return {"rel": 1e-11, "max": 1e-8}


# ---- the same in plain torch, 64 bits ----------------------------------------------
def exact(case, seed):
    """What run() returns, from the scheme's formulas in plain torch.  None
    where that takes too long, and for the learned and trained cases, whose
    results depend on BF16 networks and on the trainer's own tile order."""
    if case["kind"] not in ("solver", "seam") or case.get("learned"):
        return None
    if case["nx"] * case["ny"] * case.get("steps", 1) > 2_500_000:
        return None
    order, nx, ny = ORDERS[case["scheme"]], case["nx"], case["ny"]
    lx, ly = _lengths(nx, ny)
    m = _Plain(nx, ny, lx / nx, ly / ny, order, MODES[case["bc"]])
    u = m.fill(_case_state(case, seed))
    if case["kind"] == "seam":
        d, _ = m.residual(u)
        return {"dudt": d.reshape(8, -1), "next": None}
    t = 0.0
    for _ in range(case["steps"]):
        dt, u = m.step(u)
        t += dt
    return {"t": t, "state": u.reshape(8, -1)}


def _gauss_legendre(q):
    x, w = np.polynomial.legendre.leggauss(q)
    return (x / 2).tolist(), (w / 2).tolist()


def _average_to_point(x, h):
    """Weights over 2h + 1 cell averages of the polynomial's value at x
    (cell units from the centre cell's centre)."""
    k = np.arange(-h, h + 1)
    n = 2 * h + 1
    a = np.array([[((j + 0.5) ** (p + 1) - (j - 0.5) ** (p + 1)) / (p + 1) for p in range(n)] for j in k])
    return np.linalg.solve(a.T, np.array([x ** p for p in range(n)])).tolist()


class _Plain:
    """Ideal MHD on a Cartesian grid: MP5 / MP7 in characteristic fields or
    MUSCL-minmod in primitive ones, HLLD at the faces' transverse Gauss
    points, upwind constrained transport, SSP-RK3.  Whole arrays of shape
    [..., ny + 2g, nx + 2g]; a y sweep is an x sweep of the transpose."""

    def __init__(self, nx, ny, dx, dy, order, bc, gamma=5.0 / 3.0):
        self.n, self.d, self.order, self.bc, self.gamma = (nx, ny), (dx, dy), order, bc, gamma
        self.g = GHOSTS[order]
        self.nodes = _gauss_legendre(4 if order == 7 else 3) if order > 2 else ([0.0], [1.0])
        self.h = {2: 0, 5: 2, 7: 3}[order]
        self.pw = [_average_to_point(x, self.h) for x in self.nodes[0]]

    # boundary closure, x sides before y sides
    def fill(self, u):
        u = u.clone()
        self._fill_x(u, 0)
        t = self._turn(u).contiguous()
        self._fill_x(t, 1)
        return self._turn(t).contiguous()

    @staticmethod
    def _turn(u):
        return u[[0, 2, 1, 3, 4, 6, 5, 7]].transpose(-1, -2)

    def _fill_x(self, u, axis):
        g, n = self.g, self.n[axis]
        for k in range(1, g + 1):
            for lo in (True, False):
                dst = g - k if lo else g + n - 1 + k
                src = {0: g + n - k if lo else g + k - 1, 1: g if lo else g + n - 1,
                       2: g + k - 1 if lo else g + n - k}[self.bc]
                sign = -1.0 if self.bc == 2 else 1.0
                for c in (0, 2, 3, 4, 6, 7):
                    u[c, :, dst] = u[c, :, src]
                u[1, :, dst] = sign * u[1, :, src]
                if self.bc == 2:  # the normal field is odd about the wall's face
                    wall = g if lo else g + n
                    u[5, :, wall] = 0.0
                    if lo:
                        u[5, :, g - k] = -u[5, :, g + k]
                    elif k > 1:
                        u[5, :, g + n + k - 1] = -u[5, :, g + n - (k - 1)]
                elif self.bc == 1 and not lo:
                    if k > 1:  # the face n is evolved
                        u[5, :, g + n - 1 + k] = u[5, :, g + n]
                else:
                    u[5, :, dst] = u[5, :, src]

    def collocate(self, f):
        """Cell averages along x of the polynomial through the 2g nearest faces."""
        w, n = 2 * self.g, f.shape[-1]
        out = torch.empty_like(f)
        made = {}
        for c in range(n):
            s = min(max(c - (w // 2 - 1), 0), n - w)
            if c - s not in made:
                k = np.arange(w)
                a = np.array([k ** p for p in range(w)], dtype=float)
                b = np.array([((c - s + 1.0) ** (p + 1) - (c - s) ** (p + 1.0)) / (p + 1) for p in range(w)])
                made[c - s] = np.linalg.solve(a, b).tolist()
            out[..., c] = sum(q * f[..., s + k] for k, q in enumerate(made[c - s]))
        return out

    def cells(self, u):
        v = u.clone()
        v[5] = self.collocate(u[5])
        v[6] = self.collocate(u[6].transpose(-1, -2)).transpose(-1, -2)
        return v

    # pointwise formulas, normal along x
    def p(self, u):
        return (self.gamma - 1.0) * (u[4] - 0.5 * (u[1] ** 2 + u[2] ** 2 + u[3] ** 2) / u[0]
                                     - 0.5 * (u[5] ** 2 + u[6] ** 2 + u[7] ** 2))

    def fast(self, u):
        a2 = self.gamma * self.p(u).clamp_min(0.0) / u[0]
        bn2, bt2 = u[5] ** 2 / u[0], (u[6] ** 2 + u[7] ** 2) / u[0]
        return torch.sqrt(0.5 * (a2 + bn2 + bt2 + torch.sqrt((a2 - bn2 - bt2) ** 2 + 4.0 * a2 * bt2)))

    def good(self, u):
        p = self.p(u)
        return torch.isfinite(u).all(0) & (u[0] > 0) & torch.isfinite(p) & (p > 0)

    def flux(self, u):
        v, p = u[1:4] / u[0], self.p(u)
        pt = p + 0.5 * (u[5] ** 2 + u[6] ** 2 + u[7] ** 2)
        vb = v[0] * u[5] + v[1] * u[6] + v[2] * u[7]
        return torch.stack([u[1], u[1] * v[0] + pt - u[5] ** 2, u[1] * v[1] - u[5] * u[6],
                            u[1] * v[2] - u[5] * u[7], v[0] * (u[4] + pt) - u[5] * vb, 0.0 * u[0],
                            u[6] * v[0] - u[5] * v[1], u[7] * v[0] - u[5] * v[2]])

    def hlld(self, l, r):
        """Miyoshi and Kusano's solver; HLL where a star state is unresolved."""
        tiny = 64.0 * torch.finfo(torch.float64).eps
        same = (l == r).all(0)
        fl_same = self.flux(l)
        bn = 0.5 * l[5] + 0.5 * r[5]
        l, r = l.clone(), r.clone()
        for s in (l, r):
            s[4] = s[4] - 0.5 * s[5] ** 2 + 0.5 * bn ** 2
            s[5] = bn
        cf = torch.maximum(self.fast(l), self.fast(r))
        vl, vr = l[1:4] / l[0], r[1:4] / r[0]
        sl, sr = torch.minimum(vl[0], vr[0]) - cf, torch.maximum(vl[0], vr[0]) + cf
        pt = [self.p(s) + 0.5 * (s[5] ** 2 + s[6] ** 2 + s[7] ** 2) for s in (l, r)]
        al, ar = (sl - vl[0]) * l[0], (sr - vr[0]) * r[0]
        sm = (ar * vr[0] - al * vl[0] - pt[1] + pt[0]) / (ar - al)
        ps = (ar * pt[0] - al * pt[1] + al * ar * (vr[0] - vl[0])) / (ar - al)
        bad = ~(torch.isfinite(sm) & torch.isfinite(ps)) | ~((ar - al).abs() > tiny * (ar.abs() + al.abs()))
        ws = sl.abs() + sr.abs() + sm.abs()
        star = []
        for u, v, s, q in ((l, vl, sl, pt[0]), (r, vr, sr, pt[1])):
            bad = bad | ~((s - sm).abs() > tiny * ws)
            rs = u[0] * (s - v[0]) / (s - sm)
            bad = bad | ~(rs > 0)
            t = u[0] * (s - v[0]) * (s - sm)
            den = t - bn ** 2
            bad = bad | ~(den.abs() > tiny * (t.abs() + bn ** 2))
            fac, bc = bn * (sm - v[0]) / den, (u[0] * (s - v[0]) ** 2 - bn ** 2) / den
            vy, vz, by, bz = v[1] - u[6] * fac, v[2] - u[7] * fac, u[6] * bc, u[7] * bc
            vb, vbs = v[0] * bn + v[1] * u[6] + v[2] * u[7], sm * bn + vy * by + vz * bz
            e = ((s - v[0]) * u[4] - q * v[0] + ps * sm + bn * (vb - vbs)) / (s - sm)
            star.append((torch.stack([rs, rs * sm, rs * vy, rs * vz, e, bn, by, bz]), vy, vz, by, bz, vbs))
        (ul, vyl, vzl, byl, bzl, vbl), (ur, vyr, vzr, byr, bzr, vbr) = star
        ql, qr = ul[0].clamp_min(0).sqrt(), ur[0].clamp_min(0).sqrt()
        sal, sar = sm - bn.abs() / ql, sm + bn.abs() / qr
        sg = torch.where(bn >= 0, 1.0, -1.0).to(bn)
        vy, vz = ((ql * a + qr * b + (d - c) * sg) / (ql + qr)
                  for a, b, c, d in ((vyl, vyr, byl, byr), (vzl, vzr, bzl, bzr)))
        by, bz = ((ql * d + qr * c + ql * qr * (b - a) * sg) / (ql + qr)
                  for a, b, c, d in ((vyl, vyr, byl, byr), (vzl, vzr, bzl, bzr)))
        vb = sm * bn + vy * by + vz * bz
        ull = torch.stack([ul[0], ul[1], ul[0] * vy, ul[0] * vz, ul[4] - ql * sg * (vbl - vb), bn, by, bz])
        urr = torch.stack([ur[0], ur[1], ur[0] * vy, ur[0] * vz, ur[4] + qr * sg * (vbr - vb), bn, by, bz])
        none = bn ** 2 <= tiny * (ps.abs() + pt[0].abs() + pt[1].abs())
        fl, fr = self.flux(l), self.flux(r)
        f1l, f1r = fl + sl * (ul - l), fr + sr * (ur - r)
        left, right = torch.where(none | (0 <= sal), f1l, f1l + sal * (ull - ul)), torch.where(
            none | (0 >= sar) & ~(0 <= sar), f1r, f1r + sar * (urr - ur))
        f = torch.where(0 <= sm, left, right)
        bad = bad | ~torch.isfinite(f).all(0)
        ss = torch.maximum(sl.abs(), sr.abs())
        hll = (sr * fl - sl * fr + sl * sr * (r - l)) / (sr - sl)
        f = torch.where(bad & torch.isfinite(ss), hll, f)
        f = torch.where(sl >= 0, fl, torch.where(sr <= 0, fr, f))
        f = torch.where(same, fl_same, f)
        f[5] = 0.0
        return f

    # reconstruction of the faces between columns i - 1 and i
    def waves(self, c):
        """Left rows and right columns [wave, 7, ...] about the states c."""
        rho, v, p = c[0], c[1:4] / c[0], self.p(c).clamp_min(0.0)
        s2 = math.sqrt(0.5)
        a2, bx2 = self.gamma * p / rho, c[5] ** 2 / rho
        b2 = bx2 + (c[6] ** 2 + c[7] ** 2) / rho
        f2 = 0.5 * (a2 + b2 + torch.sqrt(((a2 + b2) ** 2 - 4.0 * a2 * bx2).clamp_min(0.0)))
        c2 = a2 * bx2 / f2
        den = f2 - c2
        eps = torch.finfo(torch.float64).eps
        tie = den <= 64.0 * eps * (f2 + c2)
        af = torch.where(tie, s2, ((a2 - c2) / den).clamp_min(0.0).sqrt())
        as_ = torch.where(tie, s2, ((f2 - a2) / den).clamp_min(0.0).sqrt())
        a, cf, cs, sr = a2.sqrt(), f2.sqrt(), c2.sqrt(), rho.sqrt()
        bt = torch.hypot(c[6], c[7])
        no = (bt == 0) | (bt / sr <= 64.0 * eps * torch.maximum(a, b2.sqrt()))
        b1, b3 = torch.where(no, s2, c[6] / bt), torch.where(no, s2, c[7] / bt)
        sg = torch.where(c[5] >= 0, 1.0, -1.0).to(rho)
        z = torch.zeros_like(rho)
        lp, rp = [], []
        for al, cc, q, w, sign in ((af, cf, cs * as_ * sg, a * as_ * sr, 1), (None,) * 5,
                                   (as_, cs, -cf * af * sg, -a * af * sr, 1)):
            if al is None:
                rp.append([z, z, -b3 * s2, b1 * s2, z, -sg * b3 * s2 * sr, sg * b1 * s2 * sr])
                lp.append([z, z, -b3 * s2, b1 * s2, z, -sg * b3 * s2 / sr, sg * b1 * s2 / sr])
            else:
                k = 0.5 / a2
                rp.append([rho * al, -al * cc, q * b1, q * b3, al * self.gamma * p, w * b1, w * b3])
                lp.append([z, -k * al * cc, k * q * b1, k * q * b3, k * al / rho, k * w * b1 / rho, k * w * b3 / rho])
        # the right-going partners: velocities reversed (the Alfven pair: fields)
        flip = lambda r: [r[0], -r[1], -r[2], -r[3], r[4], r[5], r[6]]  # noqa: E731
        odd = lambda r: r[:5] + [-r[5], -r[6]]  # noqa: E731
        rows = lambda x, e: x[:3] + [e] + [flip(x[2]), odd(x[1]), flip(x[0])]  # noqa: E731
        one = torch.ones_like(rho)
        lp = rows(lp, [one, z, z, z, -1.0 / a2, z, z])
        rp = rows(rp, [one, z, z, z, z, z, z])
        gv, hv = self.gamma - 1.0, 0.5 * (v ** 2).sum(0)
        left = [[q[0] - (q[1] * v[0] + q[2] * v[1] + q[3] * v[2]) / rho + q[4] * gv * hv]
                + [q[1 + i] / rho - q[4] * gv * v[i] for i in range(3)]
                + [q[4] * gv, q[5] - q[4] * gv * c[6], q[6] - q[4] * gv * c[7]] for q in lp]
        right = [[q[0]] + [v[i] * q[0] + rho * q[1 + i] for i in range(3)]
                 + [hv * q[0] + rho * (v[0] * q[1] + v[1] * q[2] + v[2] * q[3]) + q[4] / gv
                    + c[6] * q[5] + c[7] * q[6], q[5], q[6]] for q in rp]
        left = torch.stack([torch.stack(q) for q in left])
        right = torch.stack([torch.stack(q) for q in right])
        off = (torch.einsum("im...,jm...->ij...", left, right)
               - torch.eye(7, dtype=rho.dtype, device=rho.device).reshape(7, 7, *[1] * rho.dim()))
        ok = (off.abs() <= 1024.0 * eps).all(0).all(0)
        unit = torch.eye(7, dtype=rho.dtype, device=rho.device).reshape(7, 7, *[1] * rho.dim())
        return torch.where(ok, left, unit), torch.where(ok, right, unit)

    def limited(self, v):
        """Suresh and Huynh's limiter on the 2h + 1 samples v, left of the face."""
        w = {2: (2, -13, 47, 27, -3), 3: (-3, 25, -101, 319, 214, -38, 4)}[self.h]
        vl = sum(q * s for q, s in zip(w, v)) / (60.0 if self.h == 2 else 420.0)
        m2, m1, v0, p1, p2 = v[self.h - 2:self.h + 3]

        def mm(*t):
            t = torch.stack(t)
            return torch.where((t > 0).all(0), t.amin(0), torch.where((t < 0).all(0), t.amax(0), 0.0))
        cm = vl - (v0 + mm(p1 - v0, 4.0 * (v0 - m1)))
        cc = vl - v0
        var = torch.stack([v0 - m1, p1 - v0, cc, cm]).abs().amax(0)
        keep = (cc * cm <= 0) | ((cc / var) * (cm / var) <= 1e-10)
        dm, d0, dp = m2 - 2 * m1 + v0, m1 - 2 * v0 + p1, v0 - 2 * p1 + p2
        ph, mh = mm(4 * d0 - dp, 4 * dp - d0, d0, dp), mm(4 * d0 - dm, 4 * dm - d0, d0, dm)
        ul, md = v0 + 4.0 * (v0 - m1), 0.5 * (v0 + p1) - 0.5 * ph
        lc = v0 + 0.5 * (v0 - m1) + 4.0 / 3.0 * mh
        lo = torch.maximum(torch.stack([v0, p1, md]).amin(0), torch.stack([v0, ul, lc]).amin(0))
        hi = torch.minimum(torch.stack([v0, p1, md]).amax(0), torch.stack([v0, ul, lc]).amax(0))
        return torch.where(keep, vl, vl + mm(lo - vl, hi - vl))

    def muscl(self, q):
        def prim(u):
            return torch.stack([u[0], u[1] / u[0], u[2] / u[0], u[3] / u[0], self.p(u), u[5], u[6], u[7]])

        def slope(a, b, c, drop):
            x, y = b - a, c - b
            s = torch.where(x * y > 0, torch.where(x.abs() < y.abs(), x, y), 0.0)
            lo, hi = drop
            return torch.where(lo, y, torch.where(hi, x, s)) if drop is not None else s

        def cons(w):
            e = w[4] / (self.gamma - 1.0) + 0.5 * w[0] * (w[1] ** 2 + w[2] ** 2 + w[3] ** 2) + 0.5 * (
                w[5] ** 2 + w[6] ** 2 + w[7] ** 2)
            return torch.stack([w[0], w[0] * w[1], w[0] * w[2], w[0] * w[3], e, w[5], w[6], w[7]])
        a, b, c, d = (prim(t) for t in q)
        k = torch.arange(b.shape[-1], device=b.device)  # face index from 0
        n = b.shape[-1] - 1
        off = self.bc != 0
        at = lambda pos: ((pos <= 0) & off, (pos >= n - 1) & off)  # noqa: E731
        return cons(b + 0.5 * slope(a, b, c, at(k - 1))), cons(c - 0.5 * slope(b, c, d, at(k)))

    def faces(self, u, v, axis):
        """Left and right states of the n + 1 faces of every padded row."""
        g, n = self.g, self.n[axis]
        cut = lambda a, k: a[..., g + k:g + k + n + 1]  # noqa: E731
        q = [cut(v, k) for k in (-2, -1, 0, 1)]
        if self.order == 2:
            l, r = self.muscl(q)
        else:
            c = 0.5 * q[1] + 0.5 * q[2]
            left, right = self.waves(c)
            use = [0, 1, 2, 3, 4, 6, 7]
            ch = [torch.einsum("im...,m...->i...", left, (cut(v, k) - c)[use])
                  for k in range(-self.h - 1, self.h + 1)]
            w = 2 * self.h + 1
            dl = torch.einsum("im...,i...->m...", right, self.limited(ch[:w]))
            dr = torch.einsum("im...,i...->m...", right, self.limited(ch[:0:-1]))
            l, r = c.clone(), c.clone()
            l[use] += dl
            r[use] += dr
            bad = ~(self.good(l) & self.good(r))
            if bad.any():
                ml, mr = self.muscl(q)
                l, r = torch.where(bad, ml, l), torch.where(bad, mr, r)
        bn = cut(u[5], 0)

        def normal(s):
            s = s.clone()
            s[4] = s[4] + 0.5 * bn ** 2 - 0.5 * s[5] ** 2
            s[5] = bn
            return s
        l, r = normal(l), normal(r)
        bad = ~(self.good(l) & self.good(r))
        return torch.where(bad, normal(q[1]), l), torch.where(bad, normal(q[2]), r)

    def face_flux(self, l, r, axis):
        """Flux of the faces on the interior rows and one more (corner rows
        n), the CFL rate and whether the face's whole stencil has no jump."""
        g, h, m = self.g, self.h, self.n[1 - axis]
        rows = lambda a, k: a[..., g + k:g + k + m + 1, :]  # noqa: E731
        if self.bc == 0:  # the periodic high face repeats face 0
            l, r = (torch.cat([s[..., :-1], s[..., :1]], -1) for s in (l, r))
        cl, cr = rows(l, 0), rows(r, 0)
        pts = [(sum(w * rows(l, k - h) for k, w in enumerate(pw)), sum(w * rows(r, k - h) for k, w in enumerate(pw)))
               for pw in self.pw]
        const = [(torch.stack([rows(s, k - h) for k in range(2 * h + 1)]) == rows(s, 0)).all(0) for s in (l, r)]
        pts = [(torch.where(const[0], cl, a), torch.where(const[1], cr, b)) for a, b in pts]

        def rate(a, b):
            return 0.5 / self.d[axis] * (torch.maximum((a[1] / a[0]).abs(), (b[1] / b[0]).abs())
                                         + torch.maximum(self.fast(a), self.fast(b)))
        spd, ok = rate(cl, cr), torch.ones_like(cl[0], dtype=torch.bool)
        fluxes = []
        for a, b in pts:
            ok = ok & self.good(a) & self.good(b)
            spd = torch.where(ok, torch.maximum(spd, rate(a, b)), spd)
            fluxes.append(self.hlld(a, b))
        f = sum(w * x for w, x in zip(self.nodes[1], fluxes))
        f = torch.where((torch.stack(fluxes) == fluxes[0]).all(0), fluxes[0], f)
        f = torch.where(ok, f, self.hlld(cl, cr))
        return f, spd, (l == r).all(0)

    def cell_ez(self, v):
        g, h = self.g, self.h
        nx, ny = self.n
        ez = lambda s: s[2] / s[0] * s[5] - s[1] / s[0] * s[6]  # noqa: E731
        mid = v[:, g:g + ny + 1, g:g + nx + 1]
        if self.order == 2:
            return ez(mid)
        total, ok = 0.0, torch.ones_like(mid[0], dtype=torch.bool)
        for wx, px in zip(self.nodes[1], self.pw):
            line = sum(w * v[:, :, g + k - h:g + k - h + nx + 1] for k, w in enumerate(px))
            for wy, py in zip(self.nodes[1], self.pw):
                s = sum(w * line[:, g + k - h:g + k - h + ny + 1] for k, w in enumerate(py))
                ok = ok & self.good(s)
                total = total + wx * wy * ez(s)
        e = torch.where(ok, total, ez(mid))
        flat = torch.ones_like(ok)  # a constant stencil returns its own value
        for a in range(-h, h + 1):
            for b in range(-h, h + 1):
                flat = flat & (v[:, g + b:g + b + ny + 1, g + a:g + a + nx + 1] == mid).all(0)
        return torch.where(flat, ez(mid), e)

    def residual(self, u):
        g, (nx, ny), (dx, dy) = self.g, self.n, self.d
        v = self.cells(u)
        ut, vt = self._turn(u), self._turn(v)
        lx, rx = self.faces(u, v, 0)
        ly, ry = self.faces(ut, vt, 1)
        fx, sx, jx = self.face_flux(lx, rx, 0)
        fyt, syt, jyt = self.face_flux(ly, ry, 1)
        fy, sy, jy = self._turn(fyt), syt.transpose(-1, -2), jyt.transpose(-1, -2)
        cell, h, per = self.cell_ez(v), self.h, self.bc == 0

        def at(n, i):  # the CT tables wrap on periodic axes and clamp on others
            return torch.remainder(i, n) if per else i.clamp(0, n)
        dev = u.device
        nt = {2: 2, 5: 6, 7: 8}[self.order]
        lo = -nt // 2
        ix, iy = torch.arange(nx + 1, device=dev), torch.arange(ny + 1, device=dev)
        taps = range(lo, lo + nt)
        w = {2: (1, 1), 6: (1, -8, 37, 37, -8, 1), 8: (-3, 29, -139, 533, 533, -139, 29, -3)}[nt]
        norm = float(sum(w))

        def edge(e):
            e = torch.stack(list(e))
            return torch.where((e == e[0]).all(0), e[0], sum(q * s for q, s in zip(w, e)) / norm)
        fx_ez, fy_ez = -fx[6], fy[5]
        ex = edge(fx_ez[at(ny, iy + k)][:, at(nx, ix)] for k in taps)
        ey = edge(fy_ez[at(ny, iy)][:, at(nx, ix + k)] for k in taps)
        line = [[cell[at(ny, iy + k)][:, at(nx, ix + m)] for m in taps] for k in taps]
        cen = edge(edge(row) for row in line)
        flat_x = torch.stack([(c == row[0]) for row in line for c in row]).all(0)
        flat_y = torch.stack([(row[m] == line[0][m]) for row in line for m in range(nt)]).all(0)

        def no_jump(j, axis):  # j over padded rows of the sweep, n + 1 faces
            j = j if axis == 0 else j.transpose(-1, -2)
            n, m = self.n[axis], self.n[1 - axis]
            f, t = torch.arange(n + 1, device=dev), torch.arange(m + 1, device=dev)
            out = torch.ones(m + 1, n + 1, dtype=torch.bool, device=dev)
            for k in range(-h, h + 1):
                out = out & j[g + at(m, t + k)][:, at(n, f)]
            return out if axis == 0 else out.transpose(-1, -2)
        njx, njy = no_jump(jx, 0), no_jump(jy, 1)
        only_y = torch.stack([njx[at(ny, iy + k)][:, at(nx, ix)] for k in taps]).all(0) & flat_x
        only_x = torch.stack([njy[at(ny, iy)][:, at(nx, ix + k)] for k in taps]).all(0) & flat_y
        ez = torch.where(only_x & ~only_y, ex, torch.where(only_y & ~only_x, ey, ex + ey - cen))
        if self.bc == 2:
            ez[0], ez[ny], ez[:, 0], ez[:, nx] = 0.0, 0.0, 0.0, 0.0
        d = torch.zeros_like(u)
        for c in (0, 1, 2, 3, 4, 7):
            d[c, g:g + ny, g:g + nx] = (-(fx[c, :ny, 1:] - fx[c, :ny, :-1]) / dx
                                        - (fy[c, 1:, :nx] - fy[c, :-1, :nx]) / dy)
        d[5, g:g + ny, g:g + nx + 1] = -(ez[1:] - ez[:-1]) / dy
        d[6, g:g + ny + 1, g:g + nx] = (ez[:, 1:] - ez[:, :-1]) / dx
        rate = (sx[:ny, :nx] + sx[:ny, 1:nx + 1]) + (sy[:ny, :nx] + sy[1:ny + 1, :nx])
        return d, float(rate.max())

    def step(self, u):
        d, rate = self.residual(u)
        dt = (min(CFL, 0.2) if self.order > 2 else CFL) / rate
        a = self.fill(u + dt * d)
        b = self.fill(0.75 * u + 0.25 * a + 0.25 * dt * self.residual(a)[0])
        return dt, self.fill(u / 3.0 + 2.0 / 3.0 * b + 2.0 / 3.0 * dt * self.residual(b)[0])
