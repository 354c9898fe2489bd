"""Admissible states whose squared fast speed overflows (p / rho or B^2 / rho
above about 1e154): the CFL reduction refuses them wherever they lie, also
where only one side of each face has such a state, and the Riemann flux takes
the exit of infinite wave speeds on either side."""
import numpy as np
import pytest

import mhd_cases as M
from test_gpu_parity import gpu_solver, seed

pytestmark = pytest.mark.gpu

GAMMA = 5.0 / 3.0


def at_rest(n, order, where, what):
    ng = M.nghost(order)
    a = [np.zeros((n + 2 * ng, n + 2 * ng)) for _ in range(8)]
    a[0][:], a[4][:] = 1.0, 0.9
    j, i = where[1] + ng, where[0] + ng
    if what == "pressure":
        a[4][j, i] = 1e160
    else:  # the out-of-plane field, which no divergence restrains
        a[7][j, i], a[4][j, i] = 1e80, 1e160
    return a


@pytest.mark.parametrize("bc", [M.PERIODIC, M.OUTFLOW])
@pytest.mark.parametrize("what", ["pressure", "field"])
@pytest.mark.parametrize("order", [2, 5, 7])
def test_one_overflowing_cell_is_refused(order, what, bc):
    n = 24
    for where in ((0, 0), (n - 1, n - 1), (11, 7)):
        s = gpu_solver(n, order, bc)
        seed(s, at_rest(n, order, where, what))
        with pytest.raises(RuntimeError, match="non-finite state encountered in CFL reduction"):
            s.cfl_limit()


@pytest.mark.parametrize("order", [5, 7])
def test_one_overflowing_cell_is_refused_in_a_batch(order):
    from quasar_b200 import mhd
    n = 24
    cfg = mhd.MhdConfig()
    cfg.grid = mhd.Grid2D(n, n, 1.0, 1.0)
    cfg.reconstruction = "mp7" if order == 7 else "mp5"
    b = mhd.MhdBatch2D([cfg, cfg])
    for k in range(2):
        quiet = at_rest(n, order, (11, 7), "pressure")
        if k == 0:
            quiet[4][:] = 0.9
        for name, a in zip(M.COMPONENTS, quiet):
            b.instance(k).seed_state(name, a)
    with pytest.raises(RuntimeError, match="non-finite state encountered in CFL reduction"):
        b.advance(1)


@pytest.mark.parametrize("order", [1, 2, 5, 7])
@pytest.mark.parametrize("dir", [0, 1])
@pytest.mark.parametrize("hot", ["left", "right"])
def test_launch_interface_one_sided_overflow(order, dir, hot):
    import torch
    from quasar_b200 import launch as L
    n, ng = 24, M.nghost(order)
    m = n + 2 * ng
    quiet = [1.0, 0.0, 0.0, 0.0, 0.9, 0.1, 0.2, 0.3]
    sides = {s: [torch.full((m, m), q, dtype=torch.float64, device="cuda") for q in quiet]
             for s in ("left", "right")}
    clean = [x.clone() for x in sides["left"]]
    sides[hot][4][:] = 1e160
    grid, bc = L.Grid(n, n, ng, 1.0 / n, 1.0 / n), L.flags([1, 1, 1, 1])
    states = L.iface(sides["left"], sides["right"])
    calm = L.iface(clean, clean)
    scratch = torch.zeros(m * m, dtype=torch.float64, device="cuda")
    rate = L.cfl_max_rate(grid, states if dir == 0 else calm, calm if dir == 0 else states,
                          GAMMA, scratch, order, bc)
    assert rate.scaled_max_rate == np.inf
    if order == 1:
        return
    out = [torch.zeros((m, m), dtype=torch.float64, device="cuda") for _ in range(8)]
    L.hlld_flux(grid, states, dir, L.field(out), bc, GAMMA, order)
    rows = slice(ng, ng + n + (1 if dir == 1 else 0))
    cols = slice(ng, ng + n + (1 if dir == 0 else 0))
    got = np.array([o.cpu().numpy()[rows, cols] for o in out])
    # infinite speeds leave the HLL combination undefined: the left state's
    # physical flux, at rest its total pressure and field tensions
    e = 1e160 if hot == "left" else quiet[4]
    b = quiet[5:]
    p = (GAMMA - 1.0) * (e - 0.5 * sum(x * x for x in b))
    pt = p + 0.5 * sum(x * x for x in b)
    n_, t_ = (1, 2) if dir == 0 else (2, 1)
    want = [0.0] * 8
    bn, bt = b[dir], b[1 - dir]
    want[n_], want[t_], want[3] = pt - bn * bn, -bn * bt, -bn * b[2]
    for c in range(8):
        # rounding of the sums over the Gauss points and of the pressure
        assert np.all(np.abs(got[c] - want[c]) <= 32 * 2.0 ** -53 * max(abs(want[c]), 0.0 if c == n_ else 1.0)), c
