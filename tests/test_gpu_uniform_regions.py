"""Grids that are mostly one state: the reconstruction, the face flux and the
cell EMF finish warps and tiles without a jump early, and the result is the
oracle's wherever the disturbance lies against their edges."""
import numpy as np
import pytest

import mhd_cases as M

pytestmark = pytest.mark.gpu

NAME = {5: "mp5", 7: "mp7"}
BC = {0: "periodic", 1: "outflow"}
GAMMA = 5.0 / 3.0


def solver(nx, ny, order, bc):
    from quasar_b200 import mhd
    cfg = mhd.MhdConfig()
    cfg.grid = mhd.Grid2D(nx, ny, 1.0, 1.0)
    cfg.reconstruction = NAME[order]
    cfg.boundary = mhd.MhdBoundarySpec([BC[b] for b in bc], [BC[b] for b in bc])
    return mhd.MhdSolver2D(cfg)


def uniform(nx, ny, order):
    ng = M.nghost(order)
    one = np.ones((ny + 2 * ng, nx + 2 * ng))
    rho, v, p, b = 1.3, (0.4, -0.25, 0.1), 0.7, (0.5, -0.3, 0.2)
    e = p / (GAMMA - 1) + 0.5 * rho * sum(x * x for x in v) + 0.5 * sum(x * x for x in b)
    return [q * one for q in (rho, rho * v[0], rho * v[1], rho * v[2], e, *b)]


@pytest.mark.parametrize("order,nx,ny", [(5, 33, 17), (7, 64, 48), (7, 70, 41)])
def test_uniform_state_stays_uniform(order, nx, ny):
    s = solver(nx, ny, order, M.PERIODIC)
    state = uniform(nx, ny, order)
    for name, a in zip(M.COMPONENTS, state):
        s.seed_state(name, a)
    s.advance_auto(0.0, 1e30, 3)
    for name, a in zip(M.COMPONENTS, state):
        assert np.array_equal(s.state_component_to_host(name).reshape(a.shape), a), name


# sizes with several warps and tiles a side; positions on and beside the edges
# of 32-face warps, 8 x 4 face tiles and 16 x 14 cell tiles, and at the domain's
@pytest.mark.parametrize("bc", [M.PERIODIC, M.OUTFLOW])
@pytest.mark.parametrize("order,at", [(5, (0, 0)), (5, (32, 15)), (5, (95, 40)), (7, (0, 63)),
                                      (7, (31, 28)), (7, (32, 13)), (7, (64, 32)), (7, (95, 0)),
                                      (7, (47, 41))])
def test_local_disturbance_matches_oracle(oracle, order, at, bc):
    nx, ny = 96, 64
    ng = M.nghost(order)
    state = uniform(nx, ny, order)
    i, j = at[0] + ng, at[1] + ng
    # one cell of denser, hotter gas moving with the flow
    for c, f in ((0, 1.5), (1, 1.5), (2, 1.5), (3, 1.5), (4, 1.8)):
        state[c][j, i] *= f
    g, o = solver(nx, ny, order, bc), oracle.solver(nx, ny, order, bc=bc)
    for name, a in zip(M.COMPONENTS, state):
        g.seed_state(name, a)
    o.seed(state)
    for k in range(2):
        dt = o.cfl()
        assert abs(g.cfl_limit() - dt) <= 1e-12 * dt
        g.step_unchecked(dt)
        o.step(dt)
    got = [g.state_component_to_host(c).reshape(state[0].shape) for c in M.COMPONENTS]
    # rounding of two steps: a few hundred operations a value
    assert M.state_rel_l1(got, o.read(), ng, nx, ny) <= 500 * 2.0 ** -53


# a disturbance reaches 8 cells a stage (stencil, transverse Gauss points, CT
# corner); beyond 3 stages' reach the moving, magnetised gas keeps its bits,
# in early-finished tiles and in those beside them
@pytest.mark.parametrize("order", [5, 7])
@pytest.mark.parametrize("row", [0, 40])
def test_gas_beyond_the_disturbance_keeps_its_bits(order, row):
    nx, ny = 96, 64
    ng = M.nghost(order)
    state = uniform(nx, ny, order)
    state[0][row + ng, ng] *= 1.5
    state[4][row + ng, ng] *= 1.8
    s = solver(nx, ny, order, M.OUTFLOW)
    for name, a in zip(M.COMPONENTS, state):
        s.seed_state(name, a)
    s.advance_auto(0.0, 1e30, 1)
    for name, a in zip(M.COMPONENTS, state):
        got = s.state_component_to_host(name).reshape(a.shape)
        assert np.array_equal(got[:, ng + 25:], a[:, ng + 25:]), name
