"""The host-driven loop (cfl_limit, step_unchecked) past its 32nd step,
where it replays captured launches: limits and states are the oracle's, the
step is the one the caller asks for, and a changed window is honoured."""
import pytest

import mhd_cases as M
from test_gpu_parity import CASES, DT_TOL, STEP_TOL, gpu_solver, read, seed

pytestmark = pytest.mark.gpu


# (not the rotor: its zero transverse field turns a rounding difference into its
# square root, and forty steps gather 3e-12 in dt, with launches as with graphs)
@pytest.mark.parametrize("order,case,bc", [(2, "ot", M.PERIODIC), (5, "ot", M.PERIODIC),
                                           (7, "ot", M.PERIODIC), (7, "blast", M.OUTFLOW)])
def test_forty_steps_match_oracle(oracle, order, case, bc):
    n, ng = 32, M.nghost(order)
    ic = CASES[case](n, order=order)
    g, o = gpu_solver(n, order, bc), oracle.solver(n, n, order, bc=bc)
    seed(g, ic)
    o.seed(ic)
    for k in range(40):
        dt = o.cfl()
        if k != 35:  # a step without its limit asked for
            assert abs(g.cfl_limit() - dt) <= DT_TOL * dt
        dt *= (0.5, 1.0, 0.8)[k % 3]
        g.step_unchecked(dt)
        o.step(dt)
        assert M.state_rel_l1(read(g, ic[0].shape), o.read(), ng, n, n) <= STEP_TOL, k


def test_window_set_after_the_capture():
    n, order = 32, 5
    ic = CASES["rotor"](n, order=order)
    a = gpu_solver(n, order, M.OUTFLOW)
    seed(a, ic)
    for _ in range(36):
        a.step_unchecked(a.cfl_limit())
    whole = a.cfl_limit()
    now = read(a, ic[0].shape)
    a.set_owned_window(0, 6, 0, 6)  # the corner's gas is at rest
    b = gpu_solver(n, order, M.OUTFLOW)
    seed(b, now)
    b.set_owned_window(0, 6, 0, 6)
    for _ in range(36):
        dt = b.cfl_limit()
        assert dt > whole and abs(a.cfl_limit() - dt) <= DT_TOL * dt
        a.step_unchecked(0.5 * whole)
        b.step_unchecked(0.5 * whole)
