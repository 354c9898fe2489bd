"""Densities below the normal range, where the shortened reciprocal has no value:
such gas is admissible, has its CFL limit and steps, as far as 1 / rho exists
(rho above 5.6e-309)."""
import numpy as np
import pytest

import mhd_cases as M
from test_gpu_parity import gpu_solver, read, seed

pytestmark = pytest.mark.gpu

GAMMA = 5.0 / 3.0
RHO = [6.7e-309, 1.1e-308, 2.2250738585072014e-308, 3e-308]  # the last two are normal


def at_rest(n, order, rho, p):
    ng = M.nghost(order)
    a = [np.zeros((n + 2 * ng, n + 2 * ng)) for _ in range(8)]
    a[0][:], a[4][:] = rho, p / (GAMMA - 1.0)
    return a


@pytest.mark.parametrize("order", [2, 5, 7])
@pytest.mark.parametrize("rho", RHO)
def test_gas_at_rest_keeps_its_state_and_sound_speed(order, rho):
    n = 40  # several tiles and warps a side
    # pressure so that a^2 is of order one and p has its digits
    state = at_rest(n, order, rho, 0.6 * rho)
    g = gpu_solver(n, order, M.OUTFLOW)
    seed(g, state)
    a = np.sqrt(GAMMA * 0.6)
    eff = min(0.4, 0.2) if order >= 5 else 0.4
    # four faces of rate a / (2 h) each; a subnormal number of this size
    # carries 2^-1074 of rounding, 1e-15 of it
    dt = eff / (2.0 * a * n)
    for _ in range(2):
        assert abs(g.cfl_limit() - dt) <= 1e-13 * dt
        g.step_unchecked(dt)
    for got, want in zip(read(g, state[0].shape), state):
        assert np.all(np.abs(got - want) <= 1e-14 * np.abs(want))


@pytest.mark.parametrize("order", [2, 5, 7])
@pytest.mark.parametrize("rho", RHO)
def test_a_bump_reconstructs_and_steps(order, rho):
    """A smooth bump in density and pressure, no two faces alike."""
    n, ng = 40, M.nghost(order)
    m = n + 2 * ng
    x = (np.arange(m) - ng + 0.5) / n
    bump = 1.0 + 0.1 * np.sin(2 * np.pi * x)[None, :] * np.cos(2 * np.pi * x)[:, None]
    state = at_rest(n, order, rho, 0.6 * rho)
    state[0] *= bump
    state[4] *= bump ** GAMMA
    g = gpu_solver(n, order, M.PERIODIC)
    seed(g, state)
    unit = gpu_solver(n, order, M.PERIODIC)
    seed(unit, [a / rho for a in state])
    dt = unit.cfl_limit()
    # first-order face states are half a cell off: h u' / 2 of the sound speed,
    # whose relative amplitude is (GAMMA - 1) / 2 of the density's
    assert abs(g.cfl_limit() - dt) <= np.pi * 0.1 * 0.5 * (GAMMA - 1.0) / n * dt
    g.step_unchecked(dt)
    unit.step_unchecked(dt)
    # subnormal densities take first-order face states and the HLL flux, beside
    # faces that do not where the bump crosses into the normal range: each of a
    # cell's four faces is off by at most half a jump, c h u' / 2 with u' at most
    # 2 pi 0.17 (the energy's amplitude), and dt c / h is at most 0.2
    bound = 4 * 0.2 * 0.5 * 2 * np.pi * 0.17 / n
    for c in (0, 1, 2, 4):
        got = M.interior(read(g, state[0].shape)[c] / rho, ng)
        want = M.interior(read(unit, state[0].shape)[c], ng)
        assert np.max(np.abs(got - want)) <= bound, c
