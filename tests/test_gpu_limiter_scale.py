"""The monotonicity-preserving limiter decides alike at every magnitude: states
scaled by powers of two reconstruct to face states scaled by the same powers,
bit for bit, also where the squares of their differences leave the binary64
range."""
import numpy as np
import pytest

import mhd_cases as M

pytestmark = pytest.mark.gpu

GAMMA = 5.0 / 3.0


def gas(nx, ny, ng, seed):
    """Steps and noise in every component: the limiter fires on many faces."""
    rng = np.random.default_rng(seed)
    shape = (ny + 2 * ng, nx + 2 * ng)
    f = lambda lo, hi: np.kron(rng.uniform(lo, hi, (shape[0] // 4 + 1, shape[1] // 4 + 1)),  # noqa: E731
                               np.ones((4, 4)))[:shape[0], :shape[1]] + 0.02 * rng.normal(0, 1, shape)
    rho, p = f(0.5, 2.0), f(0.5, 2.0)
    v, b = [f(-1.0, 1.0) for _ in range(3)], [f(-0.3, 0.3) for _ in range(3)]
    e = p / (GAMMA - 1) + 0.5 * rho * sum(x * x for x in v) + 0.5 * sum(x * x for x in b)
    return [rho, *(rho * x for x in v), e, *b]


def faces(state, nx, ny, order, dir, power):
    """Face states of `state` with densities, momenta and energies scaled by
    2^power and fields by its root, scaled back."""
    import torch
    from quasar_b200 import launch as L
    ng = M.nghost(order)
    k = [power if c < 5 else power // 2 for c in range(8)]
    dev = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
    u = [dev(np.ldexp(a, n)) for a, n in zip(state, k)]
    cb = [u[5].clone(), u[6].clone()]  # the collocated field of these cells
    out = [[torch.zeros_like(u[0]) for _ in range(8)] for _ in range(2)]
    L.reconstruct(L.Grid(nx, ny, ng, 1.0 / nx, 1.0 / ny), L.field(u), *cb, dir, L.iface(*out), order,
                  L.flags([1, 1, 1, 1]), GAMMA)
    rows = slice(ng, ng + ny + (1 if dir == 1 else 0))
    cols = slice(ng, ng + nx + (1 if dir == 0 else 0))
    return np.array([[np.ldexp(o.cpu().numpy()[rows, cols], -n) for o, n in zip(side, k)] for side in out])


# 2^-200 keeps every square in range; at 2^-800 those of all differences vanish,
# at 2^500 those of the larger ones overflow (momenta stay below the root of
# the largest number, as admissible states' do)
@pytest.mark.parametrize("order", [5, 7])
@pytest.mark.parametrize("dir", [0, 1])
@pytest.mark.parametrize("a,b", [(-200, -800), (200, 500)])
def test_reconstruction_scales_with_the_state(order, dir, a, b):
    nx, ny = 61, 35
    state = gas(nx, ny, M.nghost(order), order + dir)
    near, far = (faces(state, nx, ny, order, dir, p) for p in (a, b))
    assert np.isfinite(near).all()
    assert np.array_equal(near, far)
