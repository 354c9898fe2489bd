"""Which corners take a one-dimensional value: the corner EMF calls a row or a
column of the cell table constant where its samples compare equal, so zeros of
both signs and equal infinities count as equal, along either axis alike."""
import numpy as np
import pytest

import mhd_cases as M

pytestmark = pytest.mark.gpu

EX, EY = 0.5, 0.25


def corner(order, cell, along, ex=EX, ey=EY, nx=45, ny=37):
    """Corner E_z where the no-jump proofs hold along one axis only."""
    import torch
    from quasar_b200 import launch as L
    ng = M.nghost(order)
    shape = (ny + 2 * ng, nx + 2 * ng)
    full = lambda v, t=torch.float64: torch.full(shape, v, dtype=t, device="cuda")  # noqa: E731
    cell = torch.tensor(cell(shape), dtype=torch.float64, device="cuda")
    table = [full(ex), full(ey), full(1 if along == "x" else 0, torch.int32),
             full(1 if along == "y" else 0, torch.int32), cell, full(0.0)]
    L.ct_emf_finish(L.Grid(nx, ny, ng, 1.0 / nx, 1.0 / ny), L.flags([1, 1, 1, 1]), L.emf(*table), order)
    return table[5].cpu().numpy()[ng:ng + ny + 1, ng:ng + nx + 1]


# proofs on the x faces and constant rows leave the y faces' value, proofs on
# the y faces and constant columns the x faces'
@pytest.mark.parametrize("order", [2, 5, 7])
@pytest.mark.parametrize("along,want", [("x", EY), ("y", EX)])
def test_zeros_of_both_signs_are_equal(order, along, want):
    rng = np.random.default_rng(order)
    got = corner(order, lambda s: np.where(rng.random(s) < 0.5, 0.0, -0.0), along)
    assert np.all(got == want)


@pytest.mark.parametrize("order", [2, 5, 7])
@pytest.mark.parametrize("along,want", [("x", EY), ("y", EX)])
def test_equal_infinities_are_equal(order, along, want):
    got = corner(order, lambda s: np.full(s, np.inf), along)
    assert np.all(got == want)


@pytest.mark.parametrize("order", [2, 5, 7])
@pytest.mark.parametrize("along", ["x", "y"])
def test_equal_infinite_samples_return_their_value(order, along):
    got = corner(order, np.zeros, along, ex=-np.inf, ey=np.inf)
    assert np.all(got == (np.inf if along == "x" else -np.inf))


@pytest.mark.parametrize("order", [2, 5, 7])
@pytest.mark.parametrize("along", ["x", "y"])
def test_a_jump_is_not_constant(order, along):
    """A cell that differs in one corner's stencil: e_x + e_y - centred there."""
    nx, ny, lo = 45, 37, {2: -1, 5: -3, 7: -4}[order]
    ng = M.nghost(order)
    j, i = 18, 22

    def cell(shape):
        c = np.zeros(shape)
        c[ng + j, ng + i] = 1e-300
        return c
    got = corner(order, cell, along)
    want = np.full((ny + 1, nx + 1), EY if along == "x" else EX)
    rows = slice(j + lo + 1, j - lo + 1)
    cols = slice(i + lo + 1, i - lo + 1)
    want[rows, cols] = EX + EY
    assert np.array_equal(got, want)
