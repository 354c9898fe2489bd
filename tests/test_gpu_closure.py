"""The solver's one-launch boundary closure and collocation against the
separate passes of the launch interface (fill_ghosts side by side, then
collocate_face_to_cell): the whole padded state bit for bit, over boundary
pairs, orders, sizes with partial blocks and grids barely wider than their
ghost layers (narrower ones keep the separate passes)."""
import numpy as np
import pytest

import mhd_cases as M

pytestmark = pytest.mark.gpu

NAME = {2: "muscl_minmod", 5: "mp5", 7: "mp7"}
BC = {0: "periodic", 1: "outflow", 2: "wall"}


def random_state(nx, ny, ng, bc, rng):
    """Admissible, divergence-free to the bit: Bx(y), By(x), and no normal
    field at a wall."""
    shape = (ny + 2 * ng, nx + 2 * ng)
    rho, p = rng.uniform(0.5, 2.0, shape), rng.uniform(0.5, 2.0, shape)
    v = rng.normal(0, 0.3, (3, *shape))
    bx = np.repeat(rng.normal(0, 0.5, (shape[0], 1)), shape[1], 1)
    by = np.repeat(rng.normal(0, 0.5, (1, shape[1])), shape[0], 0)
    if 2 in bc[:2]:
        bx[:] = 0.0
    if 2 in bc[2:]:
        by[:] = 0.0
    bz = rng.normal(0, 0.5, shape)
    # ample internal energy: the collocated field of random faces may exceed
    # the faces' own
    e = p * 20.0 + 0.5 * rho * (v ** 2).sum(0) + 2.0 * (bx ** 2 + by ** 2) + 0.5 * bz ** 2
    return [rho, *(rho * v), e, bx, by, bz]


@pytest.mark.parametrize("bc", [(0, 0, 0, 0), (1, 1, 1, 1), (2, 2, 2, 2), (0, 0, 2, 1), (1, 2, 0, 0),
                                (2, 1, 1, 2)])
@pytest.mark.parametrize("order,nx,ny", [(5, 33, 17), (7, 5, 70), (7, 64, 5), (5, 4, 4), (2, 45, 3),
                                         (7, 4, 40), (7, 97, 41)])
def test_closed_state_matches_separate_passes(order, nx, ny, bc):
    import torch
    from quasar_b200 import launch as L
    from quasar_b200 import mhd
    cfg = mhd.MhdConfig()
    cfg.grid = mhd.Grid2D(nx, ny, 1.0, 1.0)
    cfg.reconstruction = NAME[order]
    cfg.boundary = mhd.MhdBoundarySpec([BC[b] for b in bc], [BC[b] for b in bc])
    s = mhd.MhdSolver2D(cfg)
    ng = M.nghost(order)
    state = random_state(nx, ny, ng, bc, np.random.default_rng(nx * 100 + ny))
    for name, a in zip(M.COMPONENTS, state):
        s.seed_state(name, a)
    got = {c: s.state_component_to_host(c) for c in ("bx", "by")}  # closes and collocates
    got.update({c: s.state_component_to_host(c) for c in M.COMPONENTS})
    grid = L.Grid(nx, ny, ng, 1.0 / nx, 1.0 / ny)
    u = [torch.tensor(a.ravel(), device="cuda") for a in state]
    L.fill_ghosts(grid, L.field(u), bc)
    cell = [torch.zeros_like(u[0]) for _ in range(2)]
    L.collocate_face_to_cell(grid, 0, u[5], cell[0])
    L.collocate_face_to_cell(grid, 1, u[6], cell[1])
    torch.cuda.synchronize()
    for name, want in zip((*M.COMPONENTS, "bx", "by"), (*u, *cell)):
        assert np.array_equal(got[name], want.cpu().numpy()), name
