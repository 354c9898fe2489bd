"""Pointwise numerics of the stage kernels on the GPU: the reciprocal and
inverse square root against correctly rounded values, and the Riemann flux
against the oracle over the wave patterns it distinguishes."""
import ctypes

import numpy as np
import pytest

import mhd_cases as M

pytestmark = pytest.mark.gpu

GAMMA = 5.0 / 3.0


@pytest.mark.parametrize("lo,hi", [(-1.0, 1.0), (-300.0, 300.0)])
def test_reciprocal_and_inverse_root_within_an_ulp(lo, hi):
    from quasar_b200 import _native
    rng = np.random.default_rng(int(hi))
    x = 10.0 ** rng.uniform(lo, hi, 1 << 18)
    x[:4] = [1.0, 4.0, 1.0 + 2.0 ** -52, 2.0 - 2.0 ** -52]
    y, z = np.empty_like(x), np.empty_like(x)
    _native.check(_native.lib().qmhd_probe_roots(x.ctypes.data, x.size, y.ctypes.data,
                                                 z.ctypes.data))
    e = np.longdouble(1) / np.longdouble(x)
    r = np.longdouble(1) / np.sqrt(np.longdouble(x))
    # reciprocal: truncation 2^-59 and one final rounding.  Root: e = 1 - x y^2
    # also carries the rounding of x y, 2^-53 of one, which moves the result
    # by half of that (at most half an ulp) beside the final rounding.
    assert np.max(np.abs(np.longdouble(y) - e) / np.spacing(np.abs(np.float64(e)))) <= 0.55
    assert np.max(np.abs(np.longdouble(z) - r) / np.spacing(np.abs(np.float64(r)))) <= 1.05


def states(pattern, n, rng):
    """n pairs of conserved states with a common normal field."""
    def cons(rho, v, p, b):
        e = p / (GAMMA - 1) + 0.5 * rho * (v ** 2).sum(0) + 0.5 * (b ** 2).sum(0)
        return np.stack([rho, *(rho * v), e, *b])
    rho = rng.uniform(0.2, 3.0, (2, n))
    p = 10.0 ** rng.uniform(-1.5, 1.0, (2, n))
    v, b = rng.normal(0, 0.5, (2, 3, n)), rng.normal(0, 0.8, (2, 3, n))
    if pattern == "supersonic":
        v[:, 0] += rng.choice([-12.0, 12.0], n)
    elif pattern == "no_normal_field":
        b[:, 0] = 0.0
    elif pattern == "field_free":
        b[:] = 0.0
    elif pattern == "aligned":  # a degenerate fan: no transverse field
        b[:, 1:] = 0.0
    elif pattern == "equal":
        rho[1], p[1], v[1], b[1] = rho[0], p[0], v[0], b[0]
    elif pattern == "strong":
        p[1] *= 1e3
        rho[1] *= 0.05
    b[1, 0] = b[0, 0]
    return cons(rho[0], v[0], p[0], b[0]), cons(rho[1], v[1], p[1], b[1])


@pytest.mark.parametrize("pattern", ["general", "supersonic", "no_normal_field", "field_free",
                                     "aligned", "equal", "strong"])
@pytest.mark.parametrize("dir", [0, 1])
def test_riemann_flux_matches_oracle(oracle, pattern, dir):
    """Order 2 takes the face states themselves, so a face is one solve."""
    import torch
    from quasar_b200 import launch as L
    nx, ny, ng = 33, 17, 2
    shape = (ny + 2 * ng, nx + 2 * ng)
    n = shape[0] * shape[1]
    l, r = states(pattern, n, np.random.default_rng(dir + 7))
    swap = [0, 2, 1, 3, 4, 6, 5, 7] if dir == 1 else list(range(8))
    dev = lambda a: [torch.tensor(a[c], device="cuda") for c in swap]  # noqa: E731
    left, right = dev(l), dev(r)
    out = [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(8)]
    L.hlld_flux(L.Grid(nx, ny, ng, 1.0 / nx, 1.0 / ny), L.iface(left, right), dir, L.field(out),
                L.flags([1, 1, 1, 1]), GAMMA, 2)
    got = np.stack([out[c].cpu().numpy().reshape(shape) for c in swap])
    rows = slice(ng, ng + ny + (1 if dir == 1 else 0))
    cols = slice(ng, ng + nx + (1 if dir == 0 else 0))
    idx = np.arange(n).reshape(shape)[rows, cols].ravel()
    want = np.stack([oracle.hlld_flux_x(l[:, k], r[:, k], GAMMA) for k in idx], axis=1)
    got = got[:, rows, cols].reshape(8, -1)
    # rounding of a flux: a few hundred operations on terms of the size of
    # the states' fluxes at the fast speed, times the amplification 1 / (1 -
    # B_n^2 / t) of the star states, which random data keeps below 1e4
    u = np.maximum(np.abs(l), np.abs(r))[:, idx]
    speed = np.abs(u[1:4]).max(0) / np.minimum(l[0], r[0])[idx] + np.sqrt(
        2 * GAMMA * u[4] / np.minimum(l[0], r[0])[idx])
    scale = np.maximum(u[4], u[4] * speed) + u[0] * speed * np.maximum(1.0, speed)
    assert np.max(np.abs(got - want) / scale) <= 200 * 1e4 * 2.0 ** -53
    if pattern in ("equal", "field_free"):
        assert np.max(np.abs(got - want) / scale) <= 200 * 2.0 ** -53
    # face by face: the rounding of a solve acts like relative changes of its
    # operands, some thirty dependent operations in each of the two programs, each
    # reaching the flux through the sensitivities to the sixteen inputs, at most
    # twice: 128 u times their sum (differences of the oracle's own flux at 1e-6),
    # and 8 u of the sums that inputs equal to zero leave out
    tol = np.empty_like(want)
    for m, k in enumerate(idx):
        x = np.concatenate([l[:, k], r[:, k]])
        y = np.repeat(x[:, None], 16, axis=1)
        y[np.arange(16), np.arange(16)] *= 1.0 + 1e-6
        y[13, 5], y[5, 13] = y[5, 5], y[13, 13]  # one normal field
        s = sum(np.abs(oracle.hlld_flux_x(y[:8, q], y[8:, q], GAMMA) - want[:, m]) for q in range(16)) / 1e-6
        big = x[4] + x[12]
        speed = np.abs(np.concatenate([x[1:4] / x[0], x[9:12] / x[8]])).max() + np.sqrt(
            2 * GAMMA * big / min(x[0], x[8]))
        tol[:, m] = (128 * s + 8 * big * max(1.0, speed)) * 2.0 ** -53
    assert np.all(np.abs(got - want) <= tol), float(np.max(np.abs(got - want) / tol))


@pytest.mark.parametrize("lo,hi", [(-0.3, 0.3), (-100.0, 100.0)])
def test_shared_quotients_have_the_bits_of_division(lo, hi):
    """Random operands, divisors next to powers of two and divisors whose
    significand is all ones, against IEEE division (the eigen scalars branch on
    these bits; 1 - c_s^2 / c_f^2 is 1 - 2^-53 where c_s / c_f is near 1e-8)."""
    from quasar_b200 import _native
    rng = np.random.default_rng(5)
    n = 1 << 20
    a, b = (rng.choice([-1.0, 1.0], n) * 10.0 ** rng.uniform(lo, hi, n) for _ in range(2))
    b[: n // 8] = 2.0 ** rng.integers(-3, 4, n // 8) * (1.0 + rng.integers(-4, 5, n // 8) * 2.0 ** -52)
    a[: n // 16] = rng.integers(1, 1 << 53, n // 16).astype(np.float64)
    b[n // 8: n // 4] = 2.0 ** rng.integers(-20, 21, n // 8) * (1.0 - 2.0 ** -53)
    q = np.empty(n)
    _native.check(_native.lib().qmhd_probe_quotients(a.ctypes.data, b.ctypes.data, n, q.ctypes.data))
    differ = q != a / b
    assert not np.any(differ), int(differ.sum())
