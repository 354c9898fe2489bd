"""The bound with which the reconstruction skips the L R = I check of a face
(eig_scalars in quasar_b200/csrc/mhd_kernels.cu): wherever it holds, the check
it replaces passes (mhd_eigensystem.hpp:416-430 of the reference: every entry of
L R - I within 1024 eps).  Once restated in numpy, formed in binary64 from full
rows and columns, and once on the GPU with the kernel's own bound, rows and
columns."""
import numpy as np
import pytest

EPS = np.finfo(np.float64).eps


def scalars(rho, v, p, b, gamma):
    ir, sr = 1.0 / rho, np.sqrt(rho)
    a = np.sqrt(gamma) * (np.sqrt(p) / sr)
    ca2 = (b ** 2).sum(0) / rho
    scale = np.maximum(a, np.sqrt(ca2))
    an, bn, cn = a / scale, np.sqrt(ca2) / scale, np.abs(b[0]) / sr / scale
    s = an * an + bn * bn
    f2 = 0.5 * (s + np.sqrt(np.maximum(s * s - 4.0 * (an * an) * (cn * cn), 0.0)))
    s2 = an * an * (cn * cn) / f2
    cf, cs = scale * np.sqrt(f2), scale * np.sqrt(s2)
    cn_, an_ = cs / cf, a / cf
    den = 1.0 - cn_ * cn_
    tie = den <= 64.0 * EPS * (1.0 + cn_ * cn_)
    with np.errstate(divide="ignore", invalid="ignore"):
        af2, as2 = (an_ * an_ - cn_ * cn_) / den, (1.0 - an_ * an_) / den
        clip = np.where(tie, 0.0, np.maximum(0.0, -np.minimum(af2, as2)))
        af = np.where(tie, np.sqrt(0.5), np.sqrt(np.maximum(af2, 0.0)))
        as_ = np.where(tie, np.sqrt(0.5), np.sqrt(np.maximum(as2, 0.0)))
        bt = np.hypot(b[1], b[2])
        none = (bt == 0.0) | (bt / sr <= 64.0 * EPS * np.maximum(a, np.sqrt(ca2)))
        b1, b2 = (np.where(none, np.sqrt(0.5), x / np.where(none, 1.0, bt)) for x in b[1:])
    return dict(rho=rho, ir=ir, sr=sr, v=v, a=a, cf=cf, cs=cs, af=af, as_=as_, b1=b1, b2=b2,
                den=np.where(tie, 0.0, den), clip=clip, sb=np.where(b[0] >= 0, 1.0, -1.0), bt=b[1:],
                gm1=gamma - 1.0, hv2=0.5 * (v ** 2).sum(0), ra2=gamma * p, ia=1.0 / a)


def sure(e):
    k, g = e["cf"] * e["ia"], e["gm1"]
    m = np.abs(e["v"]).sum(0) * e["ia"]
    b = np.abs(e["bt"]).sum(0) * (e["ia"] * e["sr"] * e["ir"])
    f = 3.0 + 3.0 * (k + g * b) + 1.5 * k * k + m * (2.0 + (1.0 + 4.0 * g) * k + 2.0 * g * m)
    w = np.maximum(e["rho"], e["ir"]) * np.maximum(e["a"], e["ia"])
    return (80.0 - w * f) * e["den"] >= k * k * (1.0 + 3.8e14 * e["den"] * e["clip"])


def product_error(e):
    """max |L R - I| from the seven rows and columns in conserved variables."""
    z, one = np.zeros_like(e["rho"]), np.ones_like(e["rho"])
    nf, s2 = 0.5 * e["ia"] ** 2, np.sqrt(0.5)
    rp, lp = [], []
    for al, cc, q, w in ((e["af"], e["cf"], e["cs"] * e["as_"] * e["sb"], e["a"] * e["as_"] * e["sr"]),
                         (e["as_"], e["cs"], -e["cf"] * e["af"] * e["sb"], -e["a"] * e["af"] * e["sr"])):
        for sg in (-1.0, 1.0):
            rp.append([e["rho"] * al, sg * al * cc, -sg * q * e["b1"], -sg * q * e["b2"],
                       al * e["ra2"], w * e["b1"], w * e["b2"]])
            lp.append([z, sg * nf * al * cc, -sg * nf * q * e["b1"], -sg * nf * q * e["b2"],
                       nf * al * e["ir"], nf * w * e["b1"] * e["ir"], nf * w * e["b2"] * e["ir"]])
    for sg in (-1.0, 1.0):
        c = sg * e["sb"] * s2
        rp.append([z, z, -e["b2"] * s2, e["b1"] * s2, z, c * e["b2"] * e["sr"], -c * e["b1"] * e["sr"]])
        lp.append([z, z, -e["b2"] * s2, e["b1"] * s2, z, c * e["b2"] * e["sr"] * e["ir"],
                   -c * e["b1"] * e["sr"] * e["ir"]])
    rp.append([one, z, z, z, z, z, z])
    lp.append([one, z, z, z, -e["ia"] ** 2, z, z])
    v, g = e["v"], e["gm1"]
    left = np.array([[q[0] - (q[1] * v[0] + q[2] * v[1] + q[3] * v[2]) * e["ir"] + q[4] * g * e["hv2"]]
                     + [q[1 + i] * e["ir"] - q[4] * g * v[i] for i in range(3)]
                     + [q[4] * g, q[5] - q[4] * g * e["bt"][0], q[6] - q[4] * g * e["bt"][1]]
                     for q in lp])
    right = np.array([[q[0]] + [v[i] * q[0] + e["rho"] * q[1 + i] for i in range(3)]
                      + [e["hv2"] * q[0] + e["rho"] * (v[0] * q[1] + v[1] * q[2] + v[2] * q[3])
                         + q[4] / g + e["bt"][0] * q[5] + e["bt"][1] * q[6], q[5], q[6]] for q in rp])
    d = np.einsum("imn,jmn->ijn", left, right) - np.eye(7)[:, :, None]
    return np.abs(d).max((0, 1))


KINDS = pytest.mark.parametrize("kind", ["general", "near_degenerate", "weak_field", "strong_field"])
SPREADS = pytest.mark.parametrize("spread", [0.3, 1.0, 3.0])


def sample(kind, spread, n=60000):
    rng = np.random.default_rng(11)
    gamma = float(rng.choice([1.1, 1.4, 5.0 / 3.0, 2.0, 3.0]))
    lg = lambda s: 10.0 ** rng.uniform(-s, s, n)  # noqa: E731
    rho, p = lg(0.4 * spread), lg(0.4 * spread)
    v = rng.normal(0, 1, (3, n)) * lg(0.3 * spread)
    b = rng.normal(0, 1, (3, n)) * lg(0.4 * spread)
    if kind == "near_degenerate":  # c_f close to c_s: a = |B_n| / sqrt(rho), small B_t
        b[0] = np.sqrt(gamma * p) * (1.0 + rng.normal(0, 1, n) * 10.0 ** rng.uniform(-12, 0, n))
        b[1:] *= 10.0 ** rng.uniform(-12, 0, n)
    elif kind == "weak_field":
        b *= 10.0 ** rng.uniform(-8, 0, n)
    elif kind == "strong_field":
        b *= 10.0 ** rng.uniform(0, 3, n)
    return rho, v, p, b, gamma


@SPREADS
@KINDS
def test_bound_implies_the_check(kind, spread):
    e = scalars(*sample(kind, spread))
    ok = sure(e)
    err = product_error(e)
    assert not np.any(err[ok] > 1024 * EPS), (kind, np.max(err[ok]) / EPS)
    # it is of use everywhere, most where states are of order one
    assert ok.mean() > (0.2 if kind == "general" and spread == 0.3 else 0.01)


@pytest.mark.gpu
@SPREADS
@KINDS
def test_the_kernels_bound_implies_its_check(kind, spread):
    """The kernel's own decision and vectors; and near the threshold, where its
    decision changes along a line of states of growing velocity."""
    from quasar_b200 import _native
    rho, v, p, b, gamma = sample(kind, spread)
    line = np.outer([0.5, 1.0, -0.7], np.linspace(0.0, 40.0, 4001))
    one = np.ones(line.shape[1])
    rho, p = np.concatenate([rho, one]), np.concatenate([p, 0.8 * one])
    v, b = np.concatenate([v, line], 1), np.concatenate([b, np.outer([0.6, 0.4, -0.3], one)], 1)
    e = p / (gamma - 1) + 0.5 * rho * (v ** 2).sum(0) + 0.5 * (b ** 2).sum(0)
    states = np.ascontiguousarray(np.stack([rho, *(rho * v), e, *b]))
    n = rho.size
    ok, err = np.zeros(n, np.int32), np.zeros(n)
    _native.check(_native.lib().qmhd_probe_eigen(states.ctypes.data, n, gamma, ok.ctypes.data, err.ctypes.data))
    ok = ok != 0
    assert not np.any(err[ok] > 1024 * EPS), (kind, np.max(err[ok]) / EPS)
    assert not np.any(np.isnan(err[ok]))
    assert ok[:60000].mean() > (0.2 if kind == "general" and spread == 0.3 else 0.01)
    on_line = ok[60000:]
    assert on_line[0] and not on_line[-1]


def test_bound_refuses_what_the_check_refuses():
    rho = np.array([1.0, 1e8, 1.0, np.nan])
    v = np.array([[0.0, 0, 1e6, 0]] + [[0.0, 0, 0, 0]] * 2)
    b = np.array([[1.0, 1, 1, 1], [1e-14, 1, 1, 1], [0.0, 0, 0, 0]])
    p = np.array([1.0 / (5.0 / 3.0), 1.0, 1.0, 1.0])
    with np.errstate(invalid="ignore"):
        assert not sure(scalars(rho, v, p, b, 5.0 / 3.0)).any()
