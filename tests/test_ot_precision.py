"""sfwi_ot and its siblings where 48 bits would not do, against the formulas in long double
(64 bits of mantissa or more).  Residuals are FP32 (6e-8 of their size); the kernel's
sums and their cancellations leave no more than that, so 1e-6 of the largest.
Misfits of nearly equal densities are sums of squares of r, whose error is the
weights' (2^-53 of 1 / sigma^2) over r, here at least 1e-6: 1e-9."""
import numpy as np
import pytest

from tests.test_ot_formats import _fn

pytestmark = pytest.mark.gpu
L = np.longdouble


def _power(obs, cal, sigma, dt):
    """misfit and adjoint source of OT_power of one trace"""
    o, u, s, n = obs.astype(L), cal.astype(L), L(sigma), len(obs)
    eps = L(1e-3) * s * s
    p, g = u * u + eps, o * o + eps
    f, g = p / p.sum(), g / g.sum()
    F, G = np.cumsum(f), np.cumsum(g)
    m = np.minimum(np.searchsorted(G, F, side="right"), n - 1)
    r = np.arange(1, n + 1) - (m + (F - np.where(m > 0, G[m - 1], L(0))) / g[m])
    A = r * r - 2 * np.cumsum((r * f / g[m])[::-1])[::-1]
    d2 = L(np.float32(dt)) ** 2
    return float(d2 * (r * r * f).sum()), (d2 / 2 * (A - (f * A).sum()) / p.sum() * 2 * u).astype(np.float64)


def _run(obs, cal, dt=1e-3):
    z = np.zeros_like(obs)
    rx, _, m = _fn(2)(obs, z, cal, z, dt)
    return rx, m


@pytest.mark.parametrize("nt", [5, 40, 900, 7161])
@pytest.mark.parametrize("ratio", [300.0, 1000.0, 1e4])
def test_a_sample_that_holds_the_weight(nt, ratio):
    """a dead observed trace beside a live one: its scale is the floor, and a
    spike of the prediction holds all but some 1e-3 / ratio^2 nt of the weight"""
    rng = np.random.default_rng(nt)
    obs = np.stack([np.zeros(nt), rng.standard_normal(nt)]).astype(np.float32)
    cal = np.stack([1e-9 * rng.standard_normal(nt), rng.standard_normal(nt)]).astype(np.float32)
    top = np.abs(obs).max()
    cal[0, nt // 3] = ratio * 1.1e-3 * top
    rx, _ = _run(obs, cal)
    for k in range(2):
        _, want = _power(obs[k], cal[k], max(np.abs(obs[k]).max(), 1e-3 * float(top)), 1e-3)
        spike = int(np.abs(cal[k]).argmax())
        assert abs(rx[k, spike] - want[spike]) <= 1e-6 * abs(want[spike]), (k, rx[k, spike], want[spike])
        assert np.abs(rx[k] - want).max() <= 1e-6 * np.abs(want).max()


@pytest.mark.parametrize("nt", [5, 33])
def test_nearly_equal_densities(nt):
    rng = np.random.default_rng(nt)
    obs = np.ones((1, nt), np.float32)
    cal = (0.006 * (1 + 1e-5 * rng.standard_normal((1, nt)))).astype(np.float32)
    rx, m = _run(obs, cal)
    want_m, want = _power(obs[0], cal[0], float(np.abs(obs).max()), 1e-3)
    assert abs(m - want_m) <= 1e-9 * want_m
    assert np.abs(rx[0] - want).max() <= 1e-6 * np.abs(want).max()


@pytest.mark.parametrize("kind", [1, 2, 3])
@pytest.mark.parametrize("nt", [3, 100, 2999, 7161])
def test_constant_traces_are_transported_nowhere(kind, nt):
    """densities of equal shape and other sums"""
    obs = np.stack([np.full(nt, v, np.float32) for v in (0.7, -1.3, 0.01)])
    cal = np.stack([np.full(nt, v, np.float32) for v in (-0.11, 2.9, 0.6)])
    rx, rz, m = _fn(kind)(obs, obs, cal, cal, 1e-3)
    assert m == 0 and not rx.any() and not rz.any()
