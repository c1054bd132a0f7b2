"""One FP64 Dormand-Prince attempt (closed-form Kerr-Schild right-hand side, straight-line stages, fifth-root step
control) against the FP64 oracle, which forms the metric and its inverse in full: charge, Lambda, zero and near-maximal
spin, points near the horizon, the axis and the equator, and steps from far below to far above the accepted size.

Tolerances: both are FP64; the right-hand side's terms reach a few hundred times their sum near the horizon, so a state
after one step agrees to 1e-11 of its size. The error estimate is a sum that cancels to about 1e-6 of its terms."""
import numpy as np
import pytest

from sirius_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("a,Q,Lam", [(0.0, 0.0, 0.0), (0.9, 0.0, 0.0), (0.998, 0.05, 0.0), (0.6, 0.5, 0.0),
                                     (0.7, 0.0, 1e-4), (-0.5, 0.2, 1e-5)])
def test_attempt_matches_oracle(engine, oracle, a, Q, Lam):
    m = abi.make_metric(a=a, Q=Q, Lambda=Lam)
    cfg = abi.default_config(abs_tolerance=1e-8, rel_tolerance=1e-8, min_step=1e-9, max_step=500.0)
    engine.configure(cfg)
    rng = np.random.default_rng(7)
    n = 400
    rp = 1 + np.sqrt(1 - a * a - Q * Q)
    r = rp * np.exp(rng.uniform(np.log(1.02), np.log(60.0), n))
    mu = rng.uniform(-1, 1, n)
    mu[:40] = np.cos(rng.uniform(1e-6, 1e-3, 40))  # the axis
    mu[40:80] = rng.uniform(-1e-8, 1e-8, 40)  # the equator
    st, ph = np.sqrt(1 - mu * mu), rng.uniform(0, 2 * np.pi, n)
    x = np.stack([np.zeros(n), r * st * np.cos(ph), r * st * np.sin(ph), r * mu], 1)
    p = rng.normal(size=(n, 4))
    p[:, 0] = -1.0
    states = np.concatenate([x, p], 1)
    hs = np.exp(rng.uniform(np.log(1e-4), np.log(200.0), n))
    s0, h0, a0, e0 = oracle.dp45_step(m, cfg, states, hs)
    s1, h1, a1, e1 = engine.dp45_step(m, states, hs)
    ok = np.isfinite(e0) & (np.abs(e0 - 1) > 1e-4)
    assert ok.sum() > 0.9 * n and 0.1 < np.mean(a0[ok]) < 0.95
    np.testing.assert_array_equal(a1[ok], a0[ok])
    scale = np.abs(s0).max(1, keepdims=True)
    assert (np.abs(s1 - s0)[ok] <= 1e-11 * scale[ok]).all()
    big = ok & (e0 > 1e-3)
    np.testing.assert_allclose(e1[big], e0[big], rtol=1e-4)
    np.testing.assert_allclose(h1[big], h0[big], rtol=3e-5)
