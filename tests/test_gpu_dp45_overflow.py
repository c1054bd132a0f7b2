"""A Dormand-Prince attempt whose scaled error is beyond FP64's range: the estimate is infinite, the attempt is refused and
the step shrinks by the configured least factor, as with the oracle."""
import numpy as np
import pytest

from sirius_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tol", [1e-170, 1e-250, 1e-305])
def test_an_infinite_estimate_shrinks_the_step(engine, oracle, tol):
    m = abi.make_metric(a=0.6, Q=0.1)
    cfg = abi.default_config(abs_tolerance=tol, rel_tolerance=0.0, min_step=1e-9, max_step=50.0)
    rng = np.random.default_rng(3)
    n = 64
    x = np.concatenate([np.zeros((n, 1)), rng.normal(size=(n, 3)) * 6 + 4], 1)
    p = np.concatenate([-np.ones((n, 1)), rng.normal(size=(n, 3))], 1)
    states, hs = np.concatenate([x, p], 1), rng.uniform(0.5, 2.0, n)
    s0, h0, a0, e0 = oracle.dp45_step(m, cfg, states, hs)
    assert np.isinf(e0).all() and not a0.any()
    engine.configure(cfg)
    s1, h1, a1, e1 = engine.dp45_step(m, states, hs)
    engine.configure(abi.default_config())
    np.testing.assert_array_equal(e1, e0)
    np.testing.assert_array_equal(a1, a0)
    np.testing.assert_array_equal(s1, s0)
    np.testing.assert_allclose(h1, h0, rtol=1e-15)
    np.testing.assert_allclose(h1, hs * cfg.step_shrink_min, rtol=1e-15)
