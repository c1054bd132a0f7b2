"""The symplectic integrator with one geometry per substep, at every composition order, with charge and Lambda, against
the oracle, which evaluates the full metric at each kick and drift.

Tolerance: a fixed number of fixed steps through a smooth flow in FP64. Rounding grows along a ray by the flow's own
stretching, at most e^4 over the 2 M of affine length taken here, so terminal states agree to 1e-11 of their size; with
FP32 right-hand sides (mixed precision) each step adds up to 1e-7 of its length 0.02 M, 100 steps and the same stretching
give 1e-5 at most, and the oracle is met at 2e-6 in the mean."""
import numpy as np
import pytest

from sirius_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [4, 6, 8])
@pytest.mark.parametrize("Q,Lam", [(0.0, 0.0), (0.4, 0.0), (0.0, 1e-4)])
def test_orders_match_oracle(engine, oracle, order, Q, Lam):
    cam = abi.make_camera(r=6.0, theta_deg=70.0, width=16, height=8, projection=abi.CAMERA_EQUIRECTANGULAR)
    fr = abi.make_frame(abi.make_metric(a=0.8, Q=Q, Lambda=Lam), cam, 0.0, 20.0)

    def cfg(prec):
        return abi.default_config(integrator=abi.INTEGRATOR_SYMPLECTIC, symplectic_order=order, symplectic_step=0.02,
                                  projection_period=3, max_steps=100, escape_radius=60.0, horizon_factor=1.01,
                                  min_step=1e-9, enable_disk=0, precision=prec)

    ref, _ = oracle.trace_frame(fr, cfg(abi.PRECISION_FP64))
    scale = np.abs(ref["final_x"]).max(1, keepdims=True)
    for prec, most, mean in ((abi.PRECISION_FP64, 1e-11, 1e-12), (abi.PRECISION_MIXED, 1e-5, 2e-6)):
        engine.configure(cfg(prec))
        res, _, _ = engine.trace_frames([fr])
        np.testing.assert_array_equal(res["outcome"], ref["outcome"])
        np.testing.assert_array_equal(res["steps"], ref["steps"])
        for f in ("final_x", "final_p"):
            err = np.abs(res[f] - ref[f]) / scale
            assert err.max() <= most and err.mean() <= mean, (f, prec, err.max(), err.mean())
