"""The mixed path's projection at the horizon, where the quadratic's leading coefficient A = (r^2 - 2 M r + a^2 + Q^2) / Sigma
vanishes and in FP32 is exactly zero for some rays: a frame of the shadow's interior, every ray of which ends there.

Bound: the null value before a projection is at most 1e-6 at these tolerances and the FP32 coefficients leave ~1e-7 of it,
up to a hundredfold where B is small: 1e-11; a ray left unprojected keeps 1e-9 and more."""
import numpy as np
import pytest

from sirius_b200 import abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("a", [0.0, 0.5, 0.9])
def test_rays_into_the_horizon_stay_null(engine, a):
    engine.configure(abi.default_config(abs_tolerance=1e-8, rel_tolerance=1e-8, min_step=1e-9, horizon_factor=1.0002,
                                        escape_radius=200.0, precision=abi.PRECISION_MIXED, island_factor=0.0,
                                        critical_band=0.0, enable_disk=0))
    fr = abi.make_frame(abi.make_metric(a=a), abi.make_camera(r=60.0, theta_deg=70.0, width=400, height=400, fov=5.0),
                        0.0, 20.0)
    res, _, _ = engine.trace_frames([fr])
    hor = res["outcome"] == abi.HORIZON
    assert hor.mean() > 0.5
    assert res["null_final"][hor].max() <= 1e-11, res["null_final"][hor].max()


def test_bench_frame_rows_across_the_shadow(engine):
    """Rows of the benchmark's frame across the shadow: one of its horizon rays has A = 0 exactly at its last step."""
    engine.configure(abi.default_config(abs_tolerance=1e-8, rel_tolerance=1e-8, min_step=1e-9, max_step=2.0,
                                        escape_radius=200.0, horizon_factor=1.01, max_steps=10000,
                                        precision=abi.PRECISION_MIXED, enable_volumetric=1, n_bins=16))
    inclination = float(np.random.default_rng(0).uniform(10.0, 89.0))
    cam = abi.make_camera(r=100.0, theta_deg=inclination, fov=30.0, width=1024, height=1024)
    fr = abi.make_frame(abi.make_metric(a=0.9), cam, 0.0, 30.0, row_begin=480, row_count=80)
    res, _, _ = engine.trace_frames([fr])
    assert (res["outcome"] == abi.HORIZON).sum() > 1000
    assert res["null_final"].max() <= 1e-11, res["null_final"].max()
