"""A frame's rays do not depend on what shares their launch: a batch equals its frames traced apart bit for bit, in each
precision, integrator and register budget, with charge, Lambda of both signs and volumetric spectra. One-frame launches read
the metric from the launch's parameters and batches from memory, by kernels of the same source: their sums and products have
to be fused alike."""
import numpy as np
import pytest

from sirius_b200 import abi

pytestmark = pytest.mark.gpu


def frames():
    mets = [dict(a=0.9), dict(a=0.4, Lambda=1e-5), dict(a=-0.9, Lambda=-1e-4), dict(a=0.6, Q=0.5), dict(M=4.0, a=-0.1),
            dict(a=0.0, Lambda=3e-4)]
    return [abi.make_frame(abi.make_metric(**m), abi.make_camera(r=25.0, theta_deg=55.0 + 7 * i, width=33 + 4 * i, height=24,
                                                                 fov=30.0 if i % 2 else 100.0, projection=int(i == 4)),
                           0.0, 20.0) for i, m in enumerate(mets)]


@pytest.mark.parametrize("bins", [0, 7])
@pytest.mark.parametrize("registers", [0, 128, 168, 255])
@pytest.mark.parametrize("integrator", [abi.INTEGRATOR_DP45, abi.INTEGRATOR_SYMPLECTIC])
@pytest.mark.parametrize("precision", [abi.PRECISION_FP64, abi.PRECISION_MIXED])
def test_a_batch_equals_its_frames_apart(engine, precision, integrator, registers, bins):
    engine.configure(abi.default_config(precision=precision, integrator=integrator, max_registers=registers,
                                        symplectic_step=0.1, max_steps=1000, escape_radius=60.0, abs_tolerance=1e-8,
                                        rel_tolerance=1e-8, min_step=1e-9, horizon_factor=1.01, enable_volumetric=int(bins > 0),
                                        n_bins=bins))
    both, img, spc = engine.trace_frames(frames(), spectra=bins > 0)
    apart = [engine.trace_frames([f], spectra=bins > 0) for f in frames()]
    engine.configure(abi.default_config())
    each = np.concatenate([a[0] for a in apart])
    differ = [i for i in range(len(each)) if each[i].tobytes() != both[i].tobytes()]
    assert not differ, (len(differ), [n for n in each.dtype.names if each[differ[0]][n].tobytes() != both[differ[0]][n].tobytes()])
    np.testing.assert_array_equal(img, np.concatenate([a[1] for a in apart]))
    if bins:
        np.testing.assert_array_equal(spc, np.concatenate([a[2] for a in apart]))
