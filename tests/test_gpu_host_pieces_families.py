"""A large frame of each metric family into page-locked buffers through the host entry point equals the same frame into
pageable ones, bit for bit, whether or not it is traced in pieces."""
import ctypes as C

import numpy as np
import pytest

from sirius_b200 import abi

pytestmark = pytest.mark.gpu
METRICS = {"wormhole": dict(family=abi.MORRIS_THORNE), "warp drive": dict(family=abi.ALCUBIERRE), "Kerr": dict(a=0.9),
           "Kerr-de Sitter": dict(a=0.5, Lambda=1e-5), "naked singularity": dict(a=0.6, Q=1.1)}


@pytest.mark.parametrize("name", METRICS)
@pytest.mark.parametrize("precision", [abi.PRECISION_MIXED, abi.PRECISION_FP64])
def test_page_locked_equals_pageable(engine, name, precision):
    import torch
    width, height = 520, 540  # over 2048 tiles of 16 x 8 pixels, edge tiles cut by the frame
    engine.configure(abi.default_config(precision=precision, abs_tolerance=1e-5, rel_tolerance=1e-5, max_steps=400,
                                        escape_radius=60.0))
    fr = abi.make_frame(abi.make_metric(**METRICS[name]), abi.make_camera(r=20.0, theta_deg=70.0, width=width, height=height,
                                                                          fov=40.0), 0.0, 20.0)
    total = width * height
    res, img, _ = engine.trace_frames([fr])
    stats = engine.stats()
    h_res = torch.zeros(total * abi.result_dtype().itemsize, dtype=torch.uint8, pin_memory=True)
    h_img = torch.full((total,), float("nan"), dtype=torch.float32, pin_memory=True)
    # the device buffers hold another frame's rays before
    engine.trace_frames([abi.make_frame(abi.make_metric(a=0.1), fr.camera, 0.0, 20.0)])
    arr = (abi.Frame * 1)(fr)
    engine.trace_frames_into(C.addressof(arr), 1, h_res.data_ptr(), h_img.data_ptr(), None)
    again = engine.stats()
    engine.configure(abi.default_config())
    assert (res["steps"] > 0).all() and len(np.unique(res["steps"])) > 3
    assert h_res.numpy().tobytes() == res.tobytes()
    np.testing.assert_array_equal(h_img.numpy(), img)
    assert (again.accepted_steps, again.rejected_steps) == (stats.accepted_steps, stats.rejected_steps)
