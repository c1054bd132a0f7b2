"""Beams on lane pairs with dual-number tangents: every beam of a ragged launch (odd counts, two frames, a last block that
is partly empty, charge and Lambda) equals the one traced in a frame of its own, and its tangents match finite differences
of the escape directions of neighbouring pixels of a finer frame.

Tolerance of the second: central differences of the float32 escape directions over one pixel of a 64-fold finer frame:
direction rounding 6e-8 over a pixel step of at least 2e-5 rad leaves 3e-3, and the curvature term is below that away from
the shadow; the median over the escaped beams must be within 5e-3."""
import numpy as np
import pytest

from sirius_b200 import abi

pytestmark = pytest.mark.gpu


def config():
    return abi.default_config(abs_tolerance=1e-9, rel_tolerance=1e-9, min_step=1e-12, max_step=4.0, initial_step=0.1,
                              escape_radius=300.0, horizon_factor=1.01, max_steps=20000, enable_disk=0)


def frame(w, h, metric, **kw):
    return abi.make_frame(metric, abi.make_camera(r=40.0, theta_deg=75.0, fov=40.0, width=w, height=h), 0.0, 20.0, **kw)


@pytest.mark.parametrize("w,h", [(1, 1), (33, 1), (7, 5), (31, 3)])
def test_ragged_launch_equals_separate_frames(engine, w, h):
    engine.configure(config())
    mets = [abi.make_metric(a=0.7, Q=0.4), abi.make_metric(a=0.9, Lambda=1e-5)]
    both = engine.trace_beams([frame(w, h, m) for m in mets])
    apart = np.concatenate([engine.trace_beams([frame(w, h, m)]) for m in mets])
    assert both.tobytes() == apart.tobytes()
    rows = np.concatenate([engine.trace_beams([frame(w, h, mets[0], row_begin=y, row_count=1)]) for y in range(h)])
    assert rows.tobytes() == both[:w * h].tobytes()


def test_tangents_against_neighbouring_pixels(engine):
    engine.configure(config())
    m, n, fine = abi.make_metric(a=0.9), 12, 64
    coarse = engine.trace_beams([frame(n, n, m)]).reshape(n, n)
    rel = []
    for y in range(0, n, 3):
        # rows y fine + fine / 2 - 1, + 1 of the finer frame straddle the coarse pixel's centre
        r0 = y * fine + fine // 2 - 1
        b = engine.trace_beams([frame(n * fine, n * fine, m, row_begin=r0, row_count=2)]).reshape(2, n * fine)
        for x in range(n):
            c = coarse[y, x]
            q = b[:, x * fine + fine // 2 - 1:x * fine + fine // 2 + 1]
            if c["outcome"] != abi.ESCAPED or (q["outcome"] != abi.ESCAPED).any():
                continue
            d = q["final_dir"].astype(np.float64)
            du, dv = (d[:, 1] - d[:, 0]).mean(0), (d[1] - d[0]).mean(0)
            omega = np.linalg.norm(np.cross(du, dv)) * fine * fine
            u, v = (np.array([x, y]) + 0.5) * 2 / n - 1
            t = np.tan(np.radians(20.0))
            pixel = (2 * t / n) ** 2 / (1 + (u * t) ** 2 + (v * t) ** 2) ** 1.5
            rel.append(abs(pixel / omega / c["magnification"] - 1))
    assert len(rel) > 20 and np.median(rel) < 5e-3, np.median(rel)
