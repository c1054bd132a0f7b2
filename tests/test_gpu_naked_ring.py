"""The short form of the Kerr-Schild projection inside the ring of a naked singularity, next to its disc, where r is held at
1e-5 and no longer solves its equation: it has to be the general projection there too.

Tolerances (u = 2^-53): the null value 64 u of its terms; a projected momentum that over the root q, and the rounding of q,
whose discriminant keeps at least 1e-6 of its terms in the rows looked at (1e-8 of the correction)."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

from sirius_b200 import abi

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
U = 2.0 ** -53
METRICS = [dict(M=0.3, a=-0.9, Q=1.2), dict(M=1.0, a=1.2, Q=0.0), dict(M=1.0, a=0.0, Q=1.3), dict(M=0.5, a=0.8, Q=0.6)]


@pytest.fixture(scope="module")
def device(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc to build the forms' kernel with")
    lib = str(tmp_path_factory.mktemp("forms") / "device_roots.so")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "-I", os.path.join(ROOT, "sirius_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "cpp", "device_roots.cu"), "-o", lib], check=True)
    L = C.CDLL(lib)
    L.device_ks_projections.argtypes = [C.c_void_p, C.c_longlong, C.c_void_p, C.c_void_p]
    return L


def states(m, n=20000):
    rng = np.random.default_rng(9)
    a = abs(m["a"])
    z = np.exp(rng.uniform(np.log(1e-9), np.log(1e-1), n)) * rng.choice([-1, 1], n)
    rho = a * np.sqrt(rng.uniform(0.01, 0.99, n)) if a else np.exp(rng.uniform(np.log(1e-8), np.log(1e-1), n))
    ph = rng.uniform(0, 2 * np.pi, n)
    x = np.stack([np.zeros(n), rho * np.cos(ph), rho * np.sin(ph), z], 1)
    p = rng.normal(size=(n, 4))
    p[:, 0] = -1.0
    return np.ascontiguousarray(np.concatenate([x, p], 1))


@pytest.mark.parametrize("m", METRICS)
def test_projections_agree_next_to_the_disc(device, m):
    s = states(m)
    n = len(s)
    out = np.empty((2, n, 8))
    met = abi.make_metric(**m)
    assert device.device_ks_projections(C.addressof(met), n, s.ctypes.data, out.ctypes.data) == 0
    fast, general = out
    X, Y, Z = s[:, 1], s[:, 2], s[:, 3]
    a2 = m["a"] ** 2
    Rm2 = X * X + Y * Y + Z * Z - a2
    sd = np.sqrt(Rm2 ** 2 + 4 * a2 * Z * Z)
    r2 = np.maximum(0.5 * (Rm2 + sd), 1e-10)
    held = r2 <= 1e-10
    assert held.mean() > 0.1
    # where the quadratic is well conditioned
    np.testing.assert_allclose(fast[held, 5], general[held, 5], rtol=1e-15)
    r = np.sqrt(r2)
    l = np.stack([(r * X + m["a"] * Y) / (r2 + a2), (r * Y - m["a"] * X) / (r2 + a2), Z / r], 1)
    H = (2 * m["M"] * r - m["Q"] ** 2) * r2 / (r2 * r2 + a2 * Z * Z)
    d = np.stack([r * X / sd, r * Y / sd, Z * (r2 + a2) / (r * sd)], 1)
    if not m["a"]:
        d = s[:, 1:4] / np.linalg.norm(s[:, 1:4], axis=1, keepdims=True)
    q3 = s[:, 5:8]
    lp, ld = 1.0 + (l * q3).sum(1), (l * d).sum(1)
    size = 1 + (q3 ** 2).sum(1) + np.abs(H) * (1 + np.abs(l * q3).sum(1)) ** 2
    A = (d * d).sum(1) - H * ld ** 2
    B = 2 * ((q3 * d).sum(1) - H * lp * ld)
    null = -1 + (q3 ** 2).sum(1) - H * lp ** 2
    disc = B * B - 4 * A * null
    well = held & (np.abs(disc) > 1e-6 * (B * B + 4 * np.abs(A * null))) & (np.abs(A) > 1e-12)
    assert well.sum() > 100
    assert (np.abs(fast[:, 4] - general[:, 4]) <= 64 * U * size)[held].all()
    root = 0.5 * (np.abs(B) + np.sqrt(np.maximum(disc, 0)))
    dn = np.linalg.norm(d, axis=1)
    move = np.abs(general[:, 1:4] - q3).max(1)
    bound = 1e-8 * move + 64 * U * (size * dn / root + 1 + np.abs(q3).max(1))
    assert (np.abs(fast[:, 1:4] - general[:, 1:4]).max(1) <= bound)[well].all()


def frames():
    """Black holes, naked singularities, a hole whose horizon does not stop the rays, a wormhole; odd sizes."""
    mets = [dict(a=0.9), dict(M=0.3, a=-0.9, Q=1.2), dict(family=abi.MORRIS_THORNE), dict(a=1.3), dict(a=0.4, Lambda=1e-5),
            dict(M=-0.5, a=0.3)]
    return [abi.make_frame(abi.make_metric(**m), abi.make_camera(r=8.0, theta_deg=50.0, width=17 + 2 * i, height=9 + i,
                                                                 fov=30.0), 0.0, 15.0) for i, m in enumerate(mets)]


@pytest.mark.parametrize("precision", [abi.PRECISION_FP64, abi.PRECISION_MIXED])
@pytest.mark.parametrize("horizon", [1.01, 1e-4])
def test_a_batch_equals_its_frames_apart(engine, precision, horizon):
    """Frames that the ring's forms serve and others, in one batch (bit for bit): each class has its own launch."""
    engine.configure(abi.default_config(precision=precision, horizon_factor=horizon, max_steps=600, escape_radius=40.0))
    fs = frames()
    both, img, _ = engine.trace_frames(fs)
    apart = [engine.trace_frames([f]) for f in frames()]
    assert both.tobytes() == np.concatenate([a[0] for a in apart]).tobytes()
    np.testing.assert_array_equal(img, np.concatenate([a[1] for a in apart]))
    assert (both["steps"] > 0).all()
    ks = [f for f in frames() if f.metric.family == abi.KERR_SCHILD]
    beams = engine.trace_beams(ks)
    each = np.concatenate([engine.trace_beams([f]) for f in [g for g in frames() if g.metric.family == abi.KERR_SCHILD]])
    engine.configure(abi.default_config())
    assert beams.tobytes() == each.tobytes() and (beams["steps"] > 0).all()
