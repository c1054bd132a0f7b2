"""The device's reciprocals and roots (csrc/dual.cuh, csrc/roots.cuh) against extended precision over the arguments that
their callers form: both signs for a reciprocal, the clamps' edges (1e-280, 1e-20, 1e-10), neighbours of powers of two.

Bounds, in units of u = 2^-53: a reciprocal's step leaves the rounding of its last operation, u, and the seed's residual
cubed (2^-57 for a seed good to 2^-19); a reciprocal root has the rounding of x y besides, halved: 1.5 u. The fifth root ends
in five rounded products and a sum, 6 u. In FP32 the unit's own documented errors: 1 ulp and 2^-22.9."""
import ctypes as C
import os
import shutil
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
U = 2.0 ** -53


@pytest.fixture(scope="module")
def device(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc to build the arrays' kernel with")
    lib = str(tmp_path_factory.mktemp("roots") / "device_roots.so")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-shared", "-Xcompiler",
                    "-fPIC", "-I", os.path.join(ROOT, "sirius_b200", "csrc"), "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "cpp", "device_roots.cu"), "-o", lib], check=True)
    L = C.CDLL(lib)
    L.device_warp_centre.argtypes = [C.c_double, C.c_void_p]
    L.device_apply.argtypes = [C.c_int, C.c_longlong, C.c_void_p, C.c_void_p]

    def apply(f, x):
        x = np.ascontiguousarray(x, dtype=np.float64)
        y = np.empty_like(x)
        assert L.device_apply(f, x.size, x.ctypes.data, y.ctypes.data) == 0
        return y
    apply.lib = L
    return apply


def arguments(lo, hi, n=1 << 20):
    rng = np.random.default_rng(11)
    x = np.exp(rng.uniform(np.log(lo), np.log(hi), n))
    k = np.arange(int(np.ceil(np.log2(lo))), int(np.floor(np.log2(hi))))
    p = np.ldexp(1.0, k)
    edges = np.array([1e-280, 1e-20, 1e-10, 1e-6, 1.0, 3.0, 1e20, 1e280])
    x = np.concatenate([x, p, np.nextafter(p, 0), np.nextafter(p, np.inf), edges])
    return x[(x >= lo) & (x <= hi)]


def worst(y, exact):
    return float(np.max(np.abs(y.astype(np.longdouble) / exact - 1)))


def test_reciprocal(device):
    x = arguments(1e-300, 1e300)
    for sign in (1, -1):
        assert worst(device(0, sign * x), sign / x.astype(np.longdouble)) <= U + 2.0 ** -57


def test_reciprocal_root(device):
    x = arguments(1e-300, 1.7e308)
    assert worst(device(1, x), 1 / np.sqrt(x.astype(np.longdouble))) <= 1.5 * U + 2.0 ** -57


def test_single_precision(device):
    x = arguments(1e-30, 1e30).astype(np.float32).astype(np.float64)
    for sign in (1, -1):
        assert worst(device(2, sign * x), sign / x.astype(np.longdouble)) <= 2.0 ** -23
    assert worst(device(3, x), 1 / np.sqrt(x.astype(np.longdouble))) <= 2.0 ** -22.9 + 2.0 ** -24


def test_fifth_root(device):
    x = arguments(1e-15, 1e38)
    assert worst(device(4, x), x.astype(np.longdouble) ** (np.longdouble(-1) / 5)) <= 6 * U
    huge = device(4, [1e39, 1e150, 1.7976931348623157e308, np.inf])
    assert (huge >= 0).all() and (huge <= 1e-7).all()
    assert np.isnan(device(4, [np.nan])).all()


def test_root_of_a_sum(device):
    x = arguments(1e-279, 1.7e308)
    assert worst(device(5, x), np.sqrt(x.astype(np.longdouble))) <= 2.5 * U + 2.0 ** -57
    np.testing.assert_array_equal(device(5, [0.0, np.inf]), [0.0, np.inf])
    assert np.isnan(device(5, [np.nan])).all()


@pytest.mark.parametrize("x", [0.0, 1e-160, 1e-100, -0.3, 1.0, 50.0])
def test_warp_drive_at_its_centre(device, x):
    """The radius and its direction at the bubble's centre and beside it: zero and none at the centre, where a projection
    leaves the momentum as it is."""
    y = np.full(10, np.nan)
    assert device.lib.device_warp_centre(x, y.ctypes.data) == 0
    assert np.isfinite(y).all()
    np.testing.assert_allclose(y[0], abs(x) if abs(x) > 1e-150 else 0.0, rtol=4 * U, atol=1e-150)
    if x == 0.0:
        np.testing.assert_array_equal(y[1:5], 0)
        np.testing.assert_array_equal(y[6:], [-1.0, 0.7, 0.3, -0.2])
    elif abs(x) > 1e-150:
        np.testing.assert_allclose(y[2], np.sign(x), rtol=4 * U)
        np.testing.assert_array_equal(y[[1, 3, 4]], 0)
