"""Builds tests/cpp/test_roots.cpp (the scalar roots of the step control and the event location, as host code) with and
without fused multiply-adds and runs it: how many iterations a search takes, and how far its root is from the zero."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("flags", [["-ffp-contract=off"], ["-mfma", "-ffp-contract=fast"]])
def test_scalar_roots(tmp_path, flags):
    out = str(tmp_path / "roots")
    subprocess.run(["g++", "-std=c++17", "-O2", *flags, "-I", os.path.join(ROOT, "sirius_b200", "csrc"), "-I",
                    "/usr/local/cuda/include", os.path.join(ROOT, "tests", "cpp", "test_roots.cpp"), "-o", out], check=True)
    r = subprocess.run([out], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
