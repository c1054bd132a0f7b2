"""Builds tests/cpp/test_ks_forms.cpp (what the closed Kerr-Schild form takes from the equation of r, as host code in extended
precision) and runs it."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_closed_form_where_r_is_held(tmp_path):
    out = str(tmp_path / "ks_forms")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "sirius_b200", "csrc"), "-I",
                    os.path.join(ROOT, "include"), "-I", "/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "cpp", "test_ks_forms.cpp"), "-o", out], check=True)
    r = subprocess.run([out], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
