"""Sines and cosines of the director angles by integer turns, on the host.

``angle_host.cu`` compares the pairs formed from ``fx_angle`` (``dtmm_fx.cuh``)
with long double for angles up to 2^21 rad: 2^-48 for the pair (two 24-bit
words), 2^-64 of the angle for the rounded 1 / (2 pi).  A product of doubles
would leave 2^-53 of the angle, 2^-33 at the largest.
"""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_integer_angles_on_host(tmp_path):
    from dtmm_gb300 import _build

    try:
        nvcc = _build.nvcc_path()
    except RuntimeError:
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "angle_host")
    r = subprocess.run([nvcc, "-std=c++17", "-O2", "-Xcompiler", "-ffp-contract=off", "-I",
                        os.path.join(ROOT, "dtmm_gb300", "csrc"), "-o", exe, os.path.join(HERE, "angle_host.cu")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.splitlines()[-1] == "OK", out.stdout
