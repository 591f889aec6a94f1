"""Pair-arithmetic eigenvalues of the mixed-precision operator records, on the host.

``lean_host.cu`` runs ``dtmm_lean.cuh`` on 400,000 random uniaxial voxels and
beams and compares alpha - a with long double: each factor of the quotient is
a pair of about 46 bits (2^-46 = 1.4e-14, some ten of them), so 2e-13 absolute,
and the FP32 record is the rounding of the exact value.
"""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_pair_arithmetic_eigenvalues_on_host(tmp_path):
    from dtmm_gb300 import _build

    try:
        nvcc = _build.nvcc_path()
    except RuntimeError:
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "lean_host")
    r = subprocess.run([nvcc, "-std=c++17", "-O2", "-Xcompiler", "-ffp-contract=off", "-I",
                        os.path.join(ROOT, "dtmm_gb300", "csrc"), "-o", exe, os.path.join(HERE, "lean_host.cu")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.splitlines()[-1] == "OK", out.stdout
