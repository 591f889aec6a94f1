"""Fixed-point line transforms of the CUDA library, checked on the host.

``fx_host.cu`` runs the conversions, the register DFTs of every length and the
two-step transform of every side up to 400 (and a sample up to 1024) as the
kernels do, against a direct DFT in long double, and the same transforms in
FP64 arithmetic: relative L2 at most 5e-16 for each, and on average over each
kind of input (flat, one dominant entry, band-limited, spread over 300 orders
of magnitude, huge, tiny) no larger than FP64's.
"""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_fixed_point_transforms_on_host(tmp_path):
    from dtmm_gb300 import _build

    try:
        nvcc = _build.nvcc_path()
    except RuntimeError:
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "fx_host")
    r = subprocess.run([nvcc, "-std=c++17", "-O2", "-I", os.path.join(ROOT, "dtmm_gb300", "csrc"), "-o", exe,
                        os.path.join(HERE, "fx_host.cu")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    out = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    lines = out.stdout.splitlines()
    assert out.returncode == 0 and lines[-1] == "OK", "\n".join(li for li in lines if li.startswith("FAIL"))
    sides = {int(li.split()[2]) for li in lines if li.startswith("err")}
    assert {2, 7, 24, 30, 64, 125, 150, 210, 250, 256, 330, 512, 1024} <= sides
