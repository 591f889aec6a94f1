"""Modulus and angle of the phases formed by integer turns, on the host
(``turn_host.cu``): 2^-58 and 2^-56, so that neither accumulates over the layers
of a transfer beside the 2^-53 that FP64 phases are rounded at."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_turns_on_host(tmp_path):
    from dtmm_gb300 import _build

    try:
        nvcc = _build.nvcc_path()
    except RuntimeError:
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "turn_host")
    r = subprocess.run([nvcc, "-std=c++17", "-O2", "-Xcompiler", "-ffp-contract=off", "-I",
                        os.path.join(ROOT, "dtmm_gb300", "csrc"), "-o", exe, os.path.join(HERE, "turn_host.cu")],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout.splitlines()[-1] == "OK", out.stdout
