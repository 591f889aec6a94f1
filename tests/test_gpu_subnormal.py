"""complex128 fields in the subnormal range through the fixed-point line passes (GPU).

A field of 2^-1030 keeps about 44 bits; its transfer is that of the field itself, scaled.  An entry takes some
hundred roundings at 2^-1075 on either path (four transforms, operators and tables of two layers): 2^-1075
100 / (0.3 2^-1030) = 1e-11 of it.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("schedule", [1, 2])
@pytest.mark.parametrize("shape", [(64, 50), (150, 96)])
def test_subnormal_fields(shape, schedule):
    from test_gpu_line import _run

    want = _run(shape, "4x4", 3, schedule)
    got = _run(shape, "4x4", 3, schedule, scale=2.0 ** -1030) * 2.0 ** 1000 * 2.0 ** 30
    assert np.linalg.norm(got - want) <= 1e-11 * np.linalg.norm(want)
