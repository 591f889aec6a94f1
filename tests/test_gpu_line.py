"""Fixed-point line passes (complex128 bulk) against the FP64 shared-memory
passes of the same library (``fft_schedule`` 2): every side with kernels of its
own, run-time sides of both length classes, the smallest and the largest, the
4x4 method with windows and the 2x2 one.

Tolerance: two layers are about 20 transforms and products of relative error
below 5e-16, and phases of at most 10 rad rounded at 2^-53: 2e-14 together.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(64, 64), (80, 96), (100, 120), (128, 150), (160, 144), (180, 192), (225, 240), (256, 256), (7, 2), (5, 16),
          (45, 50), (200, 330), (250, 125), (512, 300), (24, 1024)]


def _run(shape, method, diffraction, schedule, spoil=None, scale=1.0):
    import torch

    from dtmm_gb300 import samples
    from dtmm_gb300.illumination import illumination_device
    from dtmm_gb300.transfer import plan_transfer

    wl = [450.0, 620.0]
    mat = samples.twisted_nematic_device(shape, 2, no=1.52, ne=1.71, amplitude=0.3, seed=5)
    fin = illumination_device(shape, wl, 100.0, beta=0.1, phi=0.4, precision="double") * scale
    if spoil is not None:
        fin[0, 1, 0, shape[0] // 2, shape[1] // 2] = spoil
    plan = plan_transfer(tuple(fin.shape), wl, 100.0, mat, beta=0.1, phi=0.4, method=method, diffraction=diffraction,
                         npass=1, precision="double", tuning=dict(fft_schedule=schedule))
    out = torch.empty_like(fin)
    plan.run(fin, out)
    return out.cpu().numpy()


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("method,diffraction", [("4x4", 3), ("2x2", 1)])
def test_line_passes_match_fp64_passes(shape, method, diffraction):
    a = _run(shape, method, diffraction, 0)
    b = _run(shape, method, diffraction, 2)
    assert np.linalg.norm(a - b) <= 2e-14 * np.linalg.norm(b)


@pytest.mark.parametrize("scale", [1e-120, 1e120])
def test_line_passes_scale(scale):
    # the line's own power of two: the result is the scaled result to rounding
    a = _run((64, 50), "4x4", 3, 0)
    b = _run((64, 50), "4x4", 3, 0, scale=scale) / scale
    assert np.linalg.norm(a - b) <= 2e-14 * np.linalg.norm(a)


@pytest.mark.parametrize("spoil", [np.nan, np.inf])
def test_line_passes_not_finite(spoil):
    # one bad value: its image is lost, as in FP64 arithmetic, and no other one is touched
    a = _run((64, 50), "4x4", 3, 0, spoil=spoil)
    b = _run((64, 50), "4x4", 3, 2, spoil=spoil)
    assert not np.isfinite(a[0, 1]).any() and not np.isfinite(b[0, 1]).any()
    for i in ((0, 0), (1, 0), (1, 1)):
        assert np.linalg.norm(a[i] - b[i]) <= 2e-14 * np.linalg.norm(b[i])


REG_SIDES = (64, 80, 96, 112, 128, 144, 160, 192, 224, 240, 256, 288, 320, 336, 384, 400, 432, 448, 480, 512, 1024)


def _mixed(shape, method, diffraction, schedule, pixelsize):
    import torch

    from dtmm_gb300 import samples
    from dtmm_gb300.illumination import illumination_device
    from dtmm_gb300.transfer import plan_transfer

    wl = [450.0, 620.0]
    mat = samples.twisted_nematic_device(shape, 2, no=1.52, ne=1.71, amplitude=0.3, seed=6)
    fin = illumination_device(shape, wl, pixelsize, beta=0.1, phi=0.4, precision="mixed")
    plan = plan_transfer(tuple(fin.shape), wl, pixelsize, mat, beta=0.1, phi=0.4, method=method,
                         diffraction=diffraction, npass=1, precision="mixed", tuning=dict(fft_schedule=schedule))
    out = torch.full_like(fin, float("nan"))
    plan.workspace.fill_(255)  # unwritten columns hold NaN
    plan.run(fin, out)
    return out.cpu().numpy()


@pytest.mark.parametrize("height", REG_SIDES)
@pytest.mark.parametrize("method,diffraction,pixelsize", [("4x4", 3, 50.0), ("2x2", 1, 100.0), ("4x4", 1, 220.0)])
def test_register_columns_match_shared_memory_passes(height, method, diffraction, pixelsize):
    """complex64 column pass of every register side, narrow band, wider band and (220 nm pixels) no band
    limit; the workspace starts as NaN, so nothing beyond the band may be read.  Eight transforms of
    relative error below 3e-7 on either side, at random: 3e-6."""
    shape = (height, 80 if height != 80 else 64)
    a = _mixed(shape, method, diffraction, 0, pixelsize)
    b = _mixed(shape, method, diffraction, 2, pixelsize)
    assert np.linalg.norm(a - b) <= 3e-6 * np.linalg.norm(b)


@pytest.mark.parametrize("shape", [(7, 2), (24, 30), (45, 50), (100, 210), (250, 330), (200, 125), (500, 300), (150, 64),
                                   (64, 150), (12, 900)])
@pytest.mark.parametrize("method,diffraction,pixelsize", [("4x4", 3, 50.0), ("2x2", 1, 100.0), ("4x4", 1, 220.0)])
def test_run_time_lengths_match_shared_memory_passes(shape, method, diffraction, pixelsize):
    """complex64 passes of run-time lengths, alone and beside register passes (one side each), with the
    same bound as the register columns."""
    a = _mixed(shape, method, diffraction, 0, pixelsize)
    b = _mixed(shape, method, diffraction, 2, pixelsize)
    assert np.linalg.norm(a - b) <= 3e-6 * np.linalg.norm(b)


@pytest.mark.parametrize("shape", [(45, 50), (96, 100), (150, 64), (64, 64), (250, 330)])
@pytest.mark.parametrize("precision,tol", [("double", 2e-14), ("mixed", 3e-6)])
def test_refocus_matches_fft(shape, precision, tol):
    """diffract with a random matrix per k against torch.fft in complex128 (two transforms and a 4x4
    product: the bounds above)."""
    import torch

    from dtmm_gb300 import pom

    g = torch.Generator(device="cuda").manual_seed(3)
    f = torch.randn((2, 3, 4) + shape + (2,), generator=g, device="cuda", dtype=torch.float64)
    f = torch.view_as_complex(f)
    m = torch.view_as_complex(torch.randn((3,) + shape + (4, 4, 2), generator=g, device="cuda", dtype=torch.float64))
    ref = torch.fft.ifft2(torch.einsum("lhwij,pljhw->plihw", m, torch.fft.fft2(f)))
    out = pom.diffract(f if precision == "double" else f.to(torch.complex64), m)
    assert float((out - ref).norm() / ref.norm()) <= tol


@pytest.mark.parametrize("shape", [(64, 50), (150, 96)])
def test_line_passes_read_no_column_beyond_the_band(shape):
    import torch

    from dtmm_gb300 import samples
    from dtmm_gb300.illumination import illumination_device
    from dtmm_gb300.transfer import plan_transfer

    wl = [450.0, 620.0]
    mat = samples.twisted_nematic_device(shape, 2, no=1.52, ne=1.71, amplitude=0.3, seed=6)
    fin = illumination_device(shape, wl, 50.0, precision="double")
    plan = plan_transfer(tuple(fin.shape), wl, 50.0, mat, method="4x4", diffraction=3, npass=1, precision="double")
    out = torch.empty_like(fin)
    plan.run(fin, out)
    again = torch.empty_like(fin)
    plan.workspace.fill_(255)
    plan.run(fin, again)
    assert torch.equal(out, again)


@pytest.mark.parametrize("shape", [(48, 50), (60, 72), (75, 90), (112, 135), (140, 168), (196, 210), (224, 200),
                                   (270, 288), (300, 320), (400, 384), (48, 512), (512, 48), (45, 63), (110, 125),
                                   (175, 220), (250, 280), (330, 336), (350, 352), (360, 432), (448, 480), (32, 640),
                                   (640, 32), (1024, 32)])
@pytest.mark.parametrize("method,diffraction", [("4x4", 3), ("2x2", 1)])
def test_line_passes_of_compile_time_sides(shape, method, diffraction):
    # the further sides with kernels of their own, rows and columns, the tolerance above
    a = _run(shape, method, diffraction, 0)
    b = _run(shape, method, diffraction, 2)
    assert np.linalg.norm(a - b) <= 2e-14 * np.linalg.norm(b)


@pytest.mark.parametrize("shape", [(45, 48), (60, 50), (63, 72), (90, 75), (100, 110), (125, 120), (135, 140), (168, 150),
                                   (175, 180), (200, 196), (210, 220), (250, 225), (270, 280), (330, 300), (350, 352),
                                   (45, 360), (360, 45)])
@pytest.mark.parametrize("swap", [False, True])
@pytest.mark.parametrize("method,diffraction,pixelsize", [("4x4", 3, 50.0), ("2x2", 1, 220.0)])
def test_compile_time_lines_match_shared_memory_passes(shape, swap, method, diffraction, pixelsize):
    """complex64 passes of the sides with line kernels of their own, each as rows and as columns, with the
    same bound as the register columns."""
    shape = shape[::-1] if swap else shape
    a = _mixed(shape, method, diffraction, 0, pixelsize)
    b = _mixed(shape, method, diffraction, 2, pixelsize)
    assert np.linalg.norm(a - b) <= 3e-6 * np.linalg.norm(b)
