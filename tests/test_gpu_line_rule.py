"""Sides whose two-step line transforms lose to the shared-memory passes take those (GPU).

``fft_schedule`` 0 is the engine's choice, 1 the lines wherever a side splits, 2 the shared-memory passes: the
choice, for rows and columns together or for the columns alone, shows in the bits, and all agree to the bounds of ``test_gpu_line.py`` (2e-14 in complex128, 3e-6 in
complex64; two layers here as there).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (shape, precision, method, wavelengths, polarisations, diffraction, pixel size, betamax, absorbing, reflection, shared)
CASES = [
    ((162, 162), "double", "4x4", 2, 1, 1, 220.0, 1.4, False, None, True),    # nothing cut
    ((162, 160), "double", "4x4", 2, 1, 1, 220.0, 1.4, False, None, "columns"),  # one side only
    ((125, 125), "double", "4x4", 1, 1, 3, 220.0, 1.4, False, None, True),
    ((125, 125), "double", "4x4", 2, 1, 3, 220.0, 1.4, False, None, False),   # neither few nor many lines
    ((198, 198), "double", "4x4", 2, 1, 1, 220.0, 1.4, False, None, False),   # a factor 11
    ((189, 189), "mixed", "4x4", 3, 2, 1, 220.0, 1.4, False, None, True),
    ((189, 189), "mixed", "4x4", 1, 1, 1, 220.0, 1.4, False, None, False),    # few lines
    ((125, 125), "double", "2x2", 1, 1, 3, 100.0, 0.8, False, None, True),    # cut, few lines
    ((125, 125), "double", "2x2", 3, 2, 3, 100.0, 0.8, False, None, False),
    ((162, 162), "double", "2x2", 1, 1, 1, 100.0, 0.8, False, None, True),
    ((162, 162), "double", "4x4", 1, 1, 1, 100.0, 0.8, False, None, False),
    ((243, 243), "double", "2x2", 3, 2, 1, 100.0, 0.8, False, None, True),
    ((125, 125), "double", "4x4", 3, 2, 1, 100.0, 0.8, True, None, True),     # complex records
    ((162, 162), "double", "4x4", 2, 1, 3, 100.0, 0.8, True, None, True),
    ((160, 160), "double", "4x4", 2, 1, 3, 100.0, 0.8, True, None, False),
    ((162, 162), "double", "4x4", 3, 2, 1, 100.0, 0.8, False, 2, "columns"),  # real-space steps
    ((243, 160), "double", "2x2", 1, 1, 1, 100.0, 0.8, False, 2, "columns"),
    ((160, 162), "double", "4x4", 1, 1, 1, 100.0, 0.8, False, 2, False),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "%dx%d-%s-%s-%d-d%d-%g%s%s" % (
    c[0] + (c[1], c[2], c[3] * c[4], c[5], c[6], "-absorbing" if c[8] else "", "-r2" if c[9] else "")))
def test_choice_of_the_line_passes(case):
    import torch

    from dtmm_gb300 import transfer
    from dtmm_gb300.illumination import illumination_device

    shape, precision, method, nlam, npol, diffraction, pixelsize, betamax, absorbing, reflection, shared = case
    g = torch.Generator(device="cuda").manual_seed(8)
    ea = torch.rand((2,) + shape + (3,), generator=g, device="cuda", dtype=torch.float64)
    ev = torch.tensor([2.31, 2.31, 2.92], dtype=torch.float64, device="cuda")
    mat = transfer.DeviceMaterial(np.ones(2), ev + 0.01j if absorbing else ev, ea, shape)
    wl = np.linspace(450.0, 620.0, nlam)
    fin = illumination_device(shape, wl, pixelsize, beta=0.1, phi=0.4, jones=None if npol == 2 else (1, 0),
                              precision=precision)
    out = []
    for s in (0, 1, 2):
        plan = transfer.plan_transfer(tuple(fin.shape), wl, pixelsize, mat, beta=0.1, phi=0.4, method=method,
                                      diffraction=diffraction, reflection=reflection, betamax=betamax, npass=1,
                                      precision=precision, tuning=dict(fft_schedule=s))
        o = torch.empty_like(fin)
        plan.run(fin.clone(), o)
        out.append(o)
    auto, lines, passes = out
    assert torch.equal(auto, lines) == (shared is False) and torch.equal(auto, passes) == (shared is True)
    assert not torch.equal(lines, passes)
    tol = 2e-14 if precision == "double" else 3e-6
    assert float((lines - passes).norm() / passes.norm()) <= tol
    assert float((auto - passes).norm() / passes.norm()) <= tol


@pytest.mark.parametrize("shape,images", [((162, 162), 6), ((243, 96), 6), ((96, 189), 18), ((125, 125), 18), ((512, 48), 1),
                                          ((48, 512), 1)])
@pytest.mark.parametrize("precision,tol", [("double", 2e-14), ("mixed", 3e-6)])
def test_refocus_of_such_sides(shape, images, precision, tol):
    # rows and columns choose on their own; against torch.fft in complex128
    import torch

    from dtmm_gb300 import pom

    g = torch.Generator(device="cuda").manual_seed(3)
    f = torch.view_as_complex(torch.randn((images, 4) + shape + (2,), generator=g, device="cuda", dtype=torch.float64))
    m = torch.view_as_complex(torch.randn((images,) + shape + (4, 4, 2), generator=g, device="cuda", dtype=torch.float64))
    ref = torch.fft.ifft2(torch.einsum("lhwij,ljhw->lihw", m, torch.fft.fft2(f)))
    out = pom.diffract(f if precision == "double" else f.to(torch.complex64), m)
    assert float((out - ref).norm() / ref.norm()) <= tol
