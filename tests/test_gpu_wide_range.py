"""Mixed-precision operators of materials and angles beyond the pair solve's range (GPU).

The equations keep their form when every refractive index (eps by its square),
the windows' betas and the wavelengths grow by a factor: E stays, H grows by
it.  Powers of two are exact, so a transfer far outside the exponents of FP32
products gives the ordinary one's result to rounding; likewise director angles
of many turns.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPE = (24, 40)


def _transfer(factor, method, voxel_eps, turns=0):
    import torch

    from dtmm_gb300 import samples
    from dtmm_gb300.illumination import illumination_device
    from dtmm_gb300.transfer import plan_transfer

    wl = np.array([450.0, 620.0])
    d, ev, ea = samples.twisted_nematic(SHAPE, 3, no=1.52, ne=1.71, amplitude=0.3, seed=4)
    ev = np.array(ev) * factor ** 2
    if not voxel_eps:
        ev = np.broadcast_to(ev[0, 0, 0], ev.shape)
    ea = ea + 0.0
    ea[..., 2] += 2 * np.pi * turns
    fin = illumination_device(SHAPE, wl, 100.0, beta=0.1, phi=0.4, precision="mixed")
    fin[..., 1::2, :, :] *= factor
    plan = plan_transfer(tuple(fin.shape), wl * factor, 100.0, [(d, ev, ea)], beta=0.1 * factor, phi=0.4,
                         nin=1.5 * factor, nout=1.5 * factor, betamax=0.8 * factor, method=method, diffraction=3,
                         npass=1, precision="mixed")
    out = torch.empty_like(fin)
    plan.run(fin, out)
    out[..., 1::2, :, :] /= factor
    return out.cpu().numpy()


@pytest.mark.parametrize("method", ["4x4", "2x2"])
@pytest.mark.parametrize("voxel_eps", [False, True])
@pytest.mark.parametrize("power", [-40, 22, 40])
def test_indices_beyond_the_range_of_the_pairs(method, voxel_eps, power):
    """eps of 2^-80 to 2^80: FP32 records of the FP64 solve against those of the pair solve, three layers
    of nine windows, each within a few FP32 roundings (6e-8) of the exact ones."""
    a = _transfer(1.0, method, voxel_eps)
    b = _transfer(2.0 ** power, method, voxel_eps)
    assert np.linalg.norm(a - b) <= 2e-6 * np.linalg.norm(a)


@pytest.mark.parametrize("turns", [2 ** 17, -2 ** 21])
def test_angles_of_many_turns(turns):
    """Whole turns of the director change nothing but the angle's own last place (2^-53 of 2 pi turns)."""
    a = _transfer(1.0, "4x4", True)
    b = _transfer(1.0, "4x4", True, turns)
    assert np.linalg.norm(a - b) <= 2e-6 * np.linalg.norm(a)
