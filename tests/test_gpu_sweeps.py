"""How a sweep is launched changes no bit of its result (GPU).

Small stacks form every layer's operators in one launch and launch their row and column passes with programmatic
dependencies; ``op_cache_bytes`` = 1 turns both off, a timed run the second.  ``row_group`` and ``col_tile`` choose
between accumulators in registers and in shared memory.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _plan(shape, precision, method, diffraction, npass=1, nstep=1, layers=14, nlam=2, npol=1, nray=1, equal=True):
    import torch

    from dtmm_gb300 import transfer
    from dtmm_gb300.illumination import illumination_device

    g = torch.Generator(device="cuda").manual_seed(8)
    ea = torch.rand((layers,) + shape + (3,), generator=g, device="cuda", dtype=torch.float64) * 2.0
    ev = torch.tensor([2.31, 2.31, 2.92], dtype=torch.float64, device="cuda")
    d = np.ones(layers) if equal else np.linspace(0.5, 1.5, layers)
    mat = transfer.DeviceMaterial(d, ev, ea, shape)
    wl = np.linspace(450.0, 620.0, nlam)
    beta, phi = (0.1, 0.4) if nray == 1 else (np.array([0.0, 0.1, 0.2]), np.array([0.0, 0.5, 2.0]))
    fin = illumination_device(shape, wl, 100.0, beta=beta, phi=phi, jones=None if npol == 2 else (1, 0),
                              precision=precision)
    plan = transfer.plan_transfer(tuple(fin.shape), wl, 100.0, mat, beta=beta, phi=phi, method=method,
                                  diffraction=diffraction, npass=npass, nstep=nstep, precision=precision)
    return plan, fin


def _run(plan, fin, timed=False):
    import torch

    f, out = fin.clone(), torch.full_like(fin, float("nan"))
    t = plan.run(f, out, timed=timed)
    torch.cuda.synchronize()
    return out, f, t


@pytest.mark.parametrize("shape", [(64, 64), (45, 50), (22, 26)])
@pytest.mark.parametrize("precision", ["double", "mixed"])
@pytest.mark.parametrize("method,diffraction,npass,nstep,nray", [
    ("4x4", 1, 1, 1, 1), ("4x4", 1, 1, 2, 3), ("4x4", 3, 1, 1, 1), ("4x4", 3, 1, 2, 1), ("4x4", 1, 3, 1, 1),
    ("4x4", 3, 3, 1, 1), ("2x2", 1, 1, 1, 1), ("2x2", 3, 1, 1, 3), ("2x2", 1, 3, 2, 1)])
def test_sweeps_launched_layer_by_layer(shape, precision, method, diffraction, npass, nstep, nray):
    import torch

    plan, fin = _plan(shape, precision, method, diffraction, npass, nstep, nray=nray)
    out, back, _ = _run(plan, fin)
    timed, _, t = _run(plan, fin, timed=True)
    assert torch.isfinite(torch.view_as_real(out)).all() and torch.equal(timed, out)
    # every layer at once where the stack's records (12 complex numbers a voxel, window and ray) take 32 MB at most
    records = 14 * shape[0] * shape[1] * nray * diffraction ** 2 * 12 * (16 if precision == "double" else 8)
    assert t.voxel_op_launches == (1 if npass == 1 and records <= 32 << 20 else 14)
    g = plan.capture(fin.clone(), out2 := torch.full_like(fin, float("nan")))
    if npass == 1:  # (with more passes a replay would start from the rewritten input)
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(out2, out)
    plan.desc.op_cache_bytes = 1
    plain, plain_back, _ = _run(plan, fin)
    _, _, t = _run(plan, fin, timed=True)
    assert t.voxel_op_launches == 14 * npass  # (three passes kept them in the first)
    assert torch.equal(plain, out) and torch.equal(plain_back, back)


@pytest.mark.parametrize("precision", ["double", "mixed"])
def test_layers_of_unequal_thickness_have_their_own_operators(precision):
    import torch

    plan, fin = _plan((48, 48), precision, "4x4", 1, equal=False)
    out, _, t = _run(plan, fin, timed=True)
    assert t.voxel_op_launches == 14
    one = _run(*_plan((48, 48), precision, "4x4", 1))[0]
    assert not torch.equal(out, one)
    plan.desc.op_cache_bytes = 1
    assert torch.equal(_run(plan, fin)[0], out)


@pytest.mark.parametrize("side", [64, 128, 256])
@pytest.mark.parametrize("precision,method,npol", [("mixed", "4x4", 1), ("mixed", "4x4", 2), ("mixed", "2x2", 1),
                                                   ("mixed", "2x2", 2), ("double", "4x4", 2)])
def test_row_groups_and_column_tiles_keep_the_bits(side, precision, method, npol):
    import torch

    plan, fin = _plan((32, side), precision, method, 3, layers=3, nlam=4, npol=npol)
    base = _run(plan, fin)[0]
    for rg, ct in ((1, 1), (2, 0), (3, 2), (4, 4), (8, 8)):
        plan.set_tuning(row_group=rg, col_tile=ct)
        assert torch.equal(_run(plan, fin)[0], base), (rg, ct)
