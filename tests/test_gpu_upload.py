"""Host arrays given to device entry points, while other work is queued (GPU).

The uploads need not wait for that work, but a kernel reads them only once
they are there, on whatever stream it runs, and the caller's arrays are free
when the call returns.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BUSY = 100_000_000  # clock cycles of a sleeping kernel: about 50 ms


def _spoil(n):
    """Freed device memory that holds NaN, so that a late upload shows."""
    import torch

    keep = [torch.full((n,), float("nan"), dtype=torch.float64, device="cuda") for _ in range(8)]
    torch.cuda.synchronize()
    del keep


def _image_inputs():
    import torch

    from dtmm_gb300 import pom, samples

    g = torch.Generator(device="cuda").manual_seed(2)
    f = torch.view_as_complex(torch.randn((2, 3, 4, 16, 24, 2), generator=g, device="cuda", dtype=torch.float64))
    pmat = pom.ray_jonesmat4x4(pom.polarizer(pom.jonesvec((1, -1))), epsv=(2.25,) * 3)
    return f, samples.transmission_cmf(np.linspace(400.0, 700.0, 3)), pmat


@pytest.mark.parametrize("busy", ["caller", "other"])
def test_pom_image_on_another_stream(busy):
    """The kernel's stream takes the uploads: the caller's queued work neither delays nor outruns them."""
    import torch

    from dtmm_gb300 import pom

    f, cmf, pmat = _image_inputs()
    want = pom.pom_image(f, cmf, jvec=(0.6, 0.8), pmat=pmat)
    other = torch.cuda.Stream()
    _spoil(32)
    with torch.cuda.stream(other if busy == "other" else torch.cuda.current_stream()):
        torch.cuda._sleep(BUSY)
    got = pom.pom_image(f, cmf.copy(), jvec=(0.6, 0.8), pmat=pmat.copy(), stream=other.cuda_stream)
    other.synchronize()
    assert torch.equal(got, want)


@pytest.mark.parametrize("pinned", [False, True])
def test_pom_image_arrays_are_free_after_the_call(pinned):
    import torch

    from dtmm_gb300 import pom

    f, cmf, pmat = _image_inputs()
    want = pom.pom_image(f, cmf, jvec=(0.6, 0.8), pmat=pmat)
    c = torch.from_numpy(cmf.copy())
    m = torch.from_numpy(pmat.copy())
    if pinned:
        c, m = c.pin_memory(), m.pin_memory()
    c, m = c.numpy(), m.numpy()
    torch.cuda._sleep(BUSY)
    got = pom.pom_image(f, c, jvec=(0.6, 0.8), pmat=m)
    c[...] = np.nan
    m[...] = np.nan
    assert torch.equal(got, want)


def test_pom_image_host_arrays_are_refused_in_a_capture():
    """A graph would copy from host memory that is gone when it is replayed."""
    import torch

    from dtmm_gb300 import pom

    f, cmf, pmat = _image_inputs()
    pom.pom_image(f, cmf, jvec=(0.6, 0.8), pmat=pmat)
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        with pytest.raises(RuntimeError, match="device tensors"):
            pom.pom_image(f, cmf, jvec=(0.6, 0.8), pmat=pmat)


@pytest.mark.parametrize("pinned", [False, True])
@pytest.mark.parametrize("voxel_eps", [False, True])
def test_plan_owns_its_material_when_the_call_returns(pinned, voxel_eps):
    """A plan from host arrays, made on a busy stream and run on another one: the director angles are on the
    device and the caller's arrays free.  One eps for the sample is looked through on the host, 2^18 values
    (88 x 100 x 10 voxels) and more on the device."""
    import torch

    from dtmm_gb300 import samples
    from dtmm_gb300.illumination import illumination_device
    from dtmm_gb300.transfer import plan_transfer

    shape, wl = (100, 88), [500.0]
    d, ev, ea = samples.twisted_nematic(shape, 10, no=1.52, ne=1.71, amplitude=0.3, seed=3)
    ea = np.array(np.broadcast_to(ea, (10,) + shape + (3,)))
    if voxel_eps:
        ev = np.array(np.broadcast_to(ev, (10,) + shape + (3,)))
    fin = illumination_device(shape, wl, 100.0, precision="mixed")
    opts = dict(method="4x4", diffraction=1, npass=1, precision="mixed")
    want = torch.empty_like(fin)
    plan_transfer(tuple(fin.shape), wl, 100.0, [(d, ev, ea.copy())], **opts).run(fin, want)
    torch.cuda.synchronize()
    t = torch.from_numpy(ea)
    mine = (t.pin_memory() if pinned else t.clone()).numpy()
    got = torch.empty_like(fin)
    _spoil(ea.size)
    other = torch.cuda.Stream()
    torch.cuda._sleep(BUSY)
    plan = plan_transfer(tuple(fin.shape), wl, 100.0, [(d, ev, mine)], **opts)
    mine[...] = np.nan
    with torch.cuda.stream(other):
        plan.run(fin, got)
    other.synchronize()
    assert torch.equal(got, want)
