"""The masks that an SLM and a lens return beside the light, and the quality
factor of distances on the device, against complex128 / float64 on the host:
sizes around the four-phase step, a plane per entry, planes off a 16-byte
boundary.  Tolerance: relative L2 <= 1e-6 (one float32 sincos each; the lens'
factors are rounded once to complex64 and multiplied)."""
import numpy as np
import pytest

from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lead,ny,nx,off", [((), 2, 2, False), ((), 33, 51, False), ((), 33, 51, True),
                                            ((3,), 34, 50, False), ((3,), 33, 51, True), ((1,), 1, 7, False),
                                            ((2,), 640, 520, False)])
def test_slm_mask(lead, ny, nx, off):
    import torch

    from xlumina_gb300 import optical_elements as oe, wave_optics
    x, y = np.linspace(-50, 50, max(nx, 2))[:nx], np.linspace(-50, 50, ny)
    flat = (torch.rand(int(np.prod(lead + (ny, nx))) + 1, device="cuda") - 0.5) * 20
    phase = (flat[1:] if off else flat[:-1]).reshape(lead + (ny, nx))
    if nx < 8 or ny < 2:
        mask = oe._phase_mask(phase, ny, nx)
    else:
        light = wave_optics.ScalarLight(x, y, 0.6328)
        light.field = torch.ones((ny, nx), dtype=torch.complex64, device="cuda")
        mask = oe.SLM(light, phase, nx)[1]
    assert mask.shape == phase.shape and mask.dtype == torch.complex64
    assert rel_l2(mask.cpu(), torch.exp(1j * phase.cpu().to(torch.complex128))) <= 1e-6


@pytest.mark.parametrize("ny,nx", [(2, 2), (33, 51), (64, 130)])
def test_lens_mask(ny, nx):
    import torch

    from xlumina_gb300 import optical_elements as oe, wave_optics
    x, y = np.linspace(-1100, 1050, nx), np.linspace(-950, 1000, ny)
    light = wave_optics.ScalarLight(x, y, 0.6328)
    light.field = torch.ones((ny, nx), dtype=torch.complex64, device="cuda")
    for radius, focal in [((1000.0, 1000.0), (5e4, 5e4)), ((700.0, 900.0), (4e4, 6e4)), ((1000.0, 1000.0), (6e4, 5e4))]:
        mask = oe.lens(light, radius, focal)[1]
        k = 2 * np.pi / 0.6328
        want = np.exp(-1j * k * (x[None] ** 2 / (2 * focal[0]) + y[:, None] ** 2 / (2 * focal[1])))
        want = want * (x[None] ** 2 / radius[0] ** 2 + y[:, None] ** 2 / radius[1] ** 2 < 1)
        diff = mask.cpu().to(torch.complex128) - torch.from_numpy(want)
        assert mask.shape == (ny, nx) and float(diff.norm()) <= 1e-6 * float(np.linalg.norm(want))


@pytest.mark.parametrize("n", [1, 7, 300])
def test_quality_factor(n):
    import torch

    from xlumina_gb300 import engine
    x, y = np.linspace(-300, 280, 37), np.linspace(-200, 210, 50)
    z = np.random.default_rng(0).uniform(50.0, 1e5, n)
    want = engine.quality_factor(x, y, 0.6328, z)
    got = engine.quality_factor(x, y, 0.6328, torch.tensor(z, device="cuda"))
    assert got.dtype == torch.float64 and got.shape == (n,)
    assert np.abs(got.cpu().numpy() - want).max() <= 1e-12 * np.abs(want).max()
    x[1] += 1.0                                   # a grid that was changed in place gives its own factor
    again = engine.quality_factor(x, y, 0.6328, torch.tensor(z, device="cuda")).cpu().numpy()
    assert np.abs(again - engine.quality_factor(x.copy(), y, 0.6328, z)).max() <= 1e-12 * np.abs(want).max()
    assert np.abs(again - want).max() > 1e-3 * np.abs(want).max()
