"""The two-pixel backward kernels of scalar one-op programs (a phase SLM with a
plane per entry, a thin lens) against complex128 torch, at sizes they take and
at odd ones and misaligned planes that the general kernel takes.  Tolerance:
relative L2 <= 1e-5."""
import numpy as np
import pytest

from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _cases():
    return [(1, 2, 2, False), (1, 65, 130, False), (3, 34, 50, False), (3, 33, 51, False), (1, 33, 51, False),
            (2, 257, 514, False), (2, 64, 64, True)]


def _planes(B, ny, nx, off, dtype, scale=1.0):
    """(B, ny, nx), one element off a 16-byte boundary where asked."""
    import torch
    n = B * ny * nx
    flat = torch.randn(n + 1, dtype=dtype, device="cuda") * scale
    t = (flat[1:] if off else flat[:n]).reshape(B, ny, nx)
    return t if B > 1 else t[0]


@pytest.mark.parametrize("B,ny,nx,off", _cases())
@pytest.mark.parametrize("want", [True, False])
def test_phase(B, ny, nx, off, want):
    import torch

    from xlumina_gb300 import engine
    e, g = (_planes(B, ny, nx, off, torch.complex64) for _ in range(2))
    ph = _planes(B, ny, nx, off, torch.float32, 3.0).detach().requires_grad_(True)
    gin, pg = engine.ops_backward([e], [g], [engine.op_phase(ph)], ny, nx, want_input=want)
    z = torch.exp(1j * ph.detach().double())
    y = e.to(torch.complex128) * z
    exp = (g.to(torch.complex128) * torch.conj(1j * y)).real
    assert rel_l2(pg[(0, 0)].double().cpu().numpy(), exp.cpu().numpy()) < TOL
    if want:
        assert rel_l2(gin[0].cpu().numpy(), (g.to(torch.complex128) * torch.conj(z)).cpu().numpy()) < TOL
    else:
        assert gin[0] is None


@pytest.mark.parametrize("B,ny,nx,off", _cases())
def test_lens(B, ny, nx, off):
    import torch

    from xlumina_gb300 import engine
    x, y = np.linspace(-1.0, 1.0, nx), np.linspace(-1.0, 1.0, ny)
    op = engine.op_lens(x, y, 0.6, (0.8, 0.9), (50.0, 40.0), False)
    g = _planes(B, ny, nx, off, torch.complex64)
    gin, _ = engine.ops_backward([g], [g], [op], ny, nx, want_input=True)
    cf, rf, tc, tr = engine.lens_factors(x, y, 0.6, (0.8, 0.9), (50.0, 40.0))
    m = np.where((tc[None, :] + tr[:, None]) < 1, 1, 0) * (rf[:, None] * cf[None, :])
    exp = g.cpu().numpy().astype(np.complex128) * np.conj(m)
    got = gin[0].cpu().numpy()
    assert np.array_equal(got == 0, exp == 0)
    assert np.linalg.norm(got - exp) <= TOL * np.linalg.norm(exp)   # (all zero where no pixel is in the pupil)
