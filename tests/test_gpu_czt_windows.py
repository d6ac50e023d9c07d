"""Chirp-z with a distance for each batch entry on the block engine's lengths
(the transfer functions evaluated in the kernels), over windows of a line that
begin and end anywhere between a thread's elements: short ones, a remainder of
one, odd offsets in the adjoint.  CTAs take runs of several entries' rows and
columns.  Forward against the FP64 oracle, adjoint by the dot-product identity;
relative L2 <= 1e-5, the path's bar (adjoint: 1e-4)."""
import numpy as np
import pytest

from oracle import xlumina_ref as ref
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


# x lines of 1024, 1024, 2048 and 4096 points, y lines of 1024, 2048, 1024 and 2048
@pytest.mark.parametrize("ny,nx,my,mx", [(520, 513, 37, 500), (1030, 700, 1000, 9), (257, 1025, 600, 1000),
                                         (601, 2049, 1203, 66)])
def test_one_component_with_a_distance_per_entry(ny, nx, my, mx):
    import torch

    from xlumina_gb300 import engine
    B = 5
    rng = np.random.default_rng(nx + my)
    z = [4.0e4 + 3.0e3 * b for b in range(B)]
    x, y = np.linspace(-1.0, 1.0, nx) * nx, np.linspace(-1.0, 1.0, ny) * ny
    xo, yo = np.linspace(-0.2, 0.2, mx) * nx, np.linspace(-0.3, 0.3, my) * ny
    cplx = lambda *s: (rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)  # noqa: E731
    E, W = cplx(B, ny, nx), cplx(B, my, mx)
    t, w = (torch.as_tensor(a, device="cuda") for a in (E, W))
    got = engine.czt_propagate([t], x, y, 0.633, z, xo, yo, mode="scalar")[0]
    for b in (0, B - 1):
        assert rel_l2(got[b].cpu().numpy().astype(np.complex128), ref.czt(E[b], x, y, 0.633, z[b], xo, yo)) < 1e-5
    adj = engine.CztCall([w], x, y, 0.633, z, xo, yo, "scalar", adjoint=True).run()[0]
    for b in range(B):
        lhs = torch.vdot(w[b].flatten().to(torch.complex128), got[b].flatten().to(torch.complex128))
        rhs = torch.vdot(adj[b].flatten().to(torch.complex128), t[b].flatten().to(torch.complex128))
        assert abs(lhs - rhs) < 1e-4 * abs(lhs)
