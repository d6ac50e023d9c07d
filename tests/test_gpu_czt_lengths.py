"""Chirp-z on every transform length of the block engine (1024, 1536, .. 4096
points): windows at and next to the lengths' limits, axes of different lengths
(and of different engines), against the FP64 oracle; the adjoint by the
dot-product identity.  Tolerance: relative L2 <= 1e-5, the path's bar (adjoint:
1e-4)."""
import numpy as np
import pytest

from oracle import xlumina_ref as ref
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _field(rng, ny, nx):
    import torch
    a = (rng.standard_normal((ny, nx)) + 1j * rng.standard_normal((ny, nx))).astype(np.complex64)
    return a, torch.as_tensor(a, device="cuda")


def _axis(n, h):
    return np.linspace(-h, h, n)


# (ny, nx) onto (my, mx): m + M at a length's limit, one past it, short and long axes mixed
@pytest.mark.parametrize("ny,nx,my,mx", [(512, 513, 512, 511), (1000, 1100, 536, 437), (1100, 700, 436, 837),
                                         (1300, 1537, 748, 511), (1536, 1793, 1025, 767), (2000, 2048, 1096, 1536),
                                         (200, 2047, 60, 2048), (2500, 300, 2100, 240)])
def test_scalar_lengths(ny, nx, my, mx):
    from xlumina_gb300 import engine
    rng = np.random.default_rng(ny + nx + my + mx)
    x, y, xo, yo = _axis(nx, 1.0 * nx), _axis(ny, 1.0 * ny), _axis(mx, 0.2 * nx), _axis(my, 0.3 * ny)
    a, t = _field(rng, ny, nx)
    z = 6.0e4
    got = engine.czt_propagate([t], x, y, 0.633, z, xo, yo, mode="scalar")[0]
    assert rel_l2(got.cpu().numpy().astype(np.complex128), ref.czt(a, x, y, 0.633, z, xo, yo)) < TOL


@pytest.mark.parametrize("ny,nx,my,mx", [(900, 1030, 300, 494), (1400, 1201, 700, 300)])
def test_vector_lengths_and_adjoint(ny, nx, my, mx):
    import torch

    from xlumina_gb300 import engine
    rng = np.random.default_rng(ny + 3 * nx)
    x, y, xo, yo = _axis(nx, 1.0 * nx), _axis(ny, 1.0 * ny), _axis(mx, 0.2 * nx), _axis(my, 0.3 * ny)
    (ax, tx), (ay, ty) = _field(rng, ny, nx), _field(rng, ny, nx)
    z = 5.0e4
    got = engine.czt_propagate([tx, ty], x, y, 0.633, z, xo, yo, mode="vczt")
    for g, e in zip(got, ref.vczt(ax, ay, x, y, 0.633, z, xo, yo)):
        assert rel_l2(g.cpu().numpy().astype(np.complex128), e) < TOL
    w = [_field(rng, my, mx)[1] for _ in range(3)]
    adj = engine.CztCall(w, x, y, 0.633, z, xo, yo, "vczt", adjoint=True).run()
    dot = lambda a, b: sum(torch.vdot(p.reshape(-1).to(torch.complex128), q.reshape(-1).to(torch.complex128))  # noqa: E731
                           for p, q in zip(a, b))
    lhs, rhs = dot(w, got), dot(adj, [tx, ty])
    assert abs(lhs - rhs) < 1e-4 * abs(lhs)
    # one distance per entry: spectra in natural order, the same fields
    two = engine.czt_propagate([torch.stack([tx, tx]), torch.stack([ty, ty])], x, y, 0.633, [z, z], xo, yo, mode="vczt")
    for g, h in zip(got, two):
        for b in range(2):
            assert rel_l2(h[b].cpu().numpy(), g.cpu().numpy()) < TOL
