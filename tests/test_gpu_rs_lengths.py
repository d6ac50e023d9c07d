"""RS / VRS on every transform length of the block engine (256 R points, each
axis its own): fields whose sides sit at and next to the lengths' limits,
square and not, against the FP64 oracle; the adjoint by the dot-product
identity.  Tolerance: relative L2 <= 1e-5, the path's bar (adjoint: 1e-4)."""
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


def _axes(ny, nx):
    return np.linspace(-1.0, 1.0, nx) * nx, np.linspace(-0.9, 0.9, ny) * ny


@pytest.mark.parametrize("ny,nx", [(257, 257), (2, 300), (512, 513), (768, 769), (769, 768), (1025, 60), (1000, 1280),
                                   (1281, 1536), (1537, 1100), (1792, 1793), (300, 2047)])
def test_scalar_lengths(ny, nx):
    from xlumina_gb300 import engine
    rng = np.random.default_rng(ny * 7 + nx)
    x, y = _axes(ny, nx)
    a, t = _field(rng, ny, nx)
    got = engine.rs_propagate([t], x, y, 0.633, 4.0e4, vector=False)[0]
    exp = ref.rs_propagate(a, x, y, 0.633, 4.0e4)
    assert rel_l2(got.cpu().numpy().astype(np.complex128), exp) < TOL


@pytest.mark.parametrize("ny,nx,z", [(700, 513, 3.0e4), (1025, 1281, -2.0e4), (520, 1700, 5.0e4)])
def test_vector_lengths_and_adjoint(ny, nx, z):
    import torch

    from xlumina_gb300 import engine
    rng = np.random.default_rng(ny + 3 * nx)
    x, y = _axes(ny, nx)
    (ax, tx), (ay, ty) = _field(rng, ny, nx), _field(rng, ny, nx)
    got = engine.rs_propagate([tx, ty], x, y, 0.633, z, vector=True)
    for g, e in zip(got, ref.vrs_propagate(ax, ay, x, y, 0.633, z)):
        assert rel_l2(g.cpu().numpy().astype(np.complex128), e) < TOL
    w = [_field(rng, ny, nx)[1] for _ in range(3)]
    adj = engine.RsCall(w, x, y, 0.633, z, vector=True, adjoint=True).run()
    dot = lambda a, b: sum(torch.vdot(p.reshape(-1).to(torch.complex128), q.reshape(-1).to(torch.complex128))  # noqa: E731
                           for p, q in zip(a, b))
    lhs, rhs = dot(w, got), dot(adj, [tx, ty])
    assert abs(lhs - rhs) < 1e-4 * abs(lhs)
