"""RS / VRS of sides above 2048, whose transforms (512 R points, R = 10 .. 16) run
as two halves: sides at and next to the lengths' limits, with the other axis on
either side of 2048, against the FP64 oracle; fused programs; the z-derivative's
spectrum against a central difference of the oracle; the adjoint by the
dot-product identity.  Tolerance: relative L2 <= 1e-5, the path's bar (adjoint
and derivative: 1e-4)."""
import numpy as np
import pytest

from oracle import xlumina_ref as ref
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _field(rng, lead, ny, nx):
    import torch
    a = (rng.standard_normal(lead + (ny, nx)) + 1j * rng.standard_normal(lead + (ny, nx))).astype(np.complex64)
    return a, torch.as_tensor(a, device="cuda")


def _axes(ny, nx):
    return np.linspace(-1.0, 1.0, nx) * nx, np.linspace(-0.9, 0.9, ny) * ny


def _host(t):
    return t.cpu().numpy().astype(np.complex128)


@pytest.mark.parametrize("ny,nx", [(2049, 40), (2, 2560), (130, 2561), (3073, 300), (40, 3585), (4096, 2), (601, 4095),
                                   (2049, 2050)])
def test_scalar(ny, nx):
    from xlumina_gb300 import engine
    rng = np.random.default_rng(ny * 7 + nx)
    x, y = _axes(ny, nx)
    a, t = _field(rng, (), ny, nx)
    got = engine.rs_propagate([t], x, y, 0.633, 4.0e4, vector=False)[0]
    assert rel_l2(_host(got), ref.rs_propagate(a, x, y, 0.633, 4.0e4)) < TOL


@pytest.mark.parametrize("ny,nx,z", [(60, 2561, 3.0e4), (3585, 40, -2.0e4), (2100, 2049, 5.0e4)])
def test_vector_and_adjoint(ny, nx, z):
    import torch

    from xlumina_gb300 import engine
    rng = np.random.default_rng(ny + 3 * nx)
    x, y = _axes(ny, nx)
    (ax, tx), (ay, ty) = _field(rng, (), ny, nx), _field(rng, (), ny, nx)
    got = engine.rs_propagate([tx, ty], x, y, 0.633, z, vector=True)
    for g, e in zip(got, ref.vrs_propagate(ax, ay, x, y, 0.633, z)):
        assert rel_l2(_host(g), e) < TOL
    w = [_field(rng, (), ny, nx)[1] for _ in range(3)]
    adj = engine.RsCall(w, x, y, 0.633, z, vector=True, adjoint=True).run()
    dot = lambda a, b: sum(torch.vdot(p.reshape(-1).to(torch.complex128), q.reshape(-1).to(torch.complex128))  # noqa: E731
                           for p, q in zip(a, b))
    lhs, rhs = dot(w, got), dot(adj, [tx, ty])
    assert abs(lhs - rhs) < 1e-4 * abs(lhs)


@pytest.mark.parametrize("ny,nx,vector", [(50, 2100, False), (2800, 33, False), (41, 3100, True), (2200, 270, True)])
def test_programs_and_distances(ny, nx, vector):
    """A batch at two distances behind a program and before one; the vector
    case's last op is a polarizer, which shorter rows fold into the transform."""
    import torch

    from xlumina_gb300 import engine
    rng = np.random.default_rng(nx)
    x, y = _axes(ny, nx)
    B, zs = 4, [3.0e4, 5.0e4, 3.0e4, -4.0e4]
    phase = torch.as_tensor(rng.uniform(-3, 3, (ny, nx)).astype(np.float32), device="cuda")
    fields = [_field(rng, (B,), ny, nx) for _ in range(2 if vector else 1)]
    pre, post = [engine.op_phase(phase)], [engine.op_phase(phase)]
    masked = [a * np.exp(1j * phase.cpu().numpy().astype(np.float64)) for a, _ in fields]
    if vector:
        pre, post = [engine.op_sslm(phase, 0.4), engine.op_lp(0.3)], []
        sx = fields[0][0] * np.exp(1j * phase.cpu().numpy().astype(np.float64))
        u = np.cos(0.3) * sx + np.sin(0.3) * fields[1][0] * np.exp(0.4j)
        masked = [np.cos(0.3) * u, np.sin(0.3) * u]
    got = engine.RsCall([t for _, t in fields], x, y, 0.633, zs, vector=vector, pre=pre, post=post).run()
    for b in range(B):
        if vector:
            want = ref.vrs_propagate(masked[0][b], masked[1][b], x, y, 0.633, zs[b])
        else:
            want = [ref.rs_propagate(masked[0][b], x, y, 0.633, zs[b]) *
                    np.exp(1j * phase.cpu().numpy().astype(np.float64))]
        for g, e in zip(got, want):
            assert rel_l2(_host(g[b]), e) < TOL


@pytest.mark.parametrize("ny,nx", [(2500, 20), (20, 3000)])
def test_derivative_spectrum(ny, nx):
    from xlumina_gb300 import engine
    rng = np.random.default_rng(nx)
    x, y = _axes(ny, nx)
    a, t = _field(rng, (), ny, nx)
    z, h = 4.0e4, 1e-4
    got = engine.RsCall([t], x, y, 0.633, z, vector=False, dz=True).run()[0]
    want = (ref.rs_propagate(a, x, y, 0.633, z + h) - ref.rs_propagate(a, x, y, 0.633, z - h)) / (2 * h)
    assert rel_l2(_host(got), want) < 1e-4
