"""Programs that have a kernel with their op kinds fixed, at every transform length
of the block engine: the fused call gives what the program applied by itself and
a call without it give (the general route).  Tolerance: relative L2 <= 1e-6,
float32 rounding of the same arithmetic."""
import numpy as np
import pytest

from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


def _rand(*shape):
    import torch
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    return torch.randn((2,) + shape, dtype=torch.complex64, device="cuda", generator=g)


def _plane(seed, *shape):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand(shape, device="cuda", generator=g) * 6.0


def _same(got, exp):
    for g, e in zip(got, exp):
        assert rel_l2(g.cpu().numpy(), e.cpu().numpy()) < 1e-6


# x lines of 1024, 1536, .. 4096 points
@pytest.mark.parametrize("nx,mx", [(600, 300), (1001, 500), (1400, 500), (1600, 901), (2002, 800), (2100, 1300),
                                   (2047, 1999)])
def test_chirp_z(nx, mx):
    from xlumina_gb300 import engine
    ny = my = 70
    x, y = np.linspace(-1.0, 1.0, nx + nx % 2) * nx, np.linspace(-1.0, 1.0, ny) * nx
    x = x[:nx]
    xo, yo = np.linspace(-0.2, 0.2, mx) * nx, np.linspace(-0.2, 0.2, my) * nx
    e = _rand(2, ny, nx)
    e = [e[0], e[1]]
    P = [_plane(k, 2, ny, nx) for k in range(4)]
    r, f = 0.95 * nx, 1.05 * nx
    xf, yf = np.linspace(-2.0, 2.0, mx), np.linspace(-2.0, 2.0, my)
    sslm, lcd = engine.op_sslm(P[2], P[3]), engine.op_lcd(P[0], P[1])
    for mode, before in (("high_na", [sslm]), ("high_na_ez", [lcd, sslm])):
        op, s = engine.op_high_na(x, y, r, f, ez_only=mode == "high_na_ez")
        call = lambda c, pre: engine.czt_propagate(c, x, y, 0.633, None, xf, yf, mode, pre=pre, lens=(r, f, s))  # noqa: E731
        _same(call(e, before + [op]), call(engine.apply_ops(e, before, ny, nx), [op]))
    for op in (engine.op_phase(P[0]), engine.op_lens(x, y, 0.633, (0.8 * nx, 0.9 * nx), (60.0 * nx, 70.0 * nx), False)):
        call = lambda c, pre: engine.czt_propagate(c, x, y, 0.633, 60.0 * nx, xo, yo, "scalar", pre=pre)  # noqa: E731
        _same(call(e[:1], [op]), call(engine.apply_ops(e[:1], [op], ny, nx), []))


# x transforms of 1024, 1536, .. 4096 points, then of 5120 and 8192
@pytest.mark.parametrize("nx", [300, 513, 1000, 1025, 1500, 1793, 2047, 2051, 3590])
def test_rs(nx):
    from xlumina_gb300 import engine
    ny = 41
    x, y = np.linspace(-1.0, 1.0, nx) * nx, np.linspace(-1.0, 1.0, ny) * ny
    e = _rand(2, ny, nx)
    e = [e[0], e[1]]
    P = [_plane(k, 2, ny, nx) for k in range(2)]
    call = lambda c, pre: engine.rs_propagate(c, x, y, 0.633, 5.0e4, len(c) == 2, pre=pre)  # noqa: E731
    slm = [engine.op_phase(P[0])]
    _same(call(e[:1], slm), call(engine.apply_ops(e[:1], slm, ny, nx), []))
    for ops in ([engine.op_sslm(P[0], P[1])], [engine.op_lcd(P[0], P[1]), engine.op_lp(0.3)]):
        _same(call(e, ops), call(engine.apply_ops(e, ops, ny, nx), []))
