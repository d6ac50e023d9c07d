"""The chirp-z kernels' variants at the lengths that have several (Stockham: 32 to
512 points, and 8192): x transform 0 to 3 (how much of the rows is staged, and for
how many CTAs per SM), y transform 0 and 1 (one CTA per tile, persistent), each
against the FP64 oracle and against variant 0.  Tolerance: relative L2 <= 1e-5
against the oracle (the path's bar), <= 1e-6 between variants (float32 rounding)."""
import numpy as np
import pytest

from oracle import xlumina_ref as ref
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture
def select():
    from xlumina_gb300 import _lib, engine
    lib = engine.lib()
    passes = (_lib.XL_PASS_CZT_ROWS, _lib.XL_PASS_CZT_COLS)
    saved = {(p, lg): lib.xl_get_kernel_variant(p, lg) for p in passes for lg in range(5, 14)}

    def both(rows, cols):
        for (p, lg), _ in saved.items():
            v = rows if p == passes[0] else cols
            if v < lib.xl_kernel_variant_count(p, lg):
                _lib.check(lib.xl_set_kernel_variant(p, lg, v), "xl_set_kernel_variant")

    yield both
    for (p, lg), v in saved.items():
        _lib.check(lib.xl_set_kernel_variant(p, lg, v), "xl_set_kernel_variant")


# lines of 32, 128, 512 and 8192 points (x), 64, 256, 512 and 32 points (y)
@pytest.mark.parametrize("ny,nx,my,mx", [(33, 16, 20, 10), (130, 80, 66, 40), (300, 256, 180, 128), (20, 4096, 10, 1500)])
def test_every_variant(select, ny, nx, my, mx):
    import torch

    from xlumina_gb300 import engine
    rng = np.random.default_rng(nx + my)
    x, y = np.linspace(-1.0, 1.0, nx) * nx, np.linspace(-1.0, 1.0, ny) * ny
    xo, yo = np.linspace(-0.2, 0.2, mx) * nx, np.linspace(-0.3, 0.3, my) * ny
    E = (rng.standard_normal((2, ny, nx)) + 1j * rng.standard_normal((2, ny, nx))).astype(np.complex64)
    eta = rng.uniform(0, 6, (ny, nx)).astype(np.float32)
    ex, ey, eta_d = (torch.as_tensor(a, device="cuda") for a in (E[0], E[1], eta))
    z = 5.0e4
    ax, ay = ref.lcd(E[0].astype(np.complex128), E[1].astype(np.complex128), eta.astype(np.float64), 0.4)
    exp = (ref.czt(E[0], x, y, 0.633, z, xo, yo),) + tuple(ref.vczt(ax, ay, x, y, 0.633, z, xo, yo))
    first = None
    for rows, cols in ((0, 0), (1, 0), (2, 1), (3, 1)):
        select(rows, cols)
        got = engine.czt_propagate([ex], x, y, 0.633, z, xo, yo, mode="scalar")
        got = got + engine.czt_propagate([ex, ey], x, y, 0.633, z, xo, yo, mode="vczt", pre=[engine.op_lcd(eta_d, 0.4)])
        got = [t.cpu().numpy().astype(np.complex128) for t in got]
        for g, e in zip(got, exp):
            assert rel_l2(g, e) < 1e-5, (rows, cols)
        first = first or got
        for g, e in zip(got, first):
            assert rel_l2(g, e) < 1e-6, (rows, cols)
