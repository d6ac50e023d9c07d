"""Chirp-z of several components onto a number of columns that is no multiple of
a column CTA's eight: the lanes of a warp whose column is past the edge store
nothing while the others run the epilogue, and the next component starts behind
that branch.  Batches large enough that a CTA takes an entry's components one
after the other (at least two units an SM), against the FP64 oracle; relative L2
<= 1e-5, the path's bar."""
import numpy as np
import pytest

from oracle import xlumina_ref as ref
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-5


# y transforms of 1536 and 2048 points; 39 groups of columns x 8 entries
@pytest.mark.parametrize("ny,nx,my,mx", [(800, 700, 311, 305), (1500, 600, 307, 311)])
def test_vczt_components_on_ragged_columns(ny, nx, my, mx):
    import torch

    from xlumina_gb300 import engine
    B, z = 8, 5.0e4
    rng = np.random.default_rng(ny + mx)
    x, y = np.linspace(-1.0, 1.0, nx) * nx, np.linspace(-1.0, 1.0, ny) * ny
    xo, yo = np.linspace(-0.2, 0.2, mx) * nx, np.linspace(-0.3, 0.3, my) * ny
    E = (rng.standard_normal((2, B, ny, nx)) + 1j * rng.standard_normal((2, B, ny, nx))).astype(np.complex64)
    ex, ey = (torch.as_tensor(e, device="cuda") for e in E)
    got = engine.czt_propagate([ex, ey], x, y, 0.633, z, xo, yo, mode="vczt")
    for b in (0, B - 1):
        for g, e in zip(got, ref.vczt(E[0, b], E[1, b], x, y, 0.633, z, xo, yo)):
            assert rel_l2(g[b].cpu().numpy().astype(np.complex128), e) < TOL
