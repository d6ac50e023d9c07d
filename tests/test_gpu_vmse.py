"""The vector intensity MSE's one launch for three components against the
per-component route, over the forms it takes (single and batched fields, a
target per entry or one for all, gradients of fields and targets) and some that
it leaves to that route (strided fields, targets with a leading 1).  Both run
the same sums in the same order: relative difference <= 1e-6."""
import pytest

pytestmark = pytest.mark.gpu


class _Light:
    pass


@pytest.mark.parametrize("lead,tlead,ny,nx", [((), (), 2, 3), ((), (), 33, 51), ((3,), (3,), 64, 40), ((3,), (), 65, 31),
                                              ((2, 2), (2, 2), 16, 20), ((1,), (), 300, 257), ((3,), (1,), 20, 20)])
@pytest.mark.parametrize("strided", [False, True])
@pytest.mark.parametrize("want", ["a", "b", "ex_bz"])
def test_vmse_intensity(lead, tlead, ny, nx, strided, want):
    import torch

    from xlumina_gb300 import loss_functions as lf
    torch.manual_seed(ny)

    def planes(shape):
        t = torch.randn(shape + (2 if strided else 1,), dtype=torch.complex64, device="cuda")[..., 0]
        return t.detach()

    a = [planes(lead + (ny, nx)) for _ in range(3)]
    b = [planes(tlead + (ny, nx)) for _ in range(3)]
    w = torch.randn((3,) + lead, device="cuda")
    results = []
    for fused in (True, False):
        ta, tb = [[t.clone(memory_format=torch.preserve_format) if not strided else t.detach() for t in ts] for ts in (a, b)]
        wanted = {"a": ta, "b": tb, "ex_bz": [ta[0], tb[2]]}[want]
        for t in wanted:
            t.requires_grad_(True)
        if fused:
            u, v = _Light(), _Light()
            u.Ex, u.Ey, u.Ez = ta
            v.Ex, v.Ey, v.Ez = tb
            out = lf.vMSE_Intensity(u, v)
        else:
            out = torch.stack([lf.MSE_Intensity(p, q) for p, q in zip(ta, tb)])
        (out * w).sum().backward()
        assert all((t.grad is not None) == any(t is q for q in wanted) for t in ta + tb)
        results.append([out.detach()] + [t.grad for t in wanted])
    for p, q in zip(*results):
        assert p.shape == q.shape and float((p - q).norm()) <= 1e-6 * float(q.norm())
