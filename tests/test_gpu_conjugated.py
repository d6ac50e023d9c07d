"""Lazily conjugated tensors (``t.conj()`` marks a view, its memory is that of t): a
field, a mask or a gradient given as one is used with its values.  Each call is
compared with the same one on conjugated memory, bit for bit."""
import numpy as np
import pytest
import torch


def test_as_field_resolves_the_conjugation():
    from xlumina_gb300 import engine
    t = torch.randn((2, 3, 4), dtype=torch.complex64)
    for a in (t.conj(), t[0].expand(2, 3, 4).conj(), t.to(torch.complex128).conj()):
        f = engine.as_field(a, dev=torch.device("cpu"))
        assert not f.is_conj() and torch.equal(f, a.resolve_conj().to(torch.complex64))


def _pair(*shape):
    g = torch.Generator(device="cuda").manual_seed(sum(shape))
    t = torch.randn(shape, dtype=torch.complex64, device="cuda", generator=g)
    return t.conj(), t.conj().resolve_conj()


@pytest.mark.gpu
def test_fields_masks_and_losses():
    from xlumina_gb300 import autograd, engine
    n, B = 48, 2
    x = np.linspace(-1.0, 1.0, n) * n
    res = []
    for lazy in (0, 1):
        e, f = _pair(B, n, n)[lazy], _pair(B + 1, n, n)[lazy][:B]
        m = _pair(n, n)[lazy]
        ang = torch.tensor([[0.6, 0.8j], [0.8j, 0.6]], dtype=torch.complex64, device="cuda")
        ang = ang.conj() if lazy else ang.conj().resolve_conj()
        out = engine.rs_propagate([e, f], x, x, 0.633, 5.0e4, True, pre=[engine.op_cmul(m)])
        out = out + engine.apply_ops([e[:1].expand(B, n, n)], [engine.op_phase(0.3)], n, n)
        out = out + engine.beam_splitter([e, f], None, ang)
        t = torch.rand((n, n), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
        leaf = e.detach().requires_grad_(True)
        g, = torch.autograd.grad(autograd.norm_intensity_mse(leaf, t / t.sum()).sum(), leaf)
        res.append(out + [g.resolve_conj()])
    for a, b in zip(*res):
        assert torch.equal(a, b)


@pytest.mark.gpu
def test_gradients_of_a_conjugated_output():
    from xlumina_gb300 import optical_elements as oe
    from xlumina_gb300.wave_optics import ScalarLight
    n = 48
    x = np.linspace(-1.0, 1.0, n) * n
    w = _pair(n, n)[1]
    grads = []
    for lazy in (False, True):
        light = ScalarLight(x, x, 0.633)
        light.field = _pair(n, n + 1)[1][:, :n]
        ph = torch.full((n, n), 0.4, device="cuda", requires_grad=True)
        lit = oe.SLM(light, ph, n)[0]
        a, b = lit.RS_propagation(5.0e4)[0].field, lit.field
        loss = sum((u.conj() * w if lazy else torch.complex(u.real, -u.imag) * w).real.sum() for u in (a, b))
        grads.append(torch.autograd.grad(loss, ph)[0])
    assert torch.allclose(grads[0], grads[1], rtol=1e-5, atol=1e-5 * float(grads[0].abs().max()))
