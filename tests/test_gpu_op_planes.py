"""Devices with some parameters for every batch entry and others shared by the
batch: the batch gives, entry by entry, what the entry alone gives, forward and
backward (a shared plane's gradient is the sum over the batch).  Tolerance: relative
L2 <= 1e-5; fields, <= 1e-6 (the same arithmetic in float32)."""
import pytest

from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [40, 300])
@pytest.mark.parametrize("kind", ["sslm", "amp", "lcd"])
def test_mixed_planes(n, kind):
    import torch

    from xlumina_gb300 import engine
    from xlumina_gb300 import optical_elements as oe
    from xlumina_gb300.vectorized_optics import VectorizedLight
    B = 3
    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.linspace(-1.0, 1.0, n).numpy() * n
    E = torch.randn((2, B, n, n), dtype=torch.complex64, device="cuda", generator=g)
    W = torch.randn((2, B, n, n), dtype=torch.complex64, device="cuda", generator=g)
    make = {"sslm": oe.sSLM, "amp": oe.sSLM_with_amplitude, "lcd": oe.LCD}[kind]
    count = 4 if kind == "amp" else 2
    shapes = [(B, n, n) if i % 2 else (n, n) for i in range(count)]
    P = [(torch.rand(s, device="cuda", generator=g) * 3.0).requires_grad_(True) for s in shapes]

    def run(sel):
        light = VectorizedLight(x, x, 0.633)
        light.Ex, light.Ey = E[0, sel], E[1, sel]
        out = make(light, *[p if p.dim() == 2 else p[sel] for p in P]).VRS_propagation(5.0e4)[0]
        loss = sum((torch.conj(w[sel]) * c).real.sum() for w, c in zip(W, (out.Ex, out.Ey)))
        return out, torch.autograd.grad(loss, P)

    out, grads = run(slice(None))
    one = [run(b) for b in range(B)]
    for b in range(B):
        for c in ("Ex", "Ey", "Ez"):
            assert rel_l2(getattr(out, c)[b].detach().cpu().numpy(), getattr(one[b][0], c).detach().cpu().numpy()) < 1e-6
    for i in range(count):
        exp = sum(o[1][i] for o in one)
        assert rel_l2(grads[i].cpu().numpy(), exp.cpu().numpy()) < 1e-5
    with pytest.raises(ValueError):
        engine.rs_propagate([E[0], E[1][0]], x, x, 0.633, 5.0e4, True)
