"""Calls recorded by a tracer (torch.jit.trace, make_fx, torch.compile without
graph breaks) on one input and replayed on another: the recorded graph has to
hold the arithmetic, not the memory that a kernel of the library filled behind
the tracer's back.  Tolerance: float64 1e-12, float32 masks 1e-6."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _trace(how, fn, arg):
    import torch
    if how == "jit":
        return torch.jit.trace(fn, (arg,), check_trace=False)
    if how == "compile":
        f = torch.compile(fn, backend="eager", fullgraph=True)
        f(arg)
        return f
    from torch.fx.experimental.proxy_tensor import make_fx
    return make_fx(fn)(arg)


@pytest.mark.parametrize("how", ["jit", "make_fx", "compile"])
def test_quality_factor_of_a_traced_distance(how):
    import torch

    from xlumina_gb300 import engine
    x = np.linspace(-500.0, 500.0, 96)
    z = [torch.tensor([a, 3 * a], dtype=torch.float64, device="cuda") for a in (2.0e4, 7.0e4)]
    f = _trace(how, lambda t: engine.quality_factor(x, x, 0.633, t), z[0])
    exp = engine.quality_factor(x, x, 0.633, z[1].cpu().numpy())
    assert np.allclose(f(z[1]).cpu().numpy(), exp, rtol=1e-12, atol=0)


@pytest.mark.parametrize("how", ["jit", "make_fx", "compile"])
def test_mask_of_a_traced_phase(how):
    import torch

    from xlumina_gb300 import optical_elements as oe
    rng = np.random.default_rng(5)
    ph = [torch.as_tensor(rng.uniform(-3, 3, (2, 24, 33)).astype(np.float32), device="cuda") for _ in range(2)]
    f = _trace(how, lambda t: oe._phase_mask(t, 24, 33), ph[0])
    assert np.abs(f(ph[1]).cpu().numpy() - np.exp(1j * ph[1].cpu().numpy().astype(np.float64))).max() < 1e-6
