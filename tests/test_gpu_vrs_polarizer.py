"""VRS whose program ends in a polarizer at one angle transforms two components
instead of three.  Every form the route takes, and its neighbours that it does
not take (an angle per pixel, another op last, an epilogue), against the general
path: the same program as a pass of its own, then a VRS without a program.
Tolerance: both stay within 5e-7 of the exact result, so 2e-6 of the norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 2e-6


def _planes(rng, shape, off=0, dtype="complex64"):
    """A contiguous array of the shape, ``off`` elements from its allocation's start."""
    import torch
    n = int(np.prod(shape))
    v = rng.standard_normal(n + off)
    if dtype == "complex64":
        v = v + 1j * rng.standard_normal(n + off)
    return torch.as_tensor(v.astype(dtype), device="cuda")[off:].reshape(shape)


def _program(kind, rng, ny, nx, off):
    from xlumina_gb300 import engine
    plane = lambda: _planes(rng, (ny, nx), off, "float32")   # noqa: E731
    lp = engine.op_lp(0.37)
    return {"lp": lambda: [lp], "lp0": lambda: [engine.op_lp(0.0)], "lcd_lp": lambda: [engine.op_lcd(plane(), plane()), lp],
            "lcd1_lp": lambda: [engine.op_lcd(0.7, 0.2), lp], "slm_lp": lambda: [engine.op_sslm(plane(), plane()), lp],
            "lp_lp": lambda: [engine.op_lp(-0.9), lp], "amp_lcd_lp": lambda: [
                engine.op_sslm_amp(plane(), plane(), plane(), 0.5), engine.op_lcd(plane(), 0.1), lp],
            "lp_pixel": lambda: [engine.op_lp(plane())], "lp_lcd": lambda: [lp, engine.op_lcd(plane(), plane())]}[kind]()


def _check(fields, x, y, z, ops, ny, nx, **kw):
    import torch

    from xlumina_gb300 import engine
    B = fields[0].shape[0] if fields[0].dim() == 3 else 1
    got = engine.RsCall(fields, x, y, 0.633, z, vector=True, pre=ops, **kw).run()
    # the ops are pixelwise on Ex, Ey (Ez, if any, is derived from them)
    flat = engine.apply_ops([f.contiguous() for f in fields] + [torch.zeros_like(fields[0]).contiguous()], ops, ny, nx)[:2]
    want = engine.RsCall(flat, x, y, 0.633, z, vector=True).run()
    norm = sum(float(w.to(torch.complex128).norm()) ** 2 for w in want) ** 0.5
    assert B >= 1 and norm > 0
    for g, w in zip(got, want):
        assert float((g.cpu().to(torch.complex128) - w.cpu().to(torch.complex128)).norm()) <= TOL * norm
    return got


@pytest.mark.parametrize("kind", ["lp", "lp0", "lcd_lp", "lcd1_lp", "slm_lp", "lp_lp", "amp_lcd_lp", "lp_pixel", "lp_lcd"])
@pytest.mark.parametrize("B,ny,nx,off", [(1, 2, 300, 0), (2, 301, 258, 1), (3, 70, 1025, 0), (1, 600, 2048, 1),
                                         (1, 2049, 30, 0), (1, 30, 2049, 0)])
def test_forms(kind, B, ny, nx, off):
    rng = np.random.default_rng(B + ny + nx)
    x, y = np.linspace(-1, 1, nx) * nx, np.linspace(-0.9, 0.9, ny) * ny
    ops = _program(kind, rng, ny, nx, off)
    fields = [_planes(rng, (B, ny, nx) if B > 1 else (ny, nx), off) for _ in range(2)]
    _check(fields, x, y, [3e4, -2e4, 3e4][:B] if B > 1 else 3e4, ops, ny, nx)


def test_shared_batch_outputs_and_capture():
    import torch

    from xlumina_gb300 import engine
    rng = np.random.default_rng(5)
    B, ny, nx = 3, 290, 310
    x, y = np.linspace(-1, 1, nx) * nx, np.linspace(-0.9, 0.9, ny) * ny
    ops = _program("lcd_lp", rng, ny, nx, 0)
    one = [_planes(rng, (ny, nx)) for _ in range(2)]
    shared = [f.expand(B, ny, nx) for f in one]
    zs = [3e4, 5e4, 4e4]
    first = [t.clone() for t in _check(shared, x, y, zs, ops, ny, nx)]
    pinned = [torch.empty((B, ny, nx), dtype=torch.complex64, pin_memory=True) for _ in range(3)]
    _check(shared, x, y, zs, ops, ny, nx, outs=pinned)
    torch.cuda.synchronize()
    assert all(torch.equal(p, f.cpu()) for p, f in zip(pinned, first))
    outs = [torch.empty_like(f) for f in first]
    call = engine.RsCall(shared, x, y, 0.633, zs, vector=True, pre=ops, outs=outs)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        call.run()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call.run()
    for o in outs:
        o.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(o, f) for o, f in zip(outs, first))
