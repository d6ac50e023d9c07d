"""Bounded waits that run out in the row kernels of the block engine: each form
that stages rows (scalar RS, VRS, VRS behind a polarizer, the VRS adjoint, chirp-z
of one and of three components) lets its copy land, frees what it holds, raises
the status word and returns; with the limit restored the same call gives what it
gave before."""
import ctypes

import numpy as np
import pytest

from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


def _call(kind, n):
    import torch

    from xlumina_gb300 import engine
    g = torch.Generator(device="cuda").manual_seed(n)
    x = np.linspace(-1.0, 1.0, n) * n
    xo = np.linspace(-0.2, 0.2, 400) * n
    f = [torch.randn((2, n, n), dtype=torch.complex64, device="cuda", generator=g) for _ in range(3)]
    eta = torch.rand((2, n, n), device="cuda", generator=g) * 6.0
    z = 60.0 * n
    if kind == "rs":
        return lambda: engine.rs_propagate(f[:1], x, x, 0.633, z, False, pre=[engine.op_phase(eta)])
    if kind == "vrs":
        return lambda: engine.rs_propagate(f[:2], x, x, 0.633, z, True, pre=[engine.op_lcd(eta, 0.4)])
    if kind == "polarizer":
        return lambda: engine.rs_propagate(f[:2], x, x, 0.633, z, True, pre=[engine.op_lcd(eta, 0.4), engine.op_lp(0.3)])
    if kind == "adjoint":
        return lambda: engine.RsCall(f, x, x, 0.633, z, True, adjoint=True).run()
    if kind == "czt":
        return lambda: engine.czt_propagate(f[:1], x, x, 0.633, z, xo, xo, "scalar", pre=[engine.op_phase(eta)])
    return lambda: engine.czt_propagate(f[:2], x, x, 0.633, z, xo, xo, "vczt", pre=[engine.op_lcd(eta, 0.4)])


# rows of a multiple of four samples, so that they are staged
@pytest.mark.parametrize("n", [700, 1024, 2048])
@pytest.mark.parametrize("kind", ["rs", "vrs", "polarizer", "adjoint", "czt", "vczt"])
def test_rows_return_when_their_wait_runs_out(kind, n):
    import torch

    from xlumina_gb300 import _lib, engine
    lib = engine.lib()
    call = _call(kind, n)
    flag, count = ctypes.c_uint(0), ctypes.c_uint(0)
    before = [t.cpu().numpy() for t in call()]
    _lib.check(lib.xl_device_timeouts(ctypes.byref(count), 1))
    try:
        _lib.check(lib.xl_set_wait_limit(0), "xl_set_wait_limit")
        call()
        torch.cuda.synchronize()
        _lib.check(lib.xl_device_timeouts(ctypes.byref(count), 1))
        assert count.value > 0
        with pytest.raises(_lib.XlError) as ei:
            _lib.check_device_status()
        assert ei.value.code == _lib.XL_ETIMEOUT
    finally:
        _lib.check(lib.xl_set_wait_limit(10 ** 9), "xl_set_wait_limit")
        lib.xl_device_status(ctypes.byref(flag), 1)
        lib.xl_device_timeouts(ctypes.byref(count), 1)
    for got, exp in zip(call(), before):
        assert rel_l2(got.cpu().numpy(), exp) < 1e-6
    torch.cuda.synchronize()
    _lib.check_device_status()
