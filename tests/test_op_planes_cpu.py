"""Mask parameters of one device where some have a plane for every batch entry and
others one plane for all: the kernels read every plane of an op with one batch
stride, so the shared one is laid out for every entry; too few planes for the
batch are refused.  The addresses that a launch gets are read back on the host."""
import ctypes

import numpy as np
import pytest
import torch

NY, NX = 3, 5


def _rows(op, slot, batch):
    """What a launch reads for every entry of a slot."""
    n = NY * NX
    buf = (ctypes.c_float * (n * (op.pbstride // n * (batch - 1) + 1))).from_address(op.ptr[slot])
    a = np.frombuffer(buf, dtype=np.float32)
    return [a[b * op.pbstride:b * op.pbstride + n].reshape(NY, NX) for b in range(batch)]


@pytest.mark.parametrize("batched", [(0,), (1,), (0, 2), (1, 2, 3)])
@pytest.mark.parametrize("single", ["plane", "(1, ny, nx)", "one value"])
def test_shared_planes_beside_planes_per_entry(batched, single):
    from xlumina_gb300 import _lib, engine
    B = 4
    shape = {"plane": (NY, NX), "(1, ny, nx)": (1, NY, NX), "one value": (1,)}[single]
    params = [torch.rand((B, NY, NX) if i in batched else shape) for i in range(4)]
    op = engine.JonesOp(_lib.OP_SSLM_AMP, params)
    prog = _lib.XlProg()
    engine.fill_prog(prog, [op], NY, NX, B)
    held = {t.data_ptr(): t for t in list(op.copies.values()) + list(op.planes.values()) + params}
    for i, p in enumerate(params):
        assert held[prog.ops[0].ptr[i]].numel() == B * NY * NX      # nothing is read past it
        exp = np.broadcast_to(p.numpy(), (B, NY, NX)) if p.dim() > 1 else np.full((B, NY, NX), p.numpy()[0])
        for got, e in zip(_rows(prog.ops[0], i, B), exp):
            assert np.array_equal(got, e)


def test_too_few_planes_are_refused():
    from xlumina_gb300 import _lib, engine
    prog = _lib.XlProg()
    two, three = torch.rand(2, NY, NX), torch.rand(3, NY, NX)
    with pytest.raises(ValueError):
        engine.fill_prog(prog, [engine.JonesOp(_lib.OP_PHASE, [two])], NY, NX, 3)
    with pytest.raises(ValueError):
        engine.fill_prog(prog, [engine.JonesOp(_lib.OP_SSLM, [two, three])], NY, NX, 2)
    with pytest.raises(ValueError):
        engine.fill_prog(prog, [engine.JonesOp(_lib.OP_CMUL, ptrs=[two.to(torch.complex64)])], NY, NX, 3)
    engine.fill_prog(prog, [engine.JonesOp(_lib.OP_PHASE, [three])], NY, NX, 2)   # the first two are read
    assert prog.ops[0].pbstride == NY * NX
