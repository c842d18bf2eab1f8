"""Outputs of the propagation and its adjoint in the buffers of their inputs:
the buffer itself, or shifted by some rows and a 16-byte piece.  Same bits as
with buffers of their own."""
import ctypes

import numpy as np
import pytest
import torch

from lightne_gb300._lib import PropagateParams, PropagateStats
from lightne_gb300.api import PRECISIONS, Graph
from tests.test_spmm_balance_gpu import hub_graph

pytestmark = pytest.mark.gpu

N = 3000


def buffers(dim, shift):
    """An input and a buffer of its size that starts `shift` floats into it."""
    buf = torch.zeros(N * dim + 1024, device="cuda")
    return buf[:N * dim], buf[shift:shift + N * dim]


def ptr(t):
    return ctypes.c_void_p(t.data_ptr())


@pytest.mark.parametrize("precision", ["fp32", "bf16", "fp16"])
@pytest.mark.parametrize("order", [2, 3, 5])
@pytest.mark.parametrize("dim", [33, 128])
def test_outputs_over_inputs(ctx, lib, precision, order, dim):
    off, nbrs = hub_graph(N, [2800, 700, 100], 6)
    g = Graph.from_numpy(ctx, off, nbrs)
    gen = torch.Generator().manual_seed(dim)
    a = torch.randn(N * dim, generator=gen).cuda()
    gy = torch.randn(N * dim, generator=gen).cuda()
    p = PropagateParams(dim=dim, order=order, precision=PRECISIONS[precision], mu=0.2, s=0.5)

    def forward(x, out):
        y = torch.empty_like(x)
        torch.cuda.synchronize()
        assert lib.lne_propagate(ctx.handle, g.handle, ctypes.byref(p), ptr(x), ptr(y), ptr(out),
                                 ctypes.byref(PropagateStats())) == 0, lib.lne_last_error()
        ctx.synchronize()
        return y, out.clone()

    def adjoint(x, gx, out):
        dmu, ds = ctypes.c_double(), ctypes.c_double()
        torch.cuda.synchronize()
        assert lib.lne_propagate_adjoint(ctx.handle, g.handle, ctypes.byref(p), ptr(x), ptr(gx), ptr(out),
                                         ctypes.byref(dmu), ctypes.byref(ds),
                                         ctypes.byref(PropagateStats())) == 0, lib.lne_last_error()
        ctx.synchronize()
        return out.clone(), dmu.value, ds.value

    y0, a0 = forward(a, torch.empty_like(a))
    ga0, dmu0, ds0 = adjoint(a, gy, torch.empty_like(a))
    for shift in (0, 4, 3 * dim // 4 * 4 + 4):
        x, out = buffers(dim, shift)
        x.copy_(a)
        y1, a1 = forward(x, out)
        assert torch.equal(y0, y1) and torch.equal(a0, a1)
        x.copy_(a)
        ga1, dmu1, ds1 = adjoint(x, gy, out)
        assert torch.equal(ga0, ga1) and (dmu0, ds0) == (dmu1, ds1)
        x.copy_(gy)
        ga1, dmu1, ds1 = adjoint(a, x, out)
        assert torch.equal(ga0, ga1) and (dmu0, ds0) == (dmu1, ds1)
    g.free()
