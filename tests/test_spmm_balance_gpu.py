"""The SpMM's work list at its edges: rows just below, at and above the
lengths where a row changes hands (a warp, several warps, several chunks), in
every lane layout, and the parameter gradients whose sums its epilogues take.

Tolerance of the products: a strand adds at most 2048 terms one after the
other in FP32, so |err| <= (2048 + 16) 2^-24 (|A| |X|) elementwise."""
import ctypes

import numpy as np
import pytest
import scipy.sparse as sp
import torch

from lightne_gb300 import graphs
from lightne_gb300._lib import LNE_PREC_BF16, LNE_PREC_FP8, LNE_PREC_FP16, LNE_PREC_FP32
from lightne_gb300.api import CSR, Graph, chebyshev_expansion, propagate_adjoint
from oracle import linalg_oracle as lo
from tests.test_adjoint_gpu import dense_forward

pytestmark = pytest.mark.gpu

LENS = [0, 1, 31, 32, 33, 63, 64, 65, 127, 128, 129, 511, 512, 513, 2047, 2048, 2049, 4096, 4097]
TYPES = {LNE_PREC_FP32: torch.float32, LNE_PREC_BF16: torch.bfloat16, LNE_PREC_FP8: torch.float8_e4m3fn,
         LNE_PREC_FP16: torch.float16}
BOUND = (2048 + 16) * 2.0 ** -24


@pytest.mark.parametrize("prec,d", [(LNE_PREC_FP32, 3), (LNE_PREC_FP32, 8), (LNE_PREC_FP32, 33), (LNE_PREC_FP32, 64),
                                    (LNE_PREC_FP32, 160), (LNE_PREC_FP32, 256), (LNE_PREC_FP16, 7), (LNE_PREC_FP16, 50),
                                    (LNE_PREC_FP16, 128), (LNE_PREC_BF16, 264), (LNE_PREC_FP8, 40), (LNE_PREC_FP8, 256)])
def test_row_lengths(ctx, lib, prec, d):
    n = 5000
    rng = np.random.default_rng(d)
    lens = rng.integers(0, 4, n)
    lens[np.linspace(0, n - 1, len(LENS)).astype(int)] = LENS  # first and last rows among them
    rp = np.zeros(n + 1, np.int64)
    np.cumsum(lens, out=rp[1:])
    col = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in lens]).astype(np.int32)
    val = rng.standard_normal(rp[-1]).astype(np.float32)
    ld = (d + 15) // 16 * 16
    X = torch.zeros(n, ld)
    X[:, :d] = torch.from_numpy(rng.standard_normal((n, d)).astype(np.float32))
    dX = X.to(TYPES[prec]).cuda()
    d_rp, d_col, d_val = (torch.from_numpy(a).cuda() for a in (rp, col, val))
    A = CSR.wrap_device(ctx, n, int(rp[-1]), d_rp.data_ptr(), d_col.data_ptr(), d_val.data_ptr())
    out = []
    for _ in range(2):
        Y = torch.full((n, d), 7.0, device="cuda")
        torch.cuda.synchronize()
        assert lib.lne_spmm(ctx.handle, A.handle, prec, ctypes.c_void_p(dX.data_ptr()), ld, d, 1.0, 0.0,
                            ctypes.c_void_p(Y.data_ptr()), d) == 0, lib.lne_last_error()
        ctx.synchronize()
        out.append(Y.cpu().numpy())
    Xd = dX.cpu().to(torch.float64).numpy()[:, :d]
    Am = sp.csr_matrix((val.astype(np.float64), col, rp), shape=(n, n))
    assert (np.abs(out[0] - Am @ Xd) <= BOUND * (abs(Am) @ np.abs(Xd)) + 1e-30).all()
    assert np.array_equal(out[0], out[1])
    A.free()


def hub_graph(n, degrees, seed):
    """Random sparse graph whose first vertices have about the given degrees."""
    rng = np.random.default_rng(seed)
    lo_, hi_ = [rng.integers(0, n, 3 * n)], [rng.integers(0, n, 3 * n)]
    for i, k in enumerate(degrees):
        lo_.append(np.full(k, i))
        hi_.append(rng.choice(n, k, replace=False))
    a, b = np.concatenate(lo_), np.concatenate(hi_)
    keep = a != b
    key = np.unique(np.minimum(a, b)[keep].astype(np.int64) * n + np.maximum(a, b)[keep])
    return graphs.csr_from_edges(n, key // n, key % n)


@pytest.mark.parametrize("precision,tol", [("fp32", 1e-5), ("fp16", 1e-3), ("bf16", 1e-2)])
@pytest.mark.parametrize("dim", [4, 33, 128, 136])
def test_propagate_hubs(ctx, precision, tol, dim):
    off, nbrs = hub_graph(6000, [5500, 2040, 600, 500, 60], 3)
    g = Graph.from_numpy(ctx, off, nbrs)
    a = np.random.default_rng(4).standard_normal((6000, dim)).astype(np.float32)
    y, a_out, _ = chebyshev_expansion(ctx, g, a, dim, order=5, precision=precision, return_a=True)
    ref, ref_a = lo.propagate(off, nbrs, a.astype(np.float64), order=5)
    for got, want in ((y, ref), (a_out, ref_a)):
        assert np.linalg.norm(got.double().cpu().numpy() - want) <= tol * np.linalg.norm(want)
    # a - conv may replace the input
    da = torch.from_numpy(a).cuda()
    y2, a2, _ = chebyshev_expansion(ctx, g, da, dim, order=5, precision=precision, return_a=True)
    assert torch.equal(y, y2) and torch.equal(a_out, a2)
    g.free()


@pytest.mark.parametrize("precision", ["fp32", "fp16"])
@pytest.mark.parametrize("order,dim", [(1, 8), (2, 5), (3, 8), (4, 33)])
def test_parameter_gradients(ctx, precision, order, dim):
    """dL/dmu and dL/ds from the adjoint's own recursion, at the orders where
    it is shortest, against FP64 autograd (1e-4 relative)."""
    off, nbrs = hub_graph(700, [650, 300, 70], 8)
    g = Graph.from_numpy(ctx, off, nbrs)
    rng = np.random.default_rng(order)
    a, gy = rng.standard_normal((700, dim)), rng.standard_normal((700, dim))
    at = torch.tensor(a, requires_grad=True)
    mu = torch.tensor(0.2, dtype=torch.float64, requires_grad=True)
    s = torch.tensor(0.5, dtype=torch.float64, requires_grad=True)
    (dense_forward(off, nbrs, at, mu, s, order) * torch.tensor(gy)).sum().backward()
    ga, dmu, ds = propagate_adjoint(ctx, g, a.astype(np.float32), gy.astype(np.float32), dim, order=order,
                                    precision=precision)
    ref = at.grad.numpy()
    assert np.linalg.norm(ga.double().cpu().numpy() - ref) <= (1e-4 if precision == "fp32" else 1e-3) * np.linalg.norm(ref)
    # the sums' terms cancel: relative to the size of what is added
    scale = np.linalg.norm(gy) * np.linalg.norm(a)
    assert abs(dmu - mu.grad.item()) <= 1e-4 * abs(mu.grad.item()) + 1e-6 * scale, (dmu, mu.grad.item())
    assert abs(ds - s.grad.item()) <= 1e-4 * abs(s.grad.item()) + 1e-6 * scale, (ds, s.grad.item())
    g.free()


@pytest.mark.parametrize("precision", ["fp32", "fp16"])
def test_unaligned_input(ctx, precision):
    """Rows that are not on 16-byte boundaries take the padded copies: the
    same bits."""
    off, nbrs = hub_graph(900, [800, 100], 5)
    g = Graph.from_numpy(ctx, off, nbrs)
    buf = torch.randn(900 * 16 + 1, generator=torch.Generator().manual_seed(1)).cuda()
    a = buf[1:].view(900, 16)
    y, a_out, _ = chebyshev_expansion(ctx, g, a, 16, order=4, precision=precision, return_a=True)
    y2, a2, _ = chebyshev_expansion(ctx, g, a.clone(), 16, order=4, precision=precision, return_a=True)
    assert a.data_ptr() % 16 and torch.equal(y, y2) and torch.equal(a_out, a2)
    ga = propagate_adjoint(ctx, g, a, a, 16, order=4, precision=precision)
    ga2 = propagate_adjoint(ctx, g, a.clone(), a.clone(), 16, order=4, precision=precision)
    assert torch.equal(ga[0], ga2[0]) and ga[1:] == ga2[1:]
    g.free()
