"""lne_spmm where a row belongs to one warp whatever its length: operands so
wide that a product takes 4 GB of gathers or more, and matrices of 40M entries
or more.  Against FP64 products of the same operands, and, by column slabs
(each of them narrow enough for the balanced form), bit for bit against the
form in which long rows have several warps.

Tolerance: a strand adds at most 2048 terms one after the other in FP32, so
|err| <= (2048 + 16) 2^-24 (|A| |X|) elementwise."""
import ctypes

import pytest
import torch

from lightne_gb300._lib import LNE_PREC_BF16, LNE_PREC_FP8, LNE_PREC_FP16, LNE_PREC_FP32
from lightne_gb300.api import CSR
from tests.test_spmm_balance_gpu import BOUND, LENS, TYPES

pytestmark = pytest.mark.gpu


def matrix(n, nnz, seed):
    """Row pointer, columns and values on the device; rows of every length in
    LENS among rows that bring the total to nnz or a little more."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rest = nnz // (n - len(LENS)) + 1
    lens = torch.randint(rest, rest + 3, (n,), device="cuda", generator=gen)
    lens[torch.linspace(0, n - 1, len(LENS)).long().cuda()] = torch.tensor(LENS, device="cuda")
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    rp[1:] = torch.cumsum(lens, 0)
    total = int(rp[-1])
    assert total >= nnz
    # distinct columns in a row: a random start, then every 17th vertex (n is no multiple of 17)
    row = torch.repeat_interleave(torch.arange(n, device="cuda"), lens)
    start = torch.randint(0, n, (n,), device="cuda", generator=gen)
    col = (start[row] + 17 * (torch.arange(total, device="cuda") - rp[row])) % n
    return rp, col.int(), torch.randn(total, device="cuda", generator=gen)


def product(ctx, lib, A, prec, X, c0, d):
    """Columns c0 .. c0 + d of A X."""
    n, ld = X.shape
    Y = torch.full((n, d), 7.0, device="cuda")
    torch.cuda.synchronize()
    assert lib.lne_spmm(ctx.handle, A.handle, prec, ctypes.c_void_p(X.data_ptr() + c0 * X.element_size()), ld, d, 1.0, 0.0,
                        ctypes.c_void_p(Y.data_ptr()), d) == 0, lib.lne_last_error()
    ctx.synchronize()
    return Y


def check_fp64(rp, col, val, X, Y):
    n = rp.numel() - 1
    v = val.double()
    A = torch.sparse_csr_tensor(rp, col.long(), v, size=(n, n))
    Aabs = torch.sparse_csr_tensor(rp, col.long(), v.abs(), size=(n, n))
    for c in range(0, Y.shape[1], 512):
        Xd = X[:, c:min(c + 512, Y.shape[1])].double()
        assert ((Y[:, c:c + 512].double() - A @ Xd).abs() <= BOUND * (Aabs @ Xd.abs()) + 1e-30).all()


@pytest.mark.parametrize("prec", [LNE_PREC_FP32, LNE_PREC_BF16, LNE_PREC_FP16, LNE_PREC_FP8])
def test_wide_operands(ctx, lib, prec):
    """255 16-byte vectors: slabs of 128, 64, 32, 16, 8, 4, 2 and 1."""
    n, nnz = 6000, 1_000_000
    dtype = TYPES[prec]
    E = 16 // torch.empty(0, dtype=dtype).element_size()
    assert nnz * 255 * 16 >= 4e9 and 1.1 * nnz * 32 * 16 < 4e9
    rp, col, val = matrix(n, nnz, 1)
    X = torch.randn(n, 256 * E, device="cuda", generator=torch.Generator(device="cuda").manual_seed(2)).to(dtype)
    A = CSR.wrap_device(ctx, n, col.numel(), rp.data_ptr(), col.data_ptr(), val.data_ptr())
    Y = product(ctx, lib, A, prec, X, 0, 255 * E)
    check_fp64(rp, col, val, X, Y)
    assert torch.equal(Y, product(ctx, lib, A, prec, X, 0, 255 * E))
    c = 0
    for vecs in [32] * 7 + [16, 8, 4, 2, 1]:
        assert torch.equal(Y[:, c * E:(c + vecs) * E], product(ctx, lib, A, prec, X, c * E, vecs * E)), (c, vecs)
        c += vecs
    A.free()


@pytest.mark.parametrize("prec,d", [(LNE_PREC_FP32, 28), (LNE_PREC_FP32, 128), (LNE_PREC_FP16, 138), (LNE_PREC_BF16, 50),
                                    (LNE_PREC_FP8, 144), (LNE_PREC_FP8, 60)])
def test_many_entries(ctx, lib, prec, d):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n, nnz = 24000, 2048 * sms * 128  # a warp's share of the entries reaches four rows of 2048
    rp, col, val = matrix(n, nnz, 3)
    ld = (d + 15) // 16 * 16
    X = torch.randn(n, ld, device="cuda", generator=torch.Generator(device="cuda").manual_seed(4)).to(TYPES[prec])
    A = CSR.wrap_device(ctx, n, col.numel(), rp.data_ptr(), col.data_ptr(), val.data_ptr())
    Y = product(ctx, lib, A, prec, X, 0, d)
    check_fp64(rp, col, val, X, Y)
    assert torch.equal(Y, product(ctx, lib, A, prec, X, 0, d))
    A.free()
