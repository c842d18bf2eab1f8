"""Ranks above the narrow forms' limits: the FP64 Jacobi and the Cholesky
factorisation with the matrix spread over a cluster's shared memory (up to
512 columns) and the global-memory forms above it.

Tolerances: the core SVD's as tests/test_core_svd_gpu.py (1e-12 of the
largest singular value); the dense embedding's singular values 1e-5 relative
to the largest (FP32 products), its columns 1e-3 up to sign (spectrum with
ratios of 0.97: FP32 rounding over a relative gap of 0.03)."""
import numpy as np
import pytest
import torch

from lightne_gb300.api import core_svd, get_embedding_dense

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r", [161, 162, 255, 256, 257, 512, 513])
@pytest.mark.parametrize("kind", ["decay", "deficient", "repeated"])
def test_core_svd_wide(ctx, r, kind):
    rng = np.random.default_rng(r)
    sig = {"decay": np.logspace(0.0, -3.0, r), "repeated": np.repeat(np.linspace(1.0, 0.3, 8), (r + 7) // 8)[:r],
           "deficient": np.where(np.arange(r) < r // 3, np.exp(-np.arange(r) / r), 0.0)}[kind]
    q = [np.linalg.qr(rng.standard_normal((r, r)))[0] for _ in range(2)]
    C = (q[0] * sig) @ q[1].T
    U, S, (sweeps, _) = core_svd(ctx, C)
    U, S = U.cpu().numpy(), S.cpu().numpy()
    ref = np.sort(sig)[::-1]
    assert np.all(np.diff(S) <= 0.0)
    assert np.abs(S - ref).max() <= 1e-12
    keep = ref > 1e-10
    Uk = U[:, keep]
    assert np.abs(Uk.T @ Uk - np.eye(Uk.shape[1])).max() <= 1e-12
    assert np.abs(C @ (C.T @ Uk) - Uk * S[keep] ** 2).max() <= 1e-12
    assert 1 <= sweeps <= 60


def test_core_svd_scales(ctx):
    """Scaling by a power of two scales the singular values and nothing else."""
    rng = np.random.default_rng(9)
    C = rng.standard_normal((192, 192))
    U, S, sw = core_svd(ctx, C)
    for e in (-200, 300):
        U2, S2, sw2 = core_svd(ctx, C * 2.0 ** e)
        assert torch.equal(U, U2) and torch.equal(S * 2.0 ** e, S2) and sw == sw2


@pytest.mark.parametrize("d", [144, 145, 160, 161, 256, 257, 512, 520])
def test_dense_embedding_wide(ctx, d):
    rng = np.random.default_rng(d)
    n = 3000
    q = np.linalg.qr(rng.standard_normal((n, d)))[0]
    p = np.linalg.qr(rng.standard_normal((d, d)))[0]
    sig = np.maximum(0.97 ** np.arange(d), 1e-3 * (1.0 + np.arange(d)[::-1] / d))
    x = ((q * sig) @ p.T).astype(np.float32)
    emb, S = get_embedding_dense(ctx, x, d)
    Ur, Sr, _ = np.linalg.svd(x.astype(np.float64), full_matrices=False)
    assert np.abs(S - Sr).max() <= 1e-5 * Sr[0]
    ref = Ur * np.sqrt(Sr)
    ref /= np.linalg.norm(ref, axis=1, keepdims=True)
    got = emb.double().cpu().numpy()
    k = 60  # the columns before the spectrum flattens
    sign = np.sign(np.sum(got[:, :k] * ref[:, :k], axis=0))
    err = np.linalg.norm(got[:, :k] * sign - ref[:, :k], axis=0) / np.linalg.norm(ref[:, :k], axis=0)
    assert err.max() <= 1e-3, err.max()
