"""The core SVD of a matrix that holds a NaN: its columns have norms that
compare with nothing, and every singular value and vector is written all the
same, the NaNs first."""
import numpy as np
import pytest

from lightne_gb300.api import core_svd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("r", [5, 160, 161, 256, 513])
def test_all_columns_are_written(ctx, r):
    C = np.random.default_rng(r).standard_normal((r, r))
    C[r // 2, r // 3] = np.nan
    U, S, _ = core_svd(ctx, C)
    U, S = U.cpu().numpy(), S.cpu().numpy()
    if r <= 160:  # the preconditioning multiplies by V, and the NaN's row with it
        assert np.isnan(S).all() and (U == 0.0).all()
        return
    # the sweeps leave pairs with the column alone and diagonalise the others
    assert np.isnan(S[0]) and (U[:, 0] == 0.0).all()
    ref = np.linalg.svd(np.delete(C, r // 3, axis=1), compute_uv=False)
    assert np.abs(S[1:] - ref).max() <= 1e-12 * ref[0]
    assert np.abs(U[:, 1:].T @ U[:, 1:] - np.eye(r - 1)).max() <= 1e-12
