"""The FP64 Jacobi sweeps' rotation test |x.y| > tol sqrt(x.x y.y) at the
limit itself, in both forms above 160 columns (dataflow up to 512, cluster
above).  One pair of columns is not orthogonal, with x.x, y.y and x.y exact
or rounded once, so that the limit is known to the last bit: x.y on the limit
leaves the matrix alone (one sweep), the next number above it is rotated."""
import numpy as np
import pytest

from lightne_gb300.api import core_svd

pytestmark = pytest.mark.gpu


def matrix(r, t, b, g):
    """Columns x = e0 + t e2, y = g e0 + b e1, 0, e3, e4, ..."""
    C = np.eye(r)
    C[0, 0], C[2, 0], C[2, 2] = 1.0, t, 0.0
    C[0, 1], C[1, 1] = g, b
    return C


@pytest.mark.parametrize("r", [161, 256, 257, 512, 513])
def test_rotation_at_the_limit(ctx, r):
    tol = max(1e-15, 2.220446049250313e-16 * np.sqrt(float(r)))
    rng = np.random.default_rng(r)
    sides = {-1: 0, 1: 0}  # cases where the product of the rounded roots lies below and above
    while min(sides.values()) < 3:
        t, b = rng.uniform(0.5, 2.0, 2)
        xx, yy = 1.0 + t * t, b * b
        limit = tol * np.sqrt(xx * yy)
        side = int(np.sign(tol * np.sqrt(xx) * np.sqrt(yy) - limit))
        if side == 0 or sides[side] == 3:
            continue
        sides[side] += 1
        for g, rotated in ((limit, False), (np.nextafter(limit, 1.0), True)):
            _, _, (sweeps, _) = core_svd(ctx, matrix(r, t, b, g))
            assert (sweeps > 1) == rotated, (t, b, g, sweeps)
