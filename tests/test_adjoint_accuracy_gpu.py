"""dL/dmu and dL/ds of the propagation on graphs with a hub of thousands of
neighbours, where sums over the adjoint's vectors lose digits that sums over
the forward pass keep.

L = <g, y(a; mu, s)> with random a and g; the reference is an FP64 central
difference of the FP64 map (step 1e-5: truncation and rounding below 1e-9 of
the scale).  Errors are relative to |h a| (elementwise product, 2-norm), h =
(A + I) g, the size of one order's sum, and taken as root mean square over
eight draws, since a single draw can cancel.  An FP32 forward recursion with
the tangent, rows added as the device adds them (chunks of 2048, strands),
simulated in numpy on these graphs, is off by 9e-8 and 1.8e-7 (n = 20,000, 4
columns) and 1.2e-7 and 2.2e-7 (n = 6,000, 128 columns); the weights'
rounding to FP32 adds 3e-8 at most.  Bound: 5e-7.  The sums over the adjoint's
vectors are off by 8.0e-7 and 7.3e-7 at 128 columns (on the device 7.1e-7 and
6.0e-7)."""
import numpy as np
import pytest

from lightne_gb300.api import Graph, propagate_adjoint
from oracle import linalg_oracle as lo
from tests.test_spmm_balance_gpu import hub_graph

pytestmark = pytest.mark.gpu

MU, S, H = float(np.float32(0.2)), 0.5, 1e-5


def reference(off, nbrs, a, gy, order):
    """(dL/dmu, dL/ds, |h a|) in FP64."""
    a, gy = a.astype(np.float64), gy.astype(np.float64)

    def loss(mu, s):
        return float((lo.propagate(off, nbrs, a, order=order, mu=mu, s=s, narrow=False)[0] * gy).sum())

    src = np.repeat(np.arange(off.size - 1), np.diff(off))
    h = gy.copy()
    np.add.at(h, src, gy[nbrs])
    return ((loss(MU + H, S) - loss(MU - H, S)) / (2 * H), (loss(MU, S + H) - loss(MU, S - H)) / (2 * H),
            np.linalg.norm(h * a))


@pytest.mark.parametrize("precision", ["fp32", "fp16"])
@pytest.mark.parametrize("n,hub,dim", [(20000, 19000, 4), (6000, 5500, 128)])
def test_parameter_gradients_with_a_hub(ctx, precision, n, hub, dim):
    off, nbrs = hub_graph(n, [hub], 3)
    g = Graph.from_numpy(ctx, off, nbrs)
    err = []
    for seed in range(8):
        rng = np.random.default_rng(seed)
        a = rng.standard_normal((n, dim)).astype(np.float32)
        gy = rng.standard_normal((n, dim)).astype(np.float32)
        mu_ref, s_ref, scale = reference(off, nbrs, a, gy, 10)
        _, dmu, ds = propagate_adjoint(ctx, g, a, gy, dim, order=10, mu=MU, s=S, precision=precision)
        err.append([(dmu - mu_ref) / scale, (ds - s_ref) / scale])
    rms = np.sqrt((np.array(err) ** 2).mean(0))
    print("relative errors of dL/dmu, dL/ds:", rms)
    assert (rms <= 5e-7).all(), rms
    g.free()


@pytest.mark.parametrize("dim", [5, 8])
def test_parameter_gradients_of_a_large_gradient(ctx, dim):
    """An output gradient whose sum over a hub's neighbours is above FP32's
    range: the FP16 form's scale keeps the parameter gradients finite.  Bound:
    FP32 rounding through 20 products and 20 sums of one sign, 1e-5 of |h a|."""
    off, nbrs = hub_graph(2000, [1900], 3)
    g = Graph.from_numpy(ctx, off, nbrs)
    rng = np.random.default_rng(dim)
    a = (1e-3 * rng.standard_normal((2000, dim))).astype(np.float32)
    gy = (1e37 * rng.uniform(0.5, 1.0, (2000, dim))).astype(np.float32)
    mu_ref, s_ref, scale = reference(off, nbrs, a, gy, 6)
    _, dmu, ds = propagate_adjoint(ctx, g, a, gy, dim, order=6, mu=MU, s=S, precision="fp16")
    assert abs(dmu - mu_ref) <= 1e-5 * scale and abs(ds - s_ref) <= 1e-5 * scale, (dmu, mu_ref, ds, s_ref)
    g.free()
