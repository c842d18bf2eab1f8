"""The trunc-log kernel's row counters in shared memory, which it uses from
2048 distinct pairs per block on (16 blocks per SM): graphs with a few more
pairs than that and more vertices than the tables have slots (1024), so that
most vertices meet a slot that is taken, against the port, bit for bit."""
import numpy as np
import pytest
import torch

from lightne_gb300 import graphs
from lightne_gb300.api import Graph, generate_trunc_log_matrix_v2
from oracle import port

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("upper", [False, True])
@pytest.mark.parametrize("kind", ["star", "power law"])
def test_shared_row_counters(ctx, kind, upper):
    if kind == "star":  # one hub
        (off, nbrs), walk_len, ratio = graphs.star_graph(5000), 4, 200.0
    else:
        (off, nbrs), walk_len, ratio = graphs.chung_lu(9000, 60000, 2.1, seed=3), 10, 25.0
    args = dict(walk_len=walk_len, sample_ratio=ratio)
    (rp2, col2, val2), st2 = port.sparsify(off, nbrs, 7, tablesz=40_000_000, upper=int(upper), **args)
    g = Graph.from_numpy(ctx, off, nbrs)
    csr, st = generate_trunc_log_matrix_v2(ctx, g, seed=7, table_size=40_000_000, upper=upper, **args)
    blocks = 16 * torch.cuda.get_device_properties(0).multi_processor_count
    assert st["distinct"] == st2["distinct"] >= 2048 * blocks
    rp, col, val = csr.download()
    assert np.array_equal(rp, rp2) and np.array_equal(col, col2)
    assert np.array_equal(val.view(np.uint32), val2.view(np.uint32))
    csr.free()
    g.free()
