"""The sampler's two forms (states ahead of the walks for graphs with few
directed entries, one lane per entry otherwise) on either side of the line
between them, and the small scans and histograms, against the port, bit for
bit."""
import numpy as np
import pytest
import torch

from lightne_gb300 import graphs
from lightne_gb300.api import Graph, generate_trunc_log_matrix_v2
from oracle import port

pytestmark = pytest.mark.gpu


def check(ctx, off, nbrs, **kw):
    g = Graph.from_numpy(ctx, off, nbrs)
    csr, st = generate_trunc_log_matrix_v2(ctx, g, seed=7, walk_len=kw["walk_len"], table_size=kw["tablesz"],
                                           sample_ratio=kw["sample_ratio"])
    rp, col, val = csr.download()
    (rp2, col2, val2), _ = port.sparsify(off, nbrs, 7, **kw)
    assert np.array_equal(rp, rp2) and np.array_equal(col, col2)
    assert np.array_equal(val.view(np.uint32), val2.view(np.uint32))
    csr.free()
    g.free()


@pytest.mark.parametrize("side", [-1, 0, 1])
def test_either_side_of_the_line(ctx, side):
    lanes = torch.cuda.get_device_properties(0).multi_processor_count * 6 * 256
    m = lanes // 6 + side  # directed entries 2 m: 3 * 2 m against the lanes
    off, nbrs = graphs.chung_lu(9000, m, 2.1, seed=12)
    check(ctx, off, nbrs, walk_len=10, sample_ratio=0.3, tablesz=2_000_000)


@pytest.mark.parametrize("walk_len,ratio", [(1, 1.0), (2, 0.01), (10, 1.7), (64, 0.2), (65, 0.2), (200, 0.05)])
def test_walk_lengths(ctx, walk_len, ratio):
    off, nbrs = graphs.chung_lu(300, 1500, 2.1, seed=5)
    check(ctx, off, nbrs, walk_len=walk_len, sample_ratio=ratio, tablesz=600_000)


@pytest.mark.parametrize("n", [4096, 16384, 16385])
def test_row_counts_around_a_scan(ctx, n):
    i = np.arange(n - 1)
    off, nbrs = graphs.csr_from_edges(n, i, i + 1)
    check(ctx, off, nbrs, walk_len=3, sample_ratio=0.5, tablesz=3_000_000)


@pytest.mark.parametrize("n", [900, 1025, 5000])
def test_row_counts_around_a_hub(ctx, n):
    """Every pair's walk passes the hub; more vertices than the blocks' counting
    tables have slots, and fewer."""
    off, nbrs = graphs.star_graph(n)
    check(ctx, off, nbrs, walk_len=4, sample_ratio=3.0, tablesz=3_000_000)
