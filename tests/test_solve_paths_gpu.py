"""Which kernels a plain solve runs, as the graph info reports it: small graphs
solve in one launch, larger ones sweep by sweep, with a finishing kernel where
the long rows are many. The tests that compare these paths with one another
(same ranks, bit for bit) compare nothing if a graph takes another path than
they mean."""
import numpy as np
import pytest

from nwgraph_b200 import Graph, graphs as G
from test_resident_gpu import KINDS, _graph

pytestmark = pytest.mark.gpu


def _kernels(rp, col, relabel=True, launch="graph"):
    n = len(rp) - 1
    out = np.empty(n, np.float32)
    with Graph(rp, col, relabel=relabel) as g:
        g.page_rank(np.ones(n, np.uint32), out, 0.85, 0.0, 2, launch=launch)
        return g.info()["kernels_per_sweep"]


@pytest.mark.parametrize("kind", KINDS)
def test_the_resident_tests_graphs_are_resident(gpu, kind):
    # (one vertex is not relabelled: the merge-path sweep)
    assert _kernels(*_graph(kind)) == (2 if kind == "one vertex" else 0)


def test_the_other_paths(gpu, monkeypatch):
    g = G.rmat(12, 16, 3)
    assert _kernels(g.row_ptr, g.col, launch="stream") == 1  # not looked at
    assert _kernels(g.row_ptr, g.col, relabel=False) == 2
    large = G.rmat(18, 16, 4)  # its rows do not fit the SMs' shared memory
    assert _kernels(large.row_ptr, large.col) == 1
    monkeypatch.setenv("NWGPU_SWEEP", "binned_hot")
    assert _kernels(g.row_ptr, g.col) == 1
    monkeypatch.setenv("NWGPU_SWEEP", "binned")  # the 256-thread shape
    assert _kernels(g.row_ptr, g.col) == 2
