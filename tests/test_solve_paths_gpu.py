"""Which kernels a plain solve runs, as the graph info reports it: small graphs
solve in one launch, larger ones sweep by sweep, with a finishing kernel where
the long rows are many. The tests that compare these paths with one another
(same ranks, bit for bit) compare nothing if a graph takes another path than
they mean."""
import ctypes as C

import numpy as np
import pytest

from nwgraph_b200 import Graph, graphs as G
from nwgraph_b200 import _native as N
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
    # (one vertex is not relabelled: the merge-path sweep; "warp of chunks" has four rows of 16 times a CTA's share,
    # which the loop solves faster: test_rows_of_many_chunks_in_one_launch has its chunks)
    assert _kernels(*_graph(kind)) == {"one vertex": 2, "warp of chunks": 1}.get(kind, 0)


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


def _even_rows(n, per_row, band):
    """Rows of equal length; neighbours anywhere (band 0) or at most `band` ids on."""
    rng = np.random.default_rng(7)
    rp = (np.arange(n + 1, dtype=np.int64) * per_row).astype(np.uint32)
    if band:
        col = (np.repeat(np.arange(n), per_row) + rng.integers(1, band + 1, n * per_row)) % n
    else:
        col = rng.integers(0, n, n * per_row)
    return rp, col.astype(np.uint32)


def _hubs(lens, n, rest):
    rng = np.random.default_rng(8)
    rp = np.zeros(n + 1, np.uint32)
    rp[1:] = np.cumsum(np.concatenate([lens, np.full(n - len(lens), rest)]))
    return rp, rng.integers(0, n, int(rp[-1])).astype(np.uint32)


@pytest.mark.parametrize("make,kernels", [
    (lambda: _even_rows(1 << 17, 12, 0), 0),         # 10,600 entries a CTA, few past the hubs
    (lambda: _even_rows(1 << 17, 32, 0), 1),         # 28,300, three quarters past them: the loop is 1.1 times as fast
    (lambda: _even_rows(600000, 6, 0), 1),           # 24,300, nearly all past them: 1.2 times
    (lambda: _even_rows(1 << 18, 14, 30), 0),        # 24,800, but neighbours share sectors
    (lambda: _hubs([34000] * 4, 70000, 3), 1),       # one CTA has fourteen times the average: 1.4 times
    (lambda: _hubs([14000] * 4, 70000, 3), 0),       # six times, but few
])
def test_graphs_the_sweep_loop_solves_faster_keep_it(gpu, make, kernels):
    rp, col = make()
    n = len(rp) - 1
    deg = np.bincount(col, minlength=n).astype(np.uint32)
    a, b = np.empty(n, np.float32), np.empty(n, np.float32)
    with Graph(rp, col) as g:
        sa = g.page_rank(deg, a, 0.85, 1e-6, 20)
        assert g.info()["kernels_per_sweep"] == kernels
        sb = g.page_rank(deg, b, 0.85, 1e-6, 20, launch="stream")
    assert np.array_equal(a, b, equal_nan=True) and sa.iterations == sb.iterations


def test_rows_of_many_chunks_in_one_launch(gpu, monkeypatch):
    """Rows of 32 and more chunks, which the last case above but one leaves to the loop at the default cut-offs."""
    rp, col = _hubs([8191, 8192, 8193, 12000, 16385], 70000, 3)
    n = len(rp) - 1
    deg = np.bincount(col, minlength=n).astype(np.uint32)
    a, b = np.empty(n, np.float32), np.empty(n, np.float32)
    monkeypatch.setenv("NWGPU_CHUNK_ENTRIES", "256")
    with Graph(rp, col) as g:
        sa = g.page_rank(deg, a, 0.85, 1e-6, 20)
        assert g.info()["kernels_per_sweep"] == 0
        sb = g.page_rank(deg, b, 0.85, 1e-6, 20, launch="stream")
    assert np.array_equal(a, b, equal_nan=True) and sa.iterations == sb.iterations


@pytest.mark.parametrize("edge_factor,kernels", [(20, 0), (28, 1)])  # hubs beside the rows, or no room for them
def test_hubs_without_room(gpu, edge_factor, kernels):
    g = G.rmat(17, edge_factor, 5)
    assert _kernels(g.row_ptr, g.col) == kernels


@pytest.mark.parametrize("rows,per_row,kernels", [
    (5333, 4000, 1),   # 21,332 chunks: 47,997
    (5334, 4000, 2),
    (1000, 44000, 1),  # rows of 43 chunks: 48,000
    (1001, 44000, 2),
])
def test_finishing_work(gpu, monkeypatch, rows, per_row, kernels):
    """Both sides of the line between the last CTA and a kernel for the long rows: chunks + 5 rows, against 48,000. The
    ranks depend on neither."""
    rp, col = _hubs([per_row] * rows, 60000, 2)
    chunks = rows * -(-per_row // 1024)
    assert (chunks + 5 * rows <= 48000) == (kernels == 1)
    n = len(rp) - 1
    deg = np.bincount(col, minlength=n).astype(np.uint32)
    a, b = np.empty(n, np.float32), np.empty(n, np.float32)
    with Graph(rp, col) as g:
        sa = g.page_rank(deg, a, 0.85, 0.0, 7, record_errors=True)
        assert g.info()["kernels_per_sweep"] == kernels
        for launch in ("graph", "stream"):
            sb = g.page_rank(deg, b, 0.85, 0.0, 7, launch=launch, record_errors=True)
            assert np.array_equal(a, b) and np.array_equal(sa.errors, sb.errors)
    monkeypatch.setenv("NWGPU_SWEEP", "binned")  # the 256-thread shape has a finishing kernel always
    with Graph(rp, col) as g:
        g.page_rank(deg, b, 0.85, 0.0, 7)
    assert np.array_equal(a, b)


BATCH_MEMBER, TUNE_SHAPES = 0x20000000, 0x40000000  # nwgpu_graph_create's flags of a ragged batch's own graphs


@pytest.mark.parametrize("flags", [BATCH_MEMBER, BATCH_MEMBER | TUNE_SHAPES, BATCH_MEMBER | N.GRAPH_AUTOTUNE])
@pytest.mark.parametrize("tune_all", ["0", "1"])
def test_graphs_of_a_batch_keep_the_finishing_kernel(gpu, monkeypatch, flags, tune_all):
    """Whether they are tuned or not, and through every plan the tuner builds."""
    monkeypatch.setenv("NWGPU_AUTOTUNE", tune_all)
    g = G.rmat(18, 16, 4)
    assert _kernels(g.row_ptr, g.col) <= (1 if tune_all == "0" else 2)  # a graph of its own has none in the hot shape
    for _ in range(2):  # timed, then from the cache
        h = C.c_void_p()
        N.check(N.lib().nwgpu_graph_create(g.row_ptr.ctypes.data, g.col.ctypes.data, None, g.n, g.nnz, flags, C.byref(h)))
        info = N.GraphInfo()
        N.check(N.lib().nwgpu_graph_get_info(h, C.byref(info)))
        N.lib().nwgpu_graph_destroy(h)
        assert info.kernels_per_sweep == 2


def test_device_ms_is_the_sweeps(gpu):
    """Also where one launch reads the degrees, sweeps and writes the ranks: 1 sweep takes what each of 40 takes (the
    launch's start and end take about 20 us, a sweep 14), and no sweep takes no time."""
    g = G.grid(1_000_000)
    deg = g.out_degree()
    out = np.empty(g.n, np.float32)
    with Graph(g.row_ptr, g.col) as h:
        per = {its: min(h.page_rank(deg, out, 0.85, -1.0, its).ms_per_iter for _ in range(9)) for its in (1, 40)}
        assert h.info()["kernels_per_sweep"] == 0
        none = h.page_rank(deg, out, 0.85, -1.0, 0)
        long = h.page_rank(deg, out, 0.85, -1.0, 4100)  # two launches
    print(per, long.ms_per_iter)
    assert 0.5 * per[40] < per[1] < 1.5 * per[40]
    assert 0.5 * per[40] < long.ms_per_iter < 1.5 * per[40]
    assert none.device_ms == 0.0 and none.ms_per_iter == 0.0
