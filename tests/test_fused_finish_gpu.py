"""Sweeps whose last CTA finishes the long rows, against the finishing kernel
(plans of more chunks than the fusing limit, the 256-thread shape) and the
launch modes: same ranks bit for bit, and every sweep count around the loop's
three sweeps per round."""
import numpy as np
import pytest

from nwgraph_b200 import Graph, graphs as G

pytestmark = pytest.mark.gpu


def _graph():
    """RMAT scale 18 is too large for the resident solve; with 256-entry chunks its long rows make tens of thousands."""
    g = G.rmat(18, 16, 4)
    return g.row_ptr, g.col, g.out_degree()


def test_launch_modes_and_shapes(gpu, monkeypatch):
    rp, col, deg = _graph()
    n = len(rp) - 1
    a, b = np.empty(n, np.float32), np.empty(n, np.float32)
    with Graph(rp, col) as g:
        for its in range(0, 8):
            sa = g.page_rank(deg, a, 0.85, 0.0, its, record_errors=True)
            sb = g.page_rank(deg, b, 0.85, 0.0, its, launch="stream", record_errors=True)
            assert np.array_equal(a, b) and sa.iterations == sb.iterations == its
            assert np.array_equal(sa.errors, sb.errors)
        for thr in (1e-2, 1e-3, 1e-4, 1e-5):
            sa = g.page_rank(deg, a, 0.85, thr, 100)
            sb = g.page_rank(deg, b, 0.85, thr, 100, launch="stream")
            assert np.array_equal(a, b) and sa.iterations == sb.iterations and sa.converged and sb.converged
    monkeypatch.setenv("NWGPU_SWEEP", "binned")
    with Graph(rp, col) as g:
        g.page_rank(deg, b, 0.85, 1e-5, 100)
        assert np.array_equal(a, b)


@pytest.mark.parametrize("its", [1, 8, 9, 32, 33, 70])
def test_first_loop_then_graph(gpu, its):
    """A handle's first loop launches its sweeps itself, and goes on with the loop graph after 32."""
    rp, col, deg = _graph()
    a, b = np.empty(len(deg), np.float32), np.empty(len(deg), np.float32)
    with Graph(rp, col) as g:
        s0 = g.page_rank(deg, a, 0.85, -1.0, its, record_errors=True)
        s1 = g.page_rank(deg, b, 0.85, -1.0, its, record_errors=True)
    assert np.array_equal(a, b) and s0.iterations == s1.iterations == its and np.array_equal(s0.errors, s1.errors)


def test_both_sides_of_the_chunk_limit(gpu, monkeypatch):
    """Rows of 257 to 300 entries, one or two chunks each: 2 x 16,384 chunks are finished by the last CTA, two more
    are not. The ranks may depend on neither."""
    rng = np.random.default_rng(1)
    out = []
    for rows in (16384, 16385):
        lens = np.concatenate([rng.integers(257, 301, rows), np.full(40000, 2)])
        n = len(lens)
        rp = np.zeros(n + 1, np.uint32)
        rp[1:] = np.cumsum(lens)
        col = np.random.default_rng(2).integers(0, n, int(rp[-1])).astype(np.uint32)
        deg = np.bincount(col, minlength=n).astype(np.uint32)
        monkeypatch.setenv("NWGPU_LONG_ROW", "256")
        monkeypatch.setenv("NWGPU_CHUNK_ENTRIES", "256")
        monkeypatch.setenv("NWGPU_SWEEP", "binned_hot")
        a, b = np.empty(n, np.float32), np.empty(n, np.float32)
        with Graph(rp, col) as g:
            assert g.info()["long_row_entries"] == 256
            st = g.page_rank(deg, a, 0.85, 0.0, 9)
        monkeypatch.setenv("NWGPU_SWEEP", "binned")
        with Graph(rp, col) as g:
            g.page_rank(deg, b, 0.85, 0.0, 9)
        assert st.iterations == 9 and np.array_equal(a, b)
        out.append(a)
    assert all(np.isfinite(x).all() for x in out)


def test_weighted_modes(gpu):
    rp, col, _ = _graph()
    n = len(rp) - 1
    w = G.edge_weights(len(col), seed=3)
    x = np.random.default_rng(5).standard_normal(n).astype(np.float32)
    y, a, b = (np.empty(n, np.float32) for _ in range(3))
    with Graph(rp, col, weights=w) as g:
        g.spmv(x, y)
        sa = g.weighted_page_rank(None, a, 0.85, 1e-6, 100)
        sb = g.weighted_page_rank(None, b, 0.85, 1e-6, 100, launch="stream")
    assert np.array_equal(a, b) and sa.iterations == sb.iterations
    rows = np.repeat(np.arange(n), np.diff(rp.astype(np.int64)))
    t = w.astype(np.float64) * x.astype(np.float64)[col]
    exact = np.bincount(rows, weights=t, minlength=n)
    mag = np.bincount(rows, weights=np.abs(t), minlength=n)
    assert np.all(np.abs(y - exact) <= 1e-6 * mag + 1e-30)
