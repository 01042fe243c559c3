"""The resident solve of small graphs (one cooperative launch for all sweeps,
launch="graph") against the sweep loop of the binned kernel (launch="stream"):
same ranks bit for bit, same sweep counts and stopping, the same FP64 L1
changes up to their summation order (sums of at most 2^20 doubles: 1e-12)."""
import threading
import time

import numpy as np
import pytest

from nwgraph_b200 import Graph, NwgpuError, graphs as G

pytestmark = pytest.mark.gpu


def _from_lengths(lens, n=None, seed=1):
    rng = np.random.default_rng(seed)
    lens = np.asarray(lens)
    n = n or max(len(lens), 2)
    lens = np.concatenate([lens, np.zeros(n - len(lens), int)])
    rp = np.zeros(n + 1, np.uint32)
    rp[1:] = np.cumsum(lens)
    return rp, rng.integers(0, n, int(rp[-1])).astype(np.uint32)


def _graph(kind):
    if kind.startswith("rmat"):
        g = G.rmat(int(kind[4:]), 16, 5)
        return g.row_ptr, g.col
    if kind.startswith("grid"):
        g = G.grid(int(kind[4:]))
        return g.row_ptr, g.col
    rng = np.random.default_rng(2)
    return {
        "one vertex": lambda: _from_lengths([0], 1),
        "no entries": lambda: _from_lengths([0] * 5000),
        "bin edges": lambda: _from_lengths(np.repeat([1, 2, 4, 5, 8, 9, 16, 17, 32, 33, 64, 65, 127, 128, 129, 130, 255,
                                                      256, 257, 1023, 1024, 1025, 2047, 2048, 2049, 2050, 3071, 3073,
                                                      4097], 3)),
        "warp of chunks": lambda: _from_lengths([32767, 32769, 40000, 32768] + [3] * 70000),  # rows of 32 and 33+ chunks
        "empty tail": lambda: _from_lengths(rng.integers(0, 30, 3000), 200000),
    }[kind]()


KINDS = ["one vertex", "no entries", "bin edges", "warp of chunks", "empty tail", "rmat4", "rmat10", "rmat13", "rmat16",
         "rmat17", "grid9", "grid1000", "grid1000000"]


def _same(a, b, sa, sb):
    assert np.array_equal(a, b, equal_nan=True)
    assert (sa.iterations, sa.converged) == (sb.iterations, sb.converged)
    assert np.allclose(sa.errors, sb.errors, rtol=1e-12, atol=0, equal_nan=True)


def _check(kind):
    rp, col = _graph(kind)
    n = len(rp) - 1
    deg = np.bincount(col, minlength=n).astype(np.uint32)
    a, b = np.empty(n, np.float32), np.empty(n, np.float32)
    with Graph(rp, col) as g:
        for d, thr, its in [(0.85, 0.0, 7), (0.85, 1e-4, 100), (0.5, 1e-3, 30), (0.85, 0.0, 0), (0.85, 0.0, 1), (1.0, 1e-9, 6)]:
            sa = g.page_rank(deg, a, d, thr, its, record_errors=True)
            sb = g.page_rank(deg, b, d, thr, its, launch="stream", record_errors=True)
            _same(a, b, sa, sb)
        for seed in (0, n // 2, n - 1):
            sa = g.ppr(deg, seed, a, 0.85, 1e-6, 40, record_errors=True)
            sb = g.ppr(deg, seed, b, 0.85, 1e-6, 40, launch="stream", record_errors=True)
            _same(a, b, sa, sb)


@pytest.mark.parametrize("kind", KINDS)
def test_equals_the_sweep_loop(gpu, kind):
    _check(kind)


@pytest.mark.parametrize("rows,long_row,chunk", [("1", "2048", "1024"), ("2", "256", "256"), ("1", "512", "256"),
                                                 ("2", "8192", "2048")])
def test_plan_settings(gpu, monkeypatch, rows, long_row, chunk):
    monkeypatch.setenv("NWGPU_BIN0_ROWS", rows)
    monkeypatch.setenv("NWGPU_LONG_ROW", long_row)
    monkeypatch.setenv("NWGPU_CHUNK_ENTRIES", chunk)
    for kind in ("bin edges", "rmat13", "warp of chunks"):
        _check(kind)


def test_device_arrays_streams_and_repeats(gpu):
    import torch
    g0 = G.rmat(12, 16, 3)
    deg = g0.out_degree()
    ref = np.empty(g0.n, np.float32)
    d = torch.from_numpy(deg.view(np.int32)).cuda()
    out = torch.empty(g0.n, dtype=torch.float32, device="cuda")
    s = torch.cuda.Stream()
    with Graph(g0.row_ptr, g0.col) as g:
        g.page_rank(deg, ref, 0.85, 1e-5, 50, launch="stream")
        for k in range(5):  # the two arrival counters take turns
            out.fill_(-1.0)
            torch.cuda.synchronize()
            g.page_rank(d, out, 0.85, 1e-5, 50, stream=s if k % 2 else None)
            assert np.array_equal(out.cpu().numpy(), ref)


def test_more_sweeps_than_one_launch(gpu):
    g0 = G.rmat(8, 8, 3)
    deg = g0.out_degree()
    a, b = np.empty(g0.n, np.float32), np.empty(g0.n, np.float32)
    with Graph(g0.row_ptr, g0.col) as g:
        for its in (4096, 4097, 9001):
            sa = g.page_rank(deg, a, 0.85, -1.0, its)
            sb = g.page_rank(deg, b, 0.85, -1.0, its, launch="stream")
            assert np.array_equal(a, b) and sa.iterations == sb.iterations == its


def test_abort_ends_the_solve(gpu):
    g0 = G.rmat(10, 16, 3)
    deg = g0.out_degree()
    out = np.empty(g0.n, np.float32)
    with Graph(g0.row_ptr, g0.col) as g:
        g.page_rank(deg, out, 0.85, 0.0, 1)
        t = threading.Thread(target=lambda: (time.sleep(0.2), g.abort()))
        t.start()
        with pytest.raises(NwgpuError):
            g.page_rank(deg, out, 0.85, -1.0, 1 << 40)
        t.join()
        st = g.page_rank(deg, out, 0.85, 0.0, 3)  # the handle goes on
        assert st.iterations == 3
