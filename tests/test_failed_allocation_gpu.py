"""A call that runs out of memory while it sets up its buffers fails with
NWGPU_ERR_OUT_OF_MEMORY, and the next call on the handle starts over: every
allocation of every first call in turn is made to fail, and the call after it
must give what an undisturbed handle gives, bit for bit, and hold as much."""
import numpy as np
import pytest

from nwgraph_b200 import Graph, NwgpuError, graphs as G
from nwgraph_b200 import _native as N

pytestmark = pytest.mark.gpu

RMAT = G.rmat(10, 16, 3)
DEG = RMAT.out_degree()
W = G.edge_weights(RMAT.nnz, seed=3)
T = np.random.default_rng(1).uniform(0.1, 1.0, (RMAT.n, 12)).astype(np.float32)
X = np.random.default_rng(2).standard_normal(RMAT.n).astype(np.float32)
SEEDS = np.arange(12, dtype=np.uint32)


def _solve(g):
    out = np.empty(RMAT.n, np.float32)
    g.page_rank(DEG, out, 0.85, 1e-6, 50)
    return [out]


def _loop(g):
    out = np.empty(RMAT.n, np.float32)
    g.page_rank(DEG, out, 0.85, 1e-6, 50, launch="stream")
    return [out]


def _seeds(g):
    out = np.empty((RMAT.n, 12), np.float32)
    g.ppr_batched(DEG, SEEDS, out, 0.85, 1e-6, 50)
    return [out]


def _weighted(g):
    out = np.empty(RMAT.n, np.float32)
    g.weighted_page_rank(None, out, 0.85, 1e-6, 50)
    return [out]


def _teleports(g):
    out = np.empty((RMAT.n, 12), np.float32)
    g.weighted_page_rank_batched(T, out, 0.85, 1e-6, 50)
    return [out]


def _adjoint(g):
    dw, dt = np.empty(RMAT.nnz, np.float32), np.empty(RMAT.n, np.float32)
    g.page_rank_vjp(T[:, 0].copy(), X, dw, dt, 0.85, 1e-4, 100)
    return [dw, dt]


def _spmv(g):
    y = np.empty(RMAT.n, np.float32)
    g.spmv(X, y)
    return [y]


@pytest.mark.parametrize("relabel", [True, False])
@pytest.mark.parametrize("call", [_solve, _loop, _seeds, _weighted, _teleports, _adjoint, _spmv])
def test_the_call_after_a_failed_one(gpu, call, relabel):
    weighted = call in (_weighted, _teleports, _adjoint, _spmv)
    if weighted and not relabel:
        pytest.skip("weighted solves need a relabelled graph")

    def graph():
        return Graph(RMAT.row_ptr, RMAT.col, weights=W if weighted else None, relabel=relabel)

    with graph() as g:
        want = call(g)
        held = g.info()["device_bytes"]
    failed = 0
    try:
        for after in range(200):
            with graph() as g:
                N.lib().nwgpu_selftest_fail_allocation(after)
                try:
                    call(g)
                    break  # the call makes no more than `after` allocations
                except NwgpuError as e:
                    assert e.status == N.ERR_OUT_OF_MEMORY
                    failed += 1
                N.lib().nwgpu_selftest_fail_allocation(-1)
                for a, b in zip(call(g), want):
                    assert np.array_equal(a, b, equal_nan=True), after
                if call is not _solve:  # (whose retry may go without the small-graph plan)
                    assert g.info()["device_bytes"] == held, after
    finally:
        N.lib().nwgpu_selftest_fail_allocation(-1)
    assert 10 <= failed < 200


def test_no_memory_for_the_small_graph_plan(gpu):
    """The plan of the one-launch solve is an extra: without memory for it the first solve runs the sweep loop."""
    out, want = np.empty(RMAT.n, np.float32), np.empty(RMAT.n, np.float32)
    solve_buffers = 12  # ensure_solve_buffers' allocations, before the plan's four
    try:
        for after in range(solve_buffers, solve_buffers + 5):
            with Graph(RMAT.row_ptr, RMAT.col) as g, Graph(RMAT.row_ptr, RMAT.col) as loop:
                loop.page_rank(DEG, want, 0.85, 1e-6, 50, launch="stream")
                N.lib().nwgpu_selftest_fail_allocation(after)
                g.page_rank(DEG, out, 0.85, 1e-6, 50)
                N.lib().nwgpu_selftest_fail_allocation(-1)
                without = after < solve_buffers + 4
                assert g.info()["kernels_per_sweep"] == (1 if without else 0)
                assert not without or g.info()["device_bytes"] == loop.info()["device_bytes"]
                assert np.array_equal(out, want)
    finally:
        N.lib().nwgpu_selftest_fail_allocation(-1)
