"""Batches of different widths on one handle: each must give what a handle of
its own gives, bit for bit, and once the widest has been seen the handle holds
no more and no less memory, whatever widths and kinds of batch follow (nothing
is given back and made anew)."""
import numpy as np
import pytest

from nwgraph_b200 import Graph, graphs as G

pytestmark = pytest.mark.gpu

SMALL = G.rmat(11, 16, 3)  # weighted batches: padded to 8, 16, 32, 64, 128; unweighted ones to 32, 64, 128
LARGE = G.rmat(17, 16, 3)  # 3.7M entries: unweighted batches are padded to 8 and 16 too


def _inputs(g, k):
    rng = np.random.default_rng(k)
    t = rng.uniform(0.1, 1.0, (g.n, k)).astype(np.float32)
    deg = g.out_degree()
    seeds = rng.choice(np.flatnonzero(deg), k).astype(np.uint32)
    return deg, seeds, np.ascontiguousarray(t / t.sum(axis=0, keepdims=True))


def _run(h, g, kind, k, damping=0.85):
    deg, seeds, t = _inputs(g, k)
    out = np.empty((g.n, k), np.float32)
    if kind == "seeds":
        st = h.ppr_batched(deg, seeds, out, damping, 1e-5, 60)
    elif kind == "teleports":
        st = h.ppr_batched_teleports(deg, t, out, damping, 1e-5, 60)
    else:
        st = h.weighted_page_rank_batched(t, out, damping, 1e-5, 60)
    return out, st.col_iterations


@pytest.mark.parametrize("g,kinds,widths", [
    (SMALL, ["weighted", "seeds", "teleports"], [3, 12, 20, 40, 100, 6, 20, 128, 1, 64, 9]),
    (LARGE, ["seeds", "teleports"], [6, 12, 20, 6, 12, 33, 8, 20, 1]),
], ids=["small", "large"])
def test_widths_in_turn(gpu, g, kinds, widths):
    w = G.edge_weights(g.nnz, seed=2) if "weighted" in kinds else None
    with Graph(g.row_ptr, g.col, weights=w) as h:
        held = None
        for turn in range(2):
            for i, k in enumerate(widths):
                kind = kinds[(i + turn) % len(kinds)]
                damping = 0.85 if i % 4 else 0.5
                got, iters = _run(h, g, kind, k, damping)
                with Graph(g.row_ptr, g.col, weights=w) as own:
                    want, own_iters = _run(own, g, kind, k, damping)
                assert np.array_equal(got, want, equal_nan=True), (kind, k)
                assert np.array_equal(iters, own_iters)
                if held is not None:
                    assert h.info()["device_bytes"] == held, (kind, k)
            held = h.info()["device_bytes"]
