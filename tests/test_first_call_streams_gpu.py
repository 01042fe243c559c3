"""A handle's first call of each kind, which clears its new buffers on the
handle's own stream, made on a caller's stream: it gives what the handle's own
stream gives, on host and on device arrays."""
import numpy as np
import pytest

from nwgraph_b200 import Graph, graphs as G

pytestmark = pytest.mark.gpu

RMAT = G.rmat(18, 16, 3)
W = G.edge_weights(RMAT.nnz, seed=3)
X = np.random.default_rng(2).standard_normal(RMAT.n).astype(np.float32)
T = np.random.default_rng(1).uniform(0.1, 1.0, (RMAT.n, 3)).astype(np.float32)


def _adjoint(g, on, stream):
    r, dw, dt = on(np.full(RMAT.n, 1.0 / RMAT.n, np.float32)), on(np.empty(RMAT.nnz, np.float32)), on(np.empty(RMAT.n, np.float32))
    g.page_rank_vjp(r, on(X), dw, dt, 0.85, 1.0, 60, stream=stream)
    return [dw, dt]


def _teleports(g, on, stream):
    out = on(np.empty((RMAT.n, 3), np.float32))
    g.weighted_page_rank_batched(on(T), out, 0.85, 1e-5, 50, stream=stream)
    return [out]


def _weighted(g, on, stream):
    out = on(np.empty(RMAT.n, np.float32))
    g.weighted_page_rank(None, out, 0.85, 1e-5, 50, stream=stream)
    return [out]


def _spmv(g, on, stream):
    y = on(np.empty(RMAT.n, np.float32))
    g.spmv(on(X), y, stream=stream)
    return [y]


@pytest.mark.parametrize("device", [False, True], ids=["host", "device"])
@pytest.mark.parametrize("call", [_adjoint, _teleports, _weighted, _spmv])
def test_first_call_on_a_callers_stream(gpu, call, device):
    import torch

    def on(a):
        return torch.from_numpy(a).cuda() if device else a

    def back(a):
        return a.cpu().numpy() if device else a

    with Graph(RMAT.row_ptr, RMAT.col, weights=W) as g:
        torch.cuda.synchronize()
        want = [back(a) for a in call(g, on, None)]
    s = torch.cuda.Stream()
    with Graph(RMAT.row_ptr, RMAT.col, weights=W) as g, torch.cuda.stream(s):  # inputs made on s too
        got = [back(a) for a in call(g, on, s)]
    for a, b in zip(got, want):
        assert np.array_equal(a, b, equal_nan=True)
