"""The batched gather with every lane group of every warp at work: enough tiles
that 16 groups of a warp (8 columns) walk tiles side by side and go on to
another round, in a graph whose rows without entries lie between the others.
Graphs of few tiles pad unweighted batches to 32 columns and use one group per
warp, so they do not reach this. Each column is summed in the same order at
every width, so a batch must equal the same columns of a wider batch, which the
warp-per-tile kernel sums, bit for bit; that one is checked in FP64."""
import numpy as np
import pytest
import scipy.sparse as sp

from nwgraph_b200 import Graph

pytestmark = pytest.mark.gpu
SWEEPS = 3
N = 600_000
D = 0.85


@pytest.fixture(scope="module")
def graph(gpu):
    import torch
    rng = np.random.default_rng(4)
    lens = np.where(rng.random(N) < 0.4, 0, rng.integers(1, 111, N))
    lens[rng.choice(N, 6, replace=False)] = [70000, 3000, 1023, 512, 511, 510]  # crossing tiles, ending on their edges
    lens[:3] = [0, 700, 0]
    lens[-2:] = [5, 0]
    rp = np.zeros(N + 1, np.uint32)
    rp[1:] = np.cumsum(lens)
    col = rng.integers(0, N, int(rp[-1])).astype(np.uint32)
    tiles = (N + len(col)) // 512
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert tiles > 16 * 16 * sms  # groups x warps of the 8-column gather
    w = rng.uniform(0.1, 1.0, len(col)).astype(np.float32)
    t = rng.uniform(0.1, 1.0, (N, 128)).astype(np.float32)
    return rp, col, w, t


def _f64(rp, col, w, t, columns):
    A = sp.csr_matrix((w, col.astype(np.int64), rp.astype(np.int64)), shape=(N, N))
    out = np.bincount(col, weights=w, minlength=N)
    inv = np.divide(1.0, out, out=np.zeros(N), where=out > 0)[:, None]
    base = (1 - D) * t[:, columns].astype(np.float64)
    x = t[:, columns].astype(np.float64)
    for _ in range(SWEEPS):
        x = base + D * (A @ (x * inv))
    return x


def _close(got, want):
    # A row's terms are positive, added at most 512 in a row, then by tiles of eight sums (137 of the longest row's):
    # under 560 roundings a sweep, of 2^-24 of the row's sum each
    assert np.all(np.abs(got - want) <= SWEEPS * 560 * 2.0**-24 * want)


@pytest.mark.parametrize("relabel", [True, False])
def test_unweighted(graph, relabel):
    rp, col, _, t = graph
    deg = np.bincount(col, minlength=N).astype(np.uint32)
    with Graph(rp, col, relabel=relabel) as g:
        wide = np.empty((N, 64), np.float32)
        g.ppr_batched_teleports(deg, np.ascontiguousarray(t[:, :64]), wide, D, 0.0, SWEEPS)
        _close(wide[:, [0, 31, 63]], _f64(rp, col, np.ones(len(col)), t, [0, 31, 63]))
        for k in (1, 8, 9, 16, 17, 32):
            part = np.empty((N, k), np.float32)
            g.ppr_batched_teleports(deg, np.ascontiguousarray(t[:, :k]), part, D, 0.0, SWEEPS)
            assert np.array_equal(part, wide[:, :k]), k


def test_weighted(graph):
    rp, col, w, t = graph
    with Graph(rp, col, weights=w) as g:
        wide = np.empty((N, 128), np.float32)
        g.weighted_page_rank_batched(t, wide, D, 0.0, SWEEPS)
        _close(wide[:, [0, 64, 127]], _f64(rp, col, w.astype(np.float64), t, [0, 64, 127]))
        for k in (3, 8, 16, 17, 32, 64):
            part = np.empty((N, k), np.float32)
            g.weighted_page_rank_batched(np.ascontiguousarray(t[:, :k]), part, D, 0.0, SWEEPS)
            assert np.array_equal(part, wide[:, :k]), k
