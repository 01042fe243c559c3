"""The batched gather's lane groups: batches padded to 8, 16, 32 and 64
columns, tiles whose first row started in the tile before, tiles that only
hold a row's end, rows of 0 to thousands of entries at every alignment, and
rows without entries between the others (graphs kept in input order). Each
column is summed in the same order at every width, so a batch must equal the
same columns in a 64-column batch bit for bit; columns are also checked against
the FP64 fixed-count iteration."""
import numpy as np
import pytest

import oracle as O
from nwgraph_b200 import Graph

pytestmark = pytest.mark.gpu
SWEEPS = 6


def _csr(kind):
    """Row lengths around the 512-item tiles and 16-entry blocks, in the given order."""
    rng = np.random.default_rng(3)
    if kind == "one row":
        lens = np.array([2047] + [0] * 40)
    elif kind == "exact tiles":  # 511 entries and their end fill a tile: rows end on tile boundaries
        lens = np.array([511] * 5 + [512, 510, 1023, 1024] + [0] * 60)
    else:
        lens = np.concatenate([[3000, 1500, 0, 700], rng.integers(0, 40, 900), np.zeros(50, int), rng.integers(0, 4, 500)])
    n = max(len(lens), 64)
    lens = np.concatenate([lens, np.zeros(n - len(lens), int)])
    rp = np.zeros(n + 1, np.uint32)
    rp[1:] = np.cumsum(lens)
    col = rng.integers(0, n, int(rp[-1])).astype(np.uint32)
    return rp, col, n


def _f64(rp, col, n, w, t, out, d):
    x = t.astype(np.float64)
    rows = np.repeat(np.arange(n), np.diff(rp.astype(np.int64)))
    for _ in range(SWEEPS):
        c = np.divide(x, out[:, None], out=np.zeros_like(x), where=out[:, None] > 0)
        z = np.zeros_like(x)
        np.add.at(z, rows, w[:, None] * c[col])
        x = (1 - d) * t + d * z
    return x


@pytest.mark.parametrize("relabel", [True, False])
@pytest.mark.parametrize("kind", ["one row", "exact tiles", "mixed"])
def test_every_width_sums_alike(gpu, kind, relabel):
    rp, col, n = _csr(kind)
    deg = np.bincount(col, minlength=n).astype(np.uint32)
    t = np.random.default_rng(5).uniform(0, 1, (n, 64)).astype(np.float32)
    t /= t.sum(axis=0, keepdims=True)
    with Graph(rp, col, relabel=relabel) as g:
        wide = np.empty((n, 64), np.float32)
        g.ppr_batched_teleports(deg, t, wide, 0.85, 0.0, SWEEPS)
        ref = _f64(rp, col, n, np.ones(len(col)), t, deg.astype(np.float64), 0.85)
        # FP32 serial sums of up to 3000 terms: 3000 * 2^-24 of the row sum, and the sums are at most 1
        assert np.abs(wide - ref).max() <= 2e-4 * np.abs(ref).max()
        for k in (1, 7, 8, 9, 16, 17, 32):
            part = np.empty((n, k), np.float32)
            g.ppr_batched_teleports(deg, np.ascontiguousarray(t[:, :k]), part, 0.85, 0.0, SWEEPS)
            assert np.array_equal(part, wide[:, :k]), k


@pytest.mark.parametrize("kind", ["one row", "exact tiles", "mixed"])
def test_weighted_widths(gpu, kind):
    rp, col, n = _csr(kind)
    w = np.random.default_rng(9).uniform(0.1, 1.0, len(col)).astype(np.float32)
    out = np.zeros(n)
    np.add.at(out, col, w.astype(np.float64))
    t = np.random.default_rng(5).uniform(0, 1, (n, 128)).astype(np.float32)
    t /= t.sum(axis=0, keepdims=True)
    with Graph(rp, col, weights=w) as g:
        wide = np.empty((n, 128), np.float32)
        g.weighted_page_rank_batched(t, wide, 0.85, 0.0, SWEEPS)
        ref = _f64(rp, col, n, w.astype(np.float64), t, out, 0.85)
        assert np.abs(wide - ref).max() <= 2e-4 * np.abs(ref).max()
        for k in (3, 8, 16, 24, 64):
            part = np.empty((n, k), np.float32)
            g.weighted_page_rank_batched(np.ascontiguousarray(t[:, :k]), part, 0.85, 0.0, SWEEPS)
            assert np.array_equal(part, wide[:, :k]), k
