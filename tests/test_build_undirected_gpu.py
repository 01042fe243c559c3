"""Undirected builds that sort both copies of every edge at once, and degrees
taken from the row lengths: the ends of the key range, where a dropped edge's
all-ones key meets the real ones, against oracle.build_csr."""
import numpy as np
import pytest

import oracle as O
from nwgraph_b200 import NwgpuError, construct as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 64, 65, 1 << 16])
@pytest.mark.parametrize("loops", ["none", "some", "all"])
def test_ends_of_the_key_range(gpu, n, loops):
    rng = np.random.default_rng(n)
    m = 300
    s = rng.integers(0, n, m).astype(np.uint32)
    d = rng.integers(0, n, m).astype(np.uint32)
    if loops == "none" and n > 1:
        d = ((s + 1 + rng.integers(0, n - 1, m)) % n).astype(np.uint32)
    s[-2:] = n - 1  # the last vertex's self-loop, twice: the all-ones key when n is a power of two
    if loops != "none":
        d[-2:] = n - 1
    if loops == "all":
        d = s.copy()
    for f in range(0, 0x40, 2):
        csr, deg = K.csr_from_edges(s, d, n, f)
        rp, cl, dg = O.build_csr(s, d, n, f)
        assert np.array_equal(csr.row_ptr, rp) and np.array_equal(csr.col, cl) and np.array_equal(deg, dg), (n, f)


@pytest.mark.parametrize("f", [0, K.UNDIRECTED, K.SIMPLE_UNDIRECTED, K.UNDIRECTED | K.UNIQUE, K.UNIQUE_ENTRIES])
def test_no_edges_and_bad_endpoints(gpu, f):
    none = np.zeros(0, np.uint32)
    csr, deg = K.csr_from_edges(none, none, 5, f)
    assert not csr.row_ptr.any() and len(csr.col) == 0 and not deg.any()
    with pytest.raises(NwgpuError):
        K.csr_from_edges(np.array([0, 5], np.uint32), np.array([1, 2], np.uint32), 5, f)
