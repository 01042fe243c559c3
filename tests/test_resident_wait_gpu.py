"""The grid barriers of a small graph's one-launch solve give up and say so: a
solve whose barriers wait for a CTA that does not exist ends with an error
status after its few polls, and the handle's next solves (which reuse the
arrival counters by turns) give what they gave before."""
import numpy as np
import pytest

from nwgraph_b200 import Graph, NwgpuError, graphs as G
from nwgraph_b200 import _native as N

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [4, 10, 15])  # 1, 18 and 148 CTAs
@pytest.mark.parametrize("polls", [1, 1000])
def test_gives_up_and_goes_on(gpu, scale, polls):
    g = G.rmat(scale, 16, 3)
    deg = g.out_degree()
    want, out = np.empty(g.n, np.float32), np.empty(g.n, np.float32)
    with Graph(g.row_ptr, g.col) as h:
        h.page_rank(deg, want, 0.85, 1e-6, 30)
        assert h.info()["kernels_per_sweep"] == 0
        for times in (1, 2, 3):
            for _ in range(times):
                with pytest.raises(NwgpuError) as e:
                    N.check(N.lib().nwgpu_selftest_resident_wait(h.handle, deg.ctypes.data, out.ctypes.data, polls))
                assert e.value.status == N.ERR_CUDA and "wait gave up" in str(e.value)
            for _ in range(times):
                h.page_rank(deg, out, 0.85, 1e-6, 30)
                assert np.array_equal(out, want, equal_nan=True)


def test_refuses_what_it_cannot_test(gpu):
    g = G.rmat(10, 16, 3)
    deg = g.out_degree()
    out = np.empty(g.n, np.float32)
    with Graph(g.row_ptr, g.col) as h:
        for handle, polls in ((h.handle, 10), (h.handle, 0), (None, 10)):  # no solve has run yet
            assert N.lib().nwgpu_selftest_resident_wait(handle, deg.ctypes.data, out.ctypes.data, polls) == N.ERR_INVALID_ARG
