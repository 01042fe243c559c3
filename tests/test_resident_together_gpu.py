"""Small graphs solved in one launch each, from several threads at once and
beside another stream's kernels: every such launch needs room for all its CTAs
at once, so they take turns, and each gives what it gives alone."""
import threading

import numpy as np
import pytest

from nwgraph_b200 import Graph, graphs as G

pytestmark = pytest.mark.gpu


def test_several_handles_at_once(gpu):
    import torch
    made = [G.rmat(10, 16, 1), G.rmat(13, 16, 2), G.rmat(16, 16, 3), G.grid(250_000), G.rmat(16, 8, 4)]
    handles, degs, want = [], [], []
    for g in made:
        h, deg, out = Graph(g.row_ptr, g.col), g.out_degree(), np.empty(g.n, np.float32)
        h.page_rank(deg, out, 0.85, 1e-6, 50)
        assert h.info()["kernels_per_sweep"] == 0
        handles.append(h)
        degs.append(deg)
        want.append(out)
    wrong = []
    stop = threading.Event()

    def solve(i):
        out = np.empty_like(want[i])
        for k in range(40):
            handles[i].page_rank(degs[i], out, 0.85, 1e-6, 50)
            if not np.array_equal(out, want[i]):
                wrong.append((i, k))

    def other_work():
        a = torch.rand(4096, 4096, device="cuda")
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            while not stop.is_set():
                a = torch.tanh(a @ a)
                s.synchronize()

    side = threading.Thread(target=other_work)
    threads = [threading.Thread(target=solve, args=(i,)) for i in range(len(made))]
    side.start()
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    stop.set()
    side.join()
    for h in handles:
        h.release()
    assert not wrong
