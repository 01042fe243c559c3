"""The benchmark's own count of the kernels it launches, by the path its graph takes (CPU only)."""
import argparse

import pytest

import bench


@pytest.mark.parametrize("launch,relabel,per,blocked,kernels", [
    ("graph", True, 2, 0, 44),   # 20 sweeps and finishing kernels, init, arm, degrees and ranks: RMAT scale 24
    ("stream", True, 2, 0, 43),
    ("graph", True, 1, 0, 25),   # seven rounds of three sweeps
    ("stream", True, 1, 0, 23),
    ("graph", True, 0, 0, 1),    # a small graph
    ("graph", False, 2, 0, 42),
    ("graph", True, 2, 1, 45),   # the blocked sweep checks the degrees
])
def test_kernels_of_a_step(launch, relabel, per, blocked, kernels):
    args = argparse.Namespace(launch=launch, no_relabel=not relabel)
    assert bench.SWEEPS == 20
    assert bench.launches_per_step(args, {"kernels_per_sweep": per, "blocked": blocked}) == kernels
