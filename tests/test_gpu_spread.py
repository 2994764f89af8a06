"""Blocks of throughput-bound kernels have to spread over the SMs, however the launches before them end."""

import statistics
import time

import pytest

from perf import cases

pytestmark = pytest.mark.gpu


def test_few_heavy_blocks_spread():
    """A catalogue in a cap on a coarse grid, FP64: its moments are a few blocks of many galaxies each.  Three times the
    galaxies take at most three times as long when every block has an SM's FP64 pipe to itself; packed onto a few SMs
    they took nine times as long.  The line is drawn between, at five."""
    import torch
    took = []
    for n in (100_000, 300_000):
        s = cases.prepare(dict(path="catalogue", precision="fp64", nside=16, kmax=0.03, rmin=500.0, rmax=1000.0, nr=150,
                               ngal=n, sky="cap", weights=True, window="separable"), 1)
        t = []
        for _ in range(23):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            cases.run(s)
            torch.cuda.synchronize()
            t.append(time.perf_counter() - t0)
        took.append(statistics.median(t[3:]))
    assert took[1] < 5 * took[0], took
