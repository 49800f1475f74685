"""The move of a resident step adds its agents to the scan's tile sums for the
next binning; a binning of uploaded positions sums the tiles itself.  Both ways
give the same bins, so the same agents, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("x,y,n", [
    (8, 8, 40),            # one scan tile, not full
    (64, 64, 3000),        # one full tile of 4096 cells
    (65, 127, 1),          # a tile and a rest
    (300, 517, 100001),    # a thread per agent
    (2049, 2049, 20000),   # more tiles than one launch sums up by itself
])
@pytest.mark.parametrize("wrap", [False, True])
def test_steps_equal_uploaded_steps(hal, x, y, n, wrap):
    rng = np.random.default_rng(n)
    pos = (rng.random((n, 2)) * (x, y)).astype(np.float32)
    pos = np.minimum(pos, np.nextafter(np.float32([x, y]), np.float32(0))).ravel()
    rad = (0.3 + 0.4 * rng.random(n)).astype(np.float32)
    vel = (2.0 * rng.random(2 * n) - 1.0).astype(np.float32)
    with hal.Agents(x, y, n) as a, hal.Agents(x, y, n) as b:
        a.upload(pos, rad)
        a.set_velocities(vel)
        a.step(4, 1.0, 0.1, wrap, wrap)
        p, v = pos, vel
        for _ in range(4):
            b.upload(p, rad)
            b.set_velocities(v)
            b.step(1, 1.0, 0.1, wrap, wrap)
            p, v = b.get_state()
        got_p, got_v = a.get_state()
        assert np.array_equal(got_p, p) and np.array_equal(got_v, v)
        # a dispatch takes the counted bins; one after it counts again
        for _ in range(2):
            a.dispatch(1.0, 0.1, wrap, wrap)
            b.upload(p, rad)
            b.dispatch(1.0, 0.1, wrap, wrap)
            assert np.array_equal(a.download(), b.download())
            for g, e in zip(a.get_bins(), b.get_bins()):
                assert np.array_equal(g, e)
