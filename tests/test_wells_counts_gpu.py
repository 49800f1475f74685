"""With motion a well's agents are counted into their next bins as they move.
Whatever comes between two ticks (another radius, motion off and on, new
agents, a profile), the agents go on as they do on single grids, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# one cell per bin, coarse bins, no agents, a lone one, an axis that wraps
WELLS = [(20, 24, 700, False), (128, 96, 300, True), (40, 40, 0, False), (300, 7, 1, False), (1024, 1000, 900, True)]


def _agents(rng):
    counts, pos = [], []
    for x, y, n, _ in WELLS:
        p = (rng.random((n, 2)) * (x, y)).astype(np.float32)
        pos.append(np.minimum(p, np.nextafter(np.float32([x, y]), np.float32(0))).ravel())
        counts.append(n)
    return np.array(counts, np.int32), pos, [(0.3 + 0.4 * rng.random(n)).astype(np.float32) for n in counts]


def _steps(hal, pos, rad, vel, ticks, R):
    out = []
    for (x, y, n, wrap), p, r, v in zip(WELLS, pos, rad, vel):
        if n == 0:
            out.append((p, v))
            continue
        with hal.Agents(x, y, n) as a:
            a.upload(p, r)
            a.set_velocities(v)
            a.step(ticks, R, 0.1, wrap, wrap, friction=0.95)
            out.append(a.get_state())
    return [o[0] for o in out], [o[1] for o in out]


def test_counts_survive_what_comes_between(hal):
    rng = np.random.default_rng(9)
    counts, pos, rad = _agents(rng)
    desc = [dict(xDim=x, yDim=y, kind="adi" if i % 2 else "explicit", diffRate=0.2, decay=0.0, wrapX=w, wrapY=w,
                 maxAgents=n) for i, (x, y, n, w) in enumerate(WELLS)]
    vel = [np.zeros(2 * n, np.float32) for n in counts]

    def check(b):
        p, v = b.get_agents()
        assert np.array_equal(p, np.concatenate(pos)) and np.array_equal(v, np.concatenate(vel))

    with hal.Wells(desc) as b:
        b.set_agents(counts, np.concatenate(pos), np.concatenate(rad))
        b.set_motion(True, 0.95)
        for ticks, R in ((3, 1.0), (2, 2.0), (1, 1.0)):       # each new radius is tuned for
            b.run_ticks(ticks, R, 0.1)
            pos, vel = _steps(hal, pos, rad, vel, ticks, R)
            check(b)
        b.set_motion(False)
        b.run_ticks(2, 1.0, 0.1)                              # forces only
        check(b)
        b.set_motion(True, 0.95)
        b.run_ticks(2, 1.0, 0.1)
        pos, vel = _steps(hal, pos, rad, vel, 2, 1.0)
        check(b)
        b.profile(2, 1.0, 0.1)                                # two ticks of its own
        pos, vel = _steps(hal, pos, rad, vel, 2, 1.0)
        b.run_ticks(1, 1.0, 0.1)
        pos, vel = _steps(hal, pos, rad, vel, 1, 1.0)
        check(b)
        counts, pos, rad = _agents(rng)                       # new agents, the same radius
        vel = [np.zeros(2 * n, np.float32) for n in counts]
        b.set_agents(counts, np.concatenate(pos), np.concatenate(rad))
        b.run_ticks(3, 1.0, 0.1)
        pos, vel = _steps(hal, pos, rad, vel, 3, 1.0)
        check(b)
