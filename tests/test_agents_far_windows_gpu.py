"""Agents outside the grid by more than the interaction radius, up to several
sides (uploads check no position; the binning clamps them, the windows wrap):
a group of lanes per agent (few agents) against one thread per agent (many),
forces and a step, bit for bit; also windows of more runs than a group has
lanes (radii from 4 on, and 2 at a wrapped edge) and y-ranges longer than the
side (9 cells, radius 6).  The many are a strip of agents beyond every
window (tests/test_agents_group_gpu.py)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMIT = 100_000  # agents up to which a group may take each


def _agents(dim, width, radius, rng):
    pos = (rng.random((300, 2)) * dim).astype(np.float32)
    pos[:40, 0] = rng.random(40) * 2                      # the first rows
    pos[40:80, 1] = dim - rng.random(40) * 2              # the last columns
    off = lambda side: [-radius - 1, -5.5, -side - 3, -1000.0, side + radius + 2, 3.0 * side, side + 5.0, 1e6]  # noqa: E731
    k = 80
    for y in off(dim):
        for x in (0.5, dim / 2, width - 0.5, width - 1.5):
            pos[k] = (x, y)
            k += 1
    for x in off(width):
        for y in (0.5, dim / 2, dim - 0.5):
            pos[k] = (x, y)
            k += 1
    for x, y in zip(off(width), off(dim)):
        pos[k] = (x, y)
        k += 1
    return pos


@pytest.mark.parametrize("wrap", [(False, False), (True, True), (True, False), (False, True)])
@pytest.mark.parametrize("radius", [0.75, 1.0, 2.0, 4.5, 6.0])
@pytest.mark.parametrize("dim", [9, 64])
def test_far_agents(hal, dim, radius, wrap):
    rng = np.random.default_rng(dim + int(8 * radius))
    width = dim + 64
    pos = _agents(dim, width, radius, rng)
    n = len(pos)
    rad = (0.3 + 0.4 * rng.random(n)).astype(np.float32)
    far = LIMIT + 1
    strip = np.stack([dim + 16.0 + 32.0 * rng.random(far), dim * rng.random(far)], 1).astype(np.float32)
    out = []
    for p, r in ((pos, rad), (np.concatenate([pos, strip]), np.concatenate([rad, np.full(far, 0.5, np.float32)]))):
        with hal.Agents(width, dim, len(p)) as a:
            a.upload(p.ravel(), r)
            a.dispatch(interactionRad=radius, springConstant=0.1, wrapX=wrap[0], wrapY=wrap[1])
            deltas = a.download()[: 2 * n].copy()
            a.upload(p.ravel(), r)
            a.set_velocities()
            a.step(1, radius, 0.1, wrap[0], wrap[1], friction=0.5)
            moved, vel = a.get_state()
            out.append((deltas, moved.ravel()[: 2 * n].copy(), vel.ravel()[: 2 * n].copy()))
    assert np.abs(out[1][0]).max() > 0
    for got, want in zip(out[0], out[1]):
        assert np.array_equal(got, want)
