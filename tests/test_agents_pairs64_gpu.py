"""The FP64 forces by a group of lanes per agent, with an FP32 test of which
pairs may be in range, against the CPU oracle: the same deltas bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PER_GROUP = 152 * 256  # agents from twice which on a group takes more than one


def _agents(rng, n, dim):
    pos = rng.random((n, 2)) * dim
    if n > 12:
        pos[1] = pos[0]                                  # coincident
        pos[2] = [0.0, 0.0]
        pos[3] = [dim, dim]                              # on the far edge: clamped into the last cell
        pos[4] = [3.0, 1e-300]                           # below FP32's range
        pos[5] = pos[6] + [1.0, 0.0]                     # a distance of R and one on either side of it
        pos[7] = pos[8] + [np.nextafter(1.0, 0.0), 0.0]
        pos[9] = pos[10] + [0.0, np.nextafter(1.0, 2.0)]
    return pos, 0.3 + 0.4 * rng.random(n)


@pytest.mark.parametrize("wrap", [(False, False), (True, True), (True, False), (False, True)])
@pytest.mark.parametrize("radius", [1.0, 0.75, 2.0, 3.5, 1e-3, 0.0])
@pytest.mark.parametrize("n,dim", [(1, 8), (7, 2), (15, 5), (33, 12), (900, 24), (2500, 12)])
def test_pairs_equal_oracle(hal, oracle, n, dim, radius, wrap):
    rng = np.random.default_rng(n + int(radius * 8))
    pos, rad = _agents(rng, n, dim)
    want, _, _ = oracle.accumulate_forces(pos.ravel(), rad, radius, 0.1, dim, dim, *wrap)
    with hal.Agents(dim, dim, n) as a:
        got = a.accumulate_forces(pos.ravel(), rad, radius, 0.1, dim, dim, *wrap)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("more", [2 * PER_GROUP - 700, 3 * PER_GROUP + 1, 5 * PER_GROUP])
def test_several_agents_per_group(hal, oracle, more):
    """Many far-away agents make a group take two to four agents; the ones in
    the corner keep their sums, and a lone one its zeros."""
    dim, n = 24, 900
    rng = np.random.default_rng(more)
    pos, rad = _agents(rng, n, dim)
    want, _, _ = oracle.accumulate_forces(pos.ravel(), rad, 1.0, 0.1, dim + 512, dim, False, False)
    far = np.stack([dim + 8.0 + 400.0 * rng.random(more), dim * rng.random(more)], 1)
    far[-1] = [dim + 500.0, 3.0]
    with hal.Agents(dim + 512, dim, n + more) as a:
        got = a.accumulate_forces(np.concatenate([pos, far]).ravel(), np.concatenate([rad, np.full(more, 0.5)]), 1.0,
                                  0.1, dim + 512, dim, False, False)
    assert np.array_equal(got[: 2 * n], want)
    assert np.array_equal(got[-2:], np.zeros(2))


def test_far_out_and_not_finite(hal, oracle):
    """Positions outside the grid and values FP32 cannot hold: what the FP64
    test alone decides."""
    rng = np.random.default_rng(5)
    pos, rad = _agents(rng, 64, 6)
    pos[20] = [1e39, 2.0]
    pos[21] = [1e39, 2.5]
    pos[22] = [-4.0, 5.5]
    pos[23] = [-4.25, 5.5]
    want, _, _ = oracle.accumulate_forces(pos.ravel(), rad, 1.0, 0.1, 6, 6, False, False)
    with hal.Agents(6, 6, 64) as a:
        got = a.accumulate_forces(pos.ravel(), rad, 1.0, 0.1, 6, 6, False, False)
    assert np.array_equal(got, want)
