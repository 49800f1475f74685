"""The force kernels with a group of lanes per agent (few agents) against one
thread per agent (many): the same deltas bit for bit.  Agents are padded with
far-away ones up to more than the groups' limit, which do not change the
others' windows; sizes and windows around the groups' runs of cells."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMIT = 100_000  # agents up to which a group takes each


@pytest.mark.parametrize("wrap", [(False, False), (True, True), (True, False), (False, True)])
@pytest.mark.parametrize("radius", [1.0, 0.75, 2.0, 3.5, 1e-3])
@pytest.mark.parametrize("n,dim", [(1, 8), (7, 5), (33, 12), (900, 24), (5000, 40)])
def test_group_equals_thread(hal, n, dim, radius, wrap):
    rng = np.random.default_rng(n + int(radius * 8))
    pos = (rng.random((n, 2)) * dim).astype(np.float32)
    if n > 6:
        pos[1] = pos[0]                      # coincident
        pos[2] = [0.0, 0.0]                  # corners and edges
        pos[3] = [dim, dim]                  # outside: clamped into the last cell
        pos[4] = [-0.5, dim / 2]
        pos[5] = [3.0, np.float32(1e-30)]    # a tiny coordinate (its window's rounding)
    rad = (0.3 + 0.4 * rng.random(n)).astype(np.float32)
    # a strip of columns apart, beyond every window: side dim + 64 along x
    width = dim + 64
    args = dict(interactionRad=radius, springConstant=0.1)
    wx, wy = wrap
    far = LIMIT + 1
    fpos = np.stack([dim + 16.0 + 32.0 * rng.random(far), dim * rng.random(far)], 1).astype(np.float32)
    # (x stays closed in both so that the strip is never a neighbour)
    with hal.Agents(width, dim, n + far) as a:
        a.upload(np.concatenate([pos, fpos]).ravel(), np.concatenate([rad, np.full(far, 0.5, np.float32)]))
        a.dispatch(**args, wrapX=False, wrapY=wy)
        want = a.download()[: 2 * n]
    with hal.Agents(width, dim, n) as a:
        a.upload(pos.ravel(), rad)
        a.dispatch(**args, wrapX=False, wrapY=wy)
        got = a.download()
    assert np.array_equal(got, want)
    # both axes' wraps against the FP64 interface's sums
    with hal.Agents(dim, dim, n) as a:
        a.upload(pos.ravel(), rad)
        a.dispatch(**args, wrapX=wx, wrapY=wy)
        small = a.download().astype(np.float64)
        exact = a.accumulate_forces(pos.ravel().astype(np.float64), rad.astype(np.float64), radius, 0.1, dim, dim, wx,
                                    wy)
    # (a pair at the very edge of the radius may be in for one precision only)
    bad = np.abs(small - exact) > 1e-4 * max(np.abs(exact).max(), 1e-6)
    assert bad.mean() <= 2e-3


@pytest.mark.parametrize("n", [450, 470, 1300])
def test_long_windows_equal_group(hal, n):
    """Windows around the length (64) from which a thread walks its runs one
    by one, and far past it, against the group's sums; some runs empty."""
    dim = 8
    rng = np.random.default_rng(n)
    pos = (rng.random((n, 2)) * dim).astype(np.float32)
    pos[: n // 8] = [2.5, 2.5]                       # a pile in one cell
    pos[(np.floor(pos[:, 0]) == 5)] = [0.25, 7.5]    # an empty column, a full corner
    rad = (0.3 + 0.4 * rng.random(n)).astype(np.float32)
    far = LIMIT + 1
    fpos = np.stack([dim + 16.0 + 32.0 * rng.random(far), dim * rng.random(far)], 1).astype(np.float32)
    with hal.Agents(dim + 64, dim, n + far) as a:
        a.upload(np.concatenate([pos, fpos]).ravel(), np.concatenate([rad, np.full(far, 0.5, np.float32)]))
        a.dispatch(1.0, 0.1, False, False)
        want = a.download()[: 2 * n]
    with hal.Agents(dim + 64, dim, n) as a:
        a.upload(pos.ravel(), rad)
        a.dispatch(1.0, 0.1, False, False)
        assert np.array_equal(a.download(), want)
