"""Several explicit ticks per launch (csrc/tick_patch.cu) against one tick per
launch: the same field bit for bit, over every form that a run can take."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def hal():
    import halcuda

    halcuda.lib()
    return halcuda


# (40, 32) and (24, 64) are the smallest patches' grids; (23, 200) and (200, 31)
# have none; 1031 x 517 and 700 x 800 lie above the small shape's range (odd and
# even rows); 57 = 16 * 3 + 9 and 73 leave shifted windows and strips.
SIZES = [(40, 32), (41, 33), (24, 64), (39, 65), (23, 200), (200, 31), (57, 73), (64, 64), (130, 257), (1031, 517),
         (700, 800)]
FORMS = [
    # wrapX, wrapY, dirichlet, dense, points, velocity, ticks
    (False, False, False, False, 0, (0.0, 0.0), 17),
    (True, True, False, True, 0, (0.0, 0.0), 8),
    (True, False, True, False, 9, (0.0, 0.0), 13),
    (False, True, True, True, 9, (0.05, -0.1), 9),
    (False, False, True, True, 40, (0.0, 0.0), 4),
    (False, False, True, False, 0, (-0.1, 0.05), 2),
    (True, True, False, True, 0, (0.1, 0.0), 5),
    (False, False, False, False, -6, (0.0, 0.0), 7),  # a cell listed twice
]


@pytest.mark.parametrize("form", FORMS)
@pytest.mark.parametrize("size", SIZES)
def test_patch_ticks_equal_single_ticks(hal, size, form):
    x, y = size
    wx, wy, dirichlet, dense, points, vel, ticks = form
    rng = np.random.default_rng(x * 1000 + y)
    n = x * y
    f0 = rng.random(n, dtype=np.float32)
    src = rng.random(n, dtype=np.float32) * np.float32(0.01)
    ghost = rng.random(2 * (x + y), dtype=np.float32)
    cells = rng.choice(n, abs(points), replace=False).astype(np.int32)
    if points:
        # the corners and edges, where a patch reads across the seam
        cells[:4] = [0, y - 1, n - y, n - 1]
    if points < 0:
        cells[-1] = cells[0]
    cells = cells if points < 0 else np.unique(cells).astype(np.int32)
    got = []
    for mode in (1, 0):
        with hal.Diffusion(x, y) as d:
            d.set_blocking(mode)
            d.set_field(f0)
            if dirichlet:
                d.set_dirichlet(ghost)
            if dense:
                d.set_source(src)
            if points:
                d.set_point_sources(cells, np.linspace(0.01, 0.05, cells.size).astype(np.float32))
            if vel != (0.0, 0.0):
                d.set_velocity(*vel)
            d.run_ticks(ticks, 0.2 if vel == (0.0, 0.0) else 0.1, 0.003, wx, wy)
            d.run_ticks(3, 0.2 if vel == (0.0, 0.0) else 0.1, 0.003, wx, wy)
            got.append(d.get_field())
    assert np.array_equal(got[0], got[1])


def test_patch_points_replaced_and_cleared(hal):
    """Point sources set again, beside a dense source, and taken away."""
    x, y = 96, 120
    rng = np.random.default_rng(5)
    f0 = rng.random(x * y, dtype=np.float32)
    src = rng.random(x * y, dtype=np.float32) * np.float32(0.01)
    got = []
    for mode in (1, 0):
        with hal.Diffusion(x, y) as d:
            d.set_blocking(mode)
            d.set_field(f0)
            d.set_point_sources(np.arange(5, dtype=np.int32) * 17, np.full(5, 0.1, np.float32))
            d.run_ticks(9, 0.2)
            d.set_point_sources(np.arange(7, dtype=np.int32) * 31 + 5000, np.full(7, 0.2, np.float32))
            d.set_source(src)
            d.run_ticks(9, 0.2)
            d.set_point_sources(np.zeros(0, np.int32), np.zeros(0, np.float32))
            d.run_ticks(9, 0.2)
            got.append(d.get_field())
    assert np.array_equal(got[0], got[1])


def test_patch_stops_at_an_agent_coupling(hal):
    """Ticks with agent uptake run one per launch, and several again after it."""
    x = y = 64
    rng = np.random.default_rng(6)
    f0 = rng.random(x * y, dtype=np.float32)
    got = []
    for mode in (1, 0):
        with hal.Diffusion(x, y) as d, hal.Agents(x, y, 50) as a:
            a.upload(rng.random(100, dtype=np.float32) * 0 + np.linspace(1, 60, 100, dtype=np.float32),
                     np.full(50, 0.5, np.float32))
            a.dispatch(1.0, 0.1)
            a.sync()
            d.set_blocking(mode)
            d.set_field(f0)
            d.run_ticks(6, 0.2)
            d.set_uptake(a, 0.01)
            d.run_ticks(6, 0.2)
            d.set_uptake(None, 0.0)
            d.run_ticks(6, 0.2)
            got.append(d.get_field())
    assert np.array_equal(got[0], got[1])
