"""Point sources that change between runs of several ticks per launch
(csrc/tick_patch.cu), with single ticks, repeated cells and no points in between:
the field of one tick per launch, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wrap", [(False, False), (True, True)])
@pytest.mark.parametrize("size", [(40, 32), (73, 57), (257, 130), (1031, 517), (700, 800)])
def test_points_set_between_runs(hal, size, wrap):
    x, y = size
    n = x * y
    rng = np.random.default_rng(x + y)
    f0 = rng.random(n, dtype=np.float32)
    edges = np.array([0, y - 1, n - y, n - 1, y // 2, (x // 2) * y, (x // 2) * y + y - 1], dtype=np.int32)
    plan = []
    for k, count in enumerate((9, 40, 1, 300, 0, 12, 5)):
        cells = np.unique(np.concatenate([rng.choice(n, count, replace=False), edges[: count and 7]])).astype(np.int32)
        if k == 2:
            cells = np.concatenate([cells, cells[:1]])  # a cell twice: one tick per launch
        plan.append((cells, rng.random(len(cells), dtype=np.float32), (7, 1, 5, 12, 3, 1, 16)[k]))
    got = []
    for mode in (1, 0):
        with hal.Diffusion(x, y) as d:
            d.set_blocking(mode)
            d.set_field(f0)
            for cells, values, ticks in plan:
                d.set_point_sources(cells, values)
                d.run_ticks(ticks, 0.2, 0.001, *wrap)
                d.run_ticks(2, 0.2, 0.001, *wrap)
            got.append(d.get_field())
    assert np.array_equal(got[0].view(np.uint32), got[1].view(np.uint32))
