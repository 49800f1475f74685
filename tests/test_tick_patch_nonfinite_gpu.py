"""Infinite and NaN sources and cells under several ticks per launch
(csrc/tick_patch.cu): NaN in the same cells as with one tick per launch, and the
same bits elsewhere.  A source at one edge must not reach the opposite one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wrap", [(False, False), (True, False), (False, True)])
@pytest.mark.parametrize("kind", ["dense", "points", "both", "field", "ghost"])
@pytest.mark.parametrize("size", [(40, 32), (130, 257), (1031, 517), (700, 800)])
def test_nonfinite_stays_local(hal, size, kind, wrap):
    x, y = size
    n = x * y
    rng = np.random.default_rng(x)
    f0 = rng.random(n, dtype=np.float32)
    src = rng.random(n, dtype=np.float32) * np.float32(0.01)
    at = np.array([[x // 2, y - 1], [x // 3, 0], [0, y // 3], [x - 1, y // 2], [x // 2, y // 2]])
    cells = np.unique(at[:, 0] * y + at[:, 1]).astype(np.int32)
    bad = np.array([np.inf, np.nan, -np.inf, np.inf, np.nan], dtype=np.float32)[: len(cells)]
    got = []
    for mode in (1, 0):
        rng2 = np.random.default_rng(y)
        with hal.Diffusion(x, y) as d:
            d.set_blocking(mode)
            f, s = f0.copy(), src.copy()
            if kind == "field":
                f[cells] = bad
            if kind == "dense":
                s[cells] = bad
            d.set_field(f)
            if kind == "ghost":
                g = rng2.random(2 * (x + y), dtype=np.float32)
                g[[3, y + 5, 2 * y + x // 2, 2 * y + x + x // 3]] = bad[:4]
                d.set_dirichlet(g)
            if kind != "points":
                d.set_source(s)
            if kind in ("points", "both"):
                d.set_point_sources(cells, bad)
            d.run_ticks(7, 0.2, 0.001, *wrap)
            got.append(d.get_field())
    want, have = got
    assert 0 < np.isnan(want).sum() < n
    assert np.array_equal(np.isnan(want), np.isnan(have))
    ok = ~np.isnan(want)
    assert np.array_equal(want[ok].view(np.uint32), have[ok].view(np.uint32))
