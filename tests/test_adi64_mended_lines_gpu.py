"""The FP64 ADI's split line solve on fields whose segments stay an ulp off the
serial chain (constants, ramps along one axis, steps, the tails of a point), so
that their lines are mended segment by segment: the CPU's bits, for ticks in a
row and with ordinary fields between them on the same handle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _field(kind, x, y, rng):
    i = np.arange(x)[:, None] + np.zeros(y)
    f = {"ones": np.ones((x, y)), "third": np.full((x, y), 1.0 / 3.0), "ramp": i / (x - 1.0),
         "cross": (i / (x - 1.0)).T.copy().reshape(-1)[: x * y].reshape(x, y), "step": (i < x // 2).astype(float),
         "point": ((i == x // 2) & (np.arange(y) == y // 3)).astype(float), "uniform": rng.random((x, y))}[kind]
    return np.ascontiguousarray(f).ravel()


@pytest.mark.parametrize("kind", ["ones", "third", "ramp", "cross", "step", "point"])
@pytest.mark.parametrize("rate", [0.5, 5.0, 50.0])
@pytest.mark.parametrize("shape", [(300, 263), (1024, 40), (33, 1500)])
def test_mended_lines(hal, oracle, shape, rate, kind):
    x, y = shape
    rng = np.random.default_rng(x)
    wrap = kind == "third"
    with hal.PDEGrid(x, y, wrap, wrap) as grid:
        for k in (kind, "uniform", kind):
            f = _field(k, x, y, rng)
            grid.set_state(f)
            for _ in range(5):
                grid.diffusion_adi(rate)
                grid.update()
                f = f + oracle.diffuse_adi(f, np.zeros_like(f), rate, x, y, wrap, wrap)
            got = grid.get_state()[0]
            assert np.array_equal(got.view(np.uint64), f.view(np.uint64)), k
