"""The FP64 ADI's split line solve (csrc/pdegrid.cu) against the CPU's serial
solve, bit for bit: segment lengths and remainders, rates from a fast to a slow
contraction (and one that is not split), and fields on which the segments meet
the serial chain late or never (decaying tails, zeros, sparse and huge values)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _field(kind, x, y, rng):
    if kind == "uniform":
        return rng.random(x * y)
    if kind == "signed":
        return rng.standard_normal(x * y)
    f = np.zeros((x, y))
    if kind == "corner":  # everything else is the tail of one cell
        f[0, 0] = 1.0
    elif kind == "sparse":
        at = rng.choice(x * y, 5, replace=False)
        f.ravel()[at] = rng.random(5) * 10.0 ** rng.integers(-200, 200, 5)
    elif kind == "steps":
        f[x // 3:, : y // 2] = -0.0
        f[: x // 4] = 1e-300 * rng.random((x // 4, y))
        f[x // 2, y // 3] = 1e250
        f[-1, :] = -3.0
    return f.ravel()


SHAPES = [(128, 128), (129, 64), (64, 257), (300, 517), (1000, 31), (2048, 33), (777, 640)]
RATES = [0.01, 0.5, 5.0, 60.0, 1e5]


@pytest.mark.parametrize("kind", ["uniform", "signed", "corner", "sparse", "steps", "zero"])
@pytest.mark.parametrize("shape", SHAPES)
def test_split_solve_bit_exact(hal, oracle, shape, kind):
    x, y = shape
    rng = np.random.default_rng(x + 7 * y)
    ghost = rng.random(2 * (x + y))
    for k, r in enumerate(RATES):
        wx, wy = bool(k & 1), bool(k & 2)
        g = ghost if k % 2 == 0 else None
        f = _field(kind, x, y, rng)
        with hal.PDEGrid(x, y, wx, wy) as grid:
            grid.set_state(f)
            for _ in range(3):
                grid.diffusion_adi(r, ghost=g)
                grid.update()
                f = f + oracle.diffuse_adi(f, np.zeros_like(f), r, x, y, wx, wy, ghost=g)
            got = grid.get_state()[0]
        assert np.array_equal(got.view(np.uint64), f.view(np.uint64)), f"rate {r}"


def test_split_solve_with_infinities(hal, oracle):
    """Lines that hold an infinity give the CPU's infinities and NaN, the other
    lines its bits."""
    x, y = 256, 192
    rng = np.random.default_rng(9)
    f = rng.random(x * y)
    f[100 * y + 50] = np.inf
    d = oracle.diffuse_adi(f, np.zeros_like(f), 2.0, x, y, False, False)
    with hal.PDEGrid(x, y) as grid:
        grid.set_state(f)
        grid.diffusion_adi(2.0)
        got = grid.get_state()[1]
    assert np.array_equal(np.isnan(got), np.isnan(d))
    ok = ~np.isnan(d)
    assert np.array_equal(got[ok].view(np.uint64), d[ok].view(np.uint64))


def test_split_solve_exact_mode_interface(hal, oracle):
    """DiffuseADI in exact mode on uneven sides, and twice on one handle."""
    x, y = 517, 300
    rng = np.random.default_rng(10)
    with hal.Adi(x, y) as a:
        a.set_exact()
        for r in (5.0, 0.7):
            f = rng.random(x * y)
            d = rng.random(x * y)
            want = oracle.diffuse_adi(f, d, r, x, y, False, True)
            got = a.diffuse_adi(f, d.copy(), r, x, y, False, True)
            assert np.array_equal(got.view(np.uint64), want.view(np.uint64))
