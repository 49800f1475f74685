"""FP64 forces of sparse populations around the number of agents from which a
group of lanes takes two, against the CPU oracle, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wrap", [(False, False), (True, True)])
@pytest.mark.parametrize("n", [39_999, 40_000, 40_001])
def test_sparse_populations(hal, oracle, n, wrap):
    x, y = 512, 400
    rng = np.random.default_rng(n)
    pos = rng.random((n, 2)) * (x, y)
    pos[:2000] = rng.random((2000, 2)) * 9.0  # a dense corner
    rad = np.full(n, 0.5)
    want, _, _ = oracle.accumulate_forces(pos.ravel(), rad, 1.0, 0.1, x, y, *wrap)
    with hal.Agents(x, y, n) as a:
        got = a.accumulate_forces(pos.ravel(), rad, 1.0, 0.1, x, y, *wrap)
    assert np.array_equal(got, want)
