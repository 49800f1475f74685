"""Wrapped lines of 1024 around the number of lines from which the ADI leaves the
short-line sweep, against the FP64 oracle (bounds of tests/test_adi_lines_gpu.py)."""
import numpy as np
import pytest

from conftest import max_rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(1024, 908), (1024, 912), (912, 1024), (1024, 1024)])
def test_wrapped_lines(hal, oracle, shape):
    x, y = shape
    rng = np.random.default_rng(x + y)
    f = rng.random(x * y, dtype=np.float32)
    r, ticks = 3.0, 3
    with hal.Adi(x, y) as a:
        a.set_field(f)
        a.run_ticks(ticks, r, 0.01, True, True)
        got = a.get_field()
    want = oracle.run_ticks(1, f.astype(np.float64), x, y, r, True, True, decay=0.01, ticks=ticks)
    assert max_rel(got, want) <= 2e-6 * (1 + r) * ticks
