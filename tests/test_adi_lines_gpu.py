"""The short-line ADI sweep (csrc/adi.cu, AdiLines): lengths around its chunks
of 32 and its limit of 1024, lines per warp and per CTA, uneven rows, every end
condition, against the FP64 oracle; and against the batched wells' sweep, which
computes the same operations in the same order, bit for bit."""
import numpy as np
import pytest

from conftest import max_rel

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (1, 7), (31, 33), (32, 32), (65, 3), (3, 130), (64, 2500), (33, 1217), (257, 641), (609, 1024),
          (1023, 40), (1024, 1030), (1025, 96), (96, 1025)]


@pytest.mark.parametrize("wrap", [(False, False), (True, False), (True, True)])
@pytest.mark.parametrize("shape", SHAPES)
def test_against_oracle(hal, oracle, shape, wrap):
    x, y = shape
    rng = np.random.default_rng(x * 7 + y)
    f = rng.random(x * y, dtype=np.float32)
    src = rng.random(x * y, dtype=np.float32) * np.float32(0.01)
    ghost = rng.random(2 * (x + y)) if not all(wrap) else None
    r, ticks = 3.0, 3
    with hal.Adi(x, y) as a:
        a.set_field(f)
        a.set_source(src)
        if ghost is not None:
            a.set_dirichlet(ghost)
        a.run_ticks(ticks, r, 0.01, *wrap)
        got = a.get_field()
    want = oracle.run_ticks(1, f.astype(np.float64), x, y, r, *wrap, ghost=ghost, decay=0.01,
                            src_dense=src.astype(np.float64), ticks=ticks)
    assert max_rel(got, want) <= 2e-6 * (1 + r) * ticks


@pytest.mark.parametrize("shape", [(64, 64), (100, 77), (257, 300), (641, 520), (1024, 700)])
@pytest.mark.parametrize("wrap", [(False, False), (True, True), (False, True)])
def test_equals_the_batched_sweep(hal, shape, wrap):
    x, y = shape
    rng = np.random.default_rng(x + y)
    f = rng.random(x * y, dtype=np.float32)
    src = rng.random(x * y, dtype=np.float32) * np.float32(0.01)
    with hal.Adi(x, y) as a:
        a.set_field(f)
        a.set_source(src)
        a.run_ticks(5, 2.5, 0.01, *wrap)
        single = a.get_field()
    w = dict(xDim=x, yDim=y, kind="adi", diffRate=2.5, decay=0.01, wrapX=wrap[0], wrapY=wrap[1])
    with hal.Wells([w]) as b:
        b.set_field(0, f)
        b.set_source(0, src)
        b.run_ticks(5)
        batched = b.get_field(0)
    assert np.array_equal(single, batched)


def test_padding_stays_zero_across_uses(hal):
    """Interface calls, host runs and resident ticks on one uneven grid share
    its padded buffers: each gives what a fresh handle gives."""
    x, y = 99, 101
    rng = np.random.default_rng(3)
    f, g = rng.random(x * y, dtype=np.float32), rng.random(x * y, dtype=np.float32)
    d = rng.random(x * y)
    with hal.Adi(x, y) as a:
        a.set_field(f)
        a.run_ticks(3, 2.0, 0.0, True, False)
        a.diffuse_adi(d, np.zeros_like(d), 2.0, x, y, False, True)
        a.run_ticks(3, 2.0, 0.0, True, False)
        got = a.get_field()
        host = a.run_ticks_host(g.copy(), f, 3, 2.0)
        deltas = a.diffuse_adi(d, np.zeros_like(d), 2.0, x, y, False, True)
    with hal.Adi(x, y) as b:
        b.set_field(f)
        b.run_ticks(6, 2.0, 0.0, True, False)
        assert np.array_equal(got, b.get_field())
    with hal.Adi(x, y) as b:
        assert np.array_equal(host, b.run_ticks_host(g.copy(), f, 3, 2.0))
    with hal.Adi(x, y) as b:
        assert np.array_equal(deltas, b.diffuse_adi(d, np.zeros_like(d), 2.0, x, y, False, True))
