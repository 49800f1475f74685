"""The adjoint's factored line solves (csrc/adjoint.cu) against the FP64
adjoint over line lengths around the warp's chunks (4 positions per lane up to
128, 32 up to 1024), sides that are not multiples of the CTA's four lines or of
16 bytes, and every end condition; at the bounds of tests/test_adjoint_gpu.py."""
import numpy as np
import pytest

from conftest import max_rel, rel_l2

pytestmark = pytest.mark.gpu

SHAPES = [(1, 5), (2, 7), (5, 2), (3, 3), (4, 128), (128, 129), (33, 127), (257, 64), (516, 40), (37, 513), (1024, 33),
          (30, 1021)]
WRAPS = [(False, False), (True, True), (True, False)]


@pytest.mark.parametrize("wrap", WRAPS)
@pytest.mark.parametrize("shape", SHAPES)
def test_line_lengths(hal, oracle, shape, wrap):
    xd, yd = shape
    n, steps = xd * yd, 6
    rng = np.random.default_rng(n + 3)
    f0 = rng.random(n, dtype=np.float32)
    target = rng.random(n, dtype=np.float32)
    D = (0.5 + 4.5 * rng.random(n)).astype(np.float32)
    src = (rng.random(n) * 0.01).astype(np.float32)
    loss_ref, fT_ref, gD_ref, gK_ref, gS_ref = oracle.dadi_loss_grad(f0, target, D, 0.005, src, xd, yd, steps, *wrap)
    with hal.Adjoint(xd, yd, *wrap) as a:
        a.set_problem(f0, target, steps, 2)
        loss_f, fT = a.forward(D, 0.005, src, want_field=True)
        loss, gD, gK, gS = a.gradient(D, 0.005, src)
        again = a.gradient(D, 0.005, src)
    assert max_rel(fT, fT_ref) <= 2e-6 * (1 + 5.0) * steps
    assert abs(loss - loss_ref) <= 1e-5 * loss_ref and loss_f == loss
    assert rel_l2(gD, gD_ref) <= 1e-4 or np.linalg.norm(gD_ref) < 1e-12
    assert rel_l2(gS, gS_ref) <= 1e-4
    assert abs(gK - gK_ref) <= 1e-3 * abs(gK_ref)
    # no sum depends on the order in which blocks finish
    assert again[0] == loss and again[2] == gK
    assert np.array_equal(again[1], gD) and np.array_equal(again[3], gS)


@pytest.mark.parametrize("steps,every", [(0, 3), (1, 1), (5, 5), (16, 4), (33, 11), (40, 16), (23, 1)])
def test_runs_and_segments(hal, steps, every):
    """Runs of steps as graphs, whole and partial segments: the kept-states
    gradient bit for bit, twice on one handle and after another problem."""
    xd, yd = 70, 51
    rng = np.random.default_rng(11)
    f0, target = rng.random(xd * yd, dtype=np.float32), rng.random(xd * yd, dtype=np.float32)
    D = (0.5 + 4.5 * rng.random(xd * yd)).astype(np.float32)
    src = (rng.random(xd * yd) * 0.01).astype(np.float32)
    with hal.Adjoint(xd, yd, True, False) as a:
        a.set_problem(f0, target, steps, 0)
        want = a.gradient(D, 0.005, src)
        plain = a.gradient(D, 0.02)
        a.set_problem(target, f0, 7, 3)
        a.gradient(D, 0.005, src)
        a.set_problem(f0, target, steps, every)
        for _ in range(2):
            got = a.gradient(D, 0.005, src)
            assert got[0] == want[0] and got[2] == want[2]
            assert np.array_equal(got[1], want[1]) and np.array_equal(got[3], want[3])
        # another decay and no source through the same graphs' handle
        got = a.gradient(D, 0.02)
        assert got[0] == plain[0] and np.array_equal(got[1], plain[1])
        assert a.forward(D, 0.005, src) == want[0]
