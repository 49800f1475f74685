"""The adjoint's dL/d(decay) is summed in FP64: fields scaled by a power of two,
whose products leave FP32's range, give exactly the scaled value (every operation
scales exactly), and its error is that of the FP32 states."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("every", [0, 4])
@pytest.mark.parametrize("power", [70, -60])
def test_decay_gradient_scales(hal, power, every):
    xd, yd, steps = 70, 51, 11
    rng = np.random.default_rng(5)
    f0, target = rng.random(xd * yd, dtype=np.float32), rng.random(xd * yd, dtype=np.float32)
    D = (0.5 + 4.5 * rng.random(xd * yd)).astype(np.float32)
    src = (rng.random(xd * yd) * 0.01).astype(np.float32)
    s = np.float32(2.0**power)
    out = []
    for k in (np.float32(1), s):
        with hal.Adjoint(xd, yd, False, True) as a:
            a.set_problem(f0 * k, target * k, steps, every)
            out.append(a.gradient(D, 0.005, src * k))
    assert out[1][2] == out[0][2] * 2.0 ** (2 * power)
    assert out[1][0] == out[0][0] * 2.0 ** (2 * power)


def test_decay_gradient_many_steps(hal, oracle):
    """Against the FP64 adjoint: the bound is the FP32 states' rounding, which
    random signs average over the cells and steps (6e-8 each; 1e-6 in all)."""
    xd, yd, steps = 64, 48, 60
    n = xd * yd
    rng = np.random.default_rng(6)
    f0, target = rng.random(n, dtype=np.float32), rng.random(n, dtype=np.float32)
    D = (0.5 + 4.5 * rng.random(n)).astype(np.float32)
    src = (rng.random(n) * 0.01).astype(np.float32)
    ref = oracle.dadi_loss_grad(f0, target, D, 0.005, src, xd, yd, steps, True, False)[3]
    with hal.Adjoint(xd, yd, True, False) as a:
        a.set_problem(f0, target, steps, 10)
        got = a.gradient(D, 0.005, src)[2]
    assert abs(got - ref) <= 1e-6 * abs(ref)


def test_forward_and_gradient_sum_the_loss_alike(hal):
    """The loss of a forward call and of a gradient call are the same bits, also
    with as many partial sums as there are."""
    n = 512 * 512
    rng = np.random.default_rng(7)
    f0, target = rng.random(n, dtype=np.float32), rng.random(n, dtype=np.float32)
    D = (0.5 + 4.5 * rng.random(n)).astype(np.float32)
    with hal.Adjoint(512, 512) as a:
        a.set_problem(f0, target, 3, 0)
        assert a.forward(D, 0.005) == a.gradient(D, 0.005)[0]
