"""The launch count of an adjoint whose runs are captured while another thread
launches on a handle of its own: each thread's launches are counted once."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_launch_count_beside_another_thread(hal):
    xd, yd, steps, every = 60, 44, 48, 8
    rng = np.random.default_rng(1)
    f0, target = rng.random(xd * yd, dtype=np.float32), rng.random(xd * yd, dtype=np.float32)
    D = (0.5 + rng.random(xd * yd)).astype(np.float32)

    def gradients(calls):
        with hal.Adjoint(xd, yd) as a:
            for _ in range(calls):
                a.set_problem(f0, target, steps, every)  # drops the graphs: each call captures again
                a.gradient(D, 0.01)
                a.gradient(D, 0.01)

    start = hal.launch_count()
    gradients(4)
    alone = hal.launch_count() - start
    ticks = [0]
    stop = threading.Event()

    def other():
        with hal.Diffusion(64, 64) as d:
            d.set_blocking(1)
            while not stop.is_set():
                d.run_ticks(7, 0.2)
                ticks[0] += 7
                if ticks[0] % 700 == 0:
                    d.sync()

    start = hal.launch_count()
    thread = threading.Thread(target=other)
    thread.start()
    gradients(4)
    stop.set()
    thread.join()
    assert ticks[0] > 0
    assert hal.launch_count() - start == alone + ticks[0]
