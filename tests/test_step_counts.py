"""The steps that CDKLM16.step counts in one go equal those of its step loop:
their number, the summed times and the length of the step that follows."""

from types import SimpleNamespace

import numpy as np
import pytest

from SWESimulators.CDKLM16 import CDKLM16


def _loop(dt, t, t_now, t_end, length):
    n = 0
    while t_now < t_end and np.float32(min(dt, np.float32(t_end - t_now))) == length:
        t += np.float64(length)
        t_now += np.float64(length)
        n += 1
    return n, t, t_now


@pytest.mark.parametrize("dt", [0.1, np.float32(0.1), np.float64(0.1), 1.0 / 64, np.float32(7.3), 33.3])
@pytest.mark.parametrize("steps", [0.5, 1.0, 1.0 + 6e-8, 2.0 - 1e-7, 2.0 + 1e-7, 3.0, 10.0, 999.9999, 1000.0, 4096.25])
@pytest.mark.parametrize("t", [0.0, 12.7])
def test_steps_counted_in_one_go(dt, steps, t):
    for t_end in (float(dt) * steps, float(np.float32(dt)) * steps, np.float32(dt) * np.float32(steps)):
        for length in (np.float32(dt), np.float32(min(dt, 0.01))):     # the second: a shortened step before
            sim = SimpleNamespace(dt=dt, t=np.float64(t), num_iterations=3)
            n, t_now = CDKLM16._whole_steps(sim, length, 0.0, t_end)
            want = _loop(dt, np.float64(t), 0.0, t_end, length)
            if length != np.float32(dt):
                assert n == 0 and t_now == 0.0 and sim.t == t
            else:
                assert (n, sim.t, t_now) == want
                assert sim.num_iterations == 3 + n
