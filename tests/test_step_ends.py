"""step() refuses a time step that does not advance the model time, with which
its loop would never end; one that is not a number ends it after one step."""

from types import SimpleNamespace

import numpy as np
import pytest

from SWESimulators.BatchedEnsemble import BatchedCDKLM16
from SWESimulators.CDKLM16 import CDKLM16


def _simulator(dt, update_dt=None):
    sim = SimpleNamespace(
        dt=dt, t=np.float64(10.0), num_iterations=0, small_scale_perturbation=False, hasDrifters=False,
        write_netcdf=False, wind_stress=SimpleNamespace(t=[0]),
        boundary_conditions=SimpleNamespace(isSponge=lambda: False), update_wind_stress=lambda: 1.0, launched=[])
    sim._launch_steps = lambda n, step, w: sim.launched.append((n, float(step)))
    sim._whole_steps = lambda *a: CDKLM16._whole_steps(sim, *a)

    def update():
        sim.dt = update_dt
    sim.updateDt = update
    return sim


@pytest.mark.parametrize("dt", [0.0, np.float32(0.0), -1.0, 1.0e-300])
def test_step_refuses_a_step_that_does_not_advance(dt):
    sim = _simulator(dt)
    with pytest.raises(ValueError, match="does not advance"):
        CDKLM16.step(sim, 60.0)
    assert sim.launched == [] and sim.t == 10.0 and sim.num_iterations == 0


def test_step_refuses_an_updated_step_of_zero():
    sim = _simulator(5.0, update_dt=np.float32(0.0))     # the CFL limit of an infinite speed
    with pytest.raises(ValueError, match="does not advance"):
        CDKLM16.step(sim, 60.0, update_dt=True)
    assert sim.launched == []


def test_steps_that_stop_advancing_the_sum():
    # 2^-24 advances 0 but not 2^30
    sim = _simulator(np.float32(2.0 ** -24))
    assert CDKLM16._whole_steps(sim, np.float32(2.0 ** -24), 0.0, 2.0 ** 30) == (0, 0.0)
    assert CDKLM16._whole_steps(sim, np.float32(2.0 ** -24), 0.0, 2.0 ** -20) == (16, 2.0 ** -20)


def test_step_of_no_number_takes_one_step():
    sim = _simulator(float("nan"))
    CDKLM16.step(sim, 60.0)
    assert sim.num_iterations == 1 and len(sim.launched) == 1


def test_batched_step_refuses_a_step_that_does_not_advance():
    batch = SimpleNamespace(sims=[SimpleNamespace(dt=0.0, t=0.0)] * 2, _has_model_error=lambda: False)
    with pytest.raises(ValueError, match="does not advance"):
        BatchedCDKLM16.step(batch, 60.0)
