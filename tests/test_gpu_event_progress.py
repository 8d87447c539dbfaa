"""An event that cannot end is not begun: the members keep the states, times,
step counts and time step of the events before it."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from SWESimulators import BatchedEnsemble, CDKLM16, Common, _native  # noqa: E402


def _ensemble():
    ctx = Common.CUDAContext()
    sims = []
    for nx, ny in ((40, 24), (33, 50)):
        zero = np.zeros((ny + 4, nx + 4), np.float32)
        H = np.full((ny + 5, nx + 5), 50.0, np.float32)
        sims.append(CDKLM16.CDKLM16(ctx, zero, zero, zero, H, nx, ny, 1000.0, 1000.0, 5.0, 9.81, 1.2e-4, 0.0, 0.0))
    return BatchedEnsemble.BatchedCDKLM16(sims)


def _states(ens):
    torch.cuda.synchronize()
    return [a for s in ens.sims for a in s.download()]


def test_loop_stops_before_an_event_that_cannot_end():
    ens, want = _ensemble(), _ensemble()
    # event 1 runs at dt 5; the Courant number leaves a step of some 1e-11 s for event 2
    with pytest.raises(_native.NativeError, match="event 2 not begun"):
        ens.run_events(1, 3, interval=60.0, courant=1.0e-12)
    assert want.run_events(1, 1, interval=60.0, courant=0.7) == 12
    for a, b in zip(_states(ens), _states(want)):
        assert np.array_equal(a, b)
    tiny = np.float32(1.0e-12 * float(np.min(ens.max_dt())))
    for a, b in zip(ens.sims, want.sims):
        assert (a.t, a.num_iterations, a.dt) == (b.t, 12, tiny)
    # what the loop accounts for is what the next step takes
    ens.advance(3)
    assert all(s.t == 60.0 + float(tiny) + float(tiny) + float(tiny) for s in ens.sims)
    for s in ens.sims:
        assert s.num_iterations == 15


def test_loop_goes_on_after_an_event_that_was_not_begun():
    ens, want = _ensemble(), _ensemble()
    with pytest.raises(_native.NativeError, match="event 2 not begun"):
        ens.run_events(1, 2, interval=60.0, courant=1.0e-12)
    with pytest.raises(_native.NativeError, match="event 2 not begun"):
        ens.run_events(2, 1, interval=60.0)          # the step is still too short: nothing moves
    ens.update_dt(0.7)
    ens.run_events(2, 2, interval=60.0)
    want.run_events(1, 3, interval=60.0)
    for a, b in zip(_states(ens), _states(want)):
        assert np.array_equal(a, b)
    for a, b in zip(ens.sims, want.sims):
        assert (a.t, a.num_iterations, a.dt) == (b.t, b.num_iterations, b.dt)
