"""The device event loop ends, with an error, when the common time step cannot
end an event."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from SWESimulators import BatchedEnsemble, CDKLM16, Common  # noqa: E402


def test_event_loop_ends_on_a_step_too_short():
    ctx = Common.CUDAContext()
    nx, ny = 40, 24
    zero = np.zeros((ny + 4, nx + 4), np.float32)
    H = np.full((ny + 5, nx + 5), 50.0, np.float32)
    sims = [CDKLM16.CDKLM16(ctx, zero, zero, zero, H, nx, ny, 1000.0, 1000.0, 1.0, 9.81, 1.2e-4, 0.0, 0.0)
            for _ in range(2)]
    ens = BatchedEnsemble.BatchedCDKLM16(sims)
    for s in sims:
        s.dt = np.float32(1.0e-7)
    with pytest.raises(Exception, match="too short"):
        ens.run_events(1, 1, interval=60.0)
    for s in sims:
        s.dt = np.float32(5.0)
    assert ens.run_events(1, 1, interval=60.0) == 12
