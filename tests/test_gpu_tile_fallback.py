"""Where the device refuses the one cooperative launch of all the steps of a
call, the tile kernel runs one launch per stage, with the same states."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from SWESimulators import CDKLM16, Common, SyntheticCases as SC, _native  # noqa: E402


@pytest.mark.parametrize("nx", [640, 200])       # 800 tiles, too many to be resident; 91, which fit
def test_steps_of_a_refused_cooperative_launch(nx):
    c = SC.grf(nx, dx=1000.0, seed_bathy=51000, seed_bumps=51500, steps=1)
    sims = [CDKLM16.CDKLM16(Common.CUDAContext(), dt=c.dt, **c.kwargs()) for _ in range(2)]
    sims[0]._domain.set_debug(_native.GO_DEBUG_STEPS_ANY_SIZE)
    for n in (3, 2):
        for s in sims:
            s._launch_steps(n, np.float32(c.dt), 0.0)
    torch.cuda.synchronize()
    for a, b in zip(sims[0].download(), sims[1].download()):
        assert np.array_equal(a, b)
    assert sims[0].status() == 0
