"""Which kernel the library runs by default, and the way back to it from an
explicit launch."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from SWESimulators import BatchedEnsemble, CDKLM16, Common, SyntheticCases as SC, _native  # noqa: E402

TILE, PAIR = _native.GO_KERNEL_TILE, 8


def _simulator(nx, ny=None):
    c = SC.grf(nx, ny=ny, dx=1000.0, steps=1)
    return CDKLM16.CDKLM16(Common.CUDAContext(), dt=c.dt, **c.kwargs())


@pytest.mark.parametrize("nx,kernel", [(64, TILE), (512, TILE), (1536, PAIR)])
def test_domain_returns_to_the_default(nx, kernel):
    sim, ref = _simulator(nx), _simulator(nx)
    default = sim._domain.kernel()
    assert default[0] == kernel
    sim._domain.set_launch(4, 8)
    assert sim._domain.kernel() == (4, 8)
    sim._launch_steps(2, np.float32(sim.dt), 0.0)
    sim._domain.set_launch(_native.GO_SHAPE_AUTO)
    assert sim._domain.kernel() == default
    sim._launch_steps(2, np.float32(sim.dt), 0.0)
    ref._launch_steps(4, np.float32(ref.dt), 0.0)
    torch.cuda.synchronize()
    for a, b in zip(sim.download(), ref.download()):
        assert np.array_equal(a, b)
    with pytest.raises(_native.NativeError):
        sim._domain.set_launch(_native.GO_SHAPE_AUTO, 8)
    with pytest.raises(_native.NativeError):
        sim._domain.set_launch(-2)


@pytest.mark.parametrize("n,nx,kernel", [(60, 128, TILE), (12, 700, PAIR)])
def test_batch_returns_to_the_default(n, nx, kernel):
    one = _simulator(nx)
    sims = [one] + [CDKLM16.CDKLM16(Common.CUDAContext(), dt=one.dt, **SC.grf(nx, dx=1000.0, steps=1).kwargs())
                    for _ in range(n - 1)]
    ens = BatchedEnsemble.BatchedCDKLM16(sims)
    default, tiles = ens.batch.kernel(), ens.batch.tiles()
    assert default[0] == kernel
    ens.batch.set_launch(4, 16, 0)
    assert ens.batch.kernel() == (4, 16)
    ens.advance(2)
    ens.batch.set_launch(_native.GO_SHAPE_AUTO)
    assert ens.batch.kernel() == default and ens.batch.tiles() == tiles
    ens.advance(2)
    ref = _simulator(nx)
    ref.step(4.0 * float(np.float32(ref.dt)))
    torch.cuda.synchronize()
    for a, b in zip(sims[n // 2].download(), ref.download()):
        assert np.array_equal(a, b)
