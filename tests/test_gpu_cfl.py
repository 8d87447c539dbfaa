"""The CFL reductions (csrc/cfl.cu) at the edges of their 128-column segments,
with dry and land cells: a domain's limit and every member's in a batch equal
the float32 evaluation of each cell's four quotients, bit for bit."""

import numpy as np
import pytest

from oracle import cdklm16_oracle as O

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from SWESimulators import BatchedEnsemble, CDKLM16, Common  # noqa: E402

SIZES = [(5, 4), (127, 6), (128, 9), (129, 40), (300, 7), (1400, 900)]


def _simulator(ctx, nx, ny, seed, land):
    rng = np.random.default_rng(seed)
    shape = (ny + 4, nx + 4)
    H = rng.uniform(0.2, 60.0, (ny + 5, nx + 5)).astype(np.float32)
    if land:
        H[3:4 + ny // 2, 3:4 + nx // 2] = 1.0e20
    eta = rng.uniform(-8.0, 2.0, shape).astype(np.float32)      # below -H in places: dry cells
    hu, hv = (rng.uniform(-90.0, 90.0, shape).astype(np.float32) for _ in range(2))
    zero = np.zeros(shape, np.float32)
    sim = CDKLM16.CDKLM16(ctx, zero, zero, zero, H, nx, ny, 700.0, 1300.0, 1.0, 9.81, 1.2e-4, 0.0, 0.0)
    sim.upload(eta, hu, hv)
    Bm = sim.downloadBathymetry()[1]
    want = O.max_dt(eta, hu, hv, Bm, nx, ny, np.float32(700.0), np.float32(1300.0), np.float32(9.81),
                    dtype=np.float32)
    return sim, np.float32(min(want, 1.0e5))


@pytest.mark.parametrize("land", [False, True])
def test_cfl_limits(land):
    ctx = Common.CUDAContext()
    sims, want = zip(*[_simulator(ctx, nx, ny, 7 + i, land) for i, (nx, ny) in enumerate(SIZES)])
    got = BatchedEnsemble.BatchedCDKLM16(list(sims)).max_dt()
    for m, (sim, w) in enumerate(zip(sims, want)):
        assert np.float32(got[m]) == w, SIZES[m]
        sim.updateDt(courant_number=1.0)
        assert np.float32(sim.dt) == w, SIZES[m]
