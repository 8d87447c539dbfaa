"""The tile kernel on tidal, coarse and shallow water whose least depth the
simulator tells: bit for bit the marching kernel's states, and the kernel that
runs by default."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from SWESimulators import CDKLM16, Common, _native  # noqa: E402

TILE = _native.GO_KERNEL_TILE
# (nx, ny, sides, least depth, amplitude of eta, of the currents, cell size, default kernel); the bounds of |eta|
# at 12.5 m are 7.8 m, at 30 m 19.3 m
CASES = [(97, 66, (1, 1, 1, 1), 30.0, 6.0, 1.0, 1000.0, TILE), (64, 48, (1, 2, 1, 2), 12.5, 7.6, 1.0, 1000.0, TILE),
         (65, 47, (2, 2, 2, 2), 12.5, 9.5, 1.0, 1000.0, TILE), (130, 70, (1, 1, 1, 1), 60.0, 0.5, 1.5, 30000.0, TILE),
         (96, 64, (1, 2, 1, 2), 2.0, 0.3, 0.5, 1000.0, TILE), (640, 600, (1, 1, 1, 1), 30.0, 6.0, 1.0, 1000.0, TILE),
         (640, 600, (1, 1, 1, 1), 2.0, 0.3, 0.5, 1000.0, "march"), (640, 600, (1, 2, 1, 2), 4.0, 0.3, 0.5, 30000.0, "march"),
         (640, 600, (1, 2, 1, 2), 60.0, 0.3, 0.5, 30000.0, TILE)]


def _simulator(case):
    nx, ny, sides, least, eta_amp, u_amp, dx, _ = case
    rng = np.random.default_rng(11)
    y, x = np.mgrid[0:ny + 5, 0:nx + 5]
    H = (least * (1.4 - 0.4 * np.cos(2 * np.pi * (x / (nx + 4) + 2 * y / (ny + 4))))).astype(np.float32)
    H = np.maximum(H, np.float32(least))
    y, x = y[:-1, :-1], x[:-1, :-1]
    eta = eta_amp * np.sin(2 * np.pi * x / (nx + 4) + 1.0) + 0.01 * rng.standard_normal(x.shape)
    hu = u_amp * least * np.cos(2 * np.pi * y / (ny + 4))
    hv = 0.5 * u_amp * least * np.sin(2 * np.pi * (x + y) / (nx + 4))
    dt = float(np.float32(0.1 * dx / (np.sqrt(9.81 * 2.5 * least) + 2 * u_amp)))
    return CDKLM16.CDKLM16(Common.CUDAContext(), *[a.astype(np.float32) for a in (eta, hu, hv)], H, nx, ny, dx, dx, dt,
                           9.81, 1.3e-4, 2.0e-3, boundary_conditions=Common.BoundaryConditions(*sides))


@pytest.mark.parametrize("case", CASES, ids=lambda c: "%dx%d-%gm-%gm-%gkm" % (c[0], c[1], c[3], c[4], c[6] / 1000))
def test_states_of_told_depths(case):
    sims = [_simulator(case) for _ in range(2)]
    kernel = sims[0]._domain.kernel()[0]
    assert kernel == case[-1] or (case[-1] == "march" and kernel in (4, 5, 6))
    sims[1]._domain.set_launch(4, 4)
    for n in (3, 2):
        for s in sims:
            s.step(n * float(np.float32(s.dt)))
    torch.cuda.synchronize()
    for a, b in zip(*[(s.gpu_data.h0, s.gpu_data.hu0, s.gpu_data.hv0, s.gpu_data.h1) for s in sims]):
        assert np.array_equal(a.view.cpu().numpy(), b.view.cpu().numpy())
    assert sims[0].status() == sims[1].status() == 0
