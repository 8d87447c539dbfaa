"""The tile stage kernel, the default of grids below the column-pair kernel's:
bit for bit the marching kernel's states (launch shape 4), ghost cells and
the second state included, at sizes around its 32 x 16 tiles, for every
boundary kind, with land, shallow and dry cells, per-cell wind and both
friction laws; in one launch for all the steps of a call (up to one tile per
SM) and one launch per stage; states either side of the deep-water bounds;
and no index out of bounds in the checked-index build."""

import os
import subprocess
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
PKG = os.path.join(os.path.dirname(HERE), "gpu-ocean_b200")
if __name__ == "__main__":
    sys.path[:0] = [os.path.dirname(HERE), PKG]

torch = pytest.importorskip("torch")
if __name__ != "__main__":
    pytestmark = pytest.mark.gpu
    if not torch.cuda.is_available():
        pytest.skip("needs a CUDA GPU", allow_module_level=True)

from SWESimulators import BatchedEnsemble, CDKLM16, Common, WindStress  # noqa: E402

WALLS, CHANNEL, TORUS = (1, 1, 1, 1), (1, 2, 1, 2), (2, 2, 2, 2)
# (nx, ny, sides, water, wind, friction)
CASES = [(4, 4, TORUS, "deep", "uniform", "quadratic"), (5, 11, WALLS, "deep", "none", "none"),
         (32, 16, WALLS, "deep", "uniform", "quadratic"), (31, 15, TORUS, "deep", "field", "linear"),
         (33, 17, CHANNEL, "deep", "uniform", "none"), (64, 33, (2, 1, 2, 1), "shallow", "field", "quadratic"),
         (97, 130, WALLS, "land", "field", "quadratic"), (130, 97, CHANNEL, "land", "uniform", "linear"),
         (200, 100, WALLS, "edge", "uniform", "quadratic"), (257, 9, CHANNEL, "shallow", "none", "linear"),
         (600, 131, WALLS, "land", "uniform", "quadratic"), (577, 300, TORUS, "edge", "field", "quadratic")]


def _simulator(ctx, case, dx=1000.0):
    nx, ny, sides, water, wind, friction = case
    rng = np.random.default_rng(17)

    def smooth(shape):
        a = rng.standard_normal(shape)
        for axis in (0, 1):
            a = sum(np.roll(a, s, axis) for s in range(-3, 4)) / np.sqrt(7.0)
        return a
    H = np.maximum(60.0 + 15.0 * smooth((ny + 5, nx + 5)), 12.0)
    eta, hu, hv = (s * smooth((ny + 4, nx + 4)) for s in (0.3, 4.0, 4.0))
    if water == "shallow":      # cells either side of the desingularisation depth and the cut-off
        H = 0.4 * rng.random((ny + 5, nx + 5))
        eta, hu, hv = 0.1 * eta, 0.01 * hu, 0.01 * hv
    if water == "land":
        H[smooth(H.shape) > 1.2] = 1.0e20
    if water == "edge":         # corners, eta and currents either side of the deep-water bounds
        H = np.maximum(3.6 + 0.4 * smooth(H.shape), 2.5)
        eta, hu, hv = 0.9 * smooth(eta.shape).clip(-2.2, 2.4), 2.0 * hu, 2.0 * hv
    f32 = [a.astype(np.float32) for a in (eta, hu, hv, H)]
    kw = {}
    if wind != "none":
        shape = (1, 1) if wind == "uniform" else (5, 6)
        kw["wind_stress"] = WindStress.WindStress(t=[0], X=[(1e-4 * rng.standard_normal(shape)).astype(np.float32)],
                                                  Y=[(1e-4 * rng.standard_normal(shape)).astype(np.float32)])
    dt = float(np.float32(0.1 * dx / (np.sqrt(9.81 * 150.0) + 6.0)))
    return CDKLM16.CDKLM16(ctx, f32[0], f32[1], f32[2], f32[3], nx, ny, dx, dx, dt, 9.81, 1.2e-4,
                           0.0 if friction == "none" else 2.0e-3, coriolis_beta=2.0e-11,
                           boundary_conditions=Common.BoundaryConditions(*sides),
                           linear_friction=friction == "linear", **kw)


def _run(case, launch=None, calls=(3, 1, 2)):
    sim = _simulator(Common.CUDAContext(), case)
    if launch is not None:
        sim._domain.set_launch(*launch)
    for n in calls:
        sim.step(n * float(np.float32(sim.dt)))
    torch.cuda.synchronize()
    g = sim.gpu_data
    return [a.view.cpu().numpy() for a in (g.h0, g.hu0, g.hv0, g.h1, g.hu1, g.hv1)], sim.status()


@pytest.mark.parametrize("case", CASES, ids=lambda c: "%dx%d-%s" % (c[0], c[1], c[3]))
def test_tile_kernel_equals_marching_kernel(case):
    tile, s_tile = _run(case)
    march, s_march = _run(case, launch=(4, 4))
    assert s_tile == s_march
    for a, b in zip(tile, march):
        assert np.array_equal(a, b, equal_nan=True)


# members of a batch share the friction law and the wind kind; narrow grids, so
# that the batch takes the tile kernel
BATCHES = [[(32, 16, WALLS, "deep", "uniform", "quadratic"), (33, 17, TORUS, "edge", "uniform", "quadratic"),
            (120, 50, CHANNEL, "deep", "uniform", "quadratic"), (5, 90, WALLS, "shallow", "uniform", "quadratic")],
           [(96, 31, CHANNEL, "shallow", "field", "linear"), (64, 64, WALLS, "edge", "field", "linear")]]


def _run_batch(cases, graph_steps):
    ctx = Common.CUDAContext()
    sims = [_simulator(ctx, c) for c in cases]
    ens = BatchedEnsemble.BatchedCDKLM16(sims, graph_steps=graph_steps)
    ens.advance(5)
    torch.cuda.synchronize()
    return sims, ens.member_status()


@pytest.mark.parametrize("graph_steps", [0, 2])
@pytest.mark.parametrize("cases", BATCHES, ids=["quadratic", "linear-field"])
def test_batched_tile_kernel_equals_marching_kernel(cases, graph_steps):
    sims, status = _run_batch(cases, graph_steps)
    for sim, word, case in zip(sims, status, cases):
        march, s_march = _run(case, launch=(4, 4), calls=(1,) * 5)
        g = sim.gpu_data
        assert word == s_march
        for a, b in zip((g.h0, g.hu0, g.hv0, g.h1, g.hu1, g.hv1), march):
            assert np.array_equal(a.view.cpu().numpy(), b, equal_nan=True)


def test_checked_indices_of_the_tile_kernel(tmp_path):
    if not os.path.exists(os.path.join(PKG, "lib", "libgocean_debug.so")):
        pytest.skip("lib/libgocean_debug.so not built")
    out = str(tmp_path / "debug.npz")
    subprocess.run([sys.executable, os.path.abspath(__file__), out], check=True, timeout=600,
                   env=dict(os.environ, GOCEAN_DEBUG_BOUNDS="1"))
    dbg = np.load(out)
    for i, case in enumerate(CASES):
        plain, status = _run(case)
        assert int(dbg["status%d" % i]) == status
        for k, a in enumerate(plain):
            assert np.array_equal(dbg["a%d_%d" % (i, k)], a, equal_nan=True)
    assert not dbg["batch"].any()


if __name__ == "__main__":
    res = {}
    for i, case in enumerate(CASES):
        arrays, status = _run(case)
        res["status%d" % i] = np.array(status)
        for k, a in enumerate(arrays):
            res["a%d_%d" % (i, k)] = a
    # GO_STATUS_BOUNDS of the batches' members
    res["batch"] = np.array([w & 8 for cases in BATCHES for w in _run_batch(cases, 0)[1]])
    np.savez(sys.argv[1], **res)
