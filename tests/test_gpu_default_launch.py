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


CLOSED, PERIODIC = (1, 1, 1, 1), (1, 2, 1, 2)


def _domain_kernel(nx, ny, bc, land, field, exact=False, north=(0.0, 1.0)):
    dom = _native.Domain(nx, ny, 1000.0, 1000.0, 9.81, bc=bc, north=north)
    if land is not None:
        dom.set_land(land)
    if exact:
        dom.set_arith(_native.GO_ARITH_EXACT)
    if field:
        w = torch.zeros((ny, nx), device="cuda")
        dom.set_wind_field(w, w, w, w)
        before = dom.kernel()
        dom.set_wind_uniform(0.0, 0.0, 0.0, 0.0)
        dom.set_wind_field(w, w, w, w)               # the choice follows the wind kind
        assert dom.kernel() == before
    return dom.kernel()[0]


@pytest.mark.parametrize("nx,ny,bc,land,field,kernel", [
    (500, 500, CLOSED, None, False, TILE), (500, 500, CLOSED, True, True, TILE), (700, 700, CLOSED, None, False, "march"),
    (700, 700, PERIODIC, True, False, "march"), (700, 700, CLOSED, False, True, TILE),
    (1300, 1100, PERIODIC, None, False, "march"), (1300, 1100, PERIODIC, False, False, PAIR),
    (1300, 1100, PERIODIC, False, True, "march"), (1300, 1200, PERIODIC, False, True, PAIR),
    (1300, 1100, CLOSED, False, False, "march"), (1300, 1100, PERIODIC, True, False, "march"),
    (1600, 1600, PERIODIC, None, False, PAIR), (1600, 1600, CLOSED, None, True, PAIR),
    (1600, 1600, PERIODIC, True, True, PAIR), (1600, 1600, CLOSED, False, True, PAIR),
    (1600, 1600, CLOSED, True, False, "march"), (2400, 2400, CLOSED, True, False, PAIR),
    (2400, 2400, CLOSED, True, True, "march"), (3600, 3600, CLOSED, True, True, PAIR)])
def test_default_kernel_by_sides_land_and_wind(nx, ny, bc, land, field, kernel):
    got = _domain_kernel(nx, ny, bc, land, field)
    assert got == kernel or (kernel == "march" and got in (4, 5, 6))


def test_default_kernel_of_the_forms_it_was_not_measured_for():
    """IEEE quotients and rotated grids: as before land was asked about."""
    for kw in (dict(exact=True), dict(north=(0.6, 0.8))):
        assert _domain_kernel(500, 500, CLOSED, False, False, **kw) in (4, 5, 6)
        assert _domain_kernel(1300, 1100, PERIODIC, False, False, **kw) in (4, 5, 6)
        assert _domain_kernel(1600, 1600, CLOSED, True, True, **kw) == PAIR


def _members(n, nx, land, bc, field=False):
    """n flat-bottomed members, the first `land` of them told of land."""
    ctx, sims = Common.CUDAContext(), []
    from SWESimulators import WindStress
    shape = (3, 4) if field else (1, 1)
    rng = np.random.default_rng(1)
    for m in range(n):
        H = np.full((nx + 5, nx + 5), 50.0, np.float32)
        if m < land:
            H[nx // 3:nx // 3 + 6, nx // 2:nx // 2 + 8] = 1.0e20
        eta, hu, hv = (rng.standard_normal((nx + 4, nx + 4)).astype(np.float32) * s for s in (0.1, 1.0, 1.0))
        wind = WindStress.WindStress(t=[0], X=[np.full(shape, 1e-4, np.float32)], Y=[np.full(shape, 1e-4, np.float32)])
        sims.append(CDKLM16.CDKLM16(ctx, eta, hu, hv, H, nx, nx, 1000.0, 1000.0, 5.0, 9.81, 1.2e-4, 0.0,
                                    boundary_conditions=Common.BoundaryConditions(*bc), wind_stress=wind))
    return sims


@pytest.mark.parametrize("land,bc,field,kernel", [
    (0, PERIODIC, False, (PAIR, None)), (1, PERIODIC, False, (PAIR, None)), (12, PERIODIC, True, (PAIR, None)),
    (1, CLOSED, False, (PAIR, None)), (3, CLOSED, False, (4, 16)), (12, CLOSED, False, (4, 16)),
    (1, CLOSED, True, (4, 16)), (0, CLOSED, True, (PAIR, None))])
def test_default_kernel_of_batches_with_land(land, bc, field, kernel):
    sims = _members(12, 420, land, bc, field)
    ens = BatchedEnsemble.BatchedCDKLM16(sims)
    got = ens.batch.kernel()
    assert got[0] == kernel[0] and kernel[1] in (None, got[1])
    if (land, bc) in ((1, PERIODIC), (1, CLOSED)) and not field:
        ens.advance(3)                       # a land member among others without: each as alone
        alone = [s for s in _members(2, 420, 1, bc)]
        for s in alone:
            s._domain.set_launch(4, 8)
            s.step(3.0 * float(np.float32(s.dt)))
        torch.cuda.synchronize()
        for s, w in zip(sims, alone):
            for a, b in zip(s.download(), w.download()):
                assert np.array_equal(a, b)


def test_default_kernel_of_small_batches_with_land():
    assert BatchedEnsemble.BatchedCDKLM16(_members(4, 420, 1, PERIODIC)).batch.kernel() == (4, 16)


@pytest.mark.parametrize("n,nx,bc,rows", [(12, 700, CLOSED, 29), (12, 700, PERIODIC, 22), (40, 240, CLOSED, 32),
                                             (16, 512, PERIODIC, 37), (100, 260, PERIODIC, 24)])
def test_strip_heights_of_batches_count_the_region_strips(n, nx, bc, rows):
    """Closed east and west sides: the outer column blocks are frame, and with
    two column blocks there are no others."""
    assert BatchedEnsemble.BatchedCDKLM16(_members(n, nx, 0, bc)).batch.kernel() == (PAIR, rows)


@pytest.mark.parametrize("nx,ny", [(300, 2500000), (5, 2400000), (300, 60000)])
def test_strips_of_tall_grids_fit_in_a_launch(nx, ny):
    dom = _native.Domain(nx, ny, 1000.0, 1000.0, 9.81, bc=CLOSED)
    for land in (False, True):
        dom.set_land(land)
        kernel, rows = dom.kernel()
        assert kernel == PAIR and -(-ny // rows) <= 65535 and (rows <= 36 or ny > 36 * 65535)
    dom.set_launch(4)
    assert -(-ny // dom.kernel()[1]) <= 65535
