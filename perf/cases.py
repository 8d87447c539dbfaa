"""Performance cases of the framework: what its users run, over the range of sizes they run it at.

* step       a CDKLM16 simulator advanced through ``CDKLM16.step``: closed basins, periodic channels and
             coastal domains with land, uniform or per-cell wind, quadratic or linear friction, drifters,
             model error after every step, a CFL update before the steps.
* ensemble   ``BatchedCDKLM16.run_events``: the members of an ensemble step, are perturbed, and take a new
             common time step.
* domains    ``BatchedCDKLM16.advance`` over domains of different sizes, each at its own time step, and their
             CFL limits afterwards.
* gradient   ``MisfitProblem.gradient``: forward run, misfit and reverse sweep of one domain.
* gradients  ``BatchedMisfitProblem.gradient``: the same for every member of an ensemble.

``exact`` evaluates the scheme in float64 with plain torch.
"""

import math
import os
import sys

import numpy as np
import torch

_PACKAGE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpu-ocean_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

G = 9.81
F0 = 1.2e-4
BETA = 2.0e-11
FRICTION = 3.0e-3
WIND = 0.1 * math.cos(math.pi / 4) / 1025.0      # 0.1 N/m^2 at 45 degrees
THETA = 1.3
CUTOFF = 1.0e-5
LAND = 1.0e20
MODEL_ERROR_Q0 = 1.0e-4


# ---- the cases ------------------------------------------------------------------

def _step(name, nx, ny, steps, **options):
    case = {"kind": "step", "nx": nx, "ny": ny, "steps": steps, "dx": 1000.0, "periodic_ew": False,
            "periodic_ns": False, "flat": False, "land": False, "wind": "uniform", "beta": True, "friction": "quadratic",
            "drifters": 0, "model_error": False, "update_dt": False}
    case.update(options)
    if name:
        case["name"] = name
    return case


def listed():
    return [
        # the smallest grids of the test suite: every launch is shorter than it takes to issue
        _step("basin-64x48", 64, 48, 10, dx=2000.0),
        # the bump in a closed flat basin that the scheme is validated on
        _step("bump-256", 256, 256, 10, dx=200.0, flat=True, wind="none", beta=False, friction="none"),
        # a data-assimilation cycle of a small coastal model: new time step, a few steps, drifters in the flow
        _step("coast-301x221", 301, 221, 4, land=True, wind="field", drifters=500, update_dt=True),
        # a single ensemble member stepped alone
        _step("member-512", 512, 512, 6, periodic_ew=True),
        # a regional forecast with land and wind from an atmosphere model, ragged sizes
        _step("regional-1030x771", 1030, 771, 4, land=True, wind="field"),
        # the model error after every step, as a stochastic ensemble member runs
        _step("stochastic-1501x1203", 1501, 1203, 2, periodic_ew=True, model_error=True, beta=False),
        # a large closed basin with linear friction
        _step("basin-1999x1531", 1999, 1531, 4, friction="linear"),
        # the throughput benchmark
        _step("headline-4096", 4096, 4096, 4, dx=500.0, periodic_ew=True),
        # the ensemble benchmark: 60 s of every member, model error, new time step
        {"name": "ensemble-100x512", "kind": "ensemble", "members": 100, "nx": 512, "ny": 512},
        # independent domains of different sizes, one launch per stage for all
        {"name": "domains-32", "kind": "domains", "members": 32, "smallest": 128, "largest": 640, "steps": 4},
        # gradient of an observation misfit, half of the run recomputed from a checkpoint
        {"name": "gradient-512", "kind": "gradient", "nx": 512, "ny": 512, "steps": 20, "every": 10},
        # gradients of an ensemble under a binomial schedule
        {"name": "gradients-8x1024", "kind": "gradients", "members": 8, "nx": 1024, "ny": 1024, "steps": 6,
         "snapshots": 3},
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _pair(rng, lo, hi):
    n, aspect = _size(rng, lo, hi), rng.uniform(0.6, 1.6)
    return max(lo, min(hi, int(n * math.sqrt(aspect)))), max(lo, min(hi, int(n / math.sqrt(aspect))))


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["ensemble", "domains", "gradient", "gradients"])
    if kind == "step":
        nx, ny = _pair(rng, 40, 4096)
        land = rng.random() < 0.4
        stochastic = not land and rng.random() < 0.2
        case = _step(None, nx, ny, rng.randint(1, 10 if nx * ny < 1 << 20 else 4),
                     dx=float(rng.choice([200, 500, 1000, 2000])), periodic_ew=not land and rng.random() < 0.5,
                     periodic_ns=not land and rng.random() < 0.2, land=land,
                     wind=rng.choice(["none", "uniform", "field"]), beta=not stochastic and rng.random() < 0.7,
                     friction=rng.choice(["quadratic", "quadratic", "linear", "none"]),
                     drifters=rng.choice([0, 0, 0, _size(rng, 10, 100000)]), model_error=stochastic,
                     update_dt=rng.random() < 0.3)
        return case
    if kind == "ensemble":
        nx, ny = _pair(rng, 64, 700)
        return {"kind": kind, "members": max(2, min(100, int(rng.uniform(0.2, 1.0) * 100 * 512 * 512 / (nx * ny)))),
                "nx": nx, "ny": ny}
    if kind == "domains":
        lo = _size(rng, 64, 256)
        return {"kind": kind, "members": rng.randint(4, 48), "smallest": lo, "largest": lo + _size(rng, 32, 512),
                "steps": rng.randint(1, 6)}
    steps = rng.randint(4, 16)
    if kind == "gradient":
        nx, ny = _pair(rng, 64, 1100)
        return {"kind": kind, "nx": nx, "ny": ny, "steps": steps, "every": rng.randint(2, steps)}
    nx, ny = _pair(rng, 64, 1024)
    return {"kind": kind, "members": rng.randint(2, 8), "nx": nx, "ny": ny, "steps": min(steps, 6),
            "snapshots": rng.randint(1, 4)}


# ---- inputs ---------------------------------------------------------------------

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _smooth(gen, ny, nx, corr=20.0):
    """Unit-variance random field with a correlation length of `corr` cells, periodic on the grid."""
    white = torch.randn((ny, nx), generator=gen, dtype=torch.float64, device=gen.device)
    ky = torch.fft.fftfreq(ny, dtype=torch.float64, device=gen.device)[:, None]
    kx = torch.fft.rfftfreq(nx, dtype=torch.float64, device=gen.device)[None, :]
    smooth = torch.fft.irfft2(torch.fft.rfft2(white) * torch.exp(-(math.pi * corr) ** 2 * (kx ** 2 + ky ** 2)), s=(ny, nx))
    return (smooth - smooth.mean()) / smooth.std()


def _ghosts(field, extra):
    """The periodic field on the grid with two ghost cells (extra = 4) or corners (extra = 5) added."""
    ny, nx = field.shape
    j = (torch.arange(ny + extra, device=field.device) - 2) % ny
    i = (torch.arange(nx + extra, device=field.device) - 2) % nx
    return field[j][:, i].to(torch.float32)


def _ocean(seed, nx, ny, dx=1000.0, flat=False, land=False):
    """Corner depths (land masked), initial state and a stable time step of one domain, as host arrays."""
    gen = torch.Generator(device=_device())
    gen.manual_seed(int(seed))
    if flat:
        H = torch.full((ny + 5, nx + 5), 60.0, device=gen.device)
        move, amp = torch.rand(3, generator=gen, dtype=torch.float64, device=gen.device).tolist()[:2], 0.5
        y = torch.arange(ny + 4, device=gen.device)[:, None] - 1.5 - ny * (0.4 + 0.2 * move[0])
        x = torch.arange(nx + 4, device=gen.device)[None, :] - 1.5 - nx * (0.4 + 0.2 * move[1])
        eta = (amp * torch.exp(-(x ** 2 + y ** 2) / 100.0)).to(torch.float32)
        hu = torch.zeros_like(eta)
        hv = torch.zeros_like(eta)
    else:
        H = _ghosts(100.0 + 40.0 * _smooth(gen, ny, nx), 5).clamp(min=10.0)
        eta = _ghosts(0.3 * _smooth(gen, ny, nx), 4)
        hu, hv = (_ghosts(4.0 * _smooth(gen, ny, nx), 4) for _ in range(2))
    depth = H.cpu().numpy()
    if land:
        dry = _ghosts(_smooth(gen, ny, nx), 5) > 1.1
        depth = np.ma.array(depth, mask=dry.cpu().numpy())
        inland = dry[1:, 1:] & dry[:-1, 1:] & dry[1:, :-1] & dry[:-1, :-1]
        eta, hu, hv = (torch.where(inland, torch.zeros_like(a), a) for a in (eta, hu, hv))
    # half the CFL limit of the deepest water, in 64ths of a second (exact in float32)
    dt = math.floor(64.0 * 0.5 * 0.25 * dx / (math.sqrt(G * float(H.max()) + 20.0) + 1.0)) / 64.0
    return depth, eta.cpu().numpy(), hu.cpu().numpy(), hv.cpu().numpy(), dt


def _wind_fields(seed):
    rng = np.random.default_rng(seed)
    return [(WIND * (1.0 + 0.5 * rng.standard_normal((6, 7)))).astype(np.float32) for _ in range(2)]


def _sides(case):
    """Boundary codes north, east, south, west (1 wall, 2 periodic)."""
    ns, ew = (2 if case.get("periodic_" + k) else 1 for k in ("ns", "ew"))
    return ns, ew, ns, ew


def _simulator(ctx, ocean, nx, ny, dx, sides, f, beta, r, linear=False, wind=None, **options):
    from SWESimulators import CDKLM16, Common, WindStress
    H, eta, hu, hv, dt = ocean
    if wind is not None:
        options["wind_stress"] = WindStress.WindStress(t=[0], X=[wind[0]], Y=[wind[1]])
    return CDKLM16.CDKLM16(ctx, eta, hu, hv, H, nx, ny, dx, dx, dt, G, f, r, coriolis_beta=beta,
                           boundary_conditions=Common.BoundaryConditions(*sides), linear_friction=linear, **options)


def _uniform_wind():
    return [np.array([[WIND]], dtype=np.float32) for _ in range(2)]


def _step_wind(case, seed):
    return {"none": None, "uniform": _uniform_wind(), "field": _wind_fields(seed + 1)}[case["wind"]]


def _friction(case):
    return 0.0 if case["friction"] == "none" else (1.0e-3 if case["friction"] == "linear" else FRICTION)


def _domain_sizes(case):
    lo, hi, n = case["smallest"], case["largest"], case["members"]
    return [(lo + (hi - lo) * m // max(1, n - 1), lo + (hi - lo) * ((5 * m + 3) % n) // n) for m in range(n)]


def _observed(case, seed):
    """64 observed cells at every fourth step and the last, with observed values."""
    rng = np.random.default_rng(seed + 7)
    cells = np.stack([rng.integers(0, case["nx"], 64), rng.integers(0, case["ny"], 64)], axis=1).astype(np.int32)
    steps = sorted(set(range(4, case["steps"] + 1, 4)) | {case["steps"]})
    values = rng.standard_normal((len(steps), 64, 3)) * np.array([0.3, 3.0, 3.0])
    return cells, steps, values.astype(np.float32)


def _gradient_inputs(case, seed):
    """Initial state (3, ny, nx) and wind (2, ny, nx) of one member, on the device, and its bathymetry."""
    H, eta, hu, hv, dt = _ocean(seed, case["nx"], case["ny"])
    gen = torch.Generator(device=_device())
    gen.manual_seed(seed + 3)
    x0 = torch.stack([torch.from_numpy(a[2:-2, 2:-2]).to(gen.device) for a in (eta, hu, hv)])
    wind = torch.stack([WIND * (1.0 + 0.3 * _smooth(gen, case["ny"], case["nx"])) for _ in range(2)]).to(torch.float32)
    return x0, wind, (H, eta, hu, hv, dt)


def prepare(case, seed):
    from SWESimulators import Adjoint, BatchedEnsemble, Common
    from SWESimulators.GPUDrifterCollection import GPUDrifterCollection
    seed = int(seed) % (1 << 30)
    ctx = Common.CUDAContext()
    kind = case["kind"]
    if kind == "step":
        nx, ny, dx = case["nx"], case["ny"], case["dx"]
        sim = _simulator(ctx, _ocean(seed, nx, ny, dx, case["flat"], case["land"]), nx, ny, dx, _sides(case), F0,
                         BETA if case["beta"] else 0.0, _friction(case), case["friction"] == "linear",
                         _step_wind(case, seed), small_scale_perturbation=case["model_error"],
                         small_scale_perturbation_amplitude=MODEL_ERROR_Q0, use_lcg=True, courant_number=0.5)
        if case["model_error"]:
            sim.small_scale_model_error.random_state = np.random.RandomState(seed)
            sim.small_scale_model_error.resetSeed()
        if case["drifters"]:
            drifters = GPUDrifterCollection(ctx, case["drifters"], boundaryConditions=sim.boundary_conditions,
                                            domain_size_x=nx * dx, domain_size_y=ny * dx)
            drifters.setDrifterPositions(_drifter_positions(case, seed))
            drifters.setObservationPosition(np.array([0.5 * nx * dx, 0.5 * ny * dx]))
            sim.attachDrifters(drifters)
        torch.cuda.synchronize()
        return {"case": case, "sim": sim, "t": case["steps"] * sim.dt}
    if kind == "ensemble":
        nx, ny = case["nx"], case["ny"]
        sims = [_simulator(ctx, _ocean(seed + 11 * m, nx, ny), nx, ny, 1000.0, (1, 2, 1, 2), F0, BETA, FRICTION,
                           wind=_uniform_wind()) for m in range(case["members"])]
        ens = BatchedEnsemble.BatchedCDKLM16(sims)
        ens.update_dt(0.7)
        torch.cuda.synchronize()
        return {"case": case, "ens": ens, "event": 0}
    if kind == "domains":
        sims = [_simulator(ctx, _ocean(seed + 11 * m, nx, ny), nx, ny, 1000.0, (1, 2, 1, 2), F0, BETA, FRICTION,
                           wind=_uniform_wind()) for m, (nx, ny) in enumerate(_domain_sizes(case))]
        ens = BatchedEnsemble.BatchedCDKLM16(sims)
        torch.cuda.synchronize()
        return {"case": case, "ens": ens}
    nx, ny = case["nx"], case["ny"]
    obs = Adjoint.Observations(*_observed(case, seed))
    inputs = [_gradient_inputs(case, seed + 11 * m) for m in range(case.get("members", 1))]
    dt = min(i[2][4] for i in inputs)
    sims = [_simulator(ctx, i[2][:4] + (dt,), nx, ny, 1000.0, (1, 2, 1, 2), F0, BETA, FRICTION) for i in inputs]
    if kind == "gradient":
        state = {"problem": Adjoint.MisfitProblem(sims[0], case["steps"], obs, checkpoint_every=case["every"]),
                 "x0": inputs[0][0], "wind": inputs[0][1]}
    else:
        state = {"problem": Adjoint.BatchedMisfitProblem(sims, case["steps"], obs, snapshots=case["snapshots"]),
                 "x0": torch.stack([i[0] for i in inputs]), "wind": torch.stack([i[1] for i in inputs])}
    torch.cuda.synchronize()
    return dict(state, case=case)


def _drifter_positions(case, seed):
    rng = np.random.default_rng(seed + 5)
    size = np.array([case["nx"], case["ny"]]) * case["dx"]
    return (0.1 + 0.8 * rng.random((case["drifters"], 2))) * size


# ---- one pass -------------------------------------------------------------------

def _state_of(sim):
    g = sim.gpu_data
    return [a.view[2:-2, 2:-2] for a in (g.h0, g.hu0, g.hv0)]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        sim = state["sim"]
        out = {}
        if case["update_dt"]:
            dt = sim.dt
            sim.updateDt()
            out["cfl"] = float(sim.dt)
            sim.dt = min(dt, sim.dt)
        sim.step(state["t"])
        out["state"] = _state_of(sim)
        if case["drifters"]:
            out["drifters"] = sim.drifters.driftersDevice.view
        if case["model_error"]:
            noise = sim.small_scale_model_error
            out["seeds"] = noise.seed.tensor[:, :noise.seed.nx]
        return out
    if kind == "ensemble":
        ens = state["ens"]
        state["event"] += 1
        steps = ens.run_events(state["event"], 1, interval=60.0)
        return {"steps": steps, "dt": float(ens.sims[0].dt), "members": [x for s in ens.sims[:16] for x in _state_of(s)]}
    if kind == "domains":
        ens = state["ens"]
        ens.advance(case["steps"])
        return {"limits": ens.max_dt(), "members": [x for s in ens.sims[:20] for x in _state_of(s)]}
    if kind == "gradient":
        J, ge, gu, gv, gx, gy = state["problem"].gradient(*state["x0"], *state["wind"])
        return {"J": float(J), "state": [ge, gu, gv], "wind": [gx, gy]}
    J, gs, gw = state["problem"].gradient(state["x0"], state["wind"])
    return {"J": J, "state": gs, "wind": gw}


# ---- bytes and operations -------------------------------------------------------

def work(case):
    """Per cell and step: stage one reads the state and the corners (16 bytes) and writes the state (12), stage two
    also reads the state before the step (28 + 12); about 290 additions and multiplications per stage.  A stage's
    adjoint reads the stage's input and output, the adjoint of the output and the corners and writes the adjoint of
    the input and the wind's; about three times the forward's operations."""
    kind = case["kind"]
    if kind == "step":
        cells = case["nx"] * case["ny"]
        per_step = 68.0 + (16.0 if case["wind"] == "field" else 0.0) + (52.0 if case["model_error"] else 0.0)
        b = cells * (case["steps"] * per_step + (16.0 if case["update_dt"] else 0.0))
        f = cells * case["steps"] * (580.0 + (80.0 if case["model_error"] else 0.0))
        return {"bytes": b + case["steps"] * 16.0 * case["drifters"], "flops": f}
    if kind == "ensemble":
        cells = case["members"] * case["nx"] * case["ny"]
        steps = 17.0       # 60 s at 0.7 of the CFL limit of water 200-250 m deep on a 1 km grid
        return {"bytes": cells * (68.0 * steps + 8.0 + 16.0), "flops": cells * 580.0 * steps}
    if kind == "domains":
        cells = sum(nx * ny for nx, ny in _domain_sizes(case))
        return {"bytes": cells * (68.0 * case["steps"] + 16.0), "flops": cells * 580.0 * case["steps"]}
    cells = case.get("members", 1) * case["nx"] * case["ny"]
    return {"bytes": cells * case["steps"] * (84.0 + 136.0), "flops": cells * case["steps"] * (580.0 + 1740.0)}


# ---- the scheme in float64 ------------------------------------------------------

def _minmod(b, c, f):
    sb, sc, sf = torch.sign(b), torch.sign(c), torch.sign(f)
    return 0.25 * sb * (sb + sc) * (sc + sf) * torch.minimum(torch.minimum(b.abs(), c.abs()), f.abs())


def _flux(hm, am, bm, hp, ap, bp):
    """Central-upwind flux through faces with states (depth, normal, tangential velocity) either side."""
    def side(h, a, b):
        wet = h > CUTOFF
        z = torch.zeros_like(h)
        c = torch.where(wet, torch.sqrt(G * torch.where(wet, h, torch.ones_like(h))), z)
        return [torch.where(wet, q, z) for q in (h * a, h * a * a + 0.5 * G * h * h, h * a * b, a)] + [c]
    m0, m1, m2, am_, cm = side(hm, am, bm)
    p0, p1, p2, ap_, cp = side(hp, ap, bp)
    lo = torch.minimum(am_ - cm, ap_ - cp).clamp(max=0.0)
    hi = torch.maximum(am_ + cm, ap_ + cp).clamp(min=0.0)
    still = (hi - lo).abs() < 0.1
    width = torch.where(still, torch.ones_like(hi), hi - lo)
    f0 = (hi * m0 - lo * p0 + hi * lo * (hp - hm)) / width
    f1 = (hi * m1 - lo * p1 + hi * lo * (p0 - m0)) / width
    f2 = torch.where(am + ap > 0, m2, p2)
    return [torch.where(still, torch.zeros_like(q), q) for q in (f0, f1, f2)]


def _axis(e, a, b, f, land, depth, d, wall):
    """Fluxes through the n + 1 faces along the last axis: eta, normal and tangential velocity with two ghost cells
    either side, the Coriolis parameter f (its sign turned for the y axis) and the face depths."""
    n = e.shape[-1] - 4
    ghost = torch.ones(n + 4, dtype=e.dtype, device=e.device)
    if wall:
        ghost[:2] = -1.0
        ghost[n + 2:] = -1.0
    first, last = ghost[1:n + 2], ghost[2:n + 3]       # tangential signs at the faces' low and high cells
    near = ghost[1:n + 3].clone()
    near[-1] = 1.0                                     # the slope correction leaves the far ghost cell's sign
    L, C, R = slice(0, n + 2), slice(1, n + 3), slice(2, n + 4)
    f = f.expand(e.shape)
    fb = f * b * ghost

    def slope(q):
        return _minmod(THETA * (q[..., C] - q[..., L]), 0.5 * (q[..., R] - q[..., L]), THETA * (q[..., R] - q[..., C]))
    V = d / (2.0 * G)
    K = _minmod(THETA * G * (e[..., C] - e[..., L] - V * (fb[..., C] + fb[..., L])),
                0.5 * G * (e[..., R] - e[..., L] - V * (fb[..., R] + 2.0 * fb[..., C] + fb[..., L])),
                THETA * G * (e[..., R] - e[..., C] - V * (fb[..., C] + fb[..., R])))
    turn = d * f[..., C] * b[..., C] * near
    lo, hi = e[..., C] + depth[..., 1:n + 3], e[..., C] + depth[..., 2:n + 4]
    q = (K + turn) / (2.0 * G)
    K = torch.where(lo - q > 0, K, -turn + 2.0 * G * lo)
    K = torch.where(hi + q > 0, K, -turn - 2.0 * G * hi)
    da, db = slope(a), slope(b)
    m, p = slice(1, n + 2), slice(2, n + 3)
    H = depth[..., 2:n + 3]
    hm = (e[..., m] + H + (K[..., :-1] + d * f[..., m] * b[..., m] * first) / (2.0 * G)).clamp(min=0.0)
    hp = (e[..., p] + H - (K[..., 1:] + d * f[..., p] * b[..., p] * last) / (2.0 * G)).clamp(min=0.0)
    F = _flux(hm, a[..., m] + 0.5 * da[..., :-1], b[..., m] + 0.5 * db[..., :-1],
              hp, a[..., p] - 0.5 * da[..., 1:], b[..., p] - 0.5 * db[..., 1:])
    closed = land[..., m] | land[..., p]
    return [torch.where(closed, torch.zeros_like(q), q) for q in F]


def _pad(q, periodic, sign):
    """Two ghost cells either side of the last axis: wrapped, or mirrored with the given sign."""
    if periodic:
        return torch.cat([q[..., -2:], q, q[..., :2]], dim=-1)
    return torch.cat([sign * q[..., :2].flip(-1), q, sign * q[..., -2:].flip(-1)], dim=-1)


class _Model64:
    """The scheme on one domain of water deeper than the desingularisation depth, with or without land; states are
    interior arrays (ny, nx) in float64."""

    def __init__(self, H, nx, ny, dx, sides, f, beta, r, linear=False, wind=None, wind_cells=None):
        dev = _device()
        self.nx, self.ny, self.dx, self.r, self.linear = nx, ny, float(dx), float(np.float32(r)), linear
        self.pns, self.pew = sides[0] == 2, sides[1] == 2
        H = torch.from_numpy(np.ma.filled(H, np.float32(LAND)).astype(np.float64)).to(dev)
        dry = self._corners(H > 0.1 * LAND)
        depth = torch.where(dry, torch.zeros_like(dry, dtype=H.dtype), self._corners(H))
        quad = [depth[j:j + ny + 4, i:i + nx + 4] for j in (0, 1) for i in (0, 1)]
        wet = sum((~dry[j:j + ny + 4, i:i + nx + 4]).to(torch.float64) for j in (0, 1) for i in (0, 1))
        self.land = wet == 0
        inner = (slice(2, ny + 2), slice(2, nx + 2))
        self.Hm = 0.25 * sum(quad)[inner]
        self.Bm = (sum(quad) / wet.clamp(min=1.0))[inner]
        self.depth_x = 0.5 * (depth[2:ny + 2] + depth[3:ny + 3])
        self.depth_y = (0.5 * (depth[:, 2:nx + 2] + depth[:, 3:nx + 3])).T.contiguous()
        f32 = np.float32
        rows = float(f32(f - beta * 2 * dx)) + float(f32(beta)) * (np.arange(ny + 4) - 1.5) * dx
        self.f = torch.from_numpy(rows.astype(f32).astype(np.float64)).to(dev)
        self.X, self.Y = wind_cells if wind_cells is not None else (self._wind(w) for w in (wind or (0.0, 0.0)))

    def _corners(self, a):
        """The ghost corners of a domain: wrapped, or mirrored about the wall."""
        for n, periodic in ((self.ny, self.pns), (self.nx, self.pew)):
            j = torch.arange(n + 5, device=a.device)
            if periodic:
                j = torch.where(j < 2, j + n, torch.where(j > n + 1, j - n, j))
            else:
                j = torch.where(j < 2, 4 - j, torch.where(j > n + 2, 2 * n + 4 - j, j))
            a = a[j].T
        return a.contiguous()

    def _wind(self, field):
        """A wind array at the cells: bilinear, clamped, read at ((i + 2.5) / nx, (j + 2.5) / ny)."""
        if np.size(field) == 1:
            return float(np.reshape(field, -1)[0])
        w = torch.from_numpy(field.astype(np.float64)).to(_device())

        def taps(n, size):
            x = ((torch.arange(n, device=w.device) + 2.5) / n * size - 0.5).to(torch.float64)
            lo = x.floor()
            return lo.long().clamp(0, size - 1), (lo.long() + 1).clamp(0, size - 1), x - lo
        j0, j1, wy = taps(self.ny, w.shape[0])
        i0, i1, wx = taps(self.nx, w.shape[1])
        rows = w[j0] * (1 - wy)[:, None] + w[j1] * wy[:, None]
        return rows[:, i0] * (1 - wx) + rows[:, i1] * wx

    def stage(self, q, before, dt):
        """One Runge-Kutta stage from state q; `before`: the state before the step, in the second stage."""
        nx, ny, dx = self.nx, self.ny, self.dx
        land = self.land[2:ny + 2, 2:nx + 2]
        zero = torch.zeros_like(q[0])
        h = torch.where(land, torch.ones_like(zero), q[0] + self.Bm)
        e = torch.where(land, zero, q[0])
        u, v = (torch.where(land, zero, q[k] / h) for k in (1, 2))
        f_in = self.f[2:ny + 2]
        Fx = _axis(_pad(e, self.pew, 1), _pad(u, self.pew, -1), _pad(v, self.pew, 1), f_in[:, None],
                   self.land[2:ny + 2], self.depth_x, dx, not self.pew)
        Fy = _axis(_pad(e.T, self.pns, 1), _pad(v.T, self.pns, -1), _pad(u.T, self.pns, 1), -self.f[None, :],
                   self.land[:, 2:nx + 2].T, self.depth_y, dx, not self.pns)
        Fy = [Fy[0].T, Fy[2].T, Fy[1].T]
        div = [(a[:, 1:] - a[:, :-1] + b[1:] - b[:-1]) / dx for a, b in zip(Fx, Fy)]
        h = e + self.Hm
        hu, hv = u * h, v * h
        slope_x = (self.depth_x[:, 3:nx + 3] - self.depth_x[:, 2:nx + 2]) / dx
        slope_y = (self.depth_y[:, 3:ny + 3] - self.depth_y[:, 2:ny + 2]).T / dx
        f = f_in[:, None]
        source = (~land) & (h >= CUTOFF)
        su = torch.where(source, self.X + f * hv + G * h * slope_x, zero)
        sv = torch.where(source, self.Y - f * hu + G * h * slope_y, zero)
        safe = torch.where(h > 0.1, h, torch.ones_like(h))
        if self.linear:
            C = 2.0 * self.r * dt / safe
        else:
            C = dt * self.r * torch.sqrt((hu / safe) ** 2 + (hv / safe) ** 2 + 1e-300) / safe
        new = [e - dt * div[0], hu + dt * (su - div[1]), hv + dt * (sv - div[2])]
        if before is None:
            new = [new[0], new[1] / (1.0 + C), new[2] / (1.0 + C)]
        else:
            new = [0.5 * (b + a) for b, a in zip(before, new)]
            new = [new[0], new[1] / (1.0 + 0.5 * C), new[2] / (1.0 + 0.5 * C)]
        gone = new[0] + self.Hm <= CUTOFF
        return [torch.where(gone, CUTOFF - self.Hm, new[0]), torch.where(gone, zero, new[1]),
                torch.where(gone, zero, new[2])]

    def step(self, q, dt):
        return self.stage(self.stage(q, None, dt), q, dt)

    def cfl(self, q):
        h = q[0] + self.Bm
        wet = ~self.land[2:self.ny + 2, 2:self.nx + 2] & (h > 0)
        c = torch.sqrt(G * h.clamp(min=1e-9))
        speed = torch.maximum(*((q[k] / h).abs() + c for k in (1, 2)))
        return 0.25 * self.dx / float(speed[wet].max())


def _inner(ocean):
    return [torch.from_numpy(a[2:-2, 2:-2].astype(np.float64)).to(_device()) for a in ocean[1:4]]


def _perturbed(model, q, seeds, dx):
    """One model-error perturbation of the state: two LCG draws per seed, Box-Muller, the covariance
    q0 (1 + d/L) exp(-d/L) over 5 x 5 cells, and its geostrophic balance; f-plane.  Returns the new seeds too."""
    nx, ny = model.nx, model.ny
    gx, gy = (0 if model.pew else 4), (0 if model.pns else 4)

    def lcg(s):
        s = (s * 1103515245 + 12345) % 2147483647
        return s, s.to(torch.float64) / 2147483648.0
    seeds, u1 = lcg(seeds)
    seeds, u2 = lcg(seeds)
    radius = torch.sqrt(-2.0 * torch.log(u1))
    xi = torch.stack([radius * torch.cos(2 * math.pi * u2), radius * torch.sin(2 * math.pi * u2)], dim=-1)
    xi = xi.reshape(xi.shape[0], -1)[:, :nx + 2 * gx]
    if xi.shape[1] % 2:
        xi[:, -1] = 0.0       # an odd width keeps its last column unwritten
    if xi.shape[1] < nx + 2 * gx:
        xi = torch.nn.functional.pad(xi, (0, 1))
    j = torch.arange(ny + 8, device=xi.device)
    i = torch.arange(nx + 8, device=xi.device)
    xi = xi[(j - 4) % ny if model.pns else j][:, (i - 4) % nx if model.pew else i]
    L = 0.75 * dx
    d_eta = torch.zeros((ny + 4, nx + 4), dtype=torch.float64, device=xi.device)
    for ky in range(5):
        for kx in range(5):
            dist = dx * math.hypot(kx - 2, ky - 2)
            d_eta += MODEL_ERROR_Q0 * (1.0 + dist / L) * math.exp(-dist / L) * xi[ky:ky + ny + 4, kx:kx + nx + 4]
    d = d_eta[2:-2, 2:-2]
    h = d + model.Hm + q[0]
    ex = (d_eta[2:-2, 3:-1] - d_eta[2:-2, 1:-3]) / (2.0 * dx)
    ey = (d_eta[3:-1, 2:-2] - d_eta[1:-3, 2:-2]) / (2.0 * dx)
    g_f = G / float(model.f[0])
    return [q[0] + d, q[1] - g_f * h * ey, q[2] + g_f * h * ex], seeds


def _drifted(model, q, at, dt):
    """Drifters after one Euler step through the flow, velocities bilinear between cell centres."""
    h = q[0] + model.Bm
    size = (model.nx * model.dx, model.ny * model.dx)
    i, j = ((at[:, k] / model.dx - 0.5) for k in (0, 1))
    i0, j0 = i.floor(), j.floor()
    new = []
    for k in (1, 2):
        w = q[k] / h
        value = 0.0
        for dj, wj in ((0, 1 - (j - j0)), (1, j - j0)):
            for di, wi in ((0, 1 - (i - i0)), (1, i - i0)):
                value = value + wj * wi * w[j0.long() + dj, i0.long() + di]
        x = at[:, k - 1] + dt * value
        if model.pew if k == 1 else model.pns:
            x = x % size[k - 1]
        new.append(x)
    return torch.stack(new, dim=1)


def _exact_step(case, seed):
    nx, ny, dx = case["nx"], case["ny"], case["dx"]
    ocean = _ocean(seed, nx, ny, dx, case["flat"], case["land"])
    model = _Model64(ocean[0], nx, ny, dx, _sides(case), F0, BETA if case["beta"] else 0.0, _friction(case),
                     case["friction"] == "linear", _step_wind(case, seed))
    q, dt, out = _inner(ocean), ocean[4], {}
    if case["update_dt"]:
        out["cfl"] = 0.5 * model.cfl(q)
    if case["model_error"]:
        gx, gy = (0 if model.pew else 4), (0 if model.pns else 4)
        shape = (ny + 2 * gy, math.ceil((nx + 2 * gx) / 2))
        seeds = torch.from_numpy((np.random.RandomState(seed).rand(*shape) * 2147483648.0).astype(np.int64)).to(_device())
    if case["drifters"]:
        at = np.concatenate([_drifter_positions(case, seed), [[0.5 * nx * dx, 0.5 * ny * dx]]])
        at = torch.from_numpy(at.astype(np.float32).astype(np.float64)).to(_device())
    for _ in range(case["steps"]):
        q = model.step(q, dt)
        if case["model_error"]:
            q, seeds = _perturbed(model, q, seeds, dx)
        if case["drifters"]:
            at = _drifted(model, q, at, dt)
    if case["land"]:
        # a land cell holds water of the cut-off depth over a bottom at zero, at rest
        land = model.land[2:ny + 2, 2:nx + 2]
        q = [torch.where(land, torch.full_like(a, rest), a) for a, rest in zip(q, (CUTOFF, 0.0, 0.0))]
    out["state"] = q
    if case["drifters"]:
        out["drifters"] = at
    if case["model_error"]:
        out["seeds"] = seeds
    return out


def _exact_gradient(case, seed, seed0, dt):
    from torch.utils.checkpoint import checkpoint
    x0, wind, ocean = _gradient_inputs(case, seed)
    x = [a.to(torch.float64).requires_grad_() for a in x0]
    w = [a.to(torch.float64).requires_grad_() for a in wind]
    model = _Model64(ocean[0], case["nx"], case["ny"], 1000.0, (1, 2, 1, 2), F0, BETA, FRICTION, wind_cells=w)
    cells, steps, values = _observed(case, seed0)
    cells = torch.from_numpy(cells.astype(np.int64)).to(x0.device)
    values = torch.from_numpy(values.astype(np.float64)).to(x0.device)
    weight = torch.tensor([100.0, 1.0, 1.0], dtype=torch.float64, device=x0.device)

    def advance(e, u, v, X, Y):
        model.X, model.Y = X, Y
        return tuple(model.step([e, u, v], dt))
    q, J = x, 0.0
    for n in range(1, case["steps"] + 1):
        q = checkpoint(advance, *q, *w, use_reentrant=False)
        if n in steps:
            seen = torch.stack([a[cells[:, 1], cells[:, 0]] for a in q], dim=1)
            J = J + (weight * (seen - values[steps.index(n)]) ** 2).sum()
    grads = torch.autograd.grad(J, x + w)
    return float(J.detach()), torch.stack(grads[:3]), torch.stack(grads[3:])


def exact(case, seed):
    """What run returns on a fresh state, in float64; None for the ensemble, whose perturbations are random draws."""
    seed = int(seed) % (1 << 30)
    kind = case["kind"]
    if kind == "step":
        return _exact_step(case, seed)
    if kind == "ensemble":
        return None
    if kind == "domains":
        limits, members = [], []
        for m, (nx, ny) in enumerate(_domain_sizes(case)):
            ocean = _ocean(seed + 11 * m, nx, ny)
            model = _Model64(ocean[0], nx, ny, 1000.0, (1, 2, 1, 2), F0, BETA, FRICTION, wind=_uniform_wind())
            q = _inner(ocean)
            for _ in range(case["steps"]):
                q = model.step(q, ocean[4])
            limits.append(model.cfl(q))
            members += q if m < 20 else []
        return {"limits": np.array(limits), "members": members}
    M = case.get("members", 1)
    dt = min(_ocean(seed + 11 * m, case["nx"], case["ny"])[4] for m in range(M))
    got = [_exact_gradient(case, seed + 11 * m, seed, dt) for m in range(M)]
    if kind == "gradient":
        J, gs, gw = got[0]
        return {"J": J, "state": list(gs), "wind": list(gw)}
    return {"J": np.array([g[0] for g in got]), "state": torch.stack([g[1] for g in got]),
            "wind": torch.stack([g[2] for g in got])}
