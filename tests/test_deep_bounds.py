"""The deep-water bounds of csrc/deep.cuh: for stencils at their limits, the
reconstructed face depths, the slope adjustment's depths and the cell depths
stay above the depth from which the scheme takes none of its dry, shallow and
zero-fan branches.  Float32 arithmetic in the kernels' order."""

import os
import re

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
SRC = open(os.path.join(os.path.dirname(HERE), "gpu-ocean_b200", "csrc", "deep.cuh")).read()
E, U, D = (float(re.search(r"constexpr float %s = ([0-9.]+)f" % n, SRC).group(1))
           for n in ("kDeepEta", "kDeepVel", "kDeepCor"))
f32 = np.float32


def _minmod(b, c, f):
    m = np.minimum(np.minimum(np.abs(b), np.abs(c)), np.abs(f))
    same = (np.signbit(b) == np.signbit(c)) & (np.signbit(c) == np.signbit(f))
    return np.where(same, np.copysign(m, b), f32(0))


@pytest.mark.parametrize("theta", [1.0, 1.3, 2.0])
@pytest.mark.parametrize("dx,desing,slope_eps", [(100.0, 0.1, 0.1), (2000.0, 0.1, 0.1), (20000.0, 0.01, 2.0),
                                                 (500.0, 1.0, 0.5)])
def test_deep_stencils_take_no_shallow_branch(theta, dx, desing, slope_eps):
    rng = np.random.default_rng(3)
    g, cutoff, n = f32(9.81), 1.0e-5, 200000
    least = max(cutoff, desing, (0.5 * slope_eps) ** 2 / float(g))          # deep_depth
    H0 = f32(f32(1.01) * f32(least + 1.5 * E + 2.0 * D) + f32(0.01))
    f = f32(D * 2.0 * float(g) / (U * dx))                                   # deep_coriolis

    def at_limits(size, most):
        a = rng.uniform(-most, most, size)
        pick = rng.random(size) < 0.5
        return np.where(pick, np.copysign(most, a), a).astype(f32)
    e, v = at_limits((5, n), E), at_limits((5, n), U)
    fv = v * np.where(rng.random((5, n)) < 0.5, f, -f)
    H = np.full((6, n), H0, f32) + (rng.random((6, n)) < 0.5).astype(f32) * f32(0.3)   # face depths
    two_g, half_g, theta_g = f32(2) * g, f32(0.5) * g, f32(theta) * g
    V, inv = f32(dx) / two_g, f32(1) / two_g
    K = {}
    for c in (1, 2, 3):
        back = theta_g * ((e[c] - e[c - 1]) - V * (fv[c] + fv[c - 1]))
        cent = half_g * ((e[c + 1] - e[c - 1]) - V * ((fv[c + 1] + f32(2) * fv[c]) + fv[c - 1]))
        forw = theta_g * ((e[c + 1] - e[c]) - V * (fv[c] + fv[c + 1]))
        K[c] = _minmod(back, cent, forw)
        q = (K[c] + f32(dx) * fv[c]) * inv
        lo, hi = (e[c] + H[c]) - q, (e[c] + H[c + 1]) + q
        assert lo.min() > least and hi.min() > least
        assert (e[c] + H[c]).min() > least
    for m, p in ((1, 2), (2, 3)):
        hp = (e[p] + H[p]) - (K[p] + f32(dx) * fv[p]) * inv
        hm = (e[m] + H[p]) + (K[m] + f32(dx) * fv[m]) * inv
        assert hp.min() > least and hm.min() > least
        c = np.sqrt(g * np.minimum(hp, hm))
        assert (f32(2) * c).min() > slope_eps        # ap - am is at least 2 sqrt(g h)
