"""The deep-water bounds of a domain whose least depth is told (csrc/deep.cuh,
deep_bounds): at their limits no stencil takes a dry, shallow or zero-fan
branch.  Float32 arithmetic in the kernels' order."""

import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "gpu-ocean_b200", "csrc")
U = 4.0                       # kDeepVel
f32 = np.float32

SOURCE = """
#include <math.h>
#define __host__
#define __device__
#define __forceinline__ inline
struct Scheme { float dx, dy, g, cutoff, desing_eps, flux_slope_eps, land; };
%s
extern "C" int bounds(const float* k, float least, float f, float* out) {
    const Scheme s = {k[0], k[1], k[2], k[3], k[4], k[5], 1.0e20f};
    const DeepBounds b = deep_bounds(s, least, f);
    out[0] = b.depth; out[1] = b.eta; out[2] = b.f;
    return b.told;
}
"""


@pytest.fixture(scope="module")
def bounds(tmp_path_factory):
    """deep_bounds compiled for the host."""
    if shutil.which("g++") is None:
        pytest.skip("needs g++")
    text = open(os.path.join(CSRC, "deep.cuh")).read()
    text = text[text.index("constexpr float kDeepEta"):text.index("// End of the range of deep corner depths")]
    d = tmp_path_factory.mktemp("deep")
    src = d / "deep.cpp"
    src.write_text(SOURCE % text)
    subprocess.run(["g++", "-O1", "-ffp-contract=off", "-shared", "-fPIC", str(src), "-o", str(d / "deep.so")], check=True)
    lib = ctypes.CDLL(str(d / "deep.so"))

    def call(least, f, dx=1000.0, desing=0.1, fan=0.1, g=9.81):
        k = (ctypes.c_float * 6)(dx, 0.5 * dx, g, 1.0e-5, desing, fan)
        out = (ctypes.c_float * 3)()
        told = lib.bounds(k, ctypes.c_float(least), ctypes.c_float(f), out)
        return bool(told), f32(out[0]), f32(out[1]), f32(out[2])
    return call


def _minmod(b, c, f):
    m = np.minimum(np.minimum(np.abs(b), np.abs(c)), np.abs(f))
    same = (np.signbit(b) == np.signbit(c)) & (np.signbit(c) == np.signbit(f))
    return np.where(same, np.copysign(m, b), f32(0))


@pytest.mark.parametrize("least", [3.7, 5.0, 12.0, 31.0, 400.0, 9000.0])
@pytest.mark.parametrize("dx,f,desing,fan", [(100.0, 1.4e-4, 0.1, 0.1), (2000.0, 1.4e-4, 0.1, 0.1),
                                             (20000.0, 1.4e-4, 0.01, 2.0), (50000.0, 1.4e-4, 1.0, 0.5)])
@pytest.mark.parametrize("theta", [1.0, 1.3, 2.0])
def test_told_bounds_take_no_shallow_branch(bounds, least, dx, f, desing, fan, theta):
    told, depth, E, most_f = bounds(least, f, dx, desing, fan)
    assert E >= 2.0
    if told:
        assert depth <= least and most_f >= f32(f)          # the domain's own corners and rows count
    rng = np.random.default_rng(3)
    g, n = f32(9.81), 50000
    must = max(1.0e-5, desing, (0.5 * fan) ** 2 / float(g))

    def at_limits(size, most):
        a = rng.uniform(-most, most, size)
        return np.where(rng.random(size) < 0.5, np.copysign(most, a), a).astype(f32)
    e, v = at_limits((5, n), float(E)), at_limits((5, n), U)
    fv = v * np.where(rng.random((5, n)) < 0.5, most_f, -most_f)
    H = np.full((6, n), depth, f32) + (rng.random((6, n)) < 0.5).astype(f32) * f32(0.3)
    two_g, half_g, theta_g = f32(2) * g, f32(0.5) * g, f32(theta) * g
    V, inv = f32(dx) / two_g, f32(1) / two_g
    K = {}
    for c in (1, 2, 3):
        K[c] = _minmod(theta_g * ((e[c] - e[c - 1]) - V * (fv[c] + fv[c - 1])),
                       half_g * ((e[c + 1] - e[c - 1]) - V * ((fv[c + 1] + f32(2) * fv[c]) + fv[c - 1])),
                       theta_g * ((e[c + 1] - e[c]) - V * (fv[c] + fv[c + 1])))
        q = (K[c] + f32(dx) * fv[c]) * inv
        assert ((e[c] + H[c]) - q).min() > must and ((e[c] + H[c + 1]) + q).min() > must
        assert (e[c] + H[c]).min() > must
    for m, p in ((1, 2), (2, 3)):
        hp = (e[p] + H[p]) - (K[p] + f32(dx) * fv[p]) * inv
        hm = (e[m] + H[p]) + (K[m] + f32(dx) * fv[m]) * inv
        assert hp.min() > must and hm.min() > must
        assert (f32(2) * np.sqrt(g * np.minimum(hp, hm))).min() > fan


def test_what_counts_as_told(bounds):
    assert bounds(float("nan"), 1.4e-4)[0] is False and bounds(float("nan"), 1.4e-4)[2] == 2.0
    assert bounds(3.0, 1.4e-4)[0] is False and bounds(-5.0, 1.4e-4)[0] is False
    assert bounds(3.8, 1.4e-4)[0] is True
    assert bounds(8.0, 1.4e-4, dx=50000.0)[0] is True and bounds(4.0, 1.4e-4, dx=50000.0)[0] is False
    assert bounds(9000.0, 1.4e-4)[2] == 20.0
