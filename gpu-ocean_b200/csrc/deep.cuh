// Deep water: where the scheme's dry, shallow, land and zero-fan branches
// cannot be taken.
//
// With |eta| <= E and |u|, |v| <= kDeepVel = U in the cells of a stencil and
// d |f| U / 2g <= D in its rows (d the cell size), a slope K or L is at most its
// central argument, |K| / 2g <= E/2 + D, and the Coriolis part of a face depth at
// most D.  Corner depths of at least H then leave every reconstructed face
// depth at H - 3/2 E - 2 D or more and every cell depth at H - E.  The stage kernels
// run such stencils without those branches: the results are the general form's
// bit for bit.
//
// E and D are kDeepEta and kDeepCor unless the domain's least depth is told
// (go_domain_set_depth): then D is what its Coriolis parameter needs and E what
// its depth leaves, so that tides and coarse grids in deep water count as deep.
#pragma once

#include <math.h>

#include "cdklm16_device.cuh"

namespace go {

constexpr float kDeepEta = 2.0f;           // m, E unless told otherwise, and the least E
constexpr float kDeepEtaMost = 20.0f;      // m
constexpr float kDeepVel = 4.0f;           // m/s
constexpr float kDeepCor = 0.25f;          // m, D unless told otherwise, and the least D

// Face and cell depths must exceed the cut-off and the desingularisation depth,
// and the wave speeds either side of a face, which differ by at least
// 2 sqrt(g h), the width below which a fan counts as closed (flux_slope_eps).
inline float deep_face(const Scheme& k) {
    const float fan = 0.5f * k.flux_slope_eps;
    return fmaxf(fmaxf(k.cutoff, k.desing_eps), fan * fan / k.g);
}

// The bounds of a domain: least corner depth, |eta| and |f| of deep water.
struct DeepBounds {
    float depth, eta, f;
    bool told;          // they are fitted to the domain's depth and Coriolis parameter
};

// 1% and a centimetre of slack for the rounding of the evaluated depths.
// least_depth: a NaN where it is not known; f_most: the largest |f|.
inline DeepBounds deep_bounds(const Scheme& k, float least_depth, float f_most) {
    const float d = fmaxf(k.dx, k.dy);
    float E = kDeepEta, D = kDeepCor;
    const float need = fmaxf(kDeepCor, 1.001f * d * f_most * kDeepVel / (2.0f * k.g));
    const float left = 0.999f * ((least_depth - 0.01f) / 1.01f - deep_face(k) - 2.0f * need) / 1.5f;
    DeepBounds b;
    b.told = left >= kDeepEta;
    if (b.told) {
        E = fminf(left, kDeepEtaMost);
        D = need;
    }
    b.depth = 1.01f * (deep_face(k) + 1.5f * E + 2.0f * D) + 0.01f;
    b.eta = E;
    b.f = D * 2.0f * k.g / (kDeepVel * d);
    return b;
}

// End of the range of deep corner depths: a land value inside it ends it
// below the values that count as land.
__host__ __device__ __forceinline__ float deep_end(const Scheme& k) {
    return (k.land > 0.0f && k.land < 1.0e15f) ? k.land * 0.999f - 1.0f : 1.0e15f;
}

// Whether a cell state is one of deep water (false for a NaN).
__device__ __forceinline__ bool deep_state(float e, float u, float v, float most) {
    return fabsf(e) <= most && e != kDryFlag && fabsf(u) <= kDeepVel && fabsf(v) <= kDeepVel;
}

}  // namespace go
