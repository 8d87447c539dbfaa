// Deep water: where the scheme's dry, shallow, land and zero-fan branches
// cannot be taken.
//
// With |eta| <= kDeepEta = E and |u|, |v| <= kDeepVel = U in the cells of a
// stencil and d |f| U / 2g <= kDeepCor = D in its rows (d the cell size), a
// slope K or L is at most its central argument, |K| / 2g <= E/2 + D, and the
// Coriolis part of a face depth at most D.  Corner depths of at least H then
// leave every reconstructed face depth at H - 3/2 E - 2 D or more and every
// cell depth at H - E.  The stage kernels run such stencils without those
// branches: the results are the general form's bit for bit.
#pragma once

#include <math.h>

#include "cdklm16_device.cuh"

namespace go {

constexpr float kDeepEta = 2.0f;           // m
constexpr float kDeepVel = 4.0f;           // m/s
constexpr float kDeepCor = 0.25f;          // m

// Least corner depth: face and cell depths must exceed the cut-off and the
// desingularisation depth, and the wave speeds either side of a face, which
// differ by at least 2 sqrt(g h), the width below which a fan counts as closed
// (flux_slope_eps).  1% and a centimetre of slack for the rounding of the
// evaluated depths.
inline float deep_depth(const Scheme& k) {
    const float fan = 0.5f * k.flux_slope_eps;
    const float h = fmaxf(fmaxf(k.cutoff, k.desing_eps), fan * fan / k.g);
    return 1.01f * (h + 1.5f * kDeepEta + 2.0f * kDeepCor) + 0.01f;
}

// End of the range of deep corner depths: a land value inside it ends it
// below the values that count as land.
inline float deep_end(const Scheme& k) {
    return (k.land > 0.0f && k.land < 1.0e15f) ? k.land * 0.999f - 1.0f : 1.0e15f;
}

// Largest Coriolis parameter.
__host__ __device__ __forceinline__ float deep_coriolis(const Scheme& k) {
    return kDeepCor * 2.0f * k.g / (kDeepVel * fmaxf(k.dx, k.dy));
}

// Whether a cell state is one of deep water (false for a NaN).
__device__ __forceinline__ bool deep_state(float e, float u, float v) {
    return fabsf(e) <= kDeepEta && e != kDryFlag && fabsf(u) <= kDeepVel && fabsf(v) <= kDeepVel;
}

}  // namespace go
