// CFL limit of a domain (max_dt.cu:42-141): the exact minimum of 0.25 dx/|u +- c|
// and 0.25 dy/|v +- c| over the wet interior cells.
//
// A quotient of a positive constant falls with its divisor, rounding included,
// so the least quotient is that of the largest speed: each thread keeps the
// largest |u +- c| and |v +- c| of its cells and divides once (per cell two
// IEEE quotients and a root instead of six and a root).
#pragma once

#include "cdklm16_device.cuh"

namespace go {

struct CflSpeeds {
    float x = 0.0f, y = 0.0f;
};

// A cell's speeds into s; none for a dry or land cell.  The reference builds
// max_dt.cu with nvcc's default options (CDKLM16.py:221 passes no compile
// flags): its quotients and square root are IEEE round-to-nearest, kept here
// with __fdiv_rn / __fsqrt_rn whatever this library's own flags are.
__device__ __forceinline__ void cell_speeds(float e, float hu, float hv, float H, float g, float land, CflSpeeds& s) {
    const float h = e + H;
    if (h <= 0.0f || fabsf(H - land) < kDryEps) return;
    const float u = __fdiv_rn(hu, h);
    const float v = __fdiv_rn(hv, h);
    const float c = __fsqrt_rn(g * h);
    s.x = fmaxf(s.x, fmaxf(fabsf(u + c), fabsf(u - c)));
    s.y = fmaxf(s.y, fmaxf(fabsf(v + c), fabsf(v - c)));
}

// The limit of a thread's cells, at most `none`.
__device__ __forceinline__ float cfl_dt(const CflSpeeds& s, float dx, float dy, float none) {
    return fminf(none, fminf(__fdiv_rn(0.25f * dx, s.x), __fdiv_rn(0.25f * dy, s.y)));
}

// Calls use(load(j, i)) for the interior cells of an nx x ny grid: a warp per
// 128 columns of a row, whose four loads of a lane are in flight together.
template <class Load, class Use>
__device__ __forceinline__ void cfl_cells(int nx, int ny, const Load& load, const Use& use) {
    const int lane = threadIdx.x & 31, warps = blockDim.x >> 5, segments = (nx + 127) >> 7;
    for (int u = blockIdx.x * warps + (threadIdx.x >> 5); u < segments * ny; u += gridDim.x * warps) {
        const int j = u / segments, first = (u - j * segments) << 7;
        int i = first + lane + 2;
        if (first + 128 <= nx) {
            const auto a = load(j + 2, i), b = load(j + 2, i + 32), c = load(j + 2, i + 64), d = load(j + 2, i + 96);
            use(a);
            use(b);
            use(c);
            use(d);
        } else {
            for (; i < nx + 2; i += 32) use(load(j + 2, i));
        }
    }
}

}  // namespace go
