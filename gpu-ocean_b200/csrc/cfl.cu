// The CFL reductions: one domain (go_max_dt) and every member of a batch.
#include "cfl.h"

#include <string.h>

#include <algorithm>

#include "cfl.cuh"

namespace go {
namespace {

constexpr int kCflThreads = 256;

struct CflCell {
    float eta, hu, hv, H;
};
struct CflCorners {
    float eta, hu, hv, sw, nw, se, ne;
};

// Memory-bound: 16 bytes per cell.  B200, us per call, with six IEEE quotients
// per cell, a quotient of integers for its row and one load at a time before /
// now: 2048^2 35.6 / 23.0, 4096^2 128 / 82 (two launches bound
// smaller grids: 12).
__global__ void __launch_bounds__(kCflThreads)
    k_max_dt(const float* __restrict__ eta, const float* __restrict__ hu, const float* __restrict__ hv, int p,
             const float* __restrict__ Bm, int pb, int nx, int ny, float dx, float dy, float g, float land,
             unsigned int* out) {
    CflSpeeds s;
    cfl_cells(
        nx, ny,
        [&](int j, int i) {
            const size_t o = (size_t)j * p + i;
            return CflCell{eta[o], hu[o], hv[o], Bm[(size_t)j * pb + i]};
        },
        [&](const CflCell& q) { cell_speeds(q.eta, q.hu, q.hv, q.H, g, land, s); });
    block_min_to(cfl_dt(s, dx, dy, kRefFltMax), out, kRefFltMax);
}

// Every member in one launch: blockIdx.y is the member, whose current state
// (h0) is the input of its stage-0 arguments; the cell-mean bathymetry comes
// from the corners as the set-up computes it.  100 members of 512^2: 358 / 163 us.
__global__ void __launch_bounds__(kCflThreads)
    k_batch_max_dt(const StageArgs* __restrict__ args, unsigned int* __restrict__ out) {
    const StageArgs& a = args[2 * blockIdx.y];
    const float* __restrict__ eta = a.eta_in;
    const float* __restrict__ hu = a.hu_in;
    const float* __restrict__ hv = a.hv_in;
    const float* __restrict__ Hi = a.Hi;
    const int pin = a.pin, phi = a.phi;
    const float g = a.k.g, land = a.k.land;
    CflSpeeds s;
    cfl_cells(
        a.k.nx, a.k.ny,
        [&](int j, int i) {
            const size_t o = (size_t)j * pin + i;
            const float* __restrict__ H = Hi + (size_t)j * phi + i;
            return CflCorners{eta[o], hu[o], hv[o], H[0], H[phi], H[1], H[phi + 1]};
        },
        [&](const CflCorners& q) {
            cell_speeds(q.eta, q.hu, q.hv, cell_mean_depth(q.sw, q.nw, q.se, q.ne, land), g, land, s);
        });
    block_min_to(cfl_dt(s, a.k.dx, a.k.dy, kRefFltMax), out + blockIdx.y, kRefFltMax);
}

__global__ void k_fill(unsigned int* p, unsigned int v, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) p[i] = v;
}

// Blocks for an nx x ny grid: a warp per 128 columns of a row, at most `most`.
int blocks_for(int nx, int ny, long long most) {
    const long long warps = (long long)((nx + 127) / 128) * ny, per = kCflThreads / 32;
    return (int)std::min((warps + per - 1) / per, most);
}

cudaError_t fill(unsigned int* out, int n, cudaStream_t s) {
    unsigned int bits;
    memcpy(&bits, &kRefFltMax, sizeof(bits));
    k_fill<<<(n + 255) / 256, 256, 0, s>>>(out, bits, n);
    return cudaGetLastError();
}

}  // namespace

cudaError_t cfl_launch(const Scheme& k, const float* eta, const float* hu, const float* hv, int p, const float* Bm,
                       int pb, float land, unsigned int* out, cudaStream_t s) {
    const cudaError_t e = fill(out, 1, s);
    if (e != cudaSuccess) return e;
    k_max_dt<<<blocks_for(k.nx, k.ny, 148 * 8), kCflThreads, 0, s>>>(eta, hu, hv, p, Bm, pb, k.nx, k.ny, k.dx, k.dy, k.g, land,
                                                            out);
    return cudaGetLastError();
}

cudaError_t cfl_batch_launch(const StageArgs* args, int n, int blocks, unsigned int* out, cudaStream_t s) {
    const cudaError_t e = fill(out, n, s);
    if (e != cudaSuccess) return e;
    k_batch_max_dt<<<dim3(blocks, n), kCflThreads, 0, s>>>(args, out);
    return cudaGetLastError();
}

// About 8 blocks per SM in all, spread over the members.
int cfl_batch_blocks(const Scheme& k, int n) { return blocks_for(k.nx, k.ny, (148LL * 8 + n - 1) / n); }

}  // namespace go
