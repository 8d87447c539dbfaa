// Launches of the tile stage kernels (cdklm16_tile.cuh).
#include <limits.h>

#include <vector>

#include "cdklm16_tile.cuh"
#include "pair_dispatch.cuh"
#include "tile_batch.h"

using namespace go;

namespace {

dim3 tile_grid(const Scheme& k) { return dim3((k.nx + kTileX - 1) / kTileX, (k.ny + kTileY - 1) / kTileY); }

// Allows a kernel its shared-memory size in the current context.  Done for
// each domain and batch layout, whose device memory belongs to that context
// too, and not once per process, which a reset of the device would undo.
template <class K>
cudaError_t allow_smem(K kernel) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TileSmem));
}

// 32-bit byte offsets into every array of a stage.
bool offsets_fit(const StageArgs& a) {
    auto fits = [&](int pitch) { return (long long)(a.k.ny + 5) * pitch * 4 < (1LL << 32); };
    return fits(a.pin) && fits(a.pout) && fits(a.pqn) && fits(a.phi);
}

cudaLaunchConfig_t tile_config(dim3 grid, cudaStream_t s, cudaLaunchAttribute* attr, bool follows) {
    attr->id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr->val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kTileThreads);
    cfg.dynamicSmemBytes = sizeof(TileSmem);
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = follows ? 1 : 0;
    return cfg;
}

}  // namespace

int go_tile_setup(go_domain* d) {
    if ((long long)d->k.nx * d->k.ny >= kTileCells) return GO_OK;
    GO_CUDA(allow_smem(cdklm_tile_kernel));
    GO_CUDA(allow_smem(cdklm_tile_steps_kernel));
    int sms = 0, coop = 0, per_sm = 0;
    GO_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, d->device));
    GO_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, d->device));
    GO_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, cdklm_tile_steps_kernel, kTileThreads,
                                                          sizeof(TileSmem)));
    d->tile_steps_blocks = coop && per_sm > 0 ? sms : 0;
    return GO_OK;
}

bool go_tile_stage(const go_domain* d, const StageArgs& a) { return go_tile_domain(d) && offsets_fit(a); }

// One stage.  follows: the launch before it on the stream is a tile stage of
// the same call, so this one is a programmatic dependent launch: its blocks
// are scheduled, and read the corners, while that one's last blocks run.
// Measured on a B200, us per RK2 step without / with: 64 x 48 12.4 / 9.2,
// 512^2 20.6 / 16.7, 1024^2 53.4 / 48.5.
int go_launch_tile(go_domain* d, cudaStream_t s, const StageArgs& a, bool follows) {
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = tile_config(tile_grid(a.k), s, &attr, follows);
    d->stage_launches = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, cdklm_tile_kernel, a, tile_const(a.k));
    if (e != cudaSuccess) return go_fail(GO_ERR_CUDA, "stage launch (tile) failed: %s", cudaGetErrorString(e));
    return GO_OK;
}

// Grids of at most one tile per SM run all the steps of a call in one
// cooperative launch.  Measured on a B200 for 10 steps, us per step and (three
// simulators on their own streams) us per call, against one launch per stage:
// 64 x 48 8.7 / 9.2 and 33 / 51; 256^2 10.0 / 10.6 and 57 / 59; 384^2 (288
// tiles) 11.4 / 13.2 but 114 / 76, since launches of two tiles per SM leave the
// simulators no room beside one another.
bool go_tile_steps_fit(const go_domain* d) {
    const dim3 g = tile_grid(d->k);
    const int most = (d->debug & GO_DEBUG_STEPS_ANY_SIZE) && d->tile_steps_blocks ? INT_MAX : d->tile_steps_blocks;
    return (int)(g.x * g.y) <= most;
}

// Where the process has too few SMs for the launch (a share of the device, say)
// it is refused; the domain's steps then take one launch per stage: *done 0.
int go_launch_tile_steps(go_domain* d, cudaStream_t s, const StageArgs& a, int n, bool* done) {
    *done = true;
    if (n < 1) return GO_OK;
    StageArgs args = a;
    TileConst tc = tile_const(a.k);
    void* params[] = {&args, &tc, &n};
    d->stage_launches = 1;
    const cudaError_t e = cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(cdklm_tile_steps_kernel),
                                                      tile_grid(a.k), dim3(kTileThreads), params, sizeof(TileSmem), s);
    if (e == cudaErrorCooperativeLaunchTooLarge) {
        cudaGetLastError();
        d->tile_steps_blocks = 0;
        *done = false;
        return GO_OK;
    }
    if (e != cudaSuccess) return go_fail(GO_ERR_CUDA, "step launch (tiles) failed: %s", cudaGetErrorString(e));
    return GO_OK;
}

namespace go {

void tile_batch_dims(const Scheme& k, int* columns, int* rows) {
    const dim3 g = tile_grid(k);
    *columns = (int)g.x;
    *rows = (int)g.y;
}

bool tile_batch_fits(const StageArgs& a) { return offsets_fit(a); }

cudaError_t tile_batch_consts(const std::vector<StageArgs>& args, TileConst** out) {
    std::vector<TileConst> h(args.size() / 2);
    for (size_t m = 0; m < h.size(); ++m) h[m] = tile_const(args[2 * m].k);
    *out = nullptr;
    cudaError_t e = allow_smem(cdklm_tile_batch_kernel);
    if (e == cudaSuccess) e = cudaMalloc(out, sizeof(TileConst) * h.size());
    if (e == cudaSuccess) e = cudaMemcpy(*out, h.data(), sizeof(TileConst) * h.size(), cudaMemcpyHostToDevice);
    return e;
}

cudaError_t tile_batch_launch(const TileBatchReq& r) {
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = tile_config(dim3(r.ntiles), r.s, &attr, r.follows);
    return cudaLaunchKernelEx(&cfg, cdklm_tile_batch_kernel, r.args, r.dts, r.consts, r.tiles, r.rk_step);
}

}  // namespace go
