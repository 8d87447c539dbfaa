// The batched tile stage (tile_launch.cu) as the batch launches it.
#pragma once

#include "internal.h"

namespace go {

struct TileConst;

// Tiles of one member's grid: its tile columns and rows.
void tile_batch_dims(const Scheme& k, int* columns, int* rows);
// Whether a member's arrays are within the kernel's 32-bit byte offsets.
bool tile_batch_fits(const StageArgs& a);
// The members' launch constants in device memory (cudaFree to release), and the
// kernel made ready in the current context.
cudaError_t tile_batch_consts(const std::vector<StageArgs>& args, TileConst** out);

struct TileBatchReq {
    const StageArgs* args;       // two per member
    const float* dts;
    const TileConst* consts;     // one per member
    const int4* tiles;           // (member, tile column, tile row, -)
    int ntiles, rk_step;
    cudaStream_t s;
    bool follows;                // the launch before it on the stream is a stage of the same call
};
cudaError_t tile_batch_launch(const TileBatchReq& r);

}  // namespace go
