// Launches of the CFL reductions (cfl.cu): the limits' float bits into out.
#pragma once

#include "internal.h"

namespace go {

cudaError_t cfl_launch(const Scheme& k, const float* eta, const float* hu, const float* hv, int p, const float* Bm,
                       int pb, float land, unsigned int* out, cudaStream_t s);
// args: two per member (the first holds the current state as its input);
// blocks: per member, the most of cfl_batch_blocks over the n members.
cudaError_t cfl_batch_launch(const StageArgs* args, int n, int blocks, unsigned int* out, cudaStream_t s);
int cfl_batch_blocks(const Scheme& k, int n);

}  // namespace go
