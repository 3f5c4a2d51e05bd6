// Internal interface of the entry points (api.cu) for the whole-op calls (op.cu).
#pragma once

#include "common.cuh"

namespace nsa {
int check_dims(const NsaDims* d);
AttnArgs base_args(const NsaDims* d, int Lk);
bool use_tc(const NsaDims* d, int block_size, int impl, int* err);
bool profiling();     // every launch is bracketed by events on its stream: branches must not overlap
}  // namespace nsa
