// Internal interface of the pooling kernels (pool.cu): the K and the V side of a call go through
// one launch.
#pragma once

#include "common.cuh"

namespace nsa {

// One or two tensors pooled with the same geometry (the keys and the values of the compression
// branch), each with its own parameters.  x, dx, out, d_out, pooled, d_pooled, intra and proj are read and
// written as 16-byte vectors: the calls below refuse other addresses, the entry points that take them
// go to the scalar kernels of aux.cu instead.
struct PoolSides {
  int n;                         // 1 or 2
  const void* x[2];              // [B, H, T, D]
  const float* intra[2];         // learned pooling only: [len, D], [len], [D, D]
  const float* logits[2];
  const float* proj[2];
  void* out[2];                  // forward: [B, H, n_sum, D] (null: only `pooled` is wanted)
  float* pooled[2];              // [B*H*n_sum, D] before the projection (forward: may be null)
  const void* d_out[2];          // backward
  void* dx[2];
  float* d_pooled[2];            // overlapping windows only: [B*H*n_sum, D]
  float* acc[2];                 // pool_acc_floats() zeroed floats each
  float* d_intra[2];
  float* d_logits[2];
  float* d_proj[2];
};

inline int pool_count(int T, int len, int stride) { return T >= len ? (T - len) / stride + 1 : 0; }
bool pool_learned_ok(int D, int len, int dtype);
size_t pool_acc_floats(int D, int len);        // accumulators and the arrival counter of one side
int pool_learned_fwd(const PoolSides& s, int B, int H, int T, int D, int len, int stride, cudaStream_t st);
int pool_learned_bwd(const PoolSides& s, int B, int H, int T, int D, int len, int stride, cudaStream_t st);
bool pool_mean_ok(int D, int dtype);           // sizes that pool_mean_fwd takes
int pool_mean_fwd(const PoolSides& s, int B, int H, int T, int D, int len, int dtype, cudaStream_t st);
int pool_mean_bwd(const PoolSides& s, int B, int H, int T, int D, int len, int dtype, cudaStream_t st);

}  // namespace nsa
