// Window backward on tiles of 128 keys (tc_bwd_wide.cu), launched by tc_attn_bwd (tc_bwd.cu).
#pragma once

#include "tc_common.cuh"

namespace nsa {
namespace tc {

constexpr int kWideKeys = 128;

struct WideArgs {
  const float *lse, *delta, *row_scale;   // row_scale: gate value per row of a gated branch, or null
  __nv_bfloat16 *dk, *dv;
  __nv_bfloat16* dq_part;                 // [units][T][slots][G][D]
  int* status;
  int Hq, Hkv, T, G, nq;
  int window;                             // at most T
  int n_slots;
  float scale, scale_log2;
};

int bwd_wide_launch(const AttnArgs& a, const WideArgs& p, const char* name, cudaStream_t st);

}  // namespace tc
}  // namespace nsa
