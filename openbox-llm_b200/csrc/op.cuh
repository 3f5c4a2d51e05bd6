// Internal interface of the entry points (api.cu) for the whole-op calls (op.cu).
#pragma once

#include "common.cuh"

namespace nsa {
int check_dims(const NsaDims* d);
AttnArgs base_args(const NsaDims* d, int Lk);
bool use_tc(const NsaDims* d, int block_size, int impl, int* err);
bool use_three_term(const NsaDims* d, int block_size, int S, int impl, bool bwd);
int topn_check(const NsaDims* dims, int n_cmp, int cmp_len, int cmp_stride, int sel_block, int n_sel, int n_init,
               int n_local, int impl);   // aux.cu
// What the gate kernels need of the op's output or its gradient, in the order of the heads and by tokens (either may be null)
int gate_args_ok(const NsaDims* dims, const void* heads, const void* tokens);   // aux.cu
// nsa_gate_combine_fwd, unless the block-outer kernel has served the selection (a choice without header: always)
int gate_fwd_unless_blended(const void* o_cmp, const void* o_slc, const void* o_win, const void* gate_logits, void* out,
                            const NsaDims* dims, const SelChoice& choice, bool tokens, void* stream);   // aux.cu
// nsa_gate_combine_bwd_rows; with d_heads, d_out is token-major and its rows are written there in the order of the heads;
// n_zeros floats are zeroed
int gate_bwd_rows(const void* o_cmp, const void* o_slc, const void* o_win, const void* gate_logits, const void* d_out,
                  float* row_scale, float* row_dot, void* d_gate_logits, const NsaDims* dims, void* d_heads, float* zeros, size_t n_zeros,
                  void* stream);   // aux.cu
bool profiling();     // every launch is bracketed by events on its stream: branches must not overlap
}  // namespace nsa
