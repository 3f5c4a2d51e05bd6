// Shared host/device helpers of libnsa_b200: error reporting, dtype loads, launch checks.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "../../include/nsa_b200.h"

namespace nsa {
// Compression summaries: summary j covers tokens [j * stride, j * stride + len); query t sees
// the summaries that end at or before t (nsa_model.py:233-235 for stride == len).
__host__ __device__ __forceinline__ int cmp_visible(int t, int len, int stride, int n_summaries) {
  if (t + 1 < len) return 0;
  const int n = (t + 1 - len) / stride + 1;
  return n < n_summaries ? n : n_summaries;
}

// Rank keys of forced selection blocks: above every importance (a sum of at most G <= 128
// probabilities), initial blocks ahead of local ones, exact in fp32 for counts below 2^18.
constexpr float kForcedInit = 1048576.f;    // - block index
constexpr float kForcedLocal = 524288.f;    // - distance from the block holding the query

void set_error(const char* fmt, ...);

#define NSA_CHECK_ARG(cond, ...)            \
  do {                                      \
    if (!(cond)) {                          \
      nsa::set_error(__VA_ARGS__);          \
      return NSA_ERR_BAD_ARG;               \
    }                                       \
  } while (0)

#define NSA_CUDA_OK(expr)                                                        \
  do {                                                                           \
    cudaError_t _e = (expr);                                                     \
    if (_e != cudaSuccess) {                                                     \
      nsa::set_error("%s failed: %s (%s:%d)", #expr, cudaGetErrorString(_e),     \
                     __FILE__, __LINE__);                                        \
      return NSA_ERR_CUDA;                                                       \
    }                                                                            \
  } while (0)

#define NSA_LAUNCH_OK(name)                                                      \
  do {                                                                           \
    cudaError_t _e = cudaGetLastError();                                         \
    if (_e != cudaSuccess) {                                                     \
      nsa::set_error("launch of %s failed: %s", name, cudaGetErrorString(_e));   \
      return NSA_ERR_CUDA;                                                       \
    }                                                                            \
  } while (0)

constexpr float kLseEmpty = -1.0e9f;  // nsa_selection_kernel.py:134,171
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

inline size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }
template <typename... P> inline bool aligned16(const P*... p) { return ((... | (uintptr_t)p) & 15) == 0; }

__device__ __forceinline__ float to_float(float x) { return x; }
__device__ __forceinline__ float to_float(__nv_bfloat16 x) { return __bfloat162float(x); }
template <typename T> __device__ __forceinline__ T from_float(float x);
template <> __device__ __forceinline__ float from_float<float>(float x) { return x; }
template <> __device__ __forceinline__ __nv_bfloat16 from_float<__nv_bfloat16>(float x) {
  return __float2bfloat16_rn(x);
}

__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}
__device__ __forceinline__ float warp_max(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}

// error word raised by kernels whose bounded waits run out; defined in api.cu
int* device_status_ptr();
int sm_count();                                          // multiprocessors of the current device
// lets `kernel` use `bytes` of dynamic shared memory on the current device (a driver call the
// first time only)
cudaError_t func_smem(const void* kernel, size_t bytes);

// Per-kernel accounting (api.cu): every kernel launch of the library sits inside a KernelScope,
// which counts it and, when profiling is on, brackets it with CUDA events on its stream.
void kernel_begin(const char* name, cudaStream_t st);
void kernel_end(cudaStream_t st);
struct KernelScope {
  cudaStream_t st;
  KernelScope(const char* name, cudaStream_t s) : st(s) { kernel_begin(name, s); }
  ~KernelScope() { kernel_end(st); }
};

// Chains of short kernels.  A kernel launched by launch_chained may be placed on the GPU as soon as every CTA of the kernel
// before it in the stream has called chain_go or ended; chain_wait returns once that kernel is complete and its writes are
// visible.  What lies between is hidden: the launch, and what a kernel sets up before its chain_wait.  Every thread of
// a chained kernel calls chain_wait before it touches global memory (but for the device status word) and before it ends, so
// that completion carries over to the kernels behind it.  A kernel that allocates tensor memory calls chain_go after that: the next one's CTAs take theirs
// from the same SMs.
// Measured (us per call, one after the other -> chained): forward of the operator at T = 512 44.8 -> 39.5, at
// T = 1024 53.1 -> 48.1, selection at T = 8192 forward and backward 362 -> 339 (350 with the backward's kernels
// one after the other), three branches over given lists at T = 4096 94 -> 88.8.
// From a graph, where the launches cost nothing, over given lists: T = 4096 85 us before and now (80 with plain launches of the
// present kernels), T = 5000 117 -> 106, 2 x 1000 33.5 -> 29.3, 2048 at heads of 128 59.7 -> 55.7.
// Plain launches stay where an early CTA takes a place that another stream's kernel would fill: the block-outer
// selection kernel (chained 98.6 where it is 89.3 plain) and, over given lists, the attention over pooled keys (T = 3000
// 91 against 86.3), both beside the window's kernel.  With lists of the scorer the window is launched ahead of the
// pooling, and chained is the better: forward at 512 tokens 39.3 -> 37.9 us, 2 x 300 41.1 -> 38.5, 1024 47.8 -> 46.5.
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chain_go() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// What the kernel ahead writes is read by plain loads, which stay behind the wait: the read-only path (__ldg, a const
// __restrict__ argument) takes its data not to change while the kernel is on the GPU, which includes the time before.
// So do the scalar rows of sel_row.cuh, which run in chained kernels.
__device__ __forceinline__ int32_t ld_plain(const int32_t* p) { int32_t v; asm volatile("ld.global.s32 %0, [%1];" : "=r"(v) : "l"(p)); return v; }
__device__ __forceinline__ float ld_plain(const float* p) { float v; asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p)); return v; }
__device__ __forceinline__ uint4 ld_plain(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ unsigned long long ld_plain(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.global.u64 %0, [%1];" : "=l"(v) : "l"(p));
  return v;
}
template <typename... P, typename... A>
inline cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, const A&... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// kernel names carry the branch they serve: <prefix>_win / _cmp / _slc
inline const char* branch_name(const char* const names[3], int kind) { return names[kind == 0 ? 0 : (kind == 1 ? 1 : 2)]; }

// ---- SIMT kernel family (simt.cu) ---------------------------------------------------------
struct AttnArgs {
  const void* q; const void* k; const void* v; const int32_t* block_idx;
  void* o; float* lse;
  const void* d_o; void* dq; float* dk_acc; float* dv_acc;   // backward
  const float* row_scale; const float* row_dot;   // backward of a gated branch (may be null)
  float* dq_acc;     // tcgen05 window / compression backward: fp32 accumulator [B*Hkv][T][G][D] that takes dQ (or null)
  const void* sel_plan;   // tcgen05 selection: plan built earlier (tc_sel_plan_build), or null
  bool three_term;          // tcgen05 selection on 16- and 32-token blocks: P and dS in three bf16 terms, dQ partials in fp32
  // tcgen05 selection: where the block-outer kernel serves the call its merge blends the three branches as well
  // (gate logits, the other branches' outputs, the op's output; null g_out: it does not) and keeps `o` only
  // where o_kept says so
  const void *g_cmp, *g_win, *g_logits;
  void *g_out, *o_kept;
  bool g_tokens;          // g_out is [B, T, Hq, D]
  bool plan_kept;         // the plan outlives the dQ reduction: the backward need not copy its pair map
  // window backward without a dq of its own: who reads the partials knows that they may lie in tiles of 128 keys (a caller
  // who names neither the key count nor the options to nsa_dq_reduce3 gets them in tiles of 64)
  bool wide_dq;
  bool cuda_cores;   // fp32: FFMA throughout (NSA_IMPL_SIMT), where the call would take the bf16 terms of f32_tile.cu
  bool chained;      // tcgen05 compression forward: launched into the end of the pooling (launch_chained)
  int B, Hq, Hkv, T, Lk, D, S;
  int kind;          // 0 window, 1 compress, 2 selection
  int window, block_size;
  float scale;
};
int simt_attn_fwd(const AttnArgs& a, int dtype, cudaStream_t st);
int simt_attn_bwd(const AttnArgs& a, int dtype, cudaStream_t st);
bool simt_tile_ok(const AttnArgs& a, int dtype, bool bwd);                                  // simt_tile.cu
int simt_tile_fwd(const AttnArgs& a, int dtype, cudaStream_t st);
int simt_tile_bwd(const AttnArgs& a, int dtype, cudaStream_t st);
int cast_f32_to(const float* src, void* dst, size_t n, int dtype, cudaStream_t st);

// ---- tcgen05 kernel family (tc.cu) ----------------------------------------------------------
bool tc_shape_ok(const NsaDims& d, int block_size);
int tc_attn_fwd(const AttnArgs& a, cudaStream_t st);
size_t tc_sel_fwd_workspace(const AttnArgs& a);
int tc_sel_fwd(const AttnArgs& a, void* ws, size_t ws_bytes, cudaStream_t st);
size_t tc_sel_plan_bytes(const AttnArgs& a);
// what decides on the device which of the two forward kernels serves a planned call
struct SelChoice { const struct SelPlanHeader* hdr; int nq_union, force; };
SelChoice tc_sel_choice(const AttnArgs& a, const void* plan);
int tc_sel_plan_build(const AttnArgs& a, void* plan, size_t plan_bytes, cudaStream_t st);
const int32_t* sel_plan_pair_map(const AttnArgs& a, int S, int block_size, const void* plan);
size_t tc_attn_bwd_workspace(const AttnArgs& a);
int tc_attn_bwd(const AttnArgs& a, void* ws, size_t ws_bytes, cudaStream_t st);
// api.cu: the whole op's attention over pooled keys, and its window backward (wide_dq; the workspace is nsa_range_attn_bwd's)
int compress_fwd(const void* q, const void* k, const void* v, void* o, float* lse, const NsaDims* dims, int Lk, int stride,
                 int len, int impl, bool chained, void* stream);
int window_bwd(const void* q, const void* k, const void* v, const void* o, const float* lse, const void* d_o, void* dq,
               void* dk, void* dv, const NsaDims* dims, int window, const float* row_scale, const float* row_dot,
               void* workspace, size_t workspace_bytes, int impl, cudaStream_t st);
int tc_dq_reduce3(const AttnArgs& base, int Lk_cmp, int cmp_len, int cmp_stride, int S, int block_size,
                  int window, const void* ws_cmp, const void* ws_slc, const void* ws_win,
                  const int32_t* pos, const float* dq_acc, void* dq, cudaStream_t st);

}  // namespace nsa
